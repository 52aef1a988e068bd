"""Device-pointer matrix calls report a wait of the tridiagonalisation that gave
up (budget of zero cycles: the kernel records it and returns) as the
host-pointer calls do, and the calls after it are right."""
import numpy as np
import pytest
import torch

from shrinkers_b200 import _native

pytestmark = pytest.mark.gpu
ETIMEOUT = 3
P = 200


def calls(L, a):
    s = torch.cuda.current_stream().cuda_stream
    vec = lambda: torch.empty(P, dtype=torch.float64, device="cuda")
    mat = lambda: torch.empty(P, P, dtype=torch.float64, device="cuda")
    w, v = vec(), mat()
    c, e, x, o = mat(), mat(), vec(), vec()
    q, f, pe, ce = mat(), mat(), vec(), vec()
    st = [L.shrk_symmetric_eigh_dev(a.data_ptr(), P, w.data_ptr(), v.data_ptr(), s),
          L.shrk_clean_covariance_matrix_dev(a.data_ptr(), P, 0.25, 0, c.data_ptr(), e.data_ptr(),
                                             x.data_ptr(), o.data_ptr(), None, s),
          L.shrk_estimate_precision_matrix_dev(a.data_ptr(), P, 0.25, 0, q.data_ptr(),
                                               f.data_ptr(), pe.data_ptr(), ce.data_ptr(), None, s)]
    torch.cuda.synchronize()
    return st, [t.cpu().numpy() for t in (w, v, c, q)]


def test_device_matrix_calls_time_out():
    L = _native.load()
    x = np.random.default_rng(2).standard_normal((4 * P, P))
    a = torch.from_numpy(np.ascontiguousarray(x.T @ x / (4 * P))).cuda()
    st, want = calls(L, a)
    assert st == [0, 0, 0], _native.last_error()
    old = L.shrk_diag_set_wait_limit(0)
    try:
        st, _ = calls(L, a)
        assert st == [ETIMEOUT] * 3
        assert "timeout" in _native.last_error()
    finally:
        L.shrk_diag_set_wait_limit(-1)
    assert L.shrk_diag_set_wait_limit(-1) == old
    st, got = calls(L, a)
    assert st == [0, 0, 0]
    for g, r in zip(got, want):
        np.testing.assert_array_equal(g, r)
