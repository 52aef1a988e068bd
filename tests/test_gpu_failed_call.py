"""A host-pointer call that fails writes nothing to the caller's arrays, neither
then nor in a later call on the same thread.

The outputs of a small host-pointer call travel through the context's pinned
stage and are copied to the caller at the end; a call that fails on the way
must not leave that copy to be made by whatever runs next.  The arrays are kept
alive and filled with a pattern here, so that a late copy is seen as a changed
pattern.
"""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from shrinkers_b200 import _native, spectra

pytestmark = pytest.mark.gpu
NAN = float("nan")
EWALD, BLOCKED = 17, 2  # no all-points EWALD kernel: SHRK_ENOTIMPL
_D = C.POINTER(C.c_double)
PATTERN = -12345.678


def dp(a):
    return a.ctypes.data_as(_D)


def patterned(n):
    return np.full(n, PATTERN)


def failing_all(L, ev, out):
    return L.shrk_stieltjes_all(dp(ev), ev.size, 0.1, EWALD, 0, NAN, 0, dp(out[0]), dp(out[1]))


def failing_shrink(L, ev, out):
    return L.shrk_ledoit_wolf_shrinkage(dp(ev), ev.size, 0.25, EWALD, 0, 0, 0.1, dp(out[0]))


def good_all(L, ev):
    re, im = np.empty(ev.size), np.empty(ev.size)
    _native.check(L.shrk_stieltjes_all(dp(ev), ev.size, 0.1, BLOCKED, 0, NAN, 0, dp(re), dp(im)))
    return re, im


def matrix():
    g = np.random.default_rng(3).standard_normal((40, 160))
    return np.ascontiguousarray(g @ g.T / 160.0)


def then_eigh(L):
    a, w, v = matrix(), np.empty(40), np.empty((40, 40))
    _native.check(L.shrk_symmetric_eigh(dp(a), 40, dp(w), dp(v)))
    np.testing.assert_allclose(w, np.linalg.eigvalsh(a), rtol=0, atol=1e-13 * abs(w).max())


def then_eigh_dev(L):
    a = torch.from_numpy(matrix()).cuda()
    w, v = torch.empty(40, dtype=torch.float64, device="cuda"), torch.empty_like(a)
    s = torch.cuda.current_stream().cuda_stream
    _native.check(L.shrk_symmetric_eigh_dev(a.data_ptr(), 40, w.data_ptr(), v.data_ptr(), s))
    torch.cuda.synchronize()


def then_renormalize(L):
    a, o = matrix(), np.empty((40, 40))
    _native.check(L.shrk_renormalize_to_unit_diagonal(dp(a), 40, dp(o)))
    d = np.sqrt(np.diag(a))
    np.testing.assert_allclose(o, a / np.outer(d, d), rtol=1e-13)


def then_good_call(L):
    good_all(L, spectra.config2(300, seed=4))


@pytest.mark.parametrize("then", [then_eigh, then_eigh_dev, then_renormalize, then_good_call])
@pytest.mark.parametrize("fail", [failing_all, failing_shrink])
def test_a_failed_call_leaves_the_outputs_alone(fail, then):
    L = _native.load()
    ev = spectra.config2(500, seed=9)
    want = good_all(L, ev)  # from the second call on the stage is sized for this one
    good_all(L, ev)
    out = [patterned(ev.size), patterned(ev.size)]
    assert fail(L, ev, out) != 0
    assert "no GPU implementation" in _native.last_error()
    then(L)
    for a in out:
        np.testing.assert_array_equal(a, patterned(ev.size))
    got = good_all(L, ev)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
