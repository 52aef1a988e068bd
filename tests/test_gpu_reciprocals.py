"""The branch-free reciprocals and quotient equal the IEEE results (bit for bit:
no tolerance), for both signs where they take both: fractions at and next to all
ones (the case the method treats apart) and zero over every exponent of the
range, random values, and in FP32 every fraction."""
import numpy as np
import pytest
import torch

from shrinkers_b200 import _native

pytestmark = pytest.mark.gpu


def run(a, w):
    L = _native.load()
    ta, tw = torch.from_numpy(a).cuda(), torch.from_numpy(w).cuda()
    r, q = torch.empty_like(ta), torch.empty_like(ta)
    f = torch.empty(a.size, dtype=torch.float32, device="cuda")
    _native.check(L.shrk_diag_reciprocals(ta.data_ptr(), tw.data_ptr(), a.size, r.data_ptr(),
                                          q.data_ptr(), f.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream))
    return r.cpu().numpy(), q.cpu().numpy(), f.cpu().numpy()


def values(bits, lo, hi):
    """Both signs; fractions at and next to all ones, all zeros and random ones over
    the exponents [lo, hi]."""
    g = np.random.default_rng(7)
    e = np.arange(lo, hi + 1)
    one = np.ldexp(1.0, e)
    u = 2.0 ** -bits
    near = [one * (2.0 - k * u) for k in (1, 2, 3)] + [one * (1.0 + k * u) for k in (0, 1, 2)]
    n = 1 << 21
    rnd = np.ldexp(1.0 + g.integers(0, 1 << bits, n) * u, g.integers(lo, hi, n))
    a = np.concatenate([v for v in near] + [rnd])
    return np.concatenate([a, -a])


@pytest.mark.parametrize("limit", [900, 400])
def test_double(limit):
    a = values(52, -limit, limit - 1)
    g = np.random.default_rng(8)
    w = np.ldexp(1.0 + g.random(a.size), g.integers(-400, 399, a.size)) * g.choice([-1.0, 1.0], a.size)
    w[::1001] = 0.0
    r, q, _ = run(a, w)
    np.testing.assert_array_equal(r, 1.0 / a)
    if limit == 400:
        np.testing.assert_array_equal(q, w / np.abs(a))


def test_single():
    a32 = values(23, -120, 119).astype(np.float32)
    every = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)
    a = np.concatenate([a32, every]).astype(np.float64)
    _, _, f = run(a, np.zeros(a.size))
    np.testing.assert_array_equal(f, np.float32(1.0) / np.abs(a).astype(np.float32))
