"""The paired FP64 sums: the mixed kernel's near field and the FP64 query sums.

Every target's sum is near field here (all values within 32 eta), so the mixed
result must be an FP64 result like the query one's: each pair term carries a few roundings, and a
sum of n terms of one sign (the imaginary part) at most (n + 16) 2^-53 of
itself; the real part the same against the sum of its terms' magnitudes, plus
the rounding of the block offsets, at most 2^-52 of the spectrum's width over
eta per term.  Sources closer than eta in pairs, further apart than eta (the
plain form), mixed within a block, descending, duplicates, and a spike that
widens the last block.
"""
import ctypes as C

import numpy as np
import pytest

from shrinkers_b200 import _native

pytestmark = pytest.mark.gpu
NAN = float("nan")
_D = C.POINTER(C.c_double)


def gpu_mixed(ev, eta):
    L = _native.load()
    ev = np.ascontiguousarray(ev)
    re, im = np.empty(ev.size), np.empty(ev.size)
    p = lambda a: a.ctypes.data_as(_D)
    _native.check(L.shrk_stieltjes_all(p(ev), ev.size, eta, 2, 1, NAN, 0, p(re), p(im)))
    return re * ev.size, im * ev.size


def gpu_points(q, ev, eta):
    L = _native.load()
    q, ev = np.ascontiguousarray(q), np.ascontiguousarray(ev)
    re, im = np.empty(q.size), np.empty(q.size)
    p = lambda a: a.ctypes.data_as(_D)
    _native.check(L.shrk_stieltjes_at_points(p(q), q.size, p(ev), ev.size, eta, 2, 0, NAN, 0,
                                             p(re), p(im)))
    return re, im


def spectrum(kind, p, eta):
    g = np.random.default_rng(p)
    if kind == "close":
        return np.sort(g.uniform(1.0, 1.0 + 30.0 * eta, p))
    if kind == "apart":  # neighbours 1.2 eta and more from each other, up to 30 eta wide
        v = 1.0 + 1.2 * eta * np.arange(p) * g.uniform(1.0, 1.2)
        return v[v < 1.0 + 30.0 * eta]
    if kind == "descending":
        return np.sort(g.uniform(1.0, 1.0 + 30.0 * eta, p))[::-1].copy()
    if kind == "equal":
        return np.repeat(np.sort(g.uniform(1.0, 1.0 + 30.0 * eta, (p + 2) // 3)), 3)[:p]
    v = np.sort(g.uniform(1.0, 1.0 + 10.0 * eta, p))
    v[-1] = 1.0 + 30.0 * eta
    return v


def check(q, ev, eta, re, im):
    n = ev.size
    d = q.astype(np.longdouble)[:, None] - ev.astype(np.longdouble)[None, :]
    e = d * d + np.longdouble(eta) ** 2
    want_re, want_im, mag = (d / e).sum(1), (eta / e).sum(1), (np.abs(d) / e).sum(1)
    eps = 2.0 ** -53
    assert np.all(np.abs(im - want_im) <= (n + 16) * eps * want_im)
    width = float(ev.max() - ev.min())
    assert np.all(np.abs(re - want_re) <= (n + 16) * eps * mag + 2.0 * eps * (width / eta) * n / eta)


@pytest.mark.parametrize("kind", ["close", "apart", "descending", "equal", "spike"])
@pytest.mark.parametrize("p", [2, 255, 256, 257, 511, 512, 1300, 5000])
@pytest.mark.parametrize("eta", [0.01, 3e-70])
def test_near_field_is_fp64(kind, p, eta):
    ev = spectrum(kind, p, eta if eta > 1e-3 else 0.01)
    re, im = gpu_mixed(ev, eta)
    if eta < 1e-3:
        # outside the paired form's range: the same calls as ever, finite
        assert np.all(np.isfinite(re)) and np.all(np.isfinite(im))
        return
    check(ev, ev, eta, re, im)


@pytest.mark.parametrize("kind", ["close", "apart", "descending", "equal", "spike"])
@pytest.mark.parametrize("p", [1, 63, 64, 65, 257, 1300, 20001])
def test_query_sums(kind, p):
    """One target a thread and four, groups of 64 sources and the rest."""
    ev = spectrum(kind, p, 0.01)
    q = ev if p < 2000 else np.linspace(ev.min() - 0.1, ev.max() + 0.1, p)
    re, im = gpu_points(q, ev, 0.01)
    at = np.arange(q.size) if p < 2000 else np.random.default_rng(1).integers(0, q.size, 200)
    check(q[at], ev, 0.01, re[at], im[at])


def test_query_far_outside():
    """Queries outside the paired form's range stay exact."""
    ev = np.sort(np.random.default_rng(2).uniform(1.0, 2.0, 640))
    q = np.concatenate([ev[:100], [1e70, -1e70]])
    re, im = gpu_points(q, ev, 0.05)
    assert np.all(np.isfinite(re)) and np.all(np.isfinite(im))
    np.testing.assert_allclose(re[-2:], ev.size / q[-2:], rtol=1e-12)
