"""The FP64 pair sums do not lose accuracy to values far from a target.

Spectra in which a block of sources holds values far from its others: a
descending bulk behind one or several large values, an ascending one behind a
far negative value, a gap between two blocks and inside one, a shuffled order;
through the FP64 sums at query points, the FP64 batch, and the mixed sums and
batch where the whole bulk is near field.

Tolerance, for each target and not a function of the spectrum's width or of its
largest value: n rounded additions of terms t_j are off by at most
8 sqrt(n) u sum |t_j| with a probability of failure below 1e-12 a target
(u = 2^-53; Higham and Mary, SIAM J. Sci. Comput. 41, 2019, lambda = 8), each
term carries at most 16 u of its own, and a separation may carry the rounding
of an offset of 16 eta, which changes 1/((x - s) - i eta) by 16 u relatively in
each part of (x - s) and eta: 32 u (|d| + eta)/(d^2 + eta^2).
"""
import ctypes as C
import math

import numpy as np
import pytest

from shrinkers_b200 import _native

pytestmark = pytest.mark.gpu
NAN = float("nan")
F64, MIXED, BLOCKED = 0, 1, 2
_D = C.POINTER(C.c_double)
_I64 = C.POINTER(C.c_int64)
P = 2048
ETA = 1.0 / math.sqrt(P)


def dp(a):
    return a.ctypes.data_as(_D)


def spectrum(kind, width):
    """P values; the bulk over `width` from 0.25 on."""
    g = np.random.default_rng(P)
    v = np.sort(g.uniform(0.25, 0.25 + width, P))
    name, _, what = kind.partition(":")
    if name == "lead":  # descending, one large value in front
        v = v[::-1].copy()
        v[0] = float(what)
    elif name == "spikes":  # descending, five
        v = v[::-1].copy()
        v[:5] = float(what) * np.array([5.0, 4.0, 3.0, 2.5, 2.0])
    elif name == "behind":  # ascending, one far below
        v[0] = -float(what)
    elif name == "gap":  # half of the values far off, the change inside a group
        v[1000:] += float(what)
    elif name == "blocks":  # the change between two blocks
        v[1024:] += float(what)
    elif name == "shuffled":
        v[0] = float(what)
        g.shuffle(v)
    return np.ascontiguousarray(v)


KINDS = ["lead:50", "lead:1e3", "lead:1e6", "lead:1e9", "lead:1e17", "spikes:1e2", "spikes:1e8",
         "behind:1e6", "gap:1e6", "blocks:1e6", "shuffled:1e6"]


def check(ev, eta, re, im, at):
    n = ev.size
    d = ev[at].astype(np.longdouble)[:, None] - ev.astype(np.longdouble)[None, :]
    e = d * d + np.longdouble(eta) ** 2
    want_re, want_im = (d / e).sum(1), (eta / e).sum(1)
    size = ((np.abs(d) + eta) / e).sum(1)
    tol = (8.0 * math.sqrt(n) + 16.0 + 32.0) * 2.0 ** -53 * size
    assert np.all(np.abs(re[at] - want_re) <= tol), np.max(np.abs(re[at] - want_re) / size)
    assert np.all(np.abs(im[at] - want_im) <= tol), np.max(np.abs(im[at] - want_im) / size)


def every(ev, bulk_only=False):
    """Every seventh value (and the first ones); of the bulk alone the FP64 part of
    the mixed sums: a far value's own sum over the bulk is FP32."""
    at = np.unique(np.concatenate([np.arange(8), np.arange(0, ev.size, 7)]))
    return at[(ev[at] >= 0.0) & (ev[at] < 100.0)] if bulk_only else at


@pytest.mark.parametrize("kind", KINDS)
def test_query_sums(kind):
    L = _native.load()
    ev = spectrum(kind, 2.0)
    q = ev.copy()
    for order in (1, -1):  # and the sources the other way round
        src = np.ascontiguousarray(ev[::order])
        re, im = np.empty(P), np.empty(P)
        _native.check(L.shrk_stieltjes_at_points(dp(q), P, dp(src), P, ETA, BLOCKED, F64, NAN, 0,
                                                 dp(re), dp(im)))
        check(ev, ETA, re, im, every(ev))


@pytest.mark.parametrize("kind", KINDS)
def test_fp64_batch(kind):
    L = _native.load()
    arrs = [spectrum(kind, 2.0), spectrum("none", 2.0), spectrum(kind, 2.0)[::-1].copy()]
    re, im = batch(L, arrs, ETA, F64)
    for k, a in enumerate(arrs):
        check(a, ETA, re[k], im[k], every(a))


def batch(L, arrs, eta, precision):
    n = len(arrs)
    offs = np.arange(n + 1, dtype=np.int64) * P
    vals, etas = np.concatenate(arrs), np.full(n, eta)
    re, im = np.empty(n * P), np.empty(n * P)
    _native.check(L.shrk_stieltjes_batched(dp(vals), offs.ctypes.data_as(_I64), n, dp(etas),
                                           precision, dp(re), dp(im)))
    return re.reshape(n, P) * P, im.reshape(n, P) * P


# near field everywhere in the bulk: 30 eta wide.  Values far from it are summed
# in FP32 in the blocks of their own, so only spectra whose far values share a
# block with the bulk have FP64 sums throughout.
NEAR = ["lead:50", "lead:1e3", "lead:1e6", "lead:1e9", "lead:1e17", "spikes:1e8", "behind:1e6",
        "shuffled:1e6"]


@pytest.mark.parametrize("kind", NEAR)
def test_mixed_near_field(kind):
    L = _native.load()
    eta = 0.01
    ev = spectrum(kind, 30.0 * eta)
    re, im = np.empty(P), np.empty(P)
    _native.check(L.shrk_stieltjes_all(dp(ev), P, eta, BLOCKED, MIXED, NAN, 0, dp(re), dp(im)))
    check(ev, eta, re * P, im * P, every(ev, True))
    b_re, b_im = batch(L, [ev, ev], eta, MIXED)
    for k in range(2):
        check(ev, eta, b_re[k], b_im[k], every(ev, True))


def test_range_of_the_paired_form():
    """Groups far from their block's first source, within the exponent range and
    outside it: finite and right either way."""
    L = _native.load()
    eta = 0.05
    g = np.random.default_rng(5)
    near = np.sort(g.uniform(1.0, 2.0, 256))
    for far in (1e20, 1e59, 1e70, 1e100, 1e140):
        # after the first 64 values, 64 equal ones far away (a group of its own)
        ev = np.concatenate([near[:64], np.full(64, far), near[64:]])
        re, im = np.empty(256), np.empty(256)
        _native.check(L.shrk_stieltjes_at_points(dp(near), 256, dp(ev), ev.size, eta, BLOCKED, F64,
                                                 NAN, 0, dp(re), dp(im)))
        d = near[:, None] - ev[None, :].astype(np.longdouble)
        e = d * d + np.longdouble(eta) ** 2
        np.testing.assert_allclose(re, (d / e).sum(1).astype(float), rtol=1e-11, atol=1e-9)
        np.testing.assert_allclose(im, (eta / e).sum(1).astype(float), rtol=1e-12)
