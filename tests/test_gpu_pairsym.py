"""Exact all-points FP64 sums and their adjoint (each unordered pair evaluated
once): sizes at
the edges of the units (64 sources), staged chunks (256), tiles (256, 512 and
1024 targets) and of the rule that picks the tile, a size that runs in several
phases, spectra in any order and at any alignment, against the oracle's sums
at the same points.  Tolerance: the FP64 parity bar of the exact path, 1e-12
of |S| (the sums differ from the oracle's by rounding in another order only).
"""
import math

import numpy as np
import pytest
import torch

from shrinkers_b200 import _native, spectra

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 513, 1025, 3071, 3072, 3073, 3583, 3585,
         8191, 8192, 8193, 9215, 9217, 20001, 150001]


def transform(ev, eta, offset):
    """S/p at every value, from a device array `offset` doubles past 16-byte alignment."""
    L = _native.load()
    buf = torch.empty(ev.size + 2, dtype=torch.float64, device="cuda")
    d = buf[offset:offset + ev.size]
    d.copy_(torch.from_numpy(ev))
    re, im = torch.empty_like(d), torch.empty_like(d)
    _native.check(L.shrk_stieltjes_all_dev(
        d.data_ptr(), ev.size, eta, 2, 0, float("nan"), 0, re.data_ptr(), im.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    _native.check(L.shrk_stream_check(torch.cuda.current_stream().cuda_stream))
    return re.cpu().numpy(), im.cpu().numpy()


@pytest.mark.parametrize("p", SIZES)
@pytest.mark.parametrize("order", ["ascending", "descending", "shuffled"])
def test_symmetric_sums(oracle, p, order):
    if p > 20001 and order != "ascending":
        pytest.skip("one order of the largest size")
    ev = spectra.config2(p, seed=p)
    if order == "descending":
        ev = ev[::-1].copy()
    elif order == "shuffled":
        ev = np.random.default_rng(p).permutation(ev)
    eta = 1.0 / math.sqrt(p)
    # every target of a small spectrum, the tiles' edges of a large one
    at = np.unique(np.r_[0:min(p, 300), np.arange(255, p, 256), max(0, p - 300):p])
    at = at[np.linspace(0, at.size - 1, min(at.size, 1500)).astype(int)]
    q_re, q_im = oracle.compute_at_points(ev[at], ev, eta, "blocked")
    first = transform(ev, eta, 0)
    for offset in (0, 1):
        re, im = transform(ev, eta, offset)
        err = np.hypot(re[at] * p - q_re, im[at] * p - q_im) / np.hypot(q_re, q_im)
        assert np.max(err) < 1e-12, (offset, np.max(err))
        # the order of the additions depends on the size alone
        np.testing.assert_array_equal(re, first[0])
        np.testing.assert_array_equal(im, first[1])


def test_diagonal_dominates_at_small_eta(oracle):
    """eta far below the spacing, duplicates and wide ranges: each term keeps
    its place (a pair added to the wrong end would show at once)."""
    p = 1500
    rng = np.random.default_rng(7)
    ev = np.exp(rng.uniform(-20.0, 20.0, p))
    ev[100:110] = ev[100]
    for eta in (1e-12, 1e3):
        re, im = transform(ev, eta, 0)
        q_re, q_im = oracle.compute_at_points(ev, ev, eta, "blocked")
        scale = np.hypot(q_re, q_im)
        assert np.max(np.hypot(re * p - q_re, im * p - q_im) / scale) < 1e-12


@pytest.mark.parametrize("p", [1, 2, 33, 64, 65, 257, 1025, 3071, 3073, 8193, 16383, 16385,
                               60001])
def test_symmetric_adjoint(oracle, p):
    """Against the oracle's direct gradient at the tiles' edges.  Each of the p
    terms of grad_k is a few roundings of size eps (|w_k| + |w_j| + |v_k| +
    |v_j|) / (d^2 + eta^2) (|A| and |2 eta d r^2| are at most r), so the sums
    may differ by 64 eps of the terms' bounds."""
    rng = np.random.default_rng(p)
    ev = rng.permutation(spectra.config2(p, seed=p))
    w, v = rng.standard_normal(p), rng.standard_normal(p)
    eta = 1.0 / math.sqrt(p)
    L = _native.load()
    d = [torch.from_numpy(a).cuda() for a in (ev, w, v)]
    got = torch.empty_like(d[0])
    _native.check(L.shrk_stieltjes_adjoint_dev(
        d[0].data_ptr(), p, eta, d[1].data_ptr(), d[2].data_ptr(), 0, got.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    got = got.cpu().numpy()
    at = np.unique(np.r_[0:min(p, 40), np.arange(255, p, 256), max(0, p - 40):p])[:400]
    ref = oracle.adjoint_direct(ev, eta, w, v, idx=at)
    for i, k in enumerate(at):
        r = 1.0 / ((ev[k] - ev) ** 2 + eta * eta)
        bound = np.sum((abs(w[k]) + np.abs(w) + abs(v[k]) + np.abs(v)) * r) / p
        assert abs(got[k] - ref[i]) <= 64 * np.finfo(float).eps * bound, (k, got[k], ref[i])
