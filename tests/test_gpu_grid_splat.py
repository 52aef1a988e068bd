"""The grid splat by source chunks and the FFT passes at their edges.

The splat cuts the sources in chunks of 512: runs of equal cells inside a
chunk, across one boundary and across many, more than 32 equal cells in a
row (summed by a warp) and fewer, sources off both ends of the grid, the
sources in descending order (dx < 0).  The reference is the sequential splat
(fft5.rs:175-185) in numpy with the same operations: cells of at most 32
sources are the same sums bit for bit; a denser cell of n sources differs by
the order of its sum, at most n 2^-53 times the sum of its weights' magnitudes
in either order.
"""
import math

import numpy as np
import pytest

from shrinkers_b200 import _native, spectra
from test_gpu_fft5 import close, gpu_opts

pytestmark = pytest.mark.gpu


def reference_density(v, m, lo, dx):
    """(density, count of slots, sum of |weight|) of the 4-node splat."""
    pos = (v - lo) / dx
    fl = np.floor(pos)
    t = pos - fl
    n = 4
    f = [t - float(j) + 2.0 - 1.0 for j in range(n)]
    w = []
    for j in range(n):
        pre, suf = np.ones_like(t), np.ones_like(t)
        for i in range(j):
            pre = pre * f[i]
        for i in range(n - 1, j, -1):
            suf = suf * f[i]
        w.append(pre * suf / math.prod(float(j - i) for i in range(n) if i != j))
    i0 = np.clip(fl, -n - 1, m + n).astype(np.int64)
    cells = np.clip(i0[:, None] - 1 + np.arange(n), 0, m - 1)
    dens, mag, cnt = np.zeros(m), np.zeros(m), np.zeros(m, dtype=np.int64)
    flat, wf = cells.ravel(), np.stack(w, 1).ravel()
    np.add.at(dens, flat, wf)  # source by source, slot by slot
    np.add.at(mag, flat, np.abs(wf))
    np.add.at(cnt, flat, 1)
    return dens, cnt, mag


def gpu_density(v, m, lo, dx):
    import torch

    src = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    out = torch.full((m,), float("nan"), device="cuda", dtype=torch.float64)
    _native.check(_native.load().shrk_nufft_density_dev(
        src.data_ptr(), src.numel(), m, lo, dx, out.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


def sources(kind, p):
    g = np.random.default_rng(p)
    if kind == "spread":     # a few sources in a cell, many cells empty
        return np.sort(g.uniform(0.0, 100.0, p))
    if kind == "dense":      # runs of hundreds
        return np.sort(g.uniform(50.0, 50.4, p))
    if kind == "equal":      # one run over every chunk
        return np.full(p, 37.123)
    # bunches of 1 .. 80 equal values, and sources beyond both ends
    v = np.repeat(g.uniform(-20.0, 120.0, p), g.integers(1, 80, p))[:p]
    return np.sort(v)


@pytest.mark.parametrize("kind", ["spread", "dense", "equal", "bunches"])
@pytest.mark.parametrize("p", [1, 31, 33, 511, 512, 513, 1024, 1025, 20000])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_density_against_the_sequential_splat(kind, p, sign):
    v = sources(kind, p)
    m = 1024
    dx = sign * 0.0977
    lo = 0.0 if sign > 0 else 100.0
    got = gpu_density(v, m, lo, dx)
    want, cnt, mag = reference_density(v if sign > 0 else v[::-1], m, lo, dx)
    # the bit-for-bit order holds for inner cells of at most 32 sources
    inner = np.zeros(m, dtype=bool)
    inner[1:-1] = True
    few = inner & (cnt <= 32)
    np.testing.assert_array_equal(got[few], want[few])
    assert np.all(np.abs(got - want) <= 2.0 * (cnt + 1) * 2.0 ** -53 * mag)


@pytest.mark.parametrize("m", [256, 1024, 1 << 13, 1 << 14, 1 << 15, 1 << 16, 1 << 17, 1 << 18,
                               1 << 20])
@pytest.mark.parametrize("order", [2, 6, 8])
def test_every_row_length(oracle, m, order):
    """Row lengths 16 to 1024 of both passes, the spectral product on the way
    into the inverse one; the bar of the other grid tests."""
    ev = spectra.harness_spectrum(3000)
    eta = 1.0 / math.sqrt(3000)
    re, im = gpu_opts(ev, eta, order=order, m=m)
    o_re, o_im = oracle.fft5_points(ev, ev, eta, order=order, m=m)
    assert close(re, im, o_re, o_im)
