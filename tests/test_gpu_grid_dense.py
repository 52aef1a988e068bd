"""The FFT grid's splat of many sources in one cell (a spectrum with a null
space: eigenvalues that are exactly zero): a run of equal cells that spans
chunks of 512 sources, around the number of chunks from which a warp adds the
chunks' sums.

n equal sources have the density n times that of one of them, each weight's sum
of one sign: at most 16 + 5 additions inside a chunk, C chunks added one by one
up to eight and over 32 lanes with 5 more above, the tail and four runs, so
off by at most (21 + 8 + C/32 + 5 + 5) u of itself.  The whole transform with the
8-node stencil against the oracle, 1e-10 of the largest value as in the other
tests of these methods.
"""
import math

import numpy as np
import pytest
import torch

import shrinkers_b200 as rk
from shrinkers_b200 import _native, spectra

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def density(v, m, lo, dx):
    d, out = torch.from_numpy(np.ascontiguousarray(v)).cuda(), torch.empty(m, dtype=torch.float64,
                                                                         device="cuda")
    _native.check(_native.load().shrk_nufft_density_dev(
        d.data_ptr(), d.numel(), m, lo, dx, out.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [511, 513, 4000, 4096, 4097, 4607, 4608, 4609, 5200, 20000, 300000,
                               1000003])
@pytest.mark.parametrize("before", [0, 300])
@pytest.mark.parametrize("cell", [20.4, 31.7])  # the four cells in one warp's window, in two
def test_one_dense_cell(n, before, cell):
    m, lo, dx = 256, 0.0, 1.0
    one = density(np.array([cell]), m, lo, dx)
    got = density(np.concatenate([np.full(before, 3.25), np.full(n, cell), [200.5]]), m, lo, dx)
    want = n * one
    at = np.abs(want) > 0
    at[:8] = False
    at[190:] = False
    assert at.sum() == 4
    chunks = n / 512 + 2
    assert np.all(np.abs(got[at] - want[at]) <= (39 + chunks / 32) * U * np.abs(want[at]))


@pytest.mark.parametrize("p,zeros", [(30000, 12000), (30000, 30000), (120001, 90000)])
def test_null_space(oracle, p, zeros):
    ev = np.sort(np.concatenate([np.zeros(zeros), spectra.config2(p)[:p - zeros]]))
    eta = 1.0 / math.sqrt(p)
    got = rk.stieltjes_transform(ev, eta=eta, method="fft5")
    q = ev[:: p // 500]
    re, im = oracle.fft5_points(q, ev, eta)
    scale = np.max(np.hypot(re, im))
    assert np.max(np.abs(got["real"][:: p // 500] * p - re)) <= 1e-10 * scale
    assert np.max(np.abs(got["imag"][:: p // 500] * p - im)) <= 1e-10 * scale
