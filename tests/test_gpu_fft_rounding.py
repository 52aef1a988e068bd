"""The grid methods' transforms carry no more rounding than a transform with
exact twiddles.

The convolution of a given density, read at the grid points themselves (where
the interpolation weights are exactly 0 and 1), against the same pipeline in
extended precision from the same kernel samples.

Tolerance: the rms error of an FFT in double precision with twiddles rounded
once is about 0.6 u sqrt(log2 m) (Schatzman, SIAM J. Sci. Comput. 17, 1996;
u = 2^-53).  White noise of that size after each of the two transforms of this
pipeline, with a white density as large as the kernel's spectrum, gives
0.91 u sqrt(log2 m) at the output; the product, the kernel table and its power
function add about 1.4 u: 1.02 u sqrt(log2 m) at 512 points and less above.
1.25 leaves a fifth of room; twiddles formed as powers of one another (three
products deep) give 1.6 and more.
"""
import math

import numpy as np
import pytest
import torch

from shrinkers_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [512, 1024, 2048, 4096, 65536, 1 << 18, 1 << 20])
def test_transform_rounding(m):
    L = _native.load()
    eta, dx = 0.1, 1.0
    dens = np.random.default_rng(m).standard_normal(m) * (np.pi / math.sqrt(m))
    c = np.arange(m)
    sd = np.where(c <= m // 2, c, c - m).astype(np.float64)
    odd = sd / (sd * sd + eta * eta)
    r = math.exp(-2.0 * math.pi * eta / (m * dx))
    ke = (np.pi / dx) * np.longdouble(r) ** np.minimum(c, m - c).astype(np.longdouble)
    C = np.fft.fft(dens.astype(np.clongdouble) + 1j * odd)
    Cn = np.conj(C[(m - c) % m])
    D, K = 0.5 * (C + Cn), -0.5j * (C - Cn)
    want = np.conj(np.fft.fft(np.conj(D * ke + 1j * D * K))) / m
    d = torch.from_numpy(dens).cuda()
    q = torch.arange(m, dtype=torch.float64, device="cuda")
    re, im = torch.empty_like(q), torch.empty_like(q)
    _native.check(L.shrk_nufft_eval_dev(d.data_ptr(), m, 0.0, dx, eta, q.data_ptr(), m,
                                        re.data_ptr(), im.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream))
    got = im.cpu().numpy() + 1j * re.cpu().numpy()
    rms = math.sqrt(float((np.abs(got - want) ** 2).sum() / (np.abs(want) ** 2).sum()))
    assert rms <= 1.25 * 2.0 ** -53 * math.sqrt(math.log2(m)), rms / 2.0 ** -53
