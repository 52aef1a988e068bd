"""The treecode at the sizes where its tree build changes: one CTA up to 2 048
sources, subtree by subtree up to 4 194 304, level by level above.

Forward sums and the multi-eta form bit for bit the oracle's.  The gradient
against the direct sum at sampled points: the relative error of this preset
was 1.2e-10 at 20 000 values and 7.7e-10 at 200 000 (6.4 times a decade), so
8.9e-9 is expected at 4.2 million; four times that is allowed.
"""
import ctypes as C
import math

import numpy as np
import pytest

import shrinkers_b200 as rk
from shrinkers_b200 import _native, spectra

pytestmark = pytest.mark.gpu
_D = C.POINTER(C.c_double)
PRESETS = {"chebcode": (0.5, 11, 32), "chebcode_fast": (1.0, 8, 32),
           "chebcode_xtreme": (0.25, 11, 16), "chebcode_balanced": (0.55, 11, 32)}
XTREME = 15
LAST = 4194304  # of the subtree build

_made = {}


def spectrum(p):
    if p not in _made:
        _made.clear()
        _made[p] = spectra.config3(p, seed=p % 97)
    return _made[p]


@pytest.mark.parametrize("method", PRESETS)
@pytest.mark.parametrize("p", [2048, 2049, LAST, LAST + 1])
def test_forward_bit_exact(oracle, p, method):
    ev = spectrum(p)
    eta = 1.0 / math.sqrt(p)
    if p < 10000:
        got = rk.stieltjes_transform(ev, eta=eta, method=method)
        re, im = oracle.compute_all(ev, eta, method, parallel=True)
    else:
        q = np.ascontiguousarray(ev[:: p // 1500])
        got = rk.stieltjes_at_points(q, ev, eta, method=method)
        re, im = oracle.compute_at_points(q, ev, eta, method)
    np.testing.assert_array_equal(got["real"], re)
    np.testing.assert_array_equal(got["imag"], im)


@pytest.mark.parametrize("p", [2048, 2049, LAST, LAST + 1])
def test_many_eta_bit_exact(oracle, p):
    ev = spectrum(p)
    etas = [0.5 / math.sqrt(p), 1.0 / math.sqrt(p), 0.07]
    g = rk.chebcode_evaluate_many(ev, etas, method="chebcode_fast")
    re, im = oracle.evaluate_many(ev, etas, *PRESETS["chebcode_fast"])
    np.testing.assert_array_equal(g["real"], re)
    np.testing.assert_array_equal(g["imag"], im)


@pytest.mark.parametrize("p", [2048, 2049, LAST, LAST + 1])
def test_gradient(oracle, p):
    L = _native.load()
    ev = spectra.config5(p)
    rng = np.random.default_rng(5)
    w, v, g = rng.standard_normal(p), rng.standard_normal(p), np.empty(p)
    eta = 1.0 / math.sqrt(p)
    _native.check(L.shrk_stieltjes_adjoint_treecode(ev.ctypes.data_as(_D), p, eta,
                                                    w.ctypes.data_as(_D), v.ctypes.data_as(_D),
                                                    XTREME, g.ctypes.data_as(_D)))
    assert np.all(np.isfinite(g))
    idx = np.sort(rng.choice(p, 300, replace=False))
    ref = oracle.adjoint_direct(ev, eta, w, v, idx)
    assert np.linalg.norm(g[idx] - ref) <= 3.6e-8 * np.linalg.norm(ref)
