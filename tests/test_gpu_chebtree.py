"""The treecode's tree built subtree by subtree (more than 4 096 sources): bit
for bit the oracle's sums, so the same splits, node weights and order, at the
edges of the rule, around the sizes where a subtree's capacity doubles, and on
spectra whose trees are lopsided (spikes, duplicates, clusters, a geometric
range that reaches the depth cap).  Query grids take other leaf capacities.
"""
import math

import numpy as np
import pytest

import shrinkers_b200 as rk
from shrinkers_b200 import spectra

pytestmark = pytest.mark.gpu


def geometric(n, span):
    return np.sort(np.exp(np.random.default_rng(n).uniform(-span, span, n)))


def clusters():
    rng = np.random.default_rng(3)
    return np.sort(np.concatenate([1.0 + 1e-12 * rng.random(9000), 5.0 + rng.random(4000),
                                   np.linspace(0.0, 1e6, 500), np.full(3000, 0.25)]))


SPECTRA = {
    "4096": lambda: spectra.config3(4096, seed=1),
    "4097": lambda: spectra.config3(4097, seed=2),
    "16385": lambda: spectra.config3(16385, seed=3),
    "131071": lambda: spectra.config3(131071, seed=4),
    "131073": lambda: spectra.config3(131073, seed=5),
    "262145": lambda: spectra.config3(262145, seed=6),
    "log": lambda: spectra.log_spectrum(50000),
    "linear": lambda: np.linspace(0.0, 1.0, 65537),
    "duplicates": lambda: np.repeat(np.sort(np.random.default_rng(1).random(7)), 3000),
    "integers": lambda: np.sort(np.random.default_rng(2).integers(0, 300, 30000).astype(float)),
    "geometric": lambda: geometric(5000, 300.0),
    "clusters": clusters,
}


@pytest.mark.parametrize("name", SPECTRA)
@pytest.mark.parametrize("method", ["chebcode", "chebcode_fast", "chebcode_xtreme"])
def test_tree_bit_exact(oracle, name, method):
    ev = SPECTRA[name]()
    eta = 1.0 / math.sqrt(ev.size)
    if ev.size > 20000:  # every subtree through a spread of queries
        q = np.ascontiguousarray(ev[:: ev.size // 17001 + 1])
        got = rk.stieltjes_at_points(q, ev, eta, method=method)
        re, im = oracle.compute_at_points(q, ev, eta, method)
    else:
        got = rk.stieltjes_transform(ev, eta=eta, method=method)
        re, im = oracle.compute_all(ev, eta, method, parallel=True)
    np.testing.assert_array_equal(got["real"], re)
    np.testing.assert_array_equal(got["imag"], im)


def test_eta_outside_the_branch_free_range(oracle):
    """eta and distances beyond 2^+-200: the compiler's reciprocals take over."""
    ev = np.sort(np.random.default_rng(9).random(6000))
    for scale, eta in ((1.0, 1e-70), (1e70, 1e68), (1e-70, 1e-72)):
        got = rk.stieltjes_transform(ev * scale, eta=eta, method="chebcode")
        re, im = oracle.compute_all(ev * scale, eta, "chebcode", parallel=True)
        np.testing.assert_array_equal(got["real"], re)
        np.testing.assert_array_equal(got["imag"], im)
