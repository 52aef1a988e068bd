"""Eigenvectors of numerically equal eigenvalues: the warp's Gram-Schmidt over
row counts around its 32 lanes and 256 rows in flight, clusters of different
sizes in one warp, null spaces, and blocks with and without clusters side by
side.  Against LAPACK with the bars of test_gpu_matrix.py: 1e-13 of the largest
eigenvalue, 1e-12 residual and orthogonality.
"""
import numpy as np
import pytest

import shrinkers_b200 as rk

pytestmark = pytest.mark.gpu


def check(a):
    p = a.shape[0]
    w, v = rk.symmetric_eigh(a)
    w_ref = np.linalg.eigvalsh(a)
    assert np.max(np.abs(w - w_ref)) <= 1e-13 * np.max(np.abs(w_ref))
    assert np.max(np.abs(a @ v - v * w)) <= 1e-12 * np.max(np.abs(a))
    assert np.max(np.abs(v.T @ v - np.eye(p))) <= 1e-12


def with_spectrum(ev, seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((ev.size, ev.size)))
    a = (q * ev) @ q.T
    return np.ascontiguousarray((a + a.T) / 2)


@pytest.mark.parametrize("p", [5, 31, 32, 33, 64, 100, 255, 256, 257, 300, 513])
def test_repeated(p):
    """Four values, a quarter of the spectrum each, and a few single ones."""
    ev = np.repeat([1.0, 2.0, 5.0, 9.0], (p + 3) // 4)[:p]
    ev[: p // 10] = np.linspace(0.2, 0.7, p // 10)
    check(with_spectrum(ev, p))


@pytest.mark.parametrize("sizes", [[2] * 40, [3, 17, 1, 33, 1, 1, 50, 2], [200, 1, 1]])
def test_cluster_sizes(sizes):
    ev = np.repeat(np.linspace(1.0, 4.0, len(sizes)), sizes)
    check(with_spectrum(ev * (1.0 + 1e-15 * np.arange(ev.size)), len(sizes)))


@pytest.mark.parametrize("p,rank", [(60, 20), (300, 150), (700, 233), (900, 450), (1300, 433)])
def test_null_space(p, rank):
    x = np.random.default_rng(p).standard_normal((p, rank))
    check(np.ascontiguousarray(x @ x.T / rank))


def test_blocks():
    """Decoupled blocks of one to 90 rows, every other one with equal values."""
    a = np.zeros((400, 400))
    i = 0
    for k, n in enumerate([1, 2, 33, 64, 90, 5, 80, 40, 85]):
        ev = np.full(n, 2.0 + k) if k % 2 else np.linspace(1.0, 2.0 + k, n)
        ev[: n // 4] = 0.5
        a[i:i + n, i:i + n] = with_spectrum(ev, k)
        i += n
    check(a)
