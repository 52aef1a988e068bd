"""The eigensolver's resident tridiagonalisation at the edges of its forms: row
counts around the thread blocks (256 and 512 rows a step), the step from 256 to
512 threads, the largest matrix it holds and the first sizes where it takes
over from the form that streams the matrix; reflectors that vanish; and the
bounded wait's timeout.  Against LAPACK with the bars of test_gpu_matrix.py:
1e-13 of the largest eigenvalue, 1e-12 residual and orthogonality.
"""
import ctypes as C

import numpy as np
import pytest

import shrinkers_b200 as rk
from shrinkers_b200 import _native

pytestmark = pytest.mark.gpu


def check(a):
    p = a.shape[0]
    w, v = rk.symmetric_eigh(a)
    w_ref = np.linalg.eigvalsh(a)
    scale = max(np.max(np.abs(w_ref)), 1e-300)
    assert np.max(np.abs(w - w_ref)) <= 1e-13 * scale
    assert np.max(np.abs(a @ v - v * w)) <= 1e-12 * max(np.max(np.abs(a)), 1e-300)
    assert np.max(np.abs(v.T @ v - np.eye(p))) <= 1e-12


@pytest.mark.parametrize("p", [3, 4, 5, 149, 150, 255, 257, 258, 513, 514, 1281, 1282, 1537, 2049,
                               2050, 2052])
def test_sizes(p):
    rng = np.random.default_rng(p)
    x = rng.standard_normal((2 * p, p)) + rng.standard_normal((2 * p, 1)) @ rng.standard_normal((1, p))
    check(np.ascontiguousarray(x.T @ x / (2 * p)))


@pytest.mark.parametrize("kind", ["diagonal", "blocks", "tridiagonal", "rank one", "zero column"])
def test_vanishing_reflectors(kind):
    p = 300
    rng = np.random.default_rng(1)
    a = np.zeros((p, p))
    if kind == "diagonal":
        a[np.arange(p), np.arange(p)] = rng.standard_normal(p)
    elif kind == "blocks":
        for i in range(0, p, 60):
            b = rng.standard_normal((60, 60))
            a[i:i + 60, i:i + 60] = b + b.T
    elif kind == "tridiagonal":
        a[np.arange(p), np.arange(p)] = rng.standard_normal(p)
        e = rng.standard_normal(p - 1)
        a[np.arange(p - 1), np.arange(1, p)] = a[np.arange(1, p), np.arange(p - 1)] = e
    elif kind == "rank one":
        u = rng.standard_normal(p)
        a = np.eye(p) + np.outer(u, u)
    else:
        b = rng.standard_normal((p, p))
        a = b + b.T
        a[:, 120] = a[120, :] = 0.0
    check(np.ascontiguousarray(a))


def test_wait_budget_of_zero_times_out():
    L = _native.load()
    p = 200
    x = np.random.default_rng(2).standard_normal((p, p))
    a = np.ascontiguousarray(x + x.T)
    w = np.empty(p)
    D = C.POINTER(C.c_double)
    args = (a.ctypes.data_as(D), p, w.ctypes.data_as(D), None)
    old = L.shrk_diag_set_wait_limit(0)
    try:
        assert L.shrk_symmetric_eigh(*args) == _native.SHRK_ETIMEOUT
    finally:
        L.shrk_diag_set_wait_limit(-1)
    assert old > 0
    assert L.shrk_symmetric_eigh(*args) == _native.SHRK_OK
    assert np.max(np.abs(w - np.linalg.eigvalsh(a))) <= 1e-13 * np.max(np.abs(w))
