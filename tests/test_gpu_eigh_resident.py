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


@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (129, 128, 65), (128, 131, 71), (256, 384, 64),
                                   (1200, 1111, 64), (1280, 1920, 72), (2048, 130, 600),
                                   (130, 2048, 2047)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1)])
def test_gemm_in_equal_runs(m, n, k, ta, tb):
    """The large FP64 product whose k steps are dealt out in equal runs: one
    run a tile, tiles divided among two and many CTAs, whole tiles only, ragged
    edges; with C read (beta) and not, beside a guard band that must stay.
    Each entry is a sum of k products: 4 k eps of their magnitudes."""
    import torch

    L = _native.load()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    rnd = lambda r, c: torch.randn(r, c, generator=g, device="cuda", dtype=torch.float64)
    a = rnd(m, k) if ta else rnd(k, m)  # column-major op(A) m x k
    b = rnd(k, n) if tb else rnd(n, k)
    ldc = m + 3
    opa, opb = (a if ta else a.T), (b if tb else b.T)
    for beta in (0.0, -0.75):
        c = rnd(n, ldc)
        before = c.clone()
        st = L.shrk_diag_dgemm(ta, tb, m, n, k, 1.25, a.data_ptr(), a.shape[1], b.data_ptr(),
                               b.shape[1], beta, c.data_ptr(), ldc, None)
        _native.check(st, "dgemm")
        torch.cuda.synchronize()
        ref = 1.25 * (opa @ opb) + beta * before[:, :m].T
        bound = 4 * k * np.finfo(float).eps * (1.25 * (opa.abs() @ opb.abs()) + before[:, :m].T.abs())
        assert bool(((c[:, :m].T - ref).abs() <= bound).all())
        assert torch.equal(c[:, m:], before[:, m:])
