"""The eigensolver above the size that the resident tridiagonalisation holds
(2 048 rows): the form that streams the matrix runs hundreds of columns, then
hands over.  Random covariances, and columns that vanish (no reflector) around
the hand-over.  Against LAPACK with the bars of test_gpu_matrix.py: 1e-13 of the
largest eigenvalue, 1e-12 residual and orthogonality.
"""
import numpy as np
import pytest

import shrinkers_b200 as rk

pytestmark = pytest.mark.gpu
HELD = 2048


@pytest.mark.parametrize("p,zero", [(2300, None), (2500, "before"), (2500, "at"), (2500, "after"),
                                    (3071, None)])
def test_streamed_then_resident(p, zero):
    rng = np.random.default_rng(p)
    x = rng.standard_normal((p + 500, p))
    a = x.T @ x / (p + 500)
    first = p - 2 - HELD  # the first column of the resident kernel
    if zero:
        k = first + {"before": -1, "at": 0, "after": 2}[zero]
        a[:, k:k + 2] = 0.0
        a[k:k + 2, :] = 0.0
        a[k, k], a[k + 1, k + 1] = 1.5, 0.25
    a = np.ascontiguousarray((a + a.T) / 2)
    w, v = rk.symmetric_eigh(a)
    w_ref = np.linalg.eigvalsh(a)
    assert np.max(np.abs(w - w_ref)) <= 1e-13 * np.max(np.abs(w_ref))
    assert np.max(np.abs(a @ v - v * w)) <= 1e-12 * np.max(np.abs(a))
    assert np.max(np.abs(v.T @ v - np.eye(p))) <= 1e-12
