"""The finiteness check of the Python functions answers with its ValueError, or
not at all: no numpy warning, whatever the values and numpy's error state."""
import warnings

import numpy as np
import pytest

import shrinkers_b200 as rk

FINITE = [np.empty(0), np.array([1.0, 2.0]), np.full(3, 1.7e308), np.array([1.7e308, -1.7e308] * 4),
          np.array([5e-324, 0.0, -0.0])]
NOT = [np.array([np.inf, -np.inf]), np.array([1.0, np.nan]), np.array([-np.inf, 1.0]),
       np.array([np.inf, 1.7e308, np.nan])]


@pytest.mark.parametrize("ev", FINITE + NOT, ids=str)
def test_no_warning(ev):
    with warnings.catch_warnings(), np.errstate(all="raise"):
        warnings.simplefilter("error")
        if any(ev is a for a in NOT):
            with pytest.raises(ValueError, match="must be finite"):
                rk._require_finite(ev, "eigenvalues")
        else:
            rk._require_finite(ev, "eigenvalues")
