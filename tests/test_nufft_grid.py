"""The NUFFT's grid rule ends for every spectrum, descending ones included.

A descending spectrum has a negative range, and where the padding does not make
up for it the wanted size is negative: the reference's saturating conversion
takes it as zero, so the grid is the smallest one (nufft.rs:106-126).  The rule
runs in a child process, so that one which never ends fails here.
"""
import subprocess
import sys

import pytest

from shrinkers_b200 import _native

ROOT = _native.__file__.rsplit("/", 2)[0]
CODE = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
from shrinkers_b200 import _native
L = _native.load()
m, lo, dx = C.c_int64(), C.c_double(), C.c_double()
_native.check(L.shrk_nufft_grid({first!r}, {last!r}, {eta!r}, C.byref(m), C.byref(lo), C.byref(dx)))
from oracle import oracle as O
assert O.nufft_grid_size({last!r} - {first!r}, {eta!r}) == m.value
print(m.value, repr(lo.value), repr(dx.value))
"""


@pytest.mark.parametrize("first,last,eta,m", [(530.0, 0.0, 0.1052, 8192), (20.0, 0.2, 1e-3, 8192),
                                              (1e300, -1e300, 1.0, 8192), (2.0, 0.0, 0.1, 32768),
                                              (0.0, 530.0, 0.1052, 65536), (1.0, 1.0, 0.5, 32768)])
def test_grid_size(oracle, first, last, eta, m):
    code = CODE.format(root=ROOT, first=first, last=last, eta=eta)
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    got, lo, dx = out.stdout.split()
    assert int(got) == m
    pad = max(2000.0 * eta, 0.75 * (last - first))
    assert float(lo) == first - pad
    assert float(dx) == (last + pad - (first - pad)) / m
