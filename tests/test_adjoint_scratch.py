"""The adjoint's pair scratch over all sizes: every J split has its own sums and list row an atom (836
bytes), so the lists may not grow with splits that large systems hardly gain from.  The bound is two rounds
of 12 resident 32-atom blocks on 148 SMs (113,664 rows, 95 MB), or one row an atom."""
import ctypes as C

import pytest

from tholedipoleplugin_b200 import _capi as A
from tholedipoleplugin_b200 import build as B

ROW = 8 * 8 + 4 * 193


@pytest.mark.parametrize("n", [1, 32, 33, 192, 1029, 6303, 6336, 12288, 12608, 12640, 28384, 28448, 56800, 56832, 56864,
                               56896, 98304, 200000, 1000000])
def test_pair_scratch(n):
    B.build()
    f = A.lib()._ZN3tdp20adjoint_pair_scratchEi   # tdp::adjoint_pair_scratch(int), in doubles
    f.argtypes, f.restype = [C.c_int], C.c_size_t
    rows = 8 * f(n) / ROW
    assert n <= rows + 1e-9
    assert rows <= max(n, 2 * 12 * 148 * 32) + 1.0
