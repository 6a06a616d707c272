"""Null pointers are refused as arguments, for pairs that travel as kernel arguments (up to 1,000) and
for those that are copied, and leave the context usable."""
import ctypes

import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 1001])
@pytest.mark.parametrize("null", range(5))
def test_elems_refuse_null(n, null):
    import shci_gb300
    from shci_gb300 import _lib
    c = shci_gb300.Context(0)
    c.load_fcidump(C_ATOM, 4, 2, "d2h")
    v = [np.full(n, 0b1111, np.uint64), np.full(n, 0b11, np.uint64),
         np.full(n, 0b10111, np.uint64), np.full(n, 0b11, np.uint64), np.zeros(n)]
    f = ctypes.CDLL(_lib.LIB_PATH).shci_hamiltonian_elems  # (a prototype that takes null pointers)
    p = [ctypes.c_void_p(a.ctypes.data if k != null else None) for k, a in enumerate(v)]
    assert f(c.h, p[0], p[1], p[2], p[3], ctypes.c_size_t(n), p[4]) == 2  # SHCI_ERR_ARG
    assert np.all(v[4] == 0.0)
    assert np.all(np.isfinite(c.h_elems(*v[:4])))
    c.close()
