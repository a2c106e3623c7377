"""The contact query's packed rows: more contacts than the page-locked buffer
takes (over 19/16 a rod) and fewer, arrays left out, and a short capacity."""
import ctypes

import numpy as np
import pytest

import rodgpu
from helpers import make_pair, packed_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,phi,squeeze", [(300, 0.1, 0.1, 0.9), (1200, 0.1, 0.15, 0.3), (2500, 0.2, 0.3, 0.35)])
def test_packed_rows_equal_oracle(n, d, phi, squeeze):
    sc = packed_scene(n, d=d, phi=phi, seed=81, squeeze=squeeze)
    g, o = make_pair(sc, model="nsc")
    pairs, geom, shift = o.detect(0.0)
    m = len(pairs)
    assert (16 * m > 19 * n) == (squeeze < 0.5) and m > 0
    for a, b in zip(g.detect(0.0), (pairs, geom, shift)):
        np.testing.assert_array_equal(a, b)
    found = ctypes.c_size_t()
    for keep in range(3):  # one array asked for, one row too few
        out = [np.full_like(a, -7) if k == keep else None for k, a in enumerate((pairs, geom, shift))]
        ptr = [None if a is None else a.ctypes.data_as(t) for a, t in zip(out, (
            ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_double)))]
        assert g._lib.rg_detect(g._h, 0.0, *ptr, m - 1, ctypes.byref(found)) != 0
        assert found.value == m
        np.testing.assert_array_equal(out[keep][:m - 1], (pairs, geom, shift)[keep][:m - 1])
        assert (out[keep][m - 1:] == -7).all()
