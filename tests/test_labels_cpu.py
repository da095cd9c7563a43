"""Widening and transposing of C-ordered label volumes (mcxg_widen_labels) against numpy, over every item size and
sign, and grids below, at and past the 32 x 32 tile and the size at which threads share the work."""

from __future__ import annotations

import numpy as np
import pytest

GRIDS = [(1, 1, 1), (1, 5, 3), (33, 2, 31), (32, 32, 32), (7, 1, 70), (65, 130, 67)]


@pytest.mark.parametrize("grid", GRIDS, ids=str)
@pytest.mark.parametrize("dtype", ["u1", "i1", "u2", "i2", "u4", "i4", "u8", "i8", "?"])
def test_widen_labels_is_numpys_fortran_ravel(grid, dtype):
    from mcx_gb300._lib import lib

    rng = np.random.default_rng(sum(grid))
    vol = rng.integers(-100 if "i" in dtype else 0, 2 if dtype == "?" else 120, grid).astype(dtype)
    dst = np.full(vol.size + 2, 0xABCD, np.uint32)
    rc = lib.mcxg_widen_labels(vol.ctypes.data, vol.dtype.itemsize, int(vol.dtype.kind == "i"), *grid, dst[1:].ctypes.data)
    assert rc == 0
    assert np.array_equal(dst[1:-1], vol.astype(np.uint32).ravel(order="F"))
    assert dst[0] == dst[-1] == 0xABCD


def test_prepared_volume_is_the_same_from_either_order():
    from mcx_gb300 import prepare, problems

    c = problems.workload1(10)
    rng = np.random.default_rng(3)
    c["vol"] = rng.integers(1, 3, (41, 57, 33)).astype(np.uint8)
    c["srcpos"] = [20.0, 20.0, 0.0]
    a, b = prepare(c), prepare(dict(c, vol=np.asfortranarray(c["vol"])))
    assert np.array_equal(a.vol, b.vol) and a.c.mediabyte == b.c.mediabyte and a.c.isrowmajor == b.c.isrowmajor == b"\x00"


def test_widen_labels_refuses_what_it_cannot_read():
    from mcx_gb300._lib import lib

    v = np.zeros(8, np.uint32)
    assert lib.mcxg_widen_labels(None, 1, 0, 2, 2, 2, v.ctypes.data) == -4
    assert lib.mcxg_widen_labels(v.ctypes.data, 3, 0, 2, 2, 2, v.ctypes.data) == -4
    assert lib.mcxg_widen_labels(v.ctypes.data, 1, 0, 0, 2, 2, v.ctypes.data) == -4
