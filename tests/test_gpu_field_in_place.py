"""The fluence added to the caller's host field by the GPU in place: what was there stays and is added to, nothing
beside the field is touched, whatever the field's alignment, from one voxel to many pages, over gate groups.

A field of values that are whole multiples of the sums' spacing gives exact additions, so the run into a prefilled field
is the run into zeros plus the filling to one rounding of FP32 (the order of the photons' own sums: 1e-6 of the largest)."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from mcx_gb300 import problems

pytestmark = pytest.mark.gpu


def _run_into(engine, cfg, field):
    from mcx_gb300 import api
    from mcx_gb300._lib import lib, libc

    pc = engine.prepare(cfg)
    nact, info = api._active_devices(pc.c)
    assert nact >= 1
    pc.c.exportfield = field.ctypes.data
    try:
        lib.mcx_run_simulation(C.byref(pc.c), info)
        api._check()
    finally:
        libc.free(info)
        api._take_detected(pc)
    return pc


@pytest.mark.parametrize("edge,gates,maxgate,off", [(1, 1, 0, 1), (5, 3, 0, 3), (40, 1, 0, 0), (60, 50, 0, 7), (33, 10, 4, 2)])
def test_field_is_added_to_in_place(engine, edge, gates, maxgate, off):
    cfg = problems.workload0(50_000, seed=11)
    cfg.update(vol=np.ones((edge, edge, edge), np.uint8), srcpos=[edge // 2, edge // 2, 0], tstep=5e-9 / gates, maxgate=maxgate,
               isnormalized=0)
    held = maxgate or gates
    n = edge ** 3 * held
    zero = np.zeros(n + 16, np.float32)
    _run_into(engine, cfg, zero[off:off + n])
    assert (zero[:off] == 0).all() and (zero[off + n:] == 0).all()
    total = zero[off:off + n].astype(np.float64)
    assert total.sum() > 0
    full = np.full(n + 16, 3.0, np.float32)
    _run_into(engine, cfg, full[off:off + n])
    assert (full[:off] == 3).all() and (full[off + n:] == 3).all()
    tol = 1e-6 * (total.max() + 3.0) * (1 + gates // held)
    assert np.abs(full[off:off + n] - (total + 3.0)).max() <= tol
