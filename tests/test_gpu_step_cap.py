"""The per-photon step cap ends a photon wherever its last step ends, on a periodic face too: there the photon goes on
at the other side when its time is over or it has left, but not past the cap.  A slab one voxel thick, periodic on
every axis, so that about half of all steps end on such a face; runs of one photon each, so that each has to report
the cap itself.  A photon scatters every 50 mm, and ends by its time window at a scattering if the cap fails to."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gscatter", [1_000_000_000, 15_000_000], ids=["plain path", "general kernel"])
def test_step_cap_on_periodic_faces(engine, gscatter):
    from mcx_gb300._lib import lib

    deck = {"nphoton": 1, "vol": np.ones((40, 40, 1), np.uint8), "prop": np.array([[0, 0, 1, 1], [0.001, 0.02, 0.5, 1.37]], np.float32),
            "tstart": 0.0, "tend": 2e-7, "tstep": 2e-7, "srcpos": [20.0, 20.0, 0.0], "srcdir": [0.0, 0.0, 1.0], "issrcfrom0": 1,
            "isreflect": 0, "issavedet": 0, "bc": "cccccc", "gscatter": gscatter}
    try:
        lib.mcxg_set_step_cap(100)
        for seed in range(1, 17):
            with pytest.raises(engine.MCXError, match="step cap"):
                engine.run(dict(deck, seed=seed))
    finally:
        lib.mcxg_set_step_cap(0)
    r = engine.run(dict(deck, seed=1, tend=2e-9, tstep=2e-9))
    assert r["stat"]["error_flags"] == 0 and r["stat"]["n_photon"] == 1
