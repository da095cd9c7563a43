"""The plain-path kernel's replay (transport_lean.cuh, absorption Jacobians) against the general kernel's, photon for photon.

As for the forward runs, a gscatter past any photon's count of scattering events takes a run off the plain path and changes
nothing else.  Counters and records equal bit for bit; the fields differ by the order of their FP32 sums only: 1e-5 of
the total and 1e-4 in the hottest 1% of voxels."""

from __future__ import annotations

import numpy as np
import pytest

from mcx_gb300 import problems

pytestmark = pytest.mark.gpu

WLTOF = 9


def _mixed(**kw):
    """Three indices, a void pocket and an inclusion, on a grid of odd edges."""
    vol = np.ones((37, 61, 53), np.uint8)
    vol[5:20, 20:40, 10:40] = 2
    vol[22:30, 30:45, 15:20] = 0
    return dict({"nphoton": 100_000, "seed": 77, "vol": vol,
                 "prop": np.array([[0, 0, 1, 1], [0.005, 1, 0.01, 1.37], [0.02, 3, 0.8, 1.5]], np.float32),
                 "tstart": 0.0, "tend": 5e-9, "tstep": 5e-9, "srcpos": [17.3, 29.8, 0.0], "srcdir": [0.3, 0.2, np.sqrt(0.87)],
                 "issrcfrom0": 1, "isreflect": 1, "detpos": np.array([[17, 25, 0, 2], [12, 30, 0, 2.5]], np.float32),
                 "issavedet": 1, "savedetflag": "dsp", "maxdetphoton": 100000}, **kw)


DECKS = {
    "cube": (lambda: problems.cube60b(300_000), {}),
    "time of flight": (lambda: problems.cube60b(300_000), {"outputtype": WLTOF}),
    "a few photons": (lambda: _mixed(nphoton=300), {}),
    "indices and a void": (_mixed, {}),
    "no reflection, every field of a record": (lambda: _mixed(isreflect=0, savedetflag="dspmxvw"), {}),
    "boundaries": (lambda: _mixed(bc="m_r_ca001011"), {}),
    "gates, detectors apart": (lambda: _mixed(tstep=2e-10), {"replaydet": -1}),
    "one detector": (_mixed, {"replaydet": 2}),
    "gate groups, detectors apart, time of flight": (lambda: _mixed(tstep=5e-10, maxgate=3), {"replaydet": -1, "outputtype": WLTOF}),
    "late window": (_mixed, {"tstart": 5e-10, "tend": 2e-9, "tstep": 1e-10}),
    "a chosen source": (_mixed, {"srcid": 1}),
    "no absorption": (lambda: _mixed(prop=np.array([[0, 0, 1, 1], [0, 1, 0.01, 1.37], [0.02, 3, 0.8, 1.5]], np.float32)), {}),
}


@pytest.mark.parametrize("name", DECKS)
def test_replay_runs_the_general_kernels_photons(engine, name):
    deck, extra = DECKS[name]
    cfg = deck()
    rec = engine.run(dict(cfg, issaveseed=1))
    at = np.lexsort(rec["detp"][::-1])
    cfg = dict(cfg, seed=np.asfortranarray(rec["seeds"][:, at]), detphotons=np.asfortranarray(rec["detp"][:, at]),
               outputtype="jacobian", isnormalized=0)
    cfg.update(extra)
    a = engine.run(dict(cfg))
    b = engine.run(dict(cfg, gscatter=15_000_000))
    for k in ("n_steps", "n_scatter", "n_deposit", "n_launch", "n_photon", "n_detected", "n_tile_deposit", "error_flags"):
        assert a["stat"][k] == b["stat"][k], (k, a["stat"][k], b["stat"][k])
    assert a["stat"]["n_photon"] > 0
    for k in ("energytot", "energyabs", "e_escape", "e_detect", "e_absdep", "e_absother"):
        assert abs(a["stat"][k] - b["stat"][k]) <= 1e-6 * b["stat"]["e_launch"], k
    assert np.array_equal(a["detp"][:, np.lexsort(a["detp"][::-1])], b["detp"][:, np.lexsort(b["detp"][::-1])])
    fa, fb = a["flux"].astype(np.float64), b["flux"].astype(np.float64)
    assert fa.shape == fb.shape and fb.sum() > 0
    assert abs(fa.sum() - fb.sum()) <= 1e-5 * abs(fb.sum())
    hot = fb >= np.quantile(fb, 0.99)
    assert (np.abs(fa - fb)[hot] <= 1e-4 * np.abs(fb)[hot]).all()
