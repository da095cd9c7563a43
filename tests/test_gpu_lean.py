"""The plain-path transport kernel (transport_lean.cuh) against the general one, photon for photon.

A gscatter (scattering events after which mus' replaces mus) below the step cap but past any photon's
count takes a run off the plain path and changes nothing else: the general kernel then runs the same
photons into the same FP32 field.  Every counter
must be equal and every detected record equal bit for bit; the fields differ by the order of the FP32
sums only, which the accumulation tests bound by 1e-5 of the total and 1e-4 in the hottest 1% of voxels."""

from __future__ import annotations

import numpy as np
import pytest

from mcx_gb300 import problems

pytestmark = pytest.mark.gpu


def _medium(n, row):
    c = problems.workload0(n, seed=5)
    c["prop"] = np.array([[0, 0, 1, 1], row], np.float32)
    return c


def _mixed(n, **kw):
    """Three indices, a void pocket and an inclusion, on a grid of odd edges."""
    vol = np.ones((37, 61, 53), np.uint8)
    vol[5:20, 20:40, 10:40] = 2
    vol[22:30, 30:45, 15:20] = 0
    return dict({"nphoton": n, "seed": 77, "vol": vol,
                 "prop": np.array([[0, 0, 1, 1], [0.005, 1, 0.01, 1.37], [0.02, 3, 0.8, 1.5]], np.float32),
                 "tstart": 0.0, "tend": 5e-9, "tstep": 5e-10, "srcpos": [17.3, 29.8, 0.0], "srcdir": [0.3, 0.2, np.sqrt(0.87)],
                 "issrcfrom0": 1, "isreflect": 1, "detpos": np.array([[17, 25, 0, 2], [12, 30, 0, 2.5]], np.float32),
                 "issavedet": 1, "savedetflag": "dspmxvw", "maxdetphoton": 200000}, **kw)


DECKS = {
    "one photon": lambda: problems.workload0(1),
    "a warp and one": lambda: problems.workload0(33),
    "cube": lambda: problems.workload0(300_000),
    "photons drawn ahead": lambda: problems.workload0(700_001),
    "photons drawn a warp ahead": lambda: problems.workload0(2_000_033),
    "drawn ahead among indices and a void": lambda: _mixed(700_001, isreflect=0, issavedet=0),
    "sphere, gates, detectors": lambda: problems.workload1(200_000),
    "void to skip": lambda: problems.workload2(50_000, n=64),
    "indices and a void": lambda: _mixed(200_000),
    "no reflection": lambda: _mixed(200_000, isreflect=0),
    "every boundary": lambda: _mixed(100_000, bc="m_r_ca001011", isreflect=0),
    "mirror and cyclic": lambda: _mixed(50_000, bc="mcrmcr"),
    "late window": lambda: _mixed(100_000, tstart=5e-10, tend=2e-9, tstep=1e-10),
    "gate groups": lambda: _mixed(100_000, maxgate=3),
    "energy": lambda: _mixed(100_000, outputtype="energy"),
    "no scattering": lambda: _medium(100_000, [0.01, 0, 1, 1.37]),
    "no absorption": lambda: _medium(100_000, [0, 1, 0.9, 1.37]),
    "isotropic scattering": lambda: _medium(100_000, [0.005, 1, 0, 1.37]),
    "planar": lambda: problems.cube60planar(200_000),
    "disk": lambda: _mixed(100_000, srctype="disk", srcparam1=[9, 0, 0, 0]),
    "few photons of a planar source": lambda: problems.cube60planar(5_000),
    "half a warp's photons of a disk": lambda: _mixed(20_000, srctype="disk", srcparam1=[9, 0, 0, 0]),
    "few photons, detectors": lambda: _mixed(9_001),
    "isotropic source": lambda: _mixed(100_000, srctype="isotropic", srcpos=[12.3, 14.2, 20.6]),
}


@pytest.mark.parametrize("name", DECKS)
def test_plain_path_runs_the_general_kernels_photons(engine, name):
    a = engine.run(DECKS[name]())
    b = engine.run(dict(DECKS[name](), gscatter=15_000_000))
    for k in ("n_steps", "n_scatter", "n_deposit", "n_launch", "n_photon", "n_detected", "n_tile_deposit", "error_flags"):
        assert a["stat"][k] == b["stat"][k], (k, a["stat"][k], b["stat"][k])
    for k in ("energytot", "energyabs", "e_escape", "e_detect", "e_absdep", "e_absother"):
        assert abs(a["stat"][k] - b["stat"][k]) <= 1e-6 * b["stat"]["e_launch"], k
    assert ("detp" in a) == ("detp" in b)
    if "detp" in a:
        assert np.array_equal(a["detp"][:, np.lexsort(a["detp"][::-1])], b["detp"][:, np.lexsort(b["detp"][::-1])])
    fa, fb = a["flux"].astype(np.float64), b["flux"].astype(np.float64)
    assert abs(fa.sum() - fb.sum()) <= 1e-5 * abs(fb.sum())
    hot = fb >= np.quantile(fb, 0.99)
    assert (np.abs(fa - fb)[hot] <= 1e-4 * np.abs(fb)[hot]).all()
