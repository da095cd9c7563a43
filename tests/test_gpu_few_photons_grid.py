"""The blocks that a run of few photons gets: a third of the device's where most photons soon leave through the face they came
in by, one photon a thread where they live alike (a source inside, a thin or nearly clear slab), on either kernel; and
all of them for a run that fills them."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _deck(photons, **kw):
    return dict({"nphoton": photons, "seed": 9, "vol": np.ones((60, 60, 60), np.uint8),
                 "prop": np.array([[0, 0, 1, 1], [0.005, 1.0, 0.01, 1.37]], np.float32), "tstart": 0.0, "tend": 5e-9, "tstep": 5e-9,
                 "srcpos": [29.0, 29.0, 0.0], "srcdir": [0.0, 0.0, 1.0], "issrcfrom0": 1, "isreflect": 0, "issavedet": 0}, **kw)


def _void():
    v = np.ones((60, 60, 60), np.uint8)
    v[:, :, :10] = 0
    return v


ALIKE = {
    "isotropic inside": {"srctype": "isotropic", "srcpos": [29.3, 29.3, 30.2]},
    "beam from inside": {"srcpos": [29.3, 29.3, 30.2]},
    "nearly clear": {"prop": np.array([[0, 0, 1, 1], [0.005, 0.1, 0.01, 1.37]], np.float32)},
    "forward scattering": {"prop": np.array([[0, 0, 1, 1], [0.005, 1.0, 0.9, 1.37]], np.float32)},
    "thin": {"vol": np.ones((60, 60, 6), np.uint8)},
}
FACE = {
    "beam at the face": {},
    "oblique": {"srcdir": [0.6, 0.0, 0.8]},
    "from outside": {"srctype": "planar", "srcpos": [10.0, 10.0, -10.0], "srcparam1": [40.0, 0, 0, 0], "srcparam2": [0, 40.0, 0, 0]},
    "behind a void": {"vol": _void()},
}


@pytest.mark.parametrize("gscatter", [1_000_000_000, 15_000_000], ids=["plain path", "general kernel"])
@pytest.mark.parametrize("name", [*ALIKE, *FACE])
def test_blocks_of_a_run_of_few_photons(engine, name, gscatter):
    kw = dict({**ALIKE, **FACE}[name], gscatter=gscatter)
    grid = lambda n: engine.run(_deck(n, **kw))["stat"]["grid"]  # noqa: E731
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    full, few, one = grid(4_000_000), grid(200 * 3 * sms), grid(200 * sms)
    assert full in (3 * sms, 4 * sms)
    assert (few, one) == ((sms, sms) if name in FACE else (3 * sms, sms)), (few, one, full)
