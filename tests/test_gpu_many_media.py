"""Detector runs of so many media that the plain-path kernel's records do not fit in shared memory beside its fixed arrays
run on the general kernel, at every block size it takes: the last count that fits the plain path, the first that does
not, the last that fits at all, and smaller blocks.  Every medium has the same properties, so the photons are those of one
medium and the records' columns add up to its own: the scattering counts exactly, the paths and momentum transfers
within the rounding of an FP32 sum of as many terms as there are media (2^-24 each, of at most the sum)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# media (with the background), record columns, threads a block
CASES = [(106, "dspx", 0), (107, "dspx", 0), (109, "dspx", 0), (127, "dspmx", 128), (128, "dspmx", 64)]


def _deck(media, flags):
    i, j, k = np.meshgrid(np.arange(40), np.arange(40), np.arange(40), indexing="ij")
    vol = (1 + (i + 3 * j + 7 * k) % (media - 1)).astype(np.uint8)
    return {"nphoton": 100_000, "seed": 4711, "vol": vol, "prop": np.array([[0, 0, 1, 1]] + [[0.005, 1, 0.1, 1.37]] * (media - 1), np.float32),
            "tstart": 0.0, "tend": 5e-9, "tstep": 5e-9, "srcpos": [20.0, 20.0, 0.0], "srcdir": [0.0, 0.0, 1.0], "issrcfrom0": 1,
            "isreflect": 0, "detpos": np.array([[24, 20, 0, 2], [20, 13, 0, 2]], np.float32), "issavedet": 1,
            "savedetflag": flags, "maxdetphoton": 100_000}


@pytest.mark.parametrize("media,flags,block", CASES)
def test_many_media(engine, media, flags, block):
    from mcx_gb300._lib import lib

    one = engine.run(_deck(2, flags))
    try:
        if block:
            lib.mcxg_set_launch(block, 0, 0, -1)
        many = engine.run(_deck(media, flags))
    finally:
        lib.mcxg_set_launch(0, 0, 0, -1)
    for k in ("n_steps", "n_scatter", "n_deposit", "n_photon", "n_detected", "error_flags"):
        assert many["stat"][k] == one["stat"][k], k
    assert one["stat"]["n_detected"] > 500
    # rows: detector, scatterings a medium, paths a medium, (momentum transfer a medium,) exit position
    cols, n = (3 if "m" in flags else 2), media - 1
    a, b = one["detp"].astype(np.float64), many["detp"].astype(np.float64)
    assert b.shape == (1 + cols * n + 3, a.shape[1])
    a, b = (r[:, np.lexsort(r[-3:])] for r in (a, b))
    assert (a[0] == b[0]).all() and (a[-3:] == b[-3:]).all()
    sums = b[1:1 + cols * n].reshape(cols, n, -1).sum(1)
    assert (sums[0] == a[1]).all()
    for c in range(1, cols):
        # both sides are FP32 sums along the photon: as many roundings as it has segments, at most one a step or scattering
        assert (np.abs(sums[c] - a[1 + c]) <= 2.0 ** -24 * (1000 + 2 * a[1]) * np.maximum(a[1 + c], 1e-6)).all()
