"""The run log's grid and thread count are those of the launch, for a run of so few photons that it gets fewer blocks than
fit, for one that fills the device, and for a device listed twice."""

from __future__ import annotations

import re

import pytest

from mcx_gb300 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("photons,devices", [(100_000, None), (3_000_000, None), (200_000, [0, 0])])
def test_log_states_the_launch(engine, capfd, photons, devices):
    cfg = problems.workload0(photons)
    small = engine.run(problems.workload0(100_000))["stat"]["grid"]
    assert small < engine.run(problems.workload0(3_000_000))["stat"]["grid"]
    capfd.readouterr()
    pc = engine.prepare(cfg, verbose=True)
    stat = engine.run_prepared(pc, devices=devices)["stat"]
    log = "".join(capfd.readouterr())
    grids = [int(g) for g in re.findall(r"grid=(\d+)", log)]
    threads = [int(t) for t in re.findall(r"with (\d+) threads", log)]
    assert len(grids) == len(devices or [1]) and len(threads) == 1, log
    assert all(g == stat["grid"] for g in grids), (grids, stat["grid"])
    assert threads[0] == sum(grids) * stat["block"]
    if photons != 3_000_000:
        assert stat["grid"] == small
