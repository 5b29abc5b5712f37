"""adv1, divergence and projection with several z cells a thread (grids from 0.6 and 0.7 M cells on) against the CPU oracle, on a
grid that leaves ragged rows and columns and a last thread with one cell of two and three of four.  Tolerance: the stage
parity's of tests/test_gpu_stages.py (the arithmetic is the same)."""
import numpy as np
import pytest

import fire_cases as FC
from test_gpu_stages import ATOL, OUTLIERS, OUTPUTS, RTOL

pytestmark = pytest.mark.gpu
CASE = dict(FC.C1, res=(100, 110, 71), size=(1.25, 1.375, 0.8875))


@pytest.mark.parametrize("stage", ["adv1", "div", "project"])
def test_columns_match_oracle(stage):
    sim, orc = FC.make_pair(CASE, params={"windX": 0.6, "windZ": -0.3, "gust": 0.5})
    dt = CASE["dt"]
    FC.sync_block(sim, orc, dt)
    sim.run_stage("geo", dt)
    orc.stage("geo")
    FC.put_state(sim, orc, FC.random_state(CASE["res"], 3))
    FC.sync_block(sim, orc, dt)
    if stage == "project":
        p = (FC.smooth_noise(CASE["res"][::-1], np.random.default_rng(5)) * 0.02).astype(np.float32)
        sim.set_level(0, "p", p)
        orc.put_level(0, "p", p)
    sim.run_stage(stage, dt)
    sim.sync()
    orc.stage(stage)
    if stage == "div":
        FC.compare(sim.level(0, "b"), orc.get_level(0, "b"), RTOL, ATOL, OUTLIERS, what="div")
    for name in OUTPUTS.get(stage, []):
        g, o = sim.download(name), orc.get(name)
        for c in range(4):
            FC.compare(g[..., c], o[..., c], RTOL, ATOL, OUTLIERS, what=f"{stage}:{name}[{c}]")
    sim.close()
