"""Combustion below the ignition window with a uniform that is not finite: a product with an exact 0 is then not 0, so the forces
kernel must not leave the terms out.  Against the CPU oracle, which evaluates everything; tolerance: the stage parity's of
tests/test_gpu_stages.py.  Cold gas throughout, so every cell sits below the window."""
import numpy as np
import pytest

import fire_cases as FC
from test_gpu_stages import ATOL, OUTLIERS, OUTPUTS, RTOL, _stage_case, campfire  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["rs", "kMix", "heatOut", "expansion"])
def test_cold_gas_with_an_infinite_uniform(campfire, name):  # noqa: F811
    sim, orc, dt = _stage_case(campfire, "forces", seed=5)
    state = FC.random_state(FC.C1["res"], 5)
    for key in ("SY", "S"):
        state[key][..., 0] = 0.05
    sim.set_params({name: float("inf")})
    FC.put_state(sim, orc, state)
    FC.sync_block(sim, orc, dt)
    sim.run_stage("forces", dt)
    sim.sync()
    orc.stage("curl")
    orc.stage("forces")
    for out in OUTPUTS["forces"]:
        g, o = sim.download(out), orc.get(out)
        for c in range(4):
            FC.compare(g[..., c], o[..., c], RTOL, ATOL, OUTLIERS, what=f"{name}:{out}[{c}]")
    sim.close()
