"""The terms the forces kernel leaves out where their factor is exactly 0, at and around the values where that begins: temperatures
at the ignition window's foot and at 450 K (one float below, at, above), gas without age, speeds around the limit.
Against the CPU oracle, which evaluates everything; tolerance: the stage parity's of tests/test_gpu_stages.py."""
import numpy as np
import pytest

import fire_cases as FC
from test_gpu_stages import ATOL, OUTLIERS, OUTPUTS, RTOL, _stage_case, campfire  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("age", [0.0, 0.3])
def test_forces_at_the_gates(campfire, age):  # noqa: F811
    sim, orc, dt = _stage_case(campfire, "forces", seed=4)
    state = FC.random_state(FC.C1["res"], 4)
    temps = np.array([0.0, 1e-6, 0.157, 0.9], np.float32)
    foot = np.float32((float(sim.params["ignT"]) - 50.0 - 293.0) / 1000.0)
    temps = np.concatenate([temps, [np.nextafter(foot, np.float32(0)), foot, np.nextafter(foot, np.float32(9)),
                                    np.nextafter(np.float32(0.157), np.float32(0)), np.nextafter(np.float32(0.157), np.float32(9))]]).astype(np.float32)
    nx = FC.C1["res"][0]
    for name in ("SY", "S"):
        state[name][..., 0] = temps[np.arange(nx) % len(temps)]
    for name in ("S2Y", "S2"):
        state[name][..., 1] = age
    speed = np.float32([0.0, 14.9, 15.0, 15.1, 30.0])[np.arange(nx) // len(temps) % 5]
    for name in ("velY", "vel"):
        state[name][..., 0] = speed
        state[name][..., 1:3] = 0.0
    FC.put_state(sim, orc, state)
    FC.sync_block(sim, orc, dt)
    sim.run_stage("forces", dt)
    sim.sync()
    orc.stage("curl")
    orc.stage("forces")
    for name in OUTPUTS["forces"]:
        g, o = sim.download(name), orc.get(name)
        for c in range(4):
            FC.compare(g[..., c], o[..., c], RTOL, ATOL, OUTLIERS, what=f"forces:{name}[{c}]")
