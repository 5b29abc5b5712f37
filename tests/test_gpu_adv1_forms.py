"""adv1 with two cells a thread (600,000 cells and more) against the form with one cell, with wind mixed in at the open sides.

Two grids that differ in depth only hold the same state in their common planes.  Velocities are below 3 m/s, so a back-trace of
dt = 1/120 s moves less than 2.1 cells of 12.5 mm: in planes that far (and the stencil's two cells) from the shallow grid's last
one both kernels see the same cells, and their results agree bit for bit."""
import numpy as np
import pytest

import fire_cases as FC
import fire_sim as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wind", [(0.0, 0.0), (1.5, 0.0), (1.5, -1.0)])
def test_both_forms_agree(wind):
    deep, shallow, common = (118, 96, 105), (118, 96, 48), 42
    assert np.prod(deep) >= 600000 > np.prod(shallow)
    rng = np.random.default_rng(7)
    sh = (deep[2], deep[1], deep[0])
    vel = np.stack([3.0 * FC.smooth_noise(sh, rng, 2) for _ in range(3)] + [np.zeros(sh)], -1).astype(np.float32)
    vel *= min(1.0, 2.9 / np.linalg.norm(vel, axis=-1).max())
    S, S2 = (np.stack([FC.smooth_noise(sh, rng, 1) + 1.0 for _ in range(4)], -1).astype(np.float32) for _ in range(2))
    got = []
    for res in (deep, shallow):
        sim = F.FireSim(res=res, size=tuple(0.0125 * n for n in res), vcycles=1)
        sim.set_params({"windX": wind[0], "windZ": wind[1], "ox": 0.0, "oy": 0.0, "oz": 0.0})
        for name, a in (("vel", vel), ("S", S), ("S2", S2)):
            sim.upload(name, np.ascontiguousarray(a[:res[2]]))
        sim.run_stage("adv1", 1.0 / 120.0)
        sim.sync()
        got.append({name: sim.download(name)[:common] for name in ("velX", "SX", "S2X")})
        sim.close()
    assert np.isfinite(got[0]["velX"]).all()
    for name in got[0]:
        np.testing.assert_array_equal(got[0][name], got[1][name], err_msg=name)
