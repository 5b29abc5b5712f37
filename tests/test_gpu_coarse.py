"""The register-resident coarse end of the V-cycle against the same cycle built from single multigrid operations.

On these grids the V-cycle stage is one launch of the coarse kernel; the same cycle from `sweeps`, `restrict` and
`prolong` launches performs the same operations in the same order, so with omega 1 the pressures agree bit for bit.  The grids sit at the kernel's edges: one CTA with one row per thread (8x16x8, 2x2x2) and with four (10x15x10: a
partial last group of rows), levels split over the cluster (16x32x16; 32x64x32: two of them; 12x24x12: fewer
rows than CTAs; 64x16x16: half the CTAs), odd sizes (25x49x25, 33x47x29: a single level of 64 sweeps, a row that ends at an
even x), the larger CTA sizes (40x60x40; 44x90x20), and many row groups on few columns (6x200x6).

With omega != 1 the compiler may contract the single launches' relaxation differently: one rounding (2^-24) per update, at
most 64 + 4 x 5 sweeps of which none amplifies an error in the 2-norm, so 1e-5 of the pressure's norm bounds it."""
import numpy as np
import pytest

import fire_cases as FC
import fire_sim as F

pytestmark = pytest.mark.gpu

GRIDS = [(8, 16, 8), (2, 2, 2), (10, 15, 10), (16, 32, 16), (32, 64, 32), (12, 24, 12), (64, 16, 16), (25, 49, 25), (33, 47, 29),
         (40, 60, 40), (44, 90, 20), (6, 200, 6)]


def _sim(res, omega):
    sim = F.FireSim(res=res, size=tuple(0.0125 * n for n in res), vcycles=1)
    if omega != 1.0:
        sim.set_mg_omega(omega)
    rng = np.random.default_rng(res[0] + 100 * res[1])
    shape = (res[2], res[1], res[0])
    sim.set_level(0, "p", (0.01 * rng.standard_normal(shape)).astype(np.float32))
    sim.set_level(0, "b", (50.0 * rng.standard_normal(shape)).astype(np.float32))
    return sim


def _cycle_by_launches(sim, l=0):
    last = len(sim.levels) - 1
    if l == last:
        sim.run_mg("sweeps", l, sim.coarse_iters)
        return
    sim.run_mg("sweeps", l, 2)
    sim.run_mg("restrict", l)
    _cycle_by_launches(sim, l + 1)
    sim.run_mg("prolong", l)
    sim.run_mg("sweeps", l, 2)


@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("res", GRIDS)
def test_cycle_matches_single_launches(res, omega):
    a, b = _sim(res, omega), _sim(res, omega)
    for _ in range(2):
        a.run_stage("vcycle", 0.01)
        _cycle_by_launches(b)
    a.sync()
    pa, pb = a.level(0, "p"), b.level(0, "p")
    assert np.isfinite(pb).all()
    if omega == 1.0:
        np.testing.assert_array_equal(pa, pb)
    else:
        assert FC.rel_l2(pa, pb) <= 1e-5
    a.close()
    b.close()


@pytest.mark.parametrize("res", [(16, 32, 16), (33, 47, 29)])
def test_all_cycles_of_a_step_in_one_launch(res):
    """A step whose hierarchy is on chip runs its three cycles in one launch: the same bits as three single cycles."""
    dt, state = 1.0 / 120.0, FC.random_state(res, 3)
    sims = []
    for _ in range(2):
        s = F.FireSim(res=res, size=tuple(0.0125 * n for n in res), vcycles=3)
        for k in ("vel", "S", "S2"):
            s.upload(k, state[k])
        sims.append(s)
    sims[0].step(dt, 1)
    sims[1].run_stage("geo", dt)
    for stage in ("adv1", "adv2", "forces", "div", "vcycle", "vcycle", "vcycle", "project"):
        sims[1].run_stage(stage, dt)
    for s in sims:
        s.sync()
    for name in ("p", "vel"):
        np.testing.assert_array_equal(sims[0].download(name), sims[1].download(name), err_msg=name)
    for s in sims:
        s.close()
