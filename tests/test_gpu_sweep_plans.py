"""The two-sweep kernel on the cuts and instantiations that tests/test_gpu_sweep.py's grids do not reach: coarsest levels of odd depth
whose last chunk is one plane (shorter than the halo), rows of an odd length from a zero start, and over-relaxed levels of a
batch.

With omega 1 both sides do the same operations in the same order: equal bits.  With omega != 1 the compiler may contract
the launches' relaxation differently: one rounding (2^-24) per update, at most 64 + 4 x 6 sweeps of which none amplifies an
error in the 2-norm, so 1e-5 of the pressure's norm bounds it."""
import numpy as np
import pytest

import fire_cases as FC
import fire_sim as F
import test_gpu_coarse as C

pytestmark = pytest.mark.gpu


def _swept_by_two(dims, coarsest):
    """Whether the rules of the coarse kernel and of the two-sweep kernel give a level to the latter."""
    nx, ny, nz = dims
    on_chip = (nx + 1) // 2 * nz * ((ny + 63) // 64) <= (1024 if coarsest else 512)
    return not on_chip and nx * ny * nz >= (500000 if nx % 2 else 280000 if coarsest else 150000)


@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("res", [(160, 200, 162), (112, 61, 43), (96, 68, 43), (128, 54, 43)])
def test_odd_depth_and_a_last_chunk_of_one_plane(res, omega):
    a, b = C._sim(res, omega), C._sim(res, omega)
    dims = [level["dims"] for level in a.levels]
    assert all(_swept_by_two(d, k + 1 == len(dims)) for k, d in enumerate(dims))
    a.run_stage("vcycle", 0.01)
    C._cycle_by_launches(b)
    a.sync()
    pa, pb = a.level(0, "p"), b.level(0, "p")
    assert np.isfinite(pb).all()
    if omega == 1.0:
        np.testing.assert_array_equal(pa, pb)
    else:
        assert FC.rel_l2(pa, pb) <= 1e-5
    a.close()
    b.close()


@pytest.mark.parametrize("res", [(101, 90, 95), (61, 51, 47), (43, 77, 41)])
def test_refinement_from_zero_on_odd_rows(res):
    """One refinement from x = 0 on a single level is the correction's sweeps from zero on b / RMS(b), scaled back.  Against the same
    number of colour sweeps on b: scaling rounds each value of b once and the result once (2^-24 each), and a sweep is linear and
    does not amplify in the 2-norm, so 1e-5 of the result's norm bounds the difference; a wrong cell at the end of
    a row shows at 1e-3 of the largest value."""
    torch = pytest.importorskip("torch")
    n = (res[2], res[1], res[0])
    rng = np.random.default_rng(res[0])
    b = rng.standard_normal(n).astype(np.float32)
    sim = F.FireSim(res=res, size=tuple(0.0125 * k for k in res), vcycles=1)
    assert len(sim.levels) == 1
    sim.set_level(0, "p", np.zeros(n, np.float32))
    sim.set_level(0, "b", b)
    sim.run_mg("sweeps", 0, sim.coarse_iters)
    sim.sync()
    want = sim.level(0, "p").astype(np.float64)
    ps = F.Poisson(res, sim.dx, "ir32")
    db, x, lo = torch.from_numpy(b).cuda(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    ps.solve(db, x, x_lo=lo, tol=1e-30, max_iters=1)
    ps.result()
    got = x.double().cpu().numpy() + lo.double().cpu().numpy()
    assert FC.rel_l2(got, want) <= 1e-5
    assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
    ps.close()
    sim.close()


def test_relaxed_levels_of_a_batch():
    """Members over-relaxed after the ensemble's creation: their launched levels are relaxed, their coarse ends keep omega 1.  Against
    the same cycles of a simulation alone from single launches, its omega switched where the coarse end begins."""
    import test_gpu_ensemble as E
    members = [dict(res=r, size=tuple(0.0125 * k for k in r), seed=30 + i, spots=4)
               for i, r in enumerate([(46, 92, 44), (64, 128, 64), (160, 200, 120)])]
    coarse_from = [1, 1, 3]   # 23x46x22; 32x64x32; 20x25x15: the coarse kernel takes the levels from here on
    ens = F.Ensemble(members, vcycles=2)
    for s, m in zip(ens.members, members):
        E._configure(s, m)
    for s in ens.members[1:]:
        s.set_mg_omega(1.2)
    ens.step(E.DT, 1)
    ens.sync()
    for k, m in enumerate(members):
        s = F.FireSim(res=m["res"], size=m["size"], vcycles=2)
        E._configure(s, m)
        s.run_stage("geo", E.DT)
        for stage in ("adv1", "adv2", "forces", "div"):
            s.run_stage(stage, E.DT)
        omega = 1.0 if k == 0 else 1.2

        def cycle(l):
            if l == coarse_from[k]:
                s.set_mg_omega(1.0)
                s.run_mg("tail", l)
                return
            s.set_mg_omega(omega)
            s.run_mg("sweeps", l, 2)
            s.run_mg("restrict", l)
            cycle(l + 1)
            s.set_mg_omega(omega)
            s.run_mg("prolong", l)
            s.run_mg("sweeps", l, 2)

        for _ in range(2):
            cycle(0)
        s.sync()
        pa, pb = ens.members[k].level(0, "p"), s.level(0, "p")
        assert float(np.abs(pb).max()) > 0.0
        assert FC.rel_l2(pa, pb) <= 1e-5, k
        s.close()
    ens.close()
