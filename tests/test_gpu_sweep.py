"""The two-sweep kernel of the multigrid levels (one pass for four colour launches) against the colour launches.

The V-cycle stage smooths its launched levels with the two-sweep kernel; the same cycle built from `sweeps`, `restrict` and
`prolong` uses one launch per colour.  Both do the same operations in the same order, so with omega 1 the pressures
agree bit for bit.  Grids: whole rows and two, three and more tiles in x, tiles with a ragged last row or plane
(46x92x44, 96x110x70), chunks shorter than the halo (90x200x90's second level), a hierarchy that ends at odd sizes right
below (50x98x50), an odd depth in the level's chunks (92x100x66 -> 33 planes), and a level of one chunk.

With omega != 1 the compiler may contract the launches' relaxation differently: one rounding (2^-24) per update, at most
64 + 4 x 6 sweeps of which none amplifies an error in the 2-norm, so 1e-5 of the pressure's norm bounds it."""
import numpy as np
import pytest

import fire_cases as FC
import test_gpu_coarse as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("res", [(64, 128, 64), (46, 92, 44), (50, 98, 50), (80, 120, 80), (96, 110, 70), (90, 200, 90), (92, 100, 66),
                                 (200, 60, 100)])
def test_cycle_matches_colour_launches(res, omega):
    a, b = C._sim(res, omega), C._sim(res, omega)
    for _ in range(2):
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


@pytest.mark.parametrize("res", [(120, 101, 90), (150, 100, 77), (101, 90, 95), (151, 103, 64)])
def test_single_large_level_matches_colour_launches(res):
    """A grid without coarser levels and too large for the on-chip kernel: all its sweeps are two-sweep launches, in place by
    pairs, with the odd remainder by colour; an odd row count leaves a thread row with one row in the domain.  An odd row length leaves a pair
    with one column, and pairs that are not aligned."""
    a, b = C._sim(res, 1.0), C._sim(res, 1.0)
    a.run_stage("vcycle", 0.01)
    b.run_mg("sweeps", 0, a.info().coarse_iters)
    a.sync()
    np.testing.assert_array_equal(a.level(0, "p"), b.level(0, "p"))
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp16", "bf16", "ir32"])
@pytest.mark.parametrize("res", [(46, 92, 44), (50, 98, 50), (96, 110, 70), (120, 101, 90)])
def test_refinement_forms_reach_the_tolerance(precision, res):
    """The same kernel on levels in half, bfloat16 and float: the residual that the solver reports and the one computed afresh
    from the returned pair agree (both are sums of squares in double-float of FP32 residuals of the same pair: 1e-5), and
    lie at the tolerance asked for on a hierarchy, below the start on a single level (whose sweeps only smooth)."""
    torch = pytest.importorskip("torch")
    import fire_sim as F
    ps = F.Poisson(res, 0.01, precision)
    n = (res[2], res[1], res[0])
    b, x, lo = (torch.zeros(n, device="cuda") for _ in range(3))
    ps.make_rhs(b, seed=5)
    single = bool(res[1] % 2)
    ps.solve(b, x, x_lo=lo, tol=1e-6, max_iters=4 if single else 40)
    out = ps.result()
    rel = ps.residual(b, x, x_lo=lo)
    assert abs(rel - out["rel_residual"]) <= 1e-5 * out["rel_residual"] + 1e-12
    assert out["rel_residual"] <= (0.9 * out["rel_residual_initial"] if single else 1e-6)
    ps.close()


@pytest.mark.parametrize("mixed", [False, True])
def test_batched_sweeps_match_members_alone(mixed):
    """Members of very different sizes share each batched two-sweep launch (tiles cut for a share of the SMs), one whose
    second level only it has outside its coarse end: after the first step from rest their
    pressures equal those of the same simulations stepped alone (same operations, same order).  mixed: one member's launched
    levels are over-relaxed (its coarse end is not, as descriptors are made at creation), which another kernel serves; the
    others' pressures are still their own."""
    import fire_sim as F
    import test_gpu_ensemble as E
    members = [dict(res=r, size=tuple(0.0125 * k for k in r), seed=20 + i, spots=4)
               for i, r in enumerate([(46, 92, 44), (64, 128, 64), (200, 60, 100), (160, 200, 120)])]
    ens = F.Ensemble(members, vcycles=2)
    alone = [F.FireSim(res=m["res"], size=m["size"], vcycles=2) for m in members]
    for k, m in enumerate(members):
        for s in (ens.members[k], alone[k]):
            E._configure(s, m)
    if mixed:
        ens.members[1].set_mg_omega(1.2)
    ens.step(E.DT, 1)
    ens.sync()
    for k, (a, b) in enumerate(zip(ens.members, alone)):
        b.step(E.DT, 1)
        b.sync()
        pa, pb = a.level(0, "p"), b.level(0, "p")
        assert float(np.abs(pb).max()) > 0.0
        if mixed and k == 1:   # two cycles of either smoother leave a few percent of the solution's error
            assert (pa != pb).any() and FC.rel_l2(pa, pb) < 0.2
        else:
            np.testing.assert_array_equal(pa, pb)
        b.close()
    ens.close()


@pytest.mark.parametrize("res", [(128, 42, 30), (256, 20, 17), (128, 7, 5)])
def test_refinement_residual_on_whole_warp_rows(res):
    """The residual of a pair (x, x_lo) with four cells a thread (rows of a multiple of 128 cells; rows and planes that leave ragged
    CTAs, fewer planes than one thread marches) against its FP64 form.  A residual is a sum of 14 rounded terms of at most
    |b| + 12 max|x| / h^2 and the norm adds about as much again, so 64 x 2^-24 of that size over the norm bounds the error."""
    torch = pytest.importorskip("torch")
    import fire_sim as F
    import oracle as O
    n = (res[2], res[1], res[0])
    rng = np.random.default_rng(res[0] + res[1])
    b, x = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
    lo = (1e-8 * rng.standard_normal(n)).astype(np.float32)
    h = 0.5
    ps = F.Poisson(res, h, "ir32")
    got = ps.residual(*(torch.from_numpy(v).cuda() for v in (b, x, lo)))
    r = b.astype(np.float64) - O.pressure_apply(x.astype(np.float64) + lo, h)
    want = np.linalg.norm(r) / np.linalg.norm(b)
    size = np.sqrt(r.size) * (np.abs(b).max() + 12 * np.abs(x).max() / h ** 2) / np.linalg.norm(b)
    assert abs(got - want) <= 64 * 2.0 ** -24 * size
    ps.close()
