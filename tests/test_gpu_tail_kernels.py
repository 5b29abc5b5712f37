"""The tail kernels where they still serve: refinements whose coarsest level is too large for the dense inverse (64 FP64 sweeps,
in one CTA or on a cluster) and ensemble members on flat, wide grids that the coarse kernel does not fit."""
import numpy as np
import pytest

import fire_sim as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp16", "ir32"])
@pytest.mark.parametrize("res", [(18, 22, 16), (26, 42, 22), (5, 9, 13)])
def test_refinement_with_fp64_sweeps(precision, res):
    """18x22x16: a cluster with the first level in slabs, 9x11x8 gathered; 26x42x22: one CTA from 13x21x11 below a launched level;
    5x9x13: one CTA, one level.  A Gauss-Seidel sweep leaves at most 0.953 of the slowest
    error on these coarsest levels (the square of Jacobi's factor, the mean of cos(pi / nx), cos(pi / 2 ny) and cos(pi / nz)), so
    64 leave 5 % per refinement and 20 refinements are ample.  The residual of the returned pair
    is formed anew in FP64: the solver's own is a double-float sum of FP32 residuals, good to 1e-5 of itself."""
    torch = pytest.importorskip("torch")
    import oracle as O
    n, h = (res[2], res[1], res[0]), 0.1
    b = np.random.default_rng(res[0]).standard_normal(n).astype(np.float32)
    db, x, lo = torch.from_numpy(b).cuda(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    ps = F.Poisson(res, h, precision)
    ps.solve(db, x, x_lo=lo, tol=1e-6, max_iters=20)
    out = ps.result()
    assert out["iterations"] <= 20 and out["rel_residual"] <= 1e-6
    r = b - O.pressure_apply(x.double().cpu().numpy() + lo.double().cpu().numpy(), h)
    assert np.linalg.norm(r) <= 1.0001e-6 * np.linalg.norm(b.astype(np.float64))
    ps.close()


def test_flat_members_of_an_ensemble():
    """More than 1024 columns of cells and two or three rows: the coarse kernel cannot split them, and the batched tail serves them
    beside an ordinary member.  One step from rest: the bits of each member stepped alone."""
    import test_gpu_ensemble as E
    members = [dict(res=r, size=tuple(0.0125 * k for k in r), seed=40 + i, spots=4)
               for i, r in enumerate([(32, 3, 65), (24, 48, 24), (72, 2, 32)])]
    ens = F.Ensemble(members, vcycles=2)
    alone = [F.FireSim(res=m["res"], size=m["size"], vcycles=2) for m in members]
    for k, m in enumerate(members):
        for s in (ens.members[k], alone[k]):
            E._configure(s, m)
    ens.step(E.DT, 1)
    ens.sync()
    for a, b in zip(ens.members, alone):
        b.step(E.DT, 1)
        b.sync()
        pa, pb = a.level(0, "p"), b.level(0, "p")
        assert float(np.abs(pb).max()) > 0.0
        np.testing.assert_array_equal(pa, pb)
        b.close()
    ens.close()
