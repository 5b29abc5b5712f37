"""Refinement on grids whose whole hierarchy is one level small enough for the dense FP64 inverse.

The correction is then the exact solution rounded to FP32, so an iteration leaves at most a few cond(A) x 2^-24 of the residual
(A's row sums are bounded by its diagonal: the residual of a rounding is at most |A| |e| 2^-24); these grids' condition
numbers are below 100, so two iterations reach 1e-6.  The pair then lies within cond(A) x 1e-6 of the FP64 solution."""
import numpy as np
import pytest

import fire_sim as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp16", "bf16", "ir32"])
@pytest.mark.parametrize("res", [(2, 2, 2), (5, 5, 5), (7, 7, 7), (6, 12, 6), (2, 16, 16), (5, 8, 12)])
def test_solves_in_two_iterations(precision, res):
    torch = pytest.importorskip("torch")
    import oracle as O
    n, h = (res[2], res[1], res[0]), 0.1
    cells = int(np.prod(n))
    rng = np.random.default_rng(cells)
    b = rng.standard_normal(n).astype(np.float32)
    A = np.stack([O.pressure_apply(e.reshape(n), h).ravel() for e in np.eye(cells)], axis=1)
    cond = np.linalg.cond(A)
    assert cond < 100
    want = np.linalg.solve(A, b.astype(np.float64).ravel()).reshape(n)
    ps = F.Poisson(res, h, precision)
    db, x, lo = torch.from_numpy(b).cuda(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    for _ in range(2):   # the second solve starts over with the correction array the first one left
        x.zero_()
        lo.zero_()
        ps.solve(db, x, x_lo=lo, tol=1e-6, max_iters=20)
        out = ps.result()
        assert out["iterations"] <= 2 and out["rel_residual"] <= 1e-6
        got = x.double().cpu().numpy() + lo.double().cpu().numpy()
        assert np.linalg.norm(got - want) <= cond * 1e-6 * np.linalg.norm(want)
    ps.close()
