"""The restriction and prolongation kernels against the float64 forms (numpy_fire), where a thread marches one coarse plane and
where it marches four (from 1.2 M coarse cells on), and on caller-owned arrays that are only 4-byte aligned.

Grids: the smallest that restricts, ragged rows and planes, and 200x220x230, whose 115 coarse planes leave a march of three.

Tolerances, with u = 2^-24 and one rounding per operation.  Restriction: a child's residual is six neighbour sums of at most
12 max|p| / h^2 in all (7 roundings), one product and one difference with b (2 roundings of the residual's size r =
12 max|p| / h^2 + max|b|), then eight sums of residuals, divided by 8: u (7 + 2 + 8) r.  Prolongation: a term has
three roundings, eight sums of at most max|pc|, then one sum with p: u (3 + 8) max|pc| + u (max|p| + max|pc|)."""
import ctypes

import numpy as np
import pytest

import fire_sim as F
import numpy_fire as NF

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


@pytest.mark.parametrize("res", [(8, 8, 8), (66, 90, 34), (200, 220, 230)])
def test_transfers_match_float64(res):
    nx, ny, nz = res
    rng = np.random.default_rng(nx)
    sim = F.FireSim(res=res, size=tuple(0.01 * r for r in res))
    p, b = (rng.standard_normal((nz, ny, nx)).astype(np.float32) for _ in range(2))
    pc = rng.standard_normal((nz // 2, ny // 2, nx // 2)).astype(np.float32)
    h = float(np.float32(sim.levels[0]["h"]))
    sim.set_level(0, "p", p)
    sim.set_level(0, "b", b)
    sim.set_level(1, "p", pc)
    sim.run_mg("restrict", 0)
    sim.sync()
    want = NF.restrict(p.astype(np.float64), b.astype(np.float64), h, (nx // 2, ny // 2, nz // 2))
    r = 12 * np.abs(p).max() / h ** 2 + np.abs(b).max()
    assert np.abs(sim.level(1, "b") - want).max() <= 17 * U * r
    assert not sim.level(1, "p").any()
    sim.set_level(1, "p", pc)
    sim.run_mg("prolong", 0)
    sim.sync()
    want = NF.prolong_add(p.astype(np.float64), pc.astype(np.float64))
    assert np.abs(sim.level(0, "p") - want).max() <= U * (12 * np.abs(pc).max() + np.abs(p).max())
    sim.close()


def test_four_byte_aligned_level():
    torch = pytest.importorskip("torch")
    lib = F.load_library()
    res = (64, 128, 66)
    n = res[0] * res[1] * res[2]
    gen = torch.Generator(device="cuda").manual_seed(3)
    p0, b0 = (torch.randn(n, generator=gen, device="cuda") for _ in range(2))
    got = []
    for shift in (0, 1):
        p, b = torch.zeros(n + 1, device="cuda"), torch.zeros(n + 1, device="cuda")
        p[shift:shift + n] = p0
        b[shift:shift + n] = b0
        stream = torch.cuda.current_stream().cuda_stream
        rc = lib.fire_poisson_vcycles_noalloc(ctypes.c_void_p(p.data_ptr() + 4 * shift), ctypes.c_void_p(b.data_ptr() + 4 * shift), *res,
                                              ctypes.c_float(0.01), 2, ctypes.c_void_p(stream))
        assert rc == 0
        got.append(p[shift:shift + n].cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("res", [(10, 9, 7), (66, 50, 41), (25, 30, 27)])
def test_residual_norm_matches_float64(res):
    """The residual's norm with two columns a thread (even rows; ragged ends in every direction) and with one (odd rows).  A residual
    is 9 rounded terms of at most s = max|b| + 12 max|p| / h^2 and each square and column sum of 8 adds 9 roundings, so
    32 u s sqrt(cells) / ||b|| bounds the relative norm's error."""
    nx, ny, nz = res
    rng = np.random.default_rng(ny)
    sim = F.FireSim(res=res, size=tuple(0.5 * r for r in res))
    p, b = (rng.standard_normal((nz, ny, nx)).astype(np.float32) for _ in range(2))
    h = float(np.float32(sim.levels[0]["h"]))
    sim.set_level(0, "p", p)
    sim.set_level(0, "b", b)
    q = [v.astype(np.float64) for v in NF.neighbours(p.astype(np.float64))]
    r = b - (sum(q) - 6.0 * p.astype(np.float64)) / h ** 2
    norm = np.linalg.norm(b.astype(np.float64))
    s = np.abs(b).max() + 12 * np.abs(p).max() / h ** 2
    assert abs(sim.residual() - np.linalg.norm(r) / norm) <= 32 * U * s * np.sqrt(b.size) / norm
    sim.close()
