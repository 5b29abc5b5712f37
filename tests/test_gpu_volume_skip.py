"""The march's empty-space skipping: fields of zeros with a few isolated cells (hot, sooty, blue, smoky, one at a corner) against
the CPU restatement, on a grid that is no multiple of the bricks, for the reaches a sample can have: no warp, the usual
one, one of several bricks, and the B-spline's wider taps (below).  A brick skipped in error shows in the haze (every pixel is
compared) and in the pixels that the cells touch.  Tolerances are those of tests/test_volume.py's dense fire."""
import numpy as np
import pytest

import fire_cases as FC

pytestmark = pytest.mark.gpu


RES = (37, 50, 29)


def _cells():
    S = np.zeros((RES[2], RES[1], RES[0], 4), np.float32)
    S2 = np.zeros_like(S)
    S[14, 20, 17] = (0.9, 0.0, 0.5, 0.0)
    S[7, 31, 28] = (0.0, 0.0, 0.0, 0.4)
    S[20, 12, 8] = (0.3, 0.0, 0.0, 0.0)
    S[27, 40, 35] = (0.8, 0.0, 0.8, 0.2)
    S2[10, 9, 22] = (0.0, 0.0, 0.7, 0.0)
    return S, S2


def _render(S, S2, **params):
    import fire_sim as F
    sim = F.FireSim(res=RES, size=tuple(0.02 * r for r in RES), vcycles=1)
    sim.upload("S", S)
    sim.upload("S2", S2)
    vol = F.Volume(sim, width=120, height=140, vol_scale=1.0)
    vol.set_camera((0.35, 0.55, 1.6), (0.0, 0.5, 0.0), 40.0)
    vol.set_params(dict(params, sootScat=0.03))
    U = vol.uniforms(0.4, 2)
    vol.render(0.4, 2)
    out = U, vol.image(), vol.aux(), vol.lights(), sim.download("curl").astype(np.float32)
    vol.close()
    sim.close()
    return out


@pytest.mark.parametrize("detail,smoke", [(0.0, 0.05), (0.6, 0.0), (40.0, 0.05)])
def test_isolated_cells(oracle_mod, detail, smoke):
    import fire_sim as F
    S, S2 = _cells()
    U, img, aux, lights, curl = _render(S, S2, detailAmt=detail, smokeScat=smoke)
    lut = F.blackbody_lut(1024, 400.0, 3000.0, 5000.0).reshape(-1, 4)
    want, want_aux = oracle_mod.volume_render(U, S, S2, curl, lut, lights)
    np.testing.assert_allclose(aux[..., 0], want_aux[..., 0], rtol=1e-3, atol=1e-6)
    touched = (want[..., 3] < 1.0) | (np.abs(want[..., :3]).max(-1) > 0)
    assert 10 < touched.sum() and (want_aux[..., 0] > 0).any()
    bad = np.abs(img - want) > 1e-3 * np.abs(want) + 1e-4 * max(float(np.abs(want[..., :3]).max()), 1.0)
    assert bad.any(-1)[touched].mean() < 0.005 and not bad[~touched].any()


@pytest.mark.parametrize("detail", [0.0, 0.6])
def test_b_spline_reach(detail):
    """The CPU restatement has no B-spline, so the skipping render is held to one whose every brick counts: a smoke background just
    above the bricks' limit (0.999e-4) and still below the samples' (1e-4) against one just below both.  The backgrounds
    differ by 1.5e-7, in the smoke that samples inside the fire see: 1e-6 of the image bounds that; the haze does not see it."""
    S, S2 = _cells()
    got = []
    for background in (0.9985e-4, 0.99995e-4):
        B = S2.copy()
        B[..., 2] = np.maximum(B[..., 2], np.float32(background))
        got.append(_render(S, B, detailAmt=detail, smokeScat=0.05, cubic=1.0))
    (_, a, ax, _, _), (_, b, bx, _, _) = got
    np.testing.assert_array_equal(ax, bx)
    assert (ax[..., 0] > 0).any()
    assert np.abs(a - b).max() <= 1e-6 * max(float(np.abs(b).max()), 1.0)
