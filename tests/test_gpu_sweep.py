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
