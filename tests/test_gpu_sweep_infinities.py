"""The two-sweep kernel on pressures that hold infinities and not-a-numbers, against the colour launches.

A pair or thread row that ends outside the domain (an odd row length, an odd row count) has cells there; they must stay what
a missing neighbour adds in a colour launch, zero, whatever lies next to them.  Positive infinities alone stay
infinities in every sweep, so a not-a-number shows a cell outside that did not stay zero; with both signs and a not-a-number the
patterns still agree.  Grids: one level with odd rows, with an odd row count, with both, and a coarsest level of odd row count
(160x202x160 -> 80x101x80).  With omega 1 the pressures agree bit for bit, any not-a-number standing for any other."""
import numpy as np
import pytest

import test_gpu_coarse as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("values", ["positive", "mixed"])
@pytest.mark.parametrize("res", [(101, 90, 95), (151, 103, 64), (120, 101, 90), (160, 202, 160)])
def test_broken_pressures_match_colour_launches(res, values, omega):
    a, b = C._sim(res, omega), C._sim(res, omega)
    p = a.level(0, "p").copy()   # [z, y, x]
    nx, ny, nz = res
    at = [(nz // 2, ny - 1, nx // 2), (nz // 3, ny // 2, nx - 1), (nz // 4, ny - 1, nx - 1), (0, ny - 1, 5), (nz - 1, 7, nx - 1)]
    for k, (z, y, x) in enumerate(at):   # neighbours along x: the first pass replaces one colour before it is read
        p[z, y, x - 1:x + 1] = -np.inf if values == "mixed" and k % 2 else np.inf
    if values == "mixed":
        p[nz // 2, 20, 20] = np.nan
    for s in (a, b):
        s.set_level(0, "p", p)
    a.run_stage("vcycle", 0.01)
    C._cycle_by_launches(b)
    a.sync()
    pa, pb = a.level(0, "p"), b.level(0, "p")
    if values == "positive" and omega == 1.0 and len(b.levels) == 1:
        assert np.isinf(pb).any() and not np.isnan(pb).any()
    np.testing.assert_array_equal(np.isnan(pa), np.isnan(pb))
    np.testing.assert_array_equal(np.isinf(pa), np.isinf(pb))
    if omega == 1.0:
        np.testing.assert_array_equal(pa, pb)
    a.close()
    b.close()
