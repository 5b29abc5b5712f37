"""The bounded waits of the multigrid's coarse end, run out on a healthy GPU.

A default step waits in the coarse kernel for the rows that neighbouring CTAs of its cluster send.  With a limit of 0
the first wait of every CTA gives up at once: the host must see the timeout once, a hierarchy that is all on chip keeps the
pressure it had (nothing is stored), and the next cycle with the default limit must give the bits of a simulation that
never ran out.  Grids: two split levels above gathered ones (32x64x32, and its three cycles of a step in one launch), one split
level of 64 sweeps (25x49x25), fewer rows than CTAs (12x24x12), a coarse end below launched levels (64x128x64), and one
CTA, which waits for no rows and takes the kernel that waits for bulk copies instead (8x16x8).  A limit of 1 lets
waits run out anywhere or nowhere; what follows must be clean either way."""
import numpy as np
import pytest

import fire_sim as F
import test_gpu_coarse as C

pytestmark = pytest.mark.gpu
DEFAULT = 1 << 22


def _sync_reports(sim):
    try:
        sim.sync()
    except F.FireError as e:
        assert e.code == 3 and "timed out" in str(e)
        sim.sync()   # the report cleared the flag
        return True
    return False


@pytest.mark.parametrize("polls", [0, 1])
@pytest.mark.parametrize("res,on_chip", [((32, 64, 32), True), ((25, 49, 25), True), ((12, 24, 12), True), ((64, 128, 64), False),
                                         ((8, 16, 8), True)])
def test_a_wait_that_runs_out_is_reported_and_the_next_cycle_is_clean(res, on_chip, polls):
    sim, ref = C._sim(res, 1.0), C._sim(res, 1.0)
    p0 = sim.level(0, "p")
    sim.set_tail_wait_limit(polls)
    sim.run_stage("vcycle", 0.01)
    reported = _sync_reports(sim)
    if polls == 0:
        assert reported
        if on_chip:
            np.testing.assert_array_equal(sim.level(0, "p"), p0)
    sim.set_tail_wait_limit(DEFAULT)
    sim.set_level(0, "p", p0)
    sim.run_stage("vcycle", 0.01)
    ref.run_stage("vcycle", 0.01)
    sim.sync()
    ref.sync()
    np.testing.assert_array_equal(sim.level(0, "p"), ref.level(0, "p"))
    sim.close()
    ref.close()


def test_all_cycles_of_a_step_in_one_launch():
    res = (32, 64, 32)
    sim = F.FireSim(res=res, size=tuple(0.0125 * n for n in res), vcycles=3)
    sim.step(0.01, 2)
    sim.sync()
    p0 = sim.level(0, "p")
    sim.set_tail_wait_limit(0)
    sim.step(0.01, 1)
    assert _sync_reports(sim)
    np.testing.assert_array_equal(sim.level(0, "p"), p0)
    sim.set_tail_wait_limit(DEFAULT)
    sim.step(0.01, 1)
    sim.sync()
    assert np.isfinite(sim.level(0, "p")).all() and (sim.level(0, "p") != p0).any()
    sim.close()
