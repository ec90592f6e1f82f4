"""The stages of a step: the scatter pass is timed where there is one, and priced nowhere else."""
import pytest

from epp import abi, casegen
from epp.algorithm import DeviceParticleSystem
from epp.classes import NeighbourSystem


def test_no_bytes_for_a_pass_that_does_not_run():
    from test_bench_bookkeeping import _bench
    b = _bench()
    assert b.B_ALG_STAGE["scatter"] == {2: 0.0, 3: 0.0}
    assert b.B_ALG_STAGE["rank_gather"] == {2: 80.0, 3: 104.0}


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("family", [0, 1, 4])
def test_scatter_stage(dim, family):
    case = casegen.dam_break_2d(dx=0.05, max_neighbour_number=1) if dim == 2 else casegen.dam_break_3d(dx=0.1, max_neighbour_number=1)
    d = DeviceParticleSystem(case.ps, NeighbourSystem(case.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
    d.ctx.set_tuning(family)
    d.syncto()
    d.ctx.search(abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_DAMBREAK_CONTINUITY, case.physics, 0)
    for _ in range(2):
        t = d.ctx.profile_step(case.physics)
        t = list(t.values()) if isinstance(t, dict) else list(t)
        assert (t[2] > 0) == (family == 1) and t[0] > 0 and t[1] > 0 and t[3] > 0 and t[4] > 0
    d.close()
