"""More neighbours than a list keeps (h of 2.5 to 4 dx): windows beyond the staging areas, pair passes
from the stencil.  The same neighbours and sums as the lists give, and no path that leaves most of a
warp idle: the stages of a step stay within a few times those of another pair-pass family, where the
faults these tests are for took 5 to 20 times as long."""
import numpy as np
import pytest

from epp import abi, casegen
from epp.algorithm import DeviceParticleSystem
from epp.classes import NeighbourSystem

pytestmark = pytest.mark.gpu

SYM, CONT = abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_DAMBREAK_CONTINUITY
MOMENTUM, SEARCH, CONTINUITY = 0, 4, 5   # stages of a step


def device(case, family=0):
    d = DeviceParticleSystem(case.ps, NeighbourSystem(case.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
    d.ctx.set_tuning(family)
    d.syncto()
    d.ctx.search(SYM, CONT, case.physics, 0)
    return d


def stages(case, family):
    """Least time of each stage over some steps, ms."""
    d = device(case, family)
    times = [list(t.values()) if isinstance(t, dict) else list(t) for t in (d.ctx.profile_step(case.physics) for _ in range(6))]
    d.close()
    return np.min(np.array(times), axis=0)


# the staged 2D search (above 20,000 particles) against the lockstep one
@pytest.mark.parametrize("h_factor", [2.5, 3.0, 4.0])
def test_dense_2d_search_time(h_factor):
    case = casegen.dam_break_2d(dx=0.01, h_factor=h_factor, max_neighbour_number=1)
    lists = stages(case, abi.EPP_TUNING_LISTS)
    assert stages(case, 0)[SEARCH] <= 2.0 * (lists[SEARCH] + lists[CONTINUITY])


# the staged 3D search (above 50,000 particles) against eight lanes per particle
@pytest.mark.parametrize("h_factor", [2.0, 2.5])
def test_dense_3d_search_time(h_factor):
    case = casegen.dam_break_3d(dx=0.025, h_factor=h_factor, max_neighbour_number=1)
    assert case.n > 50000
    assert stages(case, 0)[SEARCH] <= 3.0 * stages(case, 8)[SEARCH]


# eight lanes per particle (up to 50,000 particles), whose first pass has the list's entries already
def test_dense_3d_search_time_of_small_systems():
    few, many = (stages(casegen.dam_break_3d(dx=0.05, h_factor=h, max_neighbour_number=1), 0)[SEARCH] for h in (1.6, 2.5))
    assert many <= 8.0 * few   # 3.8 times the candidates


# 3D list passes of four lanes per particle whose lists overflow, against eight lanes without lists
@pytest.mark.parametrize("h_factor", [2.0, 2.5])
def test_dense_3d_list_pass_time(h_factor):
    case = casegen.dam_break_3d(dx=0.025, h_factor=h_factor, max_neighbour_number=1)
    lists, lanes = stages(case, 0), stages(case, 8)   # lanes: search and continuity are one kernel
    assert lists[MOMENTUM] <= 2.5 * lanes[MOMENTUM]
    assert lists[CONTINUITY] <= 2.5 * lanes[SEARCH]


# Overflowing 3D lists: the sums of a family that keeps no lists, to FP32 rounding of a few hundred terms
# (400 * 2^-24 of the terms' magnitudes, which the column's own pressure bounds)
@pytest.mark.parametrize("h_factor", [1.8, 2.5])
def test_dense_3d_sums(h_factor):
    got = []
    for family in (0, 8):
        case = casegen.dam_break_3d(dx=0.05, column=(0.6, 1.0, 0.5), h_factor=h_factor, max_neighbour_number=1)
        rng = np.random.default_rng(6)
        fl = case.ps["Tag"] == casegen.FLUID_TAG
        v = case.ps["VelocityVec"]
        v[fl] = rng.standard_normal(v[fl].shape)
        case.ps["VelocityVec"] = v
        d = device(case, family)
        d.ctx.interaction(abi.EPP_ACTION_DAMBREAK_MOMENTUM, case.physics)
        d.ctx.synchronize()
        d.asyncto()
        got.append({k: d.host[k].astype(np.float64) for k in ("nCount", "dDensity", "dVelocityVec")})
        d.close()
    assert np.array_equal(got[0]["nCount"], got[1]["nCount"]) and got[0]["nCount"].max() > 160
    for k in ("dDensity", "dVelocityVec"):
        scale = np.abs(got[1][k]).max()
        assert np.abs(got[0][k] - got[1][k]).max() <= 400 * 2.0 ** -24 * scale, k


# spray: few particles to a cell, warps of many cell rows; the staged search against two lanes a particle
@pytest.mark.parametrize("dim", [2, 3])
def test_spray_search_time(dim):
    from epp.classes import Domain2D, Domain3D
    times = []
    for family in (0, 2):
        case = casegen.dam_break_2d(dx=0.0045, max_neighbour_number=1) if dim == 2 else \
            casegen.dam_break_3d(dx=0.0185, max_neighbour_number=1)
        gap = float(case.domain.gap)
        side = float((case.n / 0.05) ** (1.0 / dim) * gap)
        case.domain = case.ps.domain = Domain2D(gap, 0, 0, side, side) if dim == 2 else Domain3D(gap, 0, 0, 0, side, side, side)
        rng = np.random.default_rng(3)
        case.ps["PositionVec"] = rng.uniform(0.01 * side, 0.99 * side, (case.n, dim)).astype(np.float32)
        case.physics.dt = 1e-9
        times.append(stages(case, family)[SEARCH])
    print(times)
    assert times[0] <= 1.5 * times[1]
