"""Cell lists of particles in any order and of crowded cells: the time of the sort does not hang on them
(faults these tests are for took 4 to 12 times as long), and the lists are the same."""
import ctypes as C
import time

import numpy as np
import pytest

from epp import abi
from epp import lib as epplib

pytestmark = pytest.mark.gpu


def sort_time(dim, n, per_cell, ordered, seed=1):
    """(least time of a sort, us; its ids) of n particles, about per_cell to a cell, in cell order or not."""
    import torch
    lib = epplib.load()
    rng = np.random.default_rng(seed)
    side = max(1, int(round((n / per_cell) ** (1.0 / dim))))
    x = rng.random((dim, n)).astype(np.float32)
    if ordered:
        cell = np.zeros(n, np.int64)
        for a in reversed(range(dim)):
            cell = cell * side + np.minimum((x[a] * side).astype(np.int64), side - 1)
        x = np.ascontiguousarray(x[:, np.argsort(cell, kind="stable")])
    pos = torch.from_numpy(x).cuda()
    dom = abi.make_domain(dim, float(np.float32(1.0 / (side + 0.01))), [0.0] * dim, [1.0] * dim)
    ids = torch.zeros(n, dtype=torch.int32, device="cuda")
    off = torch.zeros(side ** dim + 1, dtype=torch.int32, device="cuda")
    alive, best = C.c_int32(), 1e9
    torch.cuda.synchronize()
    for _ in range(8):
        t = time.perf_counter()
        rc = lib.epp_cell_sort_noalloc(C.byref(dom), n, C.c_void_p(pos.data_ptr()), None, C.c_void_p(off.data_ptr()),
                                       C.c_void_p(ids.data_ptr()), C.byref(alive), None)
        best = min(best, (time.perf_counter() - t) * 1e6)
        assert rc == abi.EPP_OK and alive.value == n
    off, ids = off.cpu().numpy(), ids.cpu().numpy()
    rise = np.diff(ids) > 0
    rise[off[1:-1][(off[1:-1] > 0) & (off[1:-1] < n)] - 1] = True   # ids rise inside each cell
    assert rise.all() and np.array_equal(np.sort(ids), np.arange(1, n + 1))
    return best


@pytest.mark.parametrize("dim", [2, 3])
def test_sort_time_of_shuffled_particles(dim):
    assert sort_time(dim, 1000000, 36, False) <= 2.0 * sort_time(dim, 1000000, 36, True)


@pytest.mark.parametrize("dim", [2, 3])
def test_sort_time_of_crowded_cells(dim):
    assert sort_time(dim, 300000, 300, False) <= 2.5 * sort_time(dim, 300000, 9, True)


def crowd(dim, side, n, seed=4):
    """A context of n particles at random places of side^dim cells, a tenth of them outside."""
    from collections import OrderedDict
    from epp import casegen
    from epp.algorithm import DeviceParticleSystem
    from epp.classes import Domain2D, Domain3D, NeighbourSystem, ParticleSystem
    rng = np.random.default_rng(seed)
    domain = (Domain2D if dim == 2 else Domain3D)(1.0 / (side + 0.01), *[0.0] * dim, *[1.0] * dim)
    ints, floats = casegen._layout(dim, 1)
    ps = ParticleSystem(domain, n, ints, floats, OrderedDict([("rho0", 1000.0)]))
    x = rng.random((n, dim)).astype(np.float32)
    x[rng.random(n) < 0.1] += 5.0
    one = np.ones(n, np.float32)
    ps["PositionVec"], ps["H"], ps["Density"], ps["Mass"], ps["Volume"] = x, one * 1e-3, one, one, one
    ps["Tag"], ps["IsMovable"] = np.full(n, casegen.FLUID_TAG, np.int32), np.ones(n, np.int32)
    d = DeviceParticleSystem(ps, NeighbourSystem(domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
    d.syncto()
    return d, domain, x


def numpy_cells(domain, x):
    """(counts, ids in cell order, each cell's rising) of positions, by the domain's own FP32 cell index."""
    dim = x.shape[1]
    first, last = np.array(domain.first, np.float32), np.array(domain.last, np.float32)
    inside = np.all((x >= first) & (x <= last), axis=1)
    cell, stride = np.zeros(len(x), np.int64), 1
    for a in range(dim):
        k = np.floor((x[:, a] - first[a]) * np.float32(domain.gap_inv[a])).astype(np.int64)
        cell += np.clip(k, 0, domain.n_axis[a] - 1) * stride
        stride *= domain.n_axis[a]
    ids = np.flatnonzero(inside)
    order = ids[np.argsort(cell[inside], kind="stable")]
    return np.bincount(cell[inside], minlength=stride), order + 1


# Either side of 64 particles to a cell, where the sort goes from linked lists to slots; the families that
# always take one of the two; more than one search, as the buffers alternate.
@pytest.mark.parametrize("dim,side", [(2, 6), (3, 3)])
@pytest.mark.parametrize("over", [-1, 0, 1])
@pytest.mark.parametrize("family", [0, 1, 4])
def test_cells_of_crowded_contexts(dim, side, over, family):
    d, domain, x = crowd(dim, side, 64 * side ** dim + over)
    d.ctx.set_tuning(family)
    counts, ids = numpy_cells(domain, x)
    for _ in range(3):
        d.ctx.search(abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_NONE, None, 0)
        got = d.ctx.cell_stats()
        assert np.array_equal(got[0], counts) and np.array_equal(got[2][:len(ids)], ids)
    d.close()


# Family 1 taken up by a context of a large grid: no device memory beyond the budget's, and no wait.
def test_family_one_takes_no_memory():
    import torch
    from epp import casegen
    from epp.algorithm import DeviceParticleSystem
    from epp.classes import Domain2D, NeighbourSystem
    case = casegen.dam_break_2d(dx=0.05, max_neighbour_number=1)
    first = case.domain.first
    case.ps.domain = case.domain = Domain2D(0.15, first[0], first[1], 0.15 * 8000, 0.15 * 8000)
    assert case.domain.get_n() > 60e6
    d = DeviceParticleSystem(case.ps, NeighbourSystem(case.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
    d.syncto()
    d.ctx.search(abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_DAMBREAK_CONTINUITY, case.physics, 0)
    d.ctx.step(2, case.physics)
    d.ctx.synchronize()
    free = torch.cuda.mem_get_info()[0]
    d.ctx.set_tuning(1)
    d.ctx.step(2, case.physics)
    d.ctx.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)   # graphs, not heads of 60 million cells
    d.close()


# The scan over either side of the tile counts at which its counters lie otherwise or are summed by a launch of
# their own: a small column of water in the corner of a large domain steps as in its own, whatever family
# sorted it in between, and through an upload at either parity.
@pytest.mark.parametrize("tiles", [1250, 1251, 3800, 3801, 4097, 15000, 15001])
def test_steps_in_large_grids(tiles):
    from epp import casegen
    from epp.algorithm import DeviceParticleSystem
    from epp.classes import Domain2D, NeighbourSystem
    out = []
    for far in (False, True):
        case = casegen.dam_break_2d(dx=0.05, max_neighbour_number=1)
        if far:   # the same cells on x (the same order), more of them on y
            dom = case.domain
            gap, first, last = float(dom.gap), [float(v) for v in dom.first], [float(v) for v in dom.last]
            rows = int(np.ceil((tiles * 2048 - 1) / dom.n_axis[0]))
            case.ps.domain = case.domain = Domain2D(gap, first[0], first[1], last[0], first[1] + (rows + 0.4) * float(dom.gap_axis[1]))
        d = DeviceParticleSystem(case.ps, NeighbourSystem(case.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
        d.syncto()
        d.ctx.search(abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_DAMBREAK_CONTINUITY, case.physics, 0)
        d.ctx.step(3, case.physics)
        d.ctx.set_tuning(1)
        d.ctx.step(2, case.physics)
        d.ctx.set_tuning(0)
        d.ctx.step(2, case.physics)
        d.ctx.synchronize()
        d.asyncto()
        d.syncto()
        d.ctx.search(abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_NONE, case.physics, 0)
        ids = d.ctx.cell_stats()[2]
        d.asyncto()
        out.append([d.host[k].copy() for k in ("PositionVec", "VelocityVec", "nCount", "dDensity")] + [ids])
        n = case.domain.get_n()
        d.close()
    assert (n + 2048) // 2048 >= tiles
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# the scan's time follows the number of cells (each tile adding up all counters before it made it 5 times the
# look-back scan's at this size, and growing with the square)
def test_scan_time_of_a_large_grid():
    from epp import casegen
    from epp.algorithm import DeviceParticleSystem
    from epp.classes import Domain2D, NeighbourSystem
    times = []
    for side in (4000, 16000):
        case = casegen.dam_break_2d(dx=0.05, max_neighbour_number=1)
        first = case.domain.first
        case.ps.domain = case.domain = Domain2D(0.15, first[0], first[1], 0.15 * side, 0.15 * side)
        d = DeviceParticleSystem(case.ps, NeighbourSystem(case.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
        d.syncto()
        d.ctx.search(abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_DAMBREAK_CONTINUITY, case.physics, 0)
        st = [list(s.values()) if isinstance(s, dict) else list(s) for s in (d.ctx.profile_step(case.physics) for _ in range(5))]
        times.append(np.min(np.array(st), axis=0)[1])   # the scan
        d.close()
    assert times[1] <= 2.0 * 16 * times[0]
