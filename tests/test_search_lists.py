"""Neighbour lists of every search variant against the order they are defined in: stencil rows (z, then
y), cells along x, ids inside a cell; the criterion and the active-pair matrix in FP32.  On both sides
of the particle counts that choose a variant (eight lanes per particle up to 20,000 in 2D and 50,000 in
3D, staged windows beyond)."""
import numpy as np
import pytest

from epp import abi, casegen
from epp.algorithm import DeviceParticleSystem
from epp.classes import NeighbourSystem

pytestmark = pytest.mark.gpu

SYM, DEFAULT = abi.EPP_CRITERION_SYMMETRY, abi.EPP_CRITERION_DEFAULT
f32 = np.float32
CAP = {2: 64, 3: 160}   # neighbours a list keeps


def expected(domain, x, h, tag, pairs, crit, cells, i):
    """Ids (1-based) of particle i's neighbours in list order."""
    dim = domain.dim
    counts, offsets, ids = cells
    n = list(domain.n_axis) + [1] * (3 - dim)
    at = [int(np.clip(np.floor(f32(f32(x[i, a] - f32(domain.first[a])) * f32(domain.gap_inv[a]))), 0, n[a] - 1))
          for a in range(dim)] + [0] * (3 - dim)
    cand = []
    for dz in ((-1, 0, 1) if dim == 3 else (0,)):
        for dy in (-1, 0, 1):
            y, z = at[1] + dy, at[2] + dz
            if not (0 <= y < n[1] and 0 <= z < n[2]):
                continue
            row = (y + n[1] * z) * n[0]
            lo, hi = row + max(at[0] - 1, 0), row + min(at[0] + 1, n[0] - 1)
            cand.append(ids[offsets[lo]:offsets[hi + 1]] - 1)
    j = np.concatenate(cand)
    d = (x[i] - x[j]).astype(f32)
    sq = (d * d).astype(f32)
    dr2 = (sq[:, 0] + sq[:, 1]).astype(f32)
    if dim == 3:
        dr2 = (dr2 + sq[:, 2]).astype(f32)
    if crit == DEFAULT:
        bound = np.full(len(j), f32(domain.gap_square))
    else:
        h2 = (((f32(2) * h[i] * h[j]).astype(f32) / (h[i] + h[j]).astype(f32)).astype(f32) * f32(2)).astype(f32)
        bound = (h2 * h2).astype(f32)
    ok = (dr2 <= bound) & (j != i) & np.array([(tag[i], t) in pairs for t in tag[j]])
    return j[ok] + 1


def check(case, dim, crit, tags):
    dx = case.meta["dx"]
    rng = np.random.default_rng(dim)
    ps, fl = case.ps, case.ps["Tag"] == casegen.FLUID_TAG
    x = ps["PositionVec"]
    x[fl] += (0.1 * dx * rng.uniform(-1, 1, x[fl].shape)).astype(f32)
    ps["PositionVec"] = x
    ps["H"] = np.where(rng.random(case.n) < 0.02, ps["H"] * f32(0.9), ps["H"]).astype(f32)
    tag = ps["Tag"].copy()
    pairs = list(casegen.DAM_BREAK_ACTIVE_PAIRS)
    if tags == "three":   # a third kind of particle, seen by the fluid and blind to the walls
        pairs += [(casegen.FLUID_TAG, 3), (3, casegen.FLUID_TAG), (3, 3)]
        tag[fl & (rng.random(case.n) < 0.3)] = 3
    if tags == "bad":     # tags outside the matrix: reported, nobody's neighbours and without any
        odd = rng.random(case.n) < 0.01
        tag[odd] = rng.choice([0, 7, 40, 255], int(odd.sum()))
        tag[np.flatnonzero(fl)[:200]] = 9   # and whole warps of them
    ps["Tag"] = tag
    d = DeviceParticleSystem(ps, NeighbourSystem(case.domain, pairs, max_neighbour_number=1))
    d.syncto()
    h = ps["H"]
    for action in (abi.EPP_ACTION_NONE, abi.EPP_ACTION_DAMBREAK_CONTINUITY):
        d.ctx.search(crit, action, case.physics, 0)
        status = d.ctx.synchronize(raise_on_status=False)
        assert bool(status & abi.EPP_STATUS_BAD_TAG) == (tags == "bad")
        cells = d.ctx.cell_stats()
        cnt, ids = d.ctx.neighbour_lists(case.n, CAP[dim])
        pick = np.concatenate([rng.choice(case.n, 200), np.flatnonzero(tag > 2)[:50], np.flatnonzero(tag == 0)[:5]])
        for i in pick:
            want = expected(case.domain, x, h, tag, set(pairs), crit, cells, i)
            assert cnt[i] == len(want), (i, tag[i])
            if len(want) <= CAP[dim]:   # (an overflowing list's ids are not given)
                assert np.array_equal(ids[i][:len(want)], want), (i, tag[i])
    d.close()


def column(dim, dx, **kw):
    return (casegen.dam_break_2d if dim == 2 else casegen.dam_break_3d)(dx=dx, max_neighbour_number=1, **kw)


@pytest.mark.parametrize("dim,dx,staged", [(2, 0.0231, False), (2, 0.0095, True), (3, 0.05, False), (3, 0.0262, True)])
@pytest.mark.parametrize("crit", [SYM, DEFAULT])
@pytest.mark.parametrize("tags", ["two", "three", "bad"])
def test_lists_and_their_order(dim, dx, staged, crit, tags):
    case = column(dim, dx)
    assert (case.n > {2: 20000, 3: 50000}[dim]) == staged
    check(case, dim, crit, tags)


# windows and stencils beyond the staging areas, lists beyond their capacity
@pytest.mark.parametrize("dim,dx,h_factor", [(2, 0.0231, 3.0), (2, 0.0095, 2.2), (2, 0.0095, 4.0), (3, 0.05, 2.5),
                                             (3, 0.0262, 1.8), (3, 0.0262, 2.5), (3, 0.0262, 4.0)])
@pytest.mark.parametrize("tags", ["three", "bad"])
def test_lists_of_dense_neighbourhoods(dim, dx, h_factor, tags):
    check(column(dim, dx, h_factor=h_factor), dim, SYM, tags)


# spray: warps of a few and of many parts, and of both
@pytest.mark.parametrize("dim,dx", [(2, 0.0095), (3, 0.0262)])
@pytest.mark.parametrize("per_cell", [0.05, 0.5, 2.0])
def test_lists_of_spray(dim, dx, per_cell):
    from epp.classes import Domain2D, Domain3D
    case = column(dim, dx)
    gap = float(case.domain.gap)
    side = float((case.n / per_cell) ** (1.0 / dim) * gap)
    case.domain = case.ps.domain = (Domain2D if dim == 2 else Domain3D)(gap, *[0.0] * dim, *[side] * dim)
    rng = np.random.default_rng(12)
    x = rng.uniform(0.02 * side, 0.98 * side, (case.n, dim)).astype(f32)
    x[: case.n // 4] = (0.3 * side + rng.uniform(0, 4 * gap, (case.n // 4, dim))).astype(f32)   # and a crowd
    case.ps["PositionVec"] = x
    check(case, dim, SYM, "two")
