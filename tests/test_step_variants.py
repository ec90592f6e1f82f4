"""Kernel variants the step picks by size: the same results on both sides of each rule."""
import numpy as np
import pytest

from epp import abi, casegen
from epp.algorithm import DeviceParticleSystem
from epp.classes import NeighbourSystem

SYM = abi.EPP_CRITERION_SYMMETRY
CONT = abi.EPP_ACTION_DAMBREAK_CONTINUITY


def device(case, n_instances=1, max_nb=1):
    ns = NeighbourSystem(case.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=max_nb)
    d = DeviceParticleSystem(case.ps, ns, n_instances=n_instances)
    if n_instances > 1:
        d.ctx.set_instance_physics(case.inst_dt, case.inst_c0)
    d.syncto()
    return d


def stir(case, seed, speed=0.5, jitter=0.1):
    """Random velocities and displacements of the fluid, so that every pair term is in play."""
    rng = np.random.default_rng(seed)
    x, v, fl = case.ps["PositionVec"], case.ps["VelocityVec"], case.ps["Tag"] == casegen.FLUID_TAG
    x[fl] += np.float32(jitter * case.meta["dx"]) * rng.uniform(-1, 1, x[fl].shape).astype(np.float32)
    v[fl] = speed * rng.standard_normal(v[fl].shape).astype(np.float32)
    case.ps["PositionVec"] = x
    case.ps["VelocityVec"] = v


# instances per fold warp of the CFL reduction (8 warps): one each, all taken, some twice
@pytest.mark.gpu
@pytest.mark.parametrize("n_inst", [1, 8, 17])
def test_cfl_dt_of_every_instance(n_inst):
    columns = [(0.5 + 0.04 * k, 1.0 + 0.08 * k) for k in range(n_inst)]
    b = casegen.dam_break_batch(columns=columns, dx=0.05)
    stir(b, 3)
    phys = b.physics
    phys.cfl = 0.1
    d = device(b, n_inst if n_inst > 1 else 1)
    d.ctx.search(SYM, CONT, phys, 0)
    d.ctx.step(3, phys)
    dt, _ = d.ctx.step_dt(phys, n_inst)
    d.asyncto()
    v, h = d.host["VelocityVec"].astype(np.float64), d.host["H"].astype(np.float64)
    fl = (d.host["Tag"] == casegen.FLUID_TAG) & (d.host.is_alive[: b.n] == 1)
    for k, (r0, r1) in enumerate(b.rows):
        on = np.arange(r0, r1)[fl[r0:r1]]
        c0 = np.float64(np.float32(b.inst_c0[k])) if n_inst > 1 else np.float64(np.float32(phys.c0))
        want = np.float32(np.float64(np.float32(0.1)) * h[on].min() / (c0 + np.sqrt((v[on] ** 2).sum(1).max())))
        assert dt[k] == want, (k, dt[k], want)
    d.close()


def run_alone(case, phys, steps, threads=128):
    d = device(case)
    d.ctx.set_block_threads(threads)
    d.ctx.search(SYM, CONT, phys, 0)
    d.ctx.step(steps, phys)
    d.ctx.synchronize(raise_on_status=False)
    d.asyncto()
    out = {k: d.host[k].copy() for k in ("PositionVec", "VelocityVec", "Density", "dDensity", "Pressure")}
    d.close()
    return out


# A batch beyond the particle counts that take several lanes per particle, its instances below them:
# the passes give the same bits either way.  Block sizes put the groups at other places of a block.
@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 128])
def test_batch_beyond_the_lane_rules_equals_its_instances(threads):
    dx, steps = 0.0125, 4
    columns = [(0.5 + 0.04 * k, 1.0 + 0.07 * k) for k in range(20)]   # 247,832 particles
    b = casegen.dam_break_batch(columns=columns, dx=dx)
    stir(b, 5)
    assert b.n > 200000
    d = device(b, b.n_instances)
    d.ctx.set_block_threads(threads)
    d.ctx.search(SYM, CONT, b.physics, 0)
    d.ctx.step(steps, b.physics)
    d.asyncto()
    for k in (0, 7, 19):
        c = casegen.dam_break_2d(dx=dx, column=columns[k], max_neighbour_number=1)
        r0, r1 = b.rows[k]
        fresh = casegen.dam_break_batch(columns=columns, dx=dx)
        stir(fresh, 5)
        for name in ("PositionVec", "VelocityVec"):
            c.ps[name] = fresh.ps[name][r0:r1]
        assert c.n < 60000
        alone = run_alone(c, c.physics, steps, threads)
        for name, v in alone.items():
            assert np.array_equal(d.host[name][r0:r1], v), (k, name)
    d.close()


# The eight-lane search (up to 20,000 particles) against the staged one (beyond), on windows of every
# kind: lattices that drift against the cells (windows beyond 32 candidates), fluid and walls of
# different h, sparse rows, and lists beyond their capacity (h = 3 dx).  The 20-instance batch takes the
# staged search, each instance alone the eight-lane one.
@pytest.mark.gpu
@pytest.mark.parametrize("dx,h_factor,jitter,physics", [(0.0231, 1.5, 0.1, "benchmark"), (0.03, 1.5, 0.4, "benchmark"),
                                                        (0.045, 3.0, 0.1, "benchmark"), (0.0231, 1.5, 0.1, "example")])
def test_eight_lane_search_equals_the_staged_search(dx, h_factor, jitter, physics):
    n_inst = 24
    columns = [(0.5 + 0.03 * k, 1.0 + 0.05 * k) for k in range(n_inst)]
    b = casegen.dam_break_batch(columns=columns, dx=dx, h_factor=h_factor)
    if physics == "example":   # any kernel but the specialised one
        b.physics.kernel = abi.EPP_KERNEL_CUBIC_SPLINE
    stir(b, 7, jitter=jitter)
    assert b.n > 20000
    d = device(b, n_inst)
    d.ctx.search(SYM, CONT, b.physics, 0)
    d.ctx.synchronize()
    d.asyncto()
    cnt, ids = d.ctx.neighbour_lists(b.n, 64)
    for k in (0, 11, 23):
        r0, r1 = b.rows[k]
        c = casegen.dam_break_2d(dx=dx, column=columns[k], h_factor=h_factor, max_neighbour_number=1)
        for name in ("PositionVec", "VelocityVec"):
            c.ps[name] = d.host[name][r0:r1]
        c.physics.kernel = b.physics.kernel
        assert c.n <= 20000
        a = device(c)
        a.ctx.search(SYM, CONT, c.physics, 0)
        a.ctx.synchronize()
        a.asyncto()
        acnt, aids = a.ctx.neighbour_lists(c.n, 64)
        assert np.array_equal(acnt, cnt[r0:r1])
        assert np.array_equal(np.where(aids > 0, aids + r0, 0), ids[r0:r1])
        for name in ("dDensity", "nCount"):
            assert np.array_equal(a.host[name], d.host[name][r0:r1]), (k, name)
        a.close()
    d.close()


# Three h's mixed at random (walls of a third one, or of the fluid's): staged warps then see their own,
# one other and further ones.  Same bits as the eight-lane search of each instance alone.
@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.5, 0.002])
def test_staged_search_with_three_smoothing_lengths(share):
    dx, n_inst = 0.0231, 24
    columns = [(0.5 + 0.03 * k, 1.0 + 0.05 * k) for k in range(n_inst)]
    b = casegen.dam_break_batch(columns=columns, dx=dx)
    stir(b, 17)
    rng = np.random.default_rng(4)
    h = b.ps["H"].copy()
    pick = rng.random(b.n) < share   # smaller h only: every neighbour stays inside the 9 cells
    h[pick] *= rng.choice(np.float32([0.93, 0.8]), int(pick.sum()))
    b.ps["H"] = h
    d = device(b, n_inst)
    d.ctx.search(SYM, CONT, b.physics, 0)
    d.ctx.synchronize()
    d.asyncto()
    for k in (0, 23):
        r0, r1 = b.rows[k]
        c = casegen.dam_break_2d(dx=dx, column=columns[k], max_neighbour_number=1)
        for name in ("PositionVec", "VelocityVec"):
            c.ps[name] = d.host[name][r0:r1]
        c.ps["H"] = h[r0:r1]
        a = device(c)
        a.ctx.search(SYM, CONT, c.physics, 0)
        a.ctx.synchronize()
        a.asyncto()
        for name in ("dDensity", "nCount"):
            assert np.array_equal(a.host[name], d.host[name][r0:r1]), (k, name)
        a.close()
    d.close()


# v / d by multiplication, on the CPU: the same arithmetic as csrc/epp_math.cuh FastDiv
@pytest.mark.parametrize("d", [1, 2, 3, 7, 64, 1000, 1367, 65535, 65537, (1 << 22) + 1, (1 << 30) - 1, 1 << 30])
def test_fast_division(d):
    length = 0
    while (1 << length) < d:
        length += 1
    m, s = (0, 0) if d <= 1 else ((1 << (31 + length)) // d + 1, length - 1)
    assert m < 1 << 32
    rng = np.random.default_rng(d)
    v = np.concatenate([rng.integers(0, 1 << 31, 20000), np.arange(0, min(20 * d, 1 << 31), max(1, d))[:2000],
                        np.arange(d - 1, min(20 * d, (1 << 31) - 1), d)[:2000], [0, (1 << 31) - 1]])
    for x in (int(x) for x in v):
        q = x if m == 0 else ((x * m) >> 32) >> s
        assert q == x // d, (x, d)


# 3D search: eight lanes per particle (small system) and staged planes (beyond 50,000 particles), with
# one h, the two of fluid and walls, and three mixed at random; h = 2.5 dx takes rows one by one.  The
# neighbour counts are the oracle's.
@pytest.mark.gpu
@pytest.mark.parametrize("dx,column,h_factor,kinds", [
    (0.05, (1.0, 1.0, 0.6), 1.3, 1), (0.05, (0.93, 1.0, 0.57), 1.3, 3), (0.0262, (1.0, 1.0, 0.61), 1.3, 2),
    (0.0262, (1.0, 1.0, 0.61), 1.3, 3), (0.03, (1.0, 1.0, 0.6), 2.5, 1)])
def test_3d_search_variants_count_the_oracles_neighbours(dx, column, h_factor, kinds):
    from oracle_lib import Oracle
    c = casegen.dam_break_3d(dx=dx, column=column, h_factor=h_factor, max_neighbour_number=700)
    stir(c, 11)
    if kinds == 3:   # smaller h only: every neighbour stays inside the 27 cells
        rng = np.random.default_rng(2)
        c.ps["H"] = (c.ps["H"] * rng.choice([1.0, 0.93, 0.8], c.n)).astype(np.float32)
    elif kinds == 2:
        c.ps["H"] = np.where(c.ps["Tag"] == casegen.WALL_TAG, c.ps["H"] * np.float32(0.9), c.ps["H"]).astype(np.float32)
    d = device(c, max_nb=700)
    cfg = type(d.config).from_buffer_copy(d.config)
    cfg.max_cell_particles = 400
    o = Oracle(cfg, 32)
    o.upload(c.n, c.ps.is_alive, c.ps.cell_index, c.ps.int_properties, c.ps.float_properties, d.cmap)
    o.search(SYM, CONT, c.physics)
    d.ctx.search(SYM, CONT, c.physics, 0)
    d.ctx.synchronize()
    cnt, ids = d.ctx.neighbour_lists(c.n, 160)
    want = o.field(9, 0, c.n).astype(np.int32)
    assert np.array_equal(cnt, want)
    kept = cnt <= 160
    assert np.array_equal((ids[kept] > 0).sum(1), cnt[kept])
    x = c.ps["PositionVec"].astype(np.float64)
    h = c.ps["H"].astype(np.float64)
    rows = np.random.default_rng(3).choice(np.flatnonzero(kept & (cnt > 0)), 500)
    for i in rows:   # the stored neighbours are distinct, not itself, and inside the support
        j = ids[i][ids[i] > 0] - 1
        assert len(set(j.tolist())) == len(j) and i not in j
        assert np.all(np.linalg.norm(x[j] - x[i], axis=1) <= 4 * h[i] * h[j] / (h[i] + h[j]) * (1 + 1e-6))
    assert o.status() & abi.EPP_STATUS_CELL_OVERFLOW == 0
    d.close()


# Columns travel merged when the host matrices have no rows between them, one by one otherwise; absent
# columns break a run.
@pytest.mark.gpu
@pytest.mark.parametrize("spare,drop", [(0, ()), (37, ()), (0, ("velocity", "n_count", "density")), (5, ("volume",))])
def test_upload_and_download_of_padded_and_partial_matrices(spare, drop):
    from epp.classes import ParticleSystem
    a = casegen.dam_break_2d(dx=0.1, max_neighbour_number=3)
    stir(a, 1)
    tables = a.ps.named_index
    p = ParticleSystem(a.domain, a.n, tables.int_table.capacity, tables.float_table.capacity, a.ps.basic_parameters,
                       capacityExpand=lambda n: n + spare)
    for name in list(tables.int_table.capacity) + list(tables.float_table.capacity):
        p[name] = a.ps[name]
    before_f, before_i = p.float_properties.copy(), p.int_properties.copy()
    ns = NeighbourSystem(a.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=3)
    d = DeviceParticleSystem(p, ns)
    for f in drop:
        setattr(d.cmap, f, -1)
    d.syncto()
    p.float_properties[:a.n] = -7.0
    p.int_properties[:a.n] = -7
    d.ctx.download(p.is_alive, p.cell_index, p.int_properties, p.float_properties, d.cmap)
    m = d.cmap
    fcols = [c + k for c, w in [(m.position, 2), (m.velocity, 2), (m.dvelocity, 2), (m.mass, 1), (m.volume, 1),
                                (m.density, 1), (m.ddensity, 1), (m.pressure, 1), (m.h, 1)] if c >= 0 for k in range(w)]
    icols = [c for c in (m.tag, m.is_movable, m.n_count) if c >= 0]
    for c in range(before_f.shape[1]):
        want = before_f[:a.n, c] if c in fcols else np.full(a.n, -7.0, np.float32)
        assert np.array_equal(p.float_properties[:a.n, c], want), c
    for c in range(before_i.shape[1]):
        want = before_i[:a.n, c] if c in icols else np.full(a.n, -7, np.int32)
        assert np.array_equal(p.int_properties[:a.n, c], want), c
    assert np.array_equal(p.float_properties[a.n:], before_f[a.n:])   # rows beyond the particles stay
    d.close()


# The sort's buffers alternate with the state sets: an upload at either parity, pair-pass families that
# keep other lists in them, and a dead bin of many particles leave the next cell list right.
@pytest.mark.gpu
@pytest.mark.parametrize("steps,family", [(0, 0), (1, 0), (2, 0), (3, 1), (2, 1), (1, 4)])
@pytest.mark.parametrize("dead", [0, 700])
def test_cell_lists_after_uploads_and_family_switches(steps, family, dead):
    c = casegen.dam_break_2d(dx=0.04, max_neighbour_number=1)
    stir(c, 2)
    x = c.ps["PositionVec"]
    fluid = np.flatnonzero(c.ps["Tag"] == casegen.FLUID_TAG)
    x[fluid[:dead]] = 100.0   # outside: the search kills them
    c.ps["PositionVec"] = x
    want = device(c)
    want.ctx.search(SYM, CONT, c.physics, 0)
    counts, offsets, ids = want.ctx.cell_stats()
    want.close()
    d = device(c)
    d.ctx.search(SYM, CONT, c.physics, 0)
    d.ctx.set_tuning(family)
    if steps:
        d.ctx.step(steps, c.physics)
    d.syncto()
    d.ctx.search(SYM, CONT, c.physics, 0)
    for _ in range(2):   # once more: a search! in place keeps the order
        got = d.ctx.cell_stats()
        assert np.array_equal(got[0], counts) and np.array_equal(got[1], offsets) and np.array_equal(got[2], ids)
        d.ctx.set_tuning(0)
        d.ctx.search(SYM, abi.EPP_ACTION_NONE, c.physics, 0)
    assert d.ctx.synchronize(raise_on_status=False) & ~abi.EPP_STATUS_KILLED == 0
    d.close()


# The allocation-free sort on particles in no cell order: a shuffled column, a cell of many particles, and
# some outside the domain; the context's cell lists.
@pytest.mark.gpu
@pytest.mark.parametrize("dim,dx", [(2, 0.05), (2, 0.0231), (3, 0.1), (3, 0.041)])
@pytest.mark.parametrize("crowd,outside", [(0, 0), (700, 33)])
def test_noalloc_sort_of_shuffled_particles(dim, dx, crowd, outside):
    from test_zz_no_alloc import _noalloc
    c = casegen.dam_break_2d(dx=dx, max_neighbour_number=1) if dim == 2 else \
        casegen.dam_break_3d(dx=dx, max_neighbour_number=1)
    rng = np.random.default_rng(31)
    x = c.ps["PositionVec"][rng.permutation(c.n)].copy()
    x[: min(crowd, c.n // 3)] = x[c.n // 2]
    x[c.n - outside:] = 100.0
    c.ps["PositionVec"] = x
    d = device(c)
    d.ctx.search(SYM, abi.EPP_ACTION_NONE, c.physics, 0)
    counts, offsets, ids = d.ctx.cell_stats()
    got_c, got_o, got_ids, n_alive = _noalloc(c.domain, x)
    assert n_alive == c.n - outside
    assert np.array_equal(got_c, counts) and np.array_equal(got_o[:len(offsets)], offsets[:len(got_o)])
    assert np.array_equal(got_ids[:n_alive], ids[:n_alive])
    d.close()
