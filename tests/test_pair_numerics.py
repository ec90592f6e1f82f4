"""Pair terms at the ends of FP32's range and where their parts cancel, against 64-bit arithmetic of
the same FP32 inputs: isolated pairs, so that a particle's sum is one term."""
import numpy as np
import pytest

from collections import OrderedDict

from epp import abi, casegen
from epp.algorithm import DeviceParticleSystem
from epp.classes import Domain2D, Domain3D, NeighbourSystem, ParticleSystem

pytestmark = pytest.mark.gpu

SYM, CONT = abi.EPP_CRITERION_SYMMETRY, abi.EPP_ACTION_DAMBREAK_CONTINUITY
MOMENTUM = abi.EPP_ACTION_DAMBREAK_MOMENTUM
FLUID, WALL = casegen.FLUID_TAG, casegen.WALL_TAG


def pairs(dim, h, apart, seed, tags=(FLUID, FLUID), n_pairs=200):
    """`n_pairs` isolated pairs of smoothing length h, `apart` (per pair) in units of h."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n_pairs ** (1.0 / dim)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), -1).reshape(-1, dim)[:n_pairs]
    gap = 2.0 * h
    first = (grid + 0.25) * (4 * gap)
    d = rng.standard_normal((n_pairs, dim))
    d *= (np.broadcast_to(apart, n_pairs) * h / np.linalg.norm(d, axis=1))[:, None]
    n = 2 * n_pairs
    x = np.empty((n, dim), np.float32)
    x[0::2], x[1::2] = first, first.astype(np.float32) + d
    lim = [0.0] * dim + [side * 4 * gap] * dim
    domain = (Domain2D if dim == 2 else Domain3D)(gap, *lim)
    ints, floats = casegen._layout(dim, 1)
    params = OrderedDict([("rho0", 1000.0), ("p0", 0.0), ("FLUID_TAG", FLUID), ("WALL_TAG", WALL), ("gap0", h), ("h0", h)])
    ps = ParticleSystem(domain, n, ints, floats, params)
    one = np.ones(n, np.float32)
    ps["PositionVec"] = x
    ps["Tag"] = np.tile(np.array(tags, np.int32), n_pairs)
    ps["IsMovable"] = np.ones(n, np.int32)
    ps["H"], ps["Gap"] = one * np.float32(h), one * np.float32(h)
    ps["Density"], ps["Mass"], ps["Volume"] = one, one, one
    ps["VelocityVec"] = rng.standard_normal((n, dim)).astype(np.float32)
    return ps, domain, rng


def device(ps, domain, family=0):
    d = DeviceParticleSystem(ps, NeighbourSystem(domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=1))
    d.ctx.set_tuning(family)
    d.syncto()
    return d


def physics(dim, **kw):
    p = casegen._physics(dim, 1e-9, 50.0, 0, kw.pop("viscosity", abi.EPP_VISCOSITY_REFERENCE), kw.pop("alpha", 0.1),
                         kw.pop("beta", 0.2))
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def geometry(ps, dim):
    """x_i - x_j, its length, v_i - v_j of the first particle of each pair, and (dW/dr)/r, in 64 bits."""
    x, v = ps["PositionVec"].astype(np.float64), ps["VelocityVec"].astype(np.float64)
    h = ps["H"].astype(np.float64)[0]
    dx = x[0::2] - x[1::2]
    r = np.linalg.norm(dx, axis=1)
    sigma = 7 / (4 * np.pi) if dim == 2 else 21 / (16 * np.pi)
    dwr = -sigma * 0.625 * np.maximum(2 - r / h, 0) ** 3 / h ** (dim + 2)
    return dx, r, v[0::2] - v[1::2], dwr, h


# The distance of a pair is the IEEE square root at any scale: pairs much closer than h in a system of
# atomic lengths (h = 5e-10, r down to 1e-16).  About 14 roundings to a term: 14 * 2^-24 < 1e-6.
@pytest.mark.parametrize("h,lo", [(0.01, 1e-6), (5e-10, 2e-7)])
def test_continuity_of_close_pairs(h, lo):
    apart = np.exp(np.random.default_rng(5).uniform(np.log(lo), np.log(0.5), 200))
    ps, domain, rng = pairs(2, h, apart, 1)
    if h < 1e-6:   # FP32 positions resolve such distances near the origin only: one pair there
        x = ps["PositionVec"]
        x[0], x[1] = (0.0, 0.0), (3e-17, 8e-17)
        ps["PositionVec"] = x
        v = ps["VelocityVec"]
        v[0], v[1] = (1.0, 1.5), (-0.5, -0.25)
        ps["VelocityVec"] = v
    ps["Mass"] = np.full(ps["Mass"].shape, 1e-20 if h < 1e-6 else 1.0, np.float32)
    d = device(ps, domain)
    d.ctx.search(SYM, CONT, physics(2), 0)
    d.ctx.synchronize()
    d.asyncto()
    dx, r, dv, dwr, _ = geometry(ps, 2)
    want = ps["Mass"].astype(np.float64)[0] * (dx * dv).sum(1) * dwr
    got = d.host["dDensity"][0::2].astype(np.float64)
    ok = np.abs((dx * dv).sum(1)) > 0.2 * r * np.linalg.norm(dv, axis=1)   # where dx . dv does not cancel
    assert ok.sum() > 50 and (ok[0] or h > 1e-6)
    assert np.all(np.abs(got - want)[ok] <= 1e-6 * np.abs(want[ok])), np.max(np.abs(got / want - 1)[ok])
    d.close()


# Fluid beside walls of the opposite pressure and another density: p_i + p_j is exactly zero, and so
# is the force.
@pytest.mark.parametrize("family", [0, 1, 4])
@pytest.mark.parametrize("dim", [2, 3])
def test_opposite_pressures_of_fluid_and_wall_cancel(dim, family):
    ps, domain, rng = pairs(dim, 0.01, 0.8, 2, tags=(FLUID, WALL))
    n = ps["Mass"].size
    p = rng.uniform(1.0, 1e5, n // 2).astype(np.float32)
    ps["Pressure"] = np.stack([p, -p], 1).reshape(-1)
    ps["Density"] = rng.uniform(700.0, 1300.0, n).astype(np.float32)
    ps["VelocityVec"] = np.zeros((n, dim), np.float32)
    d = device(ps, domain, family)
    phys = physics(dim)
    d.ctx.search(SYM, abi.EPP_ACTION_NONE, phys, 0)
    d.ctx.interaction(MOMENTUM, phys)
    d.ctx.synchronize()
    d.asyncto()
    assert np.array_equal(d.host["nCount"], np.ones(n, np.int32))
    assert not np.any(d.host["dVelocityVec"])
    d.close()


# The pressure and viscosity of pairs over FP32's densities, p = 0 where p / rho^2 leaves the range.  Three
# reciprocals of 1 ulp and about 25 roundings: 3 * 2^-23 + 25 * 2^-24 < 2e-6.
@pytest.mark.parametrize("viscosity", [abi.EPP_VISCOSITY_REFERENCE, abi.EPP_VISCOSITY_MONAGHAN])
@pytest.mark.parametrize("rho,mass", [(1000.0, 0.1), (2e-20, 1e-35), (1e20, 1e28)])
@pytest.mark.parametrize("dim", [2, 3])
def test_viscosity_over_the_range_of_densities(dim, rho, mass, viscosity):
    ps, domain, rng = pairs(dim, 0.01, rng_apart(dim), 3)
    n = ps["Mass"].size
    ps["Density"] = (rho * rng.uniform(0.7, 1.3, n)).astype(np.float32)
    ps["Mass"] = np.full(n, mass, np.float32)
    v, x = ps["VelocityVec"], ps["PositionVec"]
    v[0::2], v[1::2] = x[1::2] - x[0::2], 0.0   # head on: v . dx does not cancel
    ps["VelocityVec"] = v * np.float32(100.0)
    d = device(ps, domain)
    phys = physics(dim, viscosity=viscosity)
    d.ctx.search(SYM, abi.EPP_ACTION_NONE, phys, 0)
    d.ctx.interaction(MOMENTUM, phys)
    d.ctx.synchronize()
    d.asyncto()
    dx, r, dv, dwr, h = geometry(ps, dim)
    den, m = ps["Density"].astype(np.float64), ps["Mass"].astype(np.float64)[1::2]
    phi = (dx * dv).sum(1) * h / (r * r + 0.01 * h * h)
    al, be, c0 = (float(np.float32(a)) for a in (phys.alpha, phys.beta, phys.c0))
    f = (-al * c0 + be * phi) * phi / (0.5 * (den[0::2] + den[1::2])) * -m * dwr
    if viscosity == abi.EPP_VISCOSITY_REFERENCE:
        f /= den[0::2] * den[1::2]
    want = f[:, None] * dx
    got = d.host["dVelocityVec"][0::2].astype(np.float64)
    err = np.abs(got - want).max(1) / np.abs(want).max(1)
    assert np.all(np.isfinite(got)) and err.max() <= 2e-6, err.max()
    d.close()


def rng_apart(dim):
    return np.random.default_rng(dim).uniform(0.1, 1.2, 200)
