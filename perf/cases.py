"""Performance cases of the SPH backend: what a user of the framework has it do, through its public
entry points, over the range of sizes and options it is used at.

A case is a plain dict:

  kind   "steps"    a running simulation: `steps` fused time steps, then the state read back
                    (Context.step + Context.download), as a run that writes an output file now and
                    then; the context, its state and the output buffers live as long as the run
         "request"  a whole served run from host data: upload, initial search, `steps` steps, FP64
                    integrals, download
         "calls"    the reference's own loop, call by call: selfaction!, interaction!, selfaction!,
                    search! per step (main.jl:166-182), then the state read back
         "lists"    search! with the neighbour lists of the reference layout written back to the
                    host matrices (nIndex, nRVec, nR, nW, nDW, nHInv)
         "sort"     the cell-list build on caller-owned device buffers (epp_cell_sort_noalloc)
  dim, dx, column, tank   the dam break (epp.casegen), its lattice spacing and column of water
  physics  "benchmark" (Wendland C2, Tait EOS, artificial viscosity, symplectic Euler), "cfl" (the
           same with a CFL time step), "example" (the reference example's own: cubic spline, linear
           EOS, classic viscosity, kernel filter every 20 steps) or "library" (Wendland C4,
           density-weighted pressure, tensile correction, extrapolated wall pressure)
  instances  > 0: that many uneven 2D columns as one batch

The state is a collapse under way: the generator's hydrostatic column with its particles off their
lattice places, a spreading flow and a random part of the velocity, all drawn from the seed.  A pass
takes few enough steps that rounding differences have not grown into the flow by its end.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "etherparallelparticles.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from epp import abi, algorithm, casegen  # noqa: E402
from epp import lib as epplib  # noqa: E402
from epp.classes import NeighbourSystem  # noqa: E402

SYM = abi.EPP_CRITERION_SYMMETRY
CONT = abi.EPP_ACTION_DAMBREAK_CONTINUITY
LIST_WIDTH = 50   # nIndex columns of the reference layout (its default max_neighbour_number)


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest runs a user makes while setting a case up: launches and latency
        dict(name="steps 2d 1k", kind="steps", dim=2, dx=0.05, column_w=1.0, column_h=2.0, physics="benchmark",
             instances=0, steps=16),
        # one served request of the 256-instance mix, from host data to host data
        dict(name="request 2d 22k", kind="request", dim=2, dx=0.01, column_w=1.03, column_h=1.87,
             physics="benchmark", instances=0, steps=40),
        # an ordinary run with the CFL time step, odd spacing (ragged cell rows)
        dict(name="steps 2d 87k cfl", kind="steps", dim=2, dx=0.0047, column_w=0.97, column_h=1.83, physics="cfl",
             instances=0, steps=16),
        # the headline workload
        dict(name="steps 2d 515k", kind="steps", dim=2, dx=0.002, column_w=1.0, column_h=2.0, physics="benchmark",
             instances=0, steps=16),
        # the largest 2D run
        dict(name="steps 2d 2m", kind="steps", dim=2, dx=0.001, column_w=1.0, column_h=2.0, physics="benchmark",
             instances=0, steps=16),
        # 3D: a small served run, and the full-size one
        dict(name="steps 3d 166k", kind="steps", dim=3, dx=0.02, column_w=1.0, column_h=0.6, physics="benchmark",
             instances=0, steps=16),
        dict(name="steps 3d 6m", kind="steps", dim=3, dx=0.005, column_w=1.0, column_h=0.6, physics="benchmark",
             instances=0, steps=8),
        # many uneven instances in one launch per pass
        dict(name="batch 64", kind="steps", dim=2, dx=0.01, column_w=1.0, column_h=2.0, physics="benchmark",
             instances=64, steps=16),
        # the reference example's physics, its kernel filter every 20 steps on the way
        dict(name="steps 2d 133k example", kind="steps", dim=2, dx=0.004, column_w=1.0, column_h=2.0,
             physics="example", instances=0, steps=6),
        # the drop-in loop, call by call
        dict(name="calls 2d 49k", kind="calls", dim=2, dx=0.0067, column_w=1.0, column_h=2.0, physics="benchmark",
             instances=0, steps=10),
        # neighbour lists in the reference layout
        dict(name="lists 2d 23k", kind="lists", dim=2, dx=0.01, column_w=1.0, column_h=2.0, physics="benchmark",
             instances=0, steps=1),
        # the allocation-free cell list on caller-owned buffers
        dict(name="sort 3d 956k", kind="sort", dim=3, dx=0.01, column_w=1.0, column_h=0.6, physics="benchmark",
             instances=0, steps=1),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["batch", "request", "calls", "lists", "sort"])
    dim = rng.choice([2, 2, 3]) if kind in ("steps", "sort") else 2
    w, h = (round(rng.uniform(0.5, 1.5), 3), round(rng.uniform(1.0, 2.5), 3)) if dim == 2 else \
        (round(rng.uniform(0.5, 1.2), 3), round(rng.uniform(0.2, 0.8), 3))
    n = {"steps": lambda: _log(rng, 1e3, 1e6) if dim == 2 else _log(rng, 1e4, 1e6),
         "batch": lambda: _log(rng, 2e3, 3e4), "request": lambda: _log(rng, 1e3, 2e5),
         "calls": lambda: _log(rng, 1e3, 3e5), "lists": lambda: _log(rng, 1e3, 4e4),
         "sort": lambda: _log(rng, 1e3, 3e5)}[kind]()
    dx = float("%.4g" % ((w * h / n) ** 0.5 if dim == 2 else (w * 1.0 * h / n) ** (1.0 / 3.0)))
    physics = rng.choice(["benchmark", "benchmark", "cfl", "example", "library"] if dim == 2 else
                         ["benchmark", "benchmark", "cfl"]) if kind == "steps" else "benchmark"
    instances = rng.randint(4, 48) if kind == "batch" else 0
    total = n * (instances or 1)
    steps = {"request": 40, "calls": 10, "lists": 1, "sort": 1}.get(kind) or \
        (6 if physics in ("example", "library") else int(min(16, max(8, 4e6 / total))))
    return dict(kind="steps" if kind == "batch" else kind, dim=dim, dx=dx, column_w=w, column_h=h, physics=physics,
                instances=instances, steps=steps)


# -------------------------------------------------------------------------------- inputs of a case
@functools.lru_cache(maxsize=24)
def _base(kind, dim, dx, w, h, physics, instances):
    """The generator's case (lattice positions, hydrostatic state), the same for every seed."""
    nb = LIST_WIDTH if kind == "lists" else 1
    if instances:
        columns = [(round(0.5 + 0.9 * ((7 * k) % instances) / instances, 3), round(1.0 + 1.4 * k / instances, 3))
                   for k in range(instances)]
        c = casegen.dam_break_batch(instances, dx=dx, columns=columns, max_neighbour_number=nb)
    elif dim == 2:
        c = casegen.dam_break_2d(dx=dx, column=(w, h), max_neighbour_number=nb,
                                 physics="example" if physics == "example" else "benchmark")
    else:
        c = casegen.dam_break_3d(dx=dx, column=(w, 1.0, h), max_neighbour_number=nb)
    p = c.physics
    if physics == "cfl":
        p.cfl = 0.1
    if physics == "library":
        p.kernel = abi.EPP_KERNEL_WENDLAND_C4
        p.viscosity = abi.EPP_VISCOSITY_MONAGHAN
        p.pressure_ff = abi.EPP_PRESSURE_DENSITY_WEIGHTED
        p.pressure_fw = abi.EPP_PRESSURE_DENSITY_WEIGHTED
        p.tensile = 1
        p.wall_pressure = abi.EPP_WALL_PRESSURE_EXTRAPOLATE
    lattice = c.ps["PositionVec"]
    if physics == "example":   # under way the column carries its weight: the example's EOS, p = rho0 g (H - y)
        fl = c.ps["Tag"] == casegen.FLUID_TAG
        rho = c.ps["Density"].astype(np.float64)
        rho[fl] += casegen.RHO0 * casegen.EXAMPLE_G * (h - lattice[fl, 1]) / casegen.EXAMPLE_C0 ** 2
        c.ps["Density"] = rho.astype(np.float32)
        c.ps["Mass"] = c.ps["Density"] * c.ps["Volume"]
    return c, lattice, c.ps["Tag"] == casegen.FLUID_TAG


def _case(case):
    return _base(case["kind"], case["dim"], case["dx"], case["column_w"], case["column_h"], case["physics"],
                 case["instances"])


def _flow(case, seed):
    """Positions and velocities of the collapse under way (float32), from the seed."""
    _, lattice, fluid = _case(case)
    rng = np.random.default_rng([int(seed), 17])
    dim, up = case["dim"], case["dim"] - 1
    x, v = lattice.copy(), np.zeros_like(lattice)
    xf = lattice[fluid]
    rate = np.float32(rng.uniform(0.8, 1.2))
    vf = np.zeros_like(xf)
    vf[:, 0] = rate * xf[:, 0]            # spreading along x, sinking: no divergence
    vf[:, up] = -rate * xf[:, up]
    vf += np.float32(0.1) * rng.standard_normal(xf.shape, dtype=np.float32)
    x[fluid] = xf + np.float32(0.12 * case["dx"]) * (2 * rng.random(xf.shape, dtype=np.float32) - 1)
    v[fluid] = vf
    return x, v


def _pinned(shape, dtype=torch.float32):
    """A page-locked host array, column-major like the reference's matrices."""
    t = torch.empty(max(1, int(np.prod(shape))), dtype=dtype, pin_memory=True)
    return t, t.numpy()[: int(np.prod(shape))].reshape(shape, order="F")


def _pin(a):
    t, v = _pinned(a.shape, torch.int32 if a.dtype == np.int32 else torch.float32)
    v[...] = a
    return t, v


class _Out:
    """The host side of a read-back: alive flags and the columns a run writes out."""

    def __init__(self, n, dim):
        self.dim = dim
        self.keep, self.f = _pinned((n, 2 * dim + 3))
        self.keep_a, self.alive = _pinned((n,), torch.int32)
        m = abi.epp_column_map.empty()
        m.position, m.velocity, m.density, m.ddensity, m.pressure = 0, dim, 2 * dim, 2 * dim + 1, 2 * dim + 2
        self.cmap = m

    def read(self, ctx):
        ctx.download(self.alive, None, None, self.f, self.cmap)
        d = self.dim
        return {"alive": self.alive, "position": self.f[:, :d], "velocity": self.f[:, d:2 * d],
                "density": self.f[:, 2 * d], "ddensity": self.f[:, 2 * d + 1], "pressure": self.f[:, 2 * d + 2]}


def prepare(case, seed):
    c, _, _ = _case(case)
    ps, phys, dim = c.ps, c.physics, case["dim"]
    x, v = _flow(case, seed)
    if case["kind"] == "sort":
        lib = epplib.load()
        nc = c.domain.get_n()
        i32 = dict(dtype=torch.int32, device="cuda")
        dom = c.domain.to_abi()
        return {"kind": "sort", "lib": lib, "dom": dom, "n": c.n,
                "pos": torch.from_numpy(np.ascontiguousarray(x.T).reshape(-1)).cuda(),
                "counts": torch.zeros(nc, **i32), "offsets": torch.zeros(nc + 1, **i32),
                "ids": torch.zeros(c.n, **i32), "stream": torch.cuda.current_stream().cuda_stream}
    ps["PositionVec"] = x
    ps["VelocityVec"] = v
    width = LIST_WIDTH if case["kind"] == "lists" else 1
    ns = NeighbourSystem(c.domain, casegen.DAM_BREAK_ACTIVE_PAIRS, max_neighbour_number=width)
    dps = algorithm.DeviceParticleSystem(ps, ns, n_instances=case["instances"] or 1)
    dps.physics = phys
    state = {"kind": case["kind"], "dps": dps, "phys": phys, "steps": case["steps"], "n": c.n,
             "out": _Out(c.n, dim), "ps": ps}
    if case["instances"]:
        dps.ctx.set_instance_physics(c.inst_dt, c.inst_c0)
    if case["kind"] == "request":
        state["host"] = [_pin(a) for a in (ps.is_alive, ps.cell_index, ps.int_properties, ps.float_properties)]
        return state
    dps.syncto()
    if case["kind"] == "lists":
        m = dps.cmap
        state["int"], state["float"] = _pinned(ps.int_properties.shape, torch.int32), _pinned(ps.float_properties.shape)
        state["int"][1][...] = 0
        state["float"][1][...] = 0.0
        state["cols"] = (m.n_index, m.n_rvec, m.n_r, m.n_w, m.n_dw, m.n_hinv, m.n_count, m.ddensity)
        dps.ctx.synchronize()
        return state
    dps.ctx.search(SYM, CONT, phys, 0)
    dps.ctx.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "sort":
        n_alive = ctypes.c_int32(0)
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        rc = state["lib"].epp_cell_sort_noalloc(ctypes.byref(state["dom"]), state["n"], p(state["pos"]),
                                                p(state["counts"]), p(state["offsets"]), p(state["ids"]),
                                                ctypes.byref(n_alive), ctypes.c_void_p(state["stream"]))
        if rc != abi.EPP_OK:
            raise epplib.EppError(rc, "epp_cell_sort_noalloc")
        return {"counts": state["counts"], "offsets": state["offsets"], "ids": state["ids"], "alive": n_alive.value}
    dps, phys, ctx = state["dps"], state["phys"], state["dps"].ctx
    if kind == "steps":
        ctx.step(state["steps"], phys)
        return state["out"].read(ctx)
    if kind == "request":
        alive, cell, ints, floats = (v for _, v in state["host"])
        ctx.upload(state["n"], alive, cell, ints, floats, dps.cmap)
        ctx.search(SYM, CONT, phys, 0)
        ctx.step(state["steps"], phys)
        ig = ctx.integrals(phys)
        return {"state": state["out"].read(ctx), "mass": ig["mass_total"], "kinetic": ig["kinetic"],
                "potential": ig["potential"], "internal": ig["internal"]}
    if kind == "calls":
        for _ in range(state["steps"]):
            algorithm.selfaction(dps, abi.EPP_ACTION_DAMBREAK_DENSITY)
            algorithm.interaction(dps, abi.EPP_ACTION_DAMBREAK_MOMENTUM)
            algorithm.selfaction(dps, abi.EPP_ACTION_DAMBREAK_INTEGRATE)
            algorithm.search(dps, SYM, CONT, emit_list=False)
        return state["out"].read(ctx)
    algorithm.search(dps, SYM, CONT, emit_list=True)
    ints, floats = state["int"][1], state["float"][1]
    ctx.download(state["out"].alive, None, ints, floats, dps.cmap)
    nidx, nrvec, nr, nw, ndw, nh, cnt, dd = state["cols"]
    b = LIST_WIDTH
    return {"count": ints[:, cnt], "index": ints[:, nidx:nidx + b], "rvec": floats[:, nrvec:nrvec + 2 * b],
            "r": floats[:, nr:nr + b], "w": floats[:, nw:nw + b], "dw": floats[:, ndw:ndw + b],
            "hinv": floats[:, nh:nh + b], "ddensity": floats[:, dd]}


# ------------------------------------------------------------------------------------ least work
def work(case):
    """Bytes: each particle's record (position, its compensation, velocity, mass, h, density, its
    rate, pressure, tag, id) read and written once a step, and what crosses to or from the host once
    a pass.  Flops: per directed pair the criterion, continuity and momentum terms."""
    c, _, fluid = _case(case)
    dim, n = case["dim"], c.n
    h = 1.5 if dim == 2 else 1.3
    near = math.pi * (2 * h) ** 2 - 1 if dim == 2 else 4.0 / 3.0 * math.pi * (2 * h) ** 3 - 1
    pairs = near * float(fluid.sum()) + 0.2 * near * float((~fluid).sum())
    rec = 4.0 * (3 * dim + 4)
    if case["kind"] == "sort":
        return {"bytes": 4.0 * (n * (dim + 1) + 2 * c.domain.get_n()), "flops": 6.0 * n}
    if case["kind"] == "lists":
        return {"bytes": n * (rec + 4.0 * (2 + LIST_WIDTH * (3 + dim + 1))), "flops": 50.0 * pairs}
    moved = 4.0 * (2 * dim + 4) * n + (4.0 * (3 * dim + 13) * n if case["kind"] == "request" else 0.0)
    return {"bytes": moved + case["steps"] * n * 2 * rec, "flops": case["steps"] * pairs * (75.0 if dim == 2 else 95.0)}


# ------------------------------------------------------- the same results in 64 bits, plain torch
def _kernel(kind, dim):
    """(W(q), (dW/dr)/r per hinv^(dim+2)) of a kernel as functions of q, both without hinv powers."""
    if kind == abi.EPP_KERNEL_CUBIC_SPLINE:
        s = 10 / (7 * math.pi) if dim == 2 else 1 / math.pi
        return (lambda q: s * torch.where(q < 1, (3 * q * q * (q - 2) + 4) / 4, (2 - q).clamp(min=0) ** 3 / 4),
                lambda q: s * torch.where(q < 1, (3 * q - 4) * 0.75,
                                          -0.75 * (2 - q).clamp(min=0) ** 2 / q.clamp(min=1)))
    if kind == abi.EPP_KERNEL_WENDLAND_C4:
        s = 9 / (4 * math.pi) if dim == 2 else 495 / (256 * math.pi)
        return (lambda q: s * (2 - q).clamp(min=0) ** 6 * (q * (35 * q + 36) + 12) / 768,
                lambda q: -s * (35 * q + 14) / 96 * (2 - q).clamp(min=0) ** 5)
    s = 7 / (4 * math.pi) if dim == 2 else 21 / (16 * math.pi)
    return (lambda q: s * (2 - q).clamp(min=0) ** 4 * (1 + 2 * q) / 16,
            lambda q: -s * 0.625 * (2 - q).clamp(min=0) ** 3)


class _Sim:
    """The dam-break step in 64 bits: pair lists with a skin, terms scattered with index_add_."""

    def __init__(self, case, seed, chunk=1 << 26):
        c, _, fluid = _case(case)
        self.c, self.P, self.dim, self.chunk = c, c.physics, case["dim"], chunk
        ps, D = c.ps, case["dim"]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()  # noqa: E731
        x, v = _flow(case, seed)
        self.x32 = torch.from_numpy(x).cuda()
        self.x, self.v = t(x), t(v)
        self.m, self.V, self.rho, self.h, self.gap = (t(ps[k]) for k in ("Mass", "Volume", "Density", "H", "Gap"))
        self.p = t(ps["Pressure"])
        self.fluid = torch.from_numpy(fluid).cuda()
        self.inst = torch.from_numpy(ps["Instance"].astype(np.int64)).cuda() if case["instances"] else \
            torch.zeros(c.n, dtype=torch.int64, device="cuda")
        one = torch.ones(c.n, dtype=torch.float64, device="cuda")
        self.dt = t(c.inst_dt)[self.inst] if case["instances"] else one * float(self.P.dt)
        self.c0 = t(c.inst_c0)[self.inst] if case["instances"] else one * float(self.P.c0)
        self.g = [float(a) for a in self.P.gravity[:D]]
        self.drho = torch.zeros_like(self.rho)
        self.W, self.dWr = _kernel(self.P.kernel, D)
        self.built = None
        self.n_step = 0

    def eos(self, rho):
        P = self.P
        if P.eos == abi.EPP_EOS_LINEAR:
            return self.c0 ** 2 * (rho - P.rho0) + P.p0
        return P.rho0 * self.c0 ** 2 / P.gamma * ((rho / P.rho0) ** P.gamma - 1) + P.p0

    def find(self, skin=0.1):
        """Pair chunks (i, j): active pairs within (1 + skin) of the support."""
        D, x = self.dim, self.x
        R = 2 * float(self.h.max()) * (1 + skin)
        lo = x.min(0).values
        cell = ((x - lo) / R).floor().long()
        n = cell.max(0).values + 1
        key = cell[:, 0] + n[0] * (cell[:, 1] + n[1] * (cell[:, 2] if D == 3 else self.inst))
        layers = int(n[2]) if D == 3 else int(self.inst.max()) + 1
        n0, n1 = int(n[0]), int(n[1])
        order = torch.argsort(key, stable=True)
        start = torch.searchsorted(key[order], torch.arange(n0 * n1 * layers + 1, device="cuda"))
        chunks, N = [], x.shape[0]
        per = 9 * 9 if D == 2 else 27 * 27
        block = max(1, self.chunk // per)
        xs, fl, inst = x, self.fluid, self.inst
        for b in range(0, N, block):
            me = order[b:b + block]
            cb = cell[me]
            got = []
            for dz in ((-1, 0, 1) if D == 3 else (0,)):
                for dy in (-1, 0, 1):
                    yy = cb[:, 1] + dy
                    zz = cb[:, 2] + dz if D == 3 else inst[me]
                    ok = (yy >= 0) & (yy < n1) & (zz >= 0) & (zz < layers)
                    row = (yy.clamp(0, n1 - 1) + n1 * zz.clamp(0, layers - 1)) * n0
                    s = start[row + (cb[:, 0] - 1).clamp(min=0)]
                    e = start[row + (cb[:, 0] + 1).clamp(max=n0 - 1) + 1]
                    cnt = torch.where(ok, e - s, torch.zeros_like(s))
                    tot = int(cnt.sum())
                    if not tot:
                        continue
                    first = torch.cumsum(cnt, 0) - cnt
                    w = torch.repeat_interleave(torch.arange(me.shape[0], device="cuda"), cnt, output_size=tot)
                    j = order[torch.arange(tot, device="cuda") - first[w] + s[w]]
                    i = me[w]
                    d2 = ((xs[i] - xs[j]) ** 2).sum(1)
                    keep = (d2 <= R * R) & (i != j) & (fl[i] | fl[j])
                    got.append((i[keep].int(), j[keep].int()))
            chunks.append((torch.cat([a for a, _ in got]), torch.cat([a for _, a in got])))
        self.pairs, self.built, self.room = chunks, x.clone(), R - R / (1 + skin)

    def each(self):
        """Geometry of the pairs now within the criterion: i, j, r vectors, r, hinv, q."""
        if self.built is None or 2.02 * float((self.x - self.built).norm(dim=1).max()) > self.room:
            self.find()
        for i, j in self.pairs:
            hi, hj = self.h[i], self.h[j]
            d = self.x[i] - self.x[j]
            r = d.norm(dim=1)
            keep = r <= 4 * hi * hj / (hi + hj)
            i, j, d, r, hi, hj = i[keep], j[keep], d[keep], r[keep], hi[keep], hj[keep]
            hinv = (hi + hj) / (2 * hi * hj)
            yield i, j, d, r, hinv, r * hinv

    def continuity(self):
        for i, j, d, r, hinv, q in self.each():
            dwr = self.dWr(q) * hinv ** (self.dim + 2)
            vdx = (d * (self.v[i] - self.v[j])).sum(1)
            ff = self.fluid[i] & self.fluid[j]
            self.drho.index_add_(0, i, torch.where(ff, self.m[j], self.rho[i] * self.V[j]) * vdx * dwr)

    def extrapolate(self):
        wall = ~self.fluid
        a, b = torch.zeros_like(self.rho), torch.zeros_like(self.rho)
        for i, j, d, r, hinv, q in self.each():
            on = wall[i] & self.fluid[j]
            i, j, d, hinv, q = i[on], j[on], d[on], hinv[on], q[on]
            wv = self.W(q) * hinv ** self.dim * self.V[j]
            gx = sum(d[:, k] * self.g[k] for k in range(self.dim))
            a.index_add_(0, i, wv)
            b.index_add_(0, i, wv * (self.p[j].clamp(min=self.P.p0) + (self.rho[j] * gx).clamp(min=self.P.p0)))
        self.p = torch.where(wall, torch.where(a > 0, b / a.clamp(min=1e-300), torch.full_like(a, self.P.p0)), self.p)

    def pressure(self, form, i, j):
        p, rho = self.p, self.rho
        if form == abi.EPP_PRESSURE_CLASSIC:
            return p[i] / rho[i] ** 2 + p[j] / rho[j] ** 2
        if form == abi.EPP_PRESSURE_BALANCED:
            return (p[i] + p[j]) / (rho[i] * rho[j])
        return 2 * (p[i] * rho[i] + p[j] * rho[j]) / ((rho[i] + rho[j]) * rho[i] * rho[j])

    def momentum(self):
        P, D = self.P, self.dim
        du = torch.zeros_like(self.v)
        for i, j, d, r, hinv, q in self.each():
            on = self.fluid[i]
            i, j, d, r, hinv, q = i[on], j[on], d[on], r[on], hinv[on], q[on]
            dwr = self.dWr(q) * hinv ** (D + 2)
            ff = P.pressure_ff or abi.EPP_PRESSURE_CLASSIC
            fw = P.pressure_fw or abi.EPP_PRESSURE_BALANCED
            term = self.pressure(ff, i, j)
            if fw != ff:
                term = torch.where(self.fluid[j], term, self.pressure(fw, i, j))
            if P.tensile:
                wg = self.W(0.5 * (self.gap[i] + self.gap[j]) * hinv)
                term = term + term.abs() * 0.01 * self.W(q) / wg
            f = -self.m[j] * term * dwr
            dv = self.v[i] - self.v[j]
            az = r * r + 0.01 / hinv ** 2
            if P.viscosity == abi.EPP_VISCOSITY_CLASSIC:
                a = 2 * P.mu * self.m[j] * r * r * dwr / (self.rho[i] * self.rho[j] * az)
                du.index_add_(0, i, f[:, None] * d + a[:, None] * dv)
                continue
            vdx = (d * dv).sum(1)
            phi = vdx / (hinv * az)
            a = -self.m[j] * dwr * (-P.alpha * self.c0[i] + P.beta * phi) * phi / (0.5 * (self.rho[i] + self.rho[j]))
            if P.viscosity == abi.EPP_VISCOSITY_REFERENCE:
                a = a / (self.rho[i] * self.rho[j])
            f = f + torch.where(vdx < 0, a, torch.zeros_like(a))
            du.index_add_(0, i, f[:, None] * d)
        return du + torch.tensor(self.g, dtype=torch.float64, device="cuda")

    def step(self):
        P, fl = self.P, self.fluid[:, None]
        if P.cfl > 0:
            on = self.fluid
            self.dt = torch.full_like(self.dt, P.cfl * float(self.h[on].min()) /
                                      (float(P.c0) + float(self.v[on].norm(dim=1).max())))
        dt = self.dt[:, None]
        self.rho = self.rho + self.drho * self.dt
        self.V, self.p, self.drho = self.m / self.rho, self.eos(self.rho), torch.zeros_like(self.rho)
        if P.wall_pressure == abi.EPP_WALL_PRESSURE_EXTRAPOLATE:
            self.extrapolate()
        du = torch.where(fl, self.momentum(), torch.zeros_like(self.v))
        if P.motion == abi.EPP_MOTION_ACCELERATE_MOVE:
            self.x = self.x + (self.v + 0.5 * du * dt) * dt
            self.v = self.v + du * dt
        else:
            self.v = self.v + du * dt
            self.x = self.x + self.v * dt
        self.continuity()
        self.n_step += 1
        if P.filter_interval > 0 and self.n_step % P.filter_interval == 0:
            self.filter()

    def filter(self):
        w0 = self.W(torch.zeros_like(self.h)) / self.h ** self.dim
        a, b = w0 * self.V, w0 * self.m
        for i, j, d, r, hinv, q in self.each():
            on = self.fluid[i] & self.fluid[j]
            i, j, w = i[on], j[on], self.W(q[on]) * hinv[on] ** self.dim
            a.index_add_(0, i, w * self.V[j])
            b.index_add_(0, i, w * self.m[j])
        self.rho = torch.where(self.fluid, b / a, self.rho)
        self.V = torch.where(self.fluid, self.m / self.rho, self.V)
        self.p = torch.where(self.fluid, self.eos(self.rho), self.p)

    def state(self):
        return {"alive": None, **{k: v.cpu() for k, v in dict(
            position=self.x, velocity=self.v, density=self.rho, ddensity=self.drho, pressure=self.p).items()}}

    def energies(self):
        P, on = self.P, self.fluid
        m, rho, r = self.m[on], self.rho[on], self.rho[on] / P.rho0
        B, g1 = P.rho0 * float(P.c0) ** 2 / P.gamma, P.gamma - 1
        e = B / P.rho0 * (r ** g1 / g1 + 1 / r - P.gamma / g1) + P.p0 * (1 / P.rho0 - 1 / rho)
        pot = -sum(float((m * self.x[on][:, k]).sum()) * self.g[k] for k in range(self.dim))
        return {"mass": float(self.m.sum()), "kinetic": float((0.5 * m * (self.v[on] ** 2).sum(1)).sum()),
                "potential": pot, "internal": None if abs(float((m * e).sum())) < 1e-6 * abs(pot) else
                float((m * e).sum())}


def _lists64(case, seed):
    """The emitted lists: neighbours by the 32-bit criterion (the definition of the set), in the
    order of the cell stencil (x offset, y offset, id), their geometry in 64 bits."""
    s = _Sim(case, seed)
    s.find(skin=0.01)
    i, j = (torch.cat(a).long() for a in zip(*s.pairs))
    x, h = s.x32, torch.from_numpy(np.ascontiguousarray(s.c.ps["H"])).cuda()
    d = x[i] - x[j]
    e = d * d
    d2 = e[:, 0] + e[:, 1]
    hi, hj = h[i], h[j]
    R = (2 * hi) * hj / (hi + hj) * 2
    ok = d2 <= R * R
    i, j = i[ok], j[ok]
    dom = s.c.domain
    first = torch.tensor([float(a) for a in dom.first], dtype=torch.float32, device="cuda")
    inv = torch.tensor([float(a) for a in dom.gap_inv], dtype=torch.float32, device="cuda")
    top = torch.tensor([n - 1 for n in dom.n_axis], device="cuda")
    cell = torch.minimum(((x - first) * inv).floor().long().clamp(min=0), top)
    off = cell[j] - cell[i] + 1
    order = torch.argsort((off[:, 0] * 3 + off[:, 1]) * x.shape[0] + j)
    order = order[torch.argsort(i[order], stable=True)]
    i, j = i[order], j[order]
    n, b = x.shape[0], LIST_WIDTH
    cnt = torch.bincount(i, minlength=n)
    slot = torch.arange(i.shape[0], device="cuda") - (torch.cumsum(cnt, 0) - cnt)[i]
    d = s.x[i] - s.x[j]
    r = d.norm(dim=1)
    hinv = (s.h[i] + s.h[j]) / (2 * s.h[i] * s.h[j])
    q = r * hinv
    out = {k: torch.zeros(n, b, dtype=torch.float64, device="cuda") for k in ("r", "w", "dw", "hinv")}
    out["r"][i, slot], out["hinv"][i, slot] = r, hinv
    out["w"][i, slot], out["dw"][i, slot] = s.W(q) * hinv ** 2, s.dWr(q) * hinv ** 4 * r
    rv = torch.zeros(n, b, 2, dtype=torch.float64, device="cuda")
    rv[i, slot] = d
    s.continuity()
    return {"count": None, "index": None, "rvec": rv.reshape(n, 2 * b).cpu(), **{k: v.cpu() for k, v in out.items()},
            "ddensity": s.drho.cpu()}


def exact(case, seed):
    if case["kind"] == "sort":
        return None
    if case["kind"] == "lists":
        return _lists64(case, seed)
    s = _Sim(case, seed)
    s.continuity()
    for _ in range(case["steps"]):
        s.step()
    return {"state": s.state(), **s.energies()} if case["kind"] == "request" else s.state()
