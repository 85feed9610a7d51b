"""What a user of this framework has it do, as cases that can be timed and compared.

A case is one of seven kinds of call:

* ``step``: one time step of a particle set through ``Context.step``, the state carried from pass to pass as a
  time loop carries it (positions, velocities, labels and neighbour tables are the previous pass's);
* ``modules``: the same time step through the module calls the C++ drop-in forwards to, with all four moment
  kinds and the pressure solve, which ``Context.step`` leaves to its caller;
* ``solve``: the pressure solve of an assembled system, with its default options;
* ``diagnostics``: neighbour tables, labels with every diagnostic, and the virtual-light pass of a loaded state;
* ``operators`` / ``step_operators``: the differentiable operator pairs, forward and backward;
* ``batch``: many boxes stepped by one captured graph.

Particle sets are the repository's layouts: a hydrostatic ``box``, a ``dam`` break, a ``splash`` dam break (5% of the
fluid lifted above the free surface) and its ``scattered`` variant (the lifted fluid off the lattice columns), with
three wall layers, r_e = 3.1 l0, jittered positions and a seeded velocity and pressure field.
"""

import ctypes
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("lsmps-3d_b200")
abi, buffers = pkg.abi, pkg.buffers

INNER, NEAR_SURFACE, SURFACE, SPLASH = 0, 1, 2, 3
VELOCITY_A, PRESSURE_A, PRESSURE_B, FLUID_A = 0, 1, 2, 3
GRAVITY = (0.0, 0.0, -9.81)
RE = 3.1  # r_e / l0
LAYERS = 3
TUNED = {"plain": (2, 1, 1), "mixed": (1, 2, 1)}  # what the autotuner picks at 2M: moment variant, PPE and gather lanes
PER_ROW = 108  # neighbours of a bulk particle at r_e = 3.1 l0
FLUID = ("x", "y", "z", "vx", "vy", "vz", "pressure")
XYZ = ("x", "y", "z")
OPERATOR_OUT = ("grad_x", "grad_y", "grad_z", "laplacian", "divergence", "ppe_rhs")
STEP_OPERATOR_OUT = ("lap_x", "lap_y", "lap_z", "divergence", "grad_x", "grad_y", "grad_z", "ppe_rhs", "wall_rhs")


def listed():
    return [
        # A handful of particles, as in the reference's unit and hydrostatic checks: latency and launches count.
        dict(name="step_1k_plain", kind="step", form="plain", layout="box", nx=10, ny=10, nz=10, tuned=False,
             shuffled=False, sync=True),
        # A small tank of odd sizes, mixed precision, default settings.
        dict(name="step_22k_mixed", kind="step", form="mixed", layout="dam", nx=37, ny=19, nz=31, tuned=False,
             shuffled=False, sync=True),
        # The 500k dam break, FP64, in a tuned time loop that does not wait for every step.
        dict(name="step_500k_plain", kind="step", form="plain", layout="dam", nx=100, ny=50, nz=100, tuned=True,
             shuffled=False, sync=False),
        # FP64 on a state whose numbering does not follow space, with sparse splash neighbourhoods.
        dict(name="step_660k_scattered", kind="step", form="plain", layout="scattered", nx=141, ny=37, nz=127, tuned=True,
             shuffled=True, sync=False),
        # The headline workload: the 2M splash dam break in the mixed form.
        dict(name="step_2m_mixed", kind="step", form="mixed", layout="splash", nx=200, ny=50, nz=200, tuned=True,
             shuffled=False, sync=False),
        # A program on the module calls (the C++ drop-in's route), solve included.
        dict(name="modules_60k", kind="modules", layout="dam", nx=50, ny=25, nz=49),
        # The pressure solve alone: a small system, where launches and the residual's way to the host count, and a
        # large one, where the matrix has to be read.
        dict(name="solve_8k", kind="solve", layout="box", nx=20, ny=20, nz=20),
        dict(name="solve_500k", kind="solve", layout="dam", nx=100, ny=50, nz=100),
        # Post-processing of a loaded state.
        dict(name="diagnostics_250k", kind="diagnostics", layout="dam", nx=79, ny=39, nz=83),
        # Training or inversion through the operators: forward and backward, without and with the wall terms.
        dict(name="operators_262k", kind="operators", layout="box", nx=64, ny=64, nz=64),
        dict(name="step_operators_31k", kind="step_operators", layout="box", nx=31, ny=33, nz=31),
        # A parameter study: boxes of 8k to 200k particles in one graph.
        dict(name="batch_12_mixed", kind="batch", form="mixed", boxes=12, n_min=8000, n_max=120000),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def block(n, layout):
        # a block of about n particles: a cube for a box, 2:1:2 or flatter for the breaks
        if layout == "box":
            a = n ** (1 / 3)
            return dict(nx=max(5, round(a * rng.uniform(0.8, 1.25))), ny=max(5, round(a * rng.uniform(0.8, 1.25))),
                        nz=max(5, round(a)))
        a = (n / 4) ** (1 / 3)
        return dict(nx=max(8, round(2 * a * rng.uniform(0.8, 1.2))), ny=max(5, round(a * rng.uniform(0.8, 1.1))),
                    nz=max(8, round(2 * a * rng.uniform(0.9, 1.1))))

    kind = rng.choice(["step"] * 5 + ["modules", "solve", "solve", "diagnostics", "operators", "step_operators", "batch"])
    if kind == "step":
        layout = rng.choice(["box", "dam", "splash", "scattered"])
        n = log(1000, 1.5e6)
        return dict(kind=kind, form=rng.choice(["plain", "mixed"]), layout=layout, **block(n, layout),
                    tuned=rng.random() < 0.5, shuffled=rng.random() < 0.25, sync=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, form=rng.choice(["plain", "mixed"]), boxes=rng.randint(3, 12), n_min=rng.randint(3000, 9000),
                    n_max=rng.randint(20000, 120000))
    hi = {"modules": 2e5, "solve": 6e5, "diagnostics": 8e5, "operators": 3e5, "step_operators": 2e5}[kind]
    layout = "box" if "operators" in kind else rng.choice(["box", "dam", "splash"])
    return dict(kind=kind, layout=layout, **block(log(1500, hi), layout))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64)


def lattice(*axes):
    """Points of a grid, first axis fastest, [n, 3]."""
    z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)


def tank(nx, ny, nz):
    """Wall samples (in units of l0) of an open tank [0, nx] x [0, ny] with walls up to nz, and their normals."""
    def span(lo, hi):
        return torch.arange(lo, hi, device="cuda", dtype=torch.float64)

    low, rim = span(-LAYERS + 1, 1), span(0, LAYERS)
    zs = span(1 - LAYERS, nz + 1)
    parts = [(lattice(low, span(1 - LAYERS, ny + LAYERS), zs), (1, 0, 0)),
             (lattice(nx + rim, span(1 - LAYERS, ny + LAYERS), zs), (-1, 0, 0)),
             (lattice(span(1, nx), low, zs), (0, 1, 0)), (lattice(span(1, nx), ny + rim, zs), (0, -1, 0)),
             (lattice(span(1, nx), span(1, ny), low), (0, 0, 1))]
    points = torch.cat([p for p, _ in parts])
    normals = torch.cat([torch.tensor(n, device="cuda", dtype=torch.float64).expand(len(p), 3) for p, n in parts])
    return points, normals.contiguous()


def particles(case, seed, l0=0.005):
    """The particle set of a case: positions, velocities, pressure, labels, walls and the physical parameters."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ar = [torch.arange(k, device="cuda", dtype=torch.float64) + 0.5 for k in (nx, ny, nz)]
    at = lattice(*ar)
    n = len(at)
    surface = at[:, 2] > nz - 1
    near = at[:, 2] > nz - 3
    if case["layout"] != "box":
        surface |= at[:, 0] > nx - 1
        near |= at[:, 0] > nx - 3
    label = torch.where(surface, SURFACE, torch.where(near, NEAR_SURFACE, INNER)).to(torch.int32)
    at = at + 0.1 * (uniform(gen, n, 3) - 0.5)
    size = {"box": (nx, ny, nz + 4), "dam": (2 * nx, ny, nz + 4)}.get(case["layout"], (2 * nx, 2 * ny, max(nx, nz + 14)))
    if case["layout"] in ("splash", "scattered"):
        lift = uniform(gen, n) < 0.05
        u = uniform(gen, n, 3)
        if case["layout"] == "scattered":
            at[:, 0] = torch.where(lift, 0.5 + u[:, 0] * (size[0] - 1), at[:, 0])
            at[:, 1] = torch.where(lift, 0.5 + u[:, 1] * (size[1] - 1), at[:, 1])
        at[:, 2] = torch.where(lift, nz + u[:, 2] * 10, at[:, 2])
        label = torch.where(lift, torch.where(uniform(gen, n) < 0.05, SPLASH, SURFACE), label).to(torch.int32)
    x = at * l0
    length = nx * l0
    vel = 0.1 * torch.stack([torch.sin(2 * math.pi * x[:, 1] / length), 0.5 * torch.cos(2 * math.pi * x[:, 2] / length),
                             0.3 * torch.sin(2 * math.pi * x[:, 0] / length)], 1) + 0.01 * (uniform(gen, n, 3) - 0.5)
    pressure = 9810.0 * torch.clamp((nz - 0.5) * l0 - x[:, 2], min=0.0) * (1 + 0.002 * (uniform(gen, n) - 0.5))
    if case.get("shuffled"):
        p = torch.randperm(n, generator=gen, device="cuda")
        x, vel, pressure, label = x[p], vel[p], pressure[p], label[p]
    wx, wn = tank(*size)
    return dict(x=x.contiguous(), u=vel.contiguous(), p=pressure.contiguous(), label=label.contiguous(), wx=wx * l0, wn=wn,
                l0=l0, dt=1e-4 if case["kind"] == "modules" else 1e-5, n=n, nw=len(wx))


def parameters(s):
    p = abi.default_params()
    p.particle_spacing, p.support_radius, p.near_surface_radius = s["l0"], RE * s["l0"], 1.5 * s["l0"]
    p.grid.cell_size = p.support_radius
    p.density, p.time_step = 1000.0, s["dt"]
    p.gravity[:] = GRAVITY
    origin, dims = grid_of(s)
    for d in range(3):
        p.grid.origin[d], p.grid.dims[d] = origin[d], dims[d]
    return p


def grid_of(s):
    h = RE * s["l0"]
    both = torch.cat([s["x"], s["wx"]])
    lo, hi = both.min(0).values.tolist(), both.max(0).values.tolist()
    return [a - h for a in lo], [int(math.ceil((b + h - (a - h)) / h)) + 1 for a, b in zip(lo, hi)]


def loaded(s, alloc=None):
    """StepBuffers on the device that hold the particle set, and the params of its calls."""
    prm = parameters(s)
    b = buffers.StepBuffers(alloc or buffers.TorchAlloc("cuda"), s["n"], s["nw"], math.prod(prm.grid.dims))
    for d, k in enumerate(XYZ):
        b.fluid[k].copy_(s["x"][:, d])
        b.fluid["v" + k].copy_(s["u"][:, d])
        b.walls[k].copy_(s["wx"][:, d])
        b.walls["normal_" + k].copy_(s["wn"][:, d])
    b.fluid["pressure"].copy_(s["p"])
    b.fluid["surface_type"].copy_(s["label"])
    return b, prm


def context(b, prm, form="plain", sync=True, tuned=False):
    api = pkg.api
    ctx = api.Context(0, precision=abi.PRECISION_MIXED if form == "mixed" else abi.PRECISION_PLAIN, synchronous=sync)
    ctx.reserve(b.n_fluid, b.n_wall, b.n_cells)
    if tuned:
        for k, v in enumerate(TUNED[form]):
            ctx.set_knob(k, v)
    return ctx


def normal(gen, n):
    return torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)


def boxes_of(case):
    """The boxes of a batch: fluid counts spread over the range, every other one a dam break."""
    out = []
    for k in range(case["boxes"]):
        n = case["n_min"] * (case["n_max"] / case["n_min"]) ** ((k + 0.5) / case["boxes"])
        if k % 2:
            a = max(3, round((n / 4) ** (1 / 3)))
            out.append(dict(kind="step", layout="dam", nx=2 * a, ny=a, nz=2 * a + k % 3))
        else:
            a = round(n ** (1 / 3))
            out.append(dict(kind="step", layout="box", nx=a, ny=a, nz=a + k % 3))
    return out


class Together(buffers.TorchAlloc):
    """Device allocation of one box of a study: its arrays one after another in a few large tensors."""

    def fluid(self, b):
        pad = -(-b.n_fluid // 32) * 32
        self.flat = torch.zeros(7 * pad, dtype=torch.float64, device="cuda")
        for k, name in enumerate(FLUID):
            b.fluid[name] = self.flat[k * pad:k * pad + b.n_fluid]


def prepare(case, seed):
    api = pkg.api
    kind = case["kind"]
    if kind == "batch":
        batch, kept = api.Batch(0, streams=8), []
        for k, c in enumerate(boxes_of(case)):
            s = particles(c, 1000 * seed + k)
            alloc = Together("cuda")
            b, prm = loaded(s, alloc)
            own = {name: b.fluid[name] for name in FLUID}
            alloc.fluid(b)
            for name in FLUID:
                b.fluid[name].copy_(own[name])
            ctx = api.Context(0)
            ctx.build_neighbor_lists(b, prm)
            ctx.close()
            batch.add(b, prm)
            kept.append((b, alloc))
        batch.capture(precision=abi.PRECISION_MIXED if case["form"] == "mixed" else abi.PRECISION_PLAIN)
        return dict(kind=kind, batch=batch, boxes=kept)
    s = particles(case, seed)
    b, prm = loaded(s)
    ctx = context(b, prm, case.get("form", "plain"), case.get("sync", True), case.get("tuned", False))
    st = dict(kind=kind, ctx=ctx, b=b, prm=prm)
    ctx.build_neighbor_lists(b, prm)
    if kind == "step":
        st["state"] = b.step_state(prm)
    elif kind == "modules":
        for k in (PRESSURE_B, FLUID_A):
            b.add_moment(k)
    elif kind == "solve":
        ctx.prepare_moments(b, prm, [VELOCITY_A, PRESSURE_A])
        ctx.provision(b, prm)
        ctx.assemble_ppe(b, prm)
        b.moments.clear()  # the program has the system, not what it was made from
    elif kind == "diagnostics":
        n = s["n"]
        names = [k for k, _ in abi.SurfaceDiagnostics._fields_]
        st["out"] = {k: torch.zeros(n, dtype=torch.int32 if "count" in k else torch.float64, device="cuda") for k in names}
        st["diag"] = abi.SurfaceDiagnostics(*(st["out"][k].data_ptr() for k in names))
        st["open"] = (torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda"))
    else:
        prepare_operators(st, s, seed)
    return st


def prepare_operators(st, s, seed):
    b, n, step = st["b"], s["n"], st["kind"] == "step_operators"
    slots = b.nnz_cap  # the matrix arrays are as long as the table's capacity asks, as in a step
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    names = STEP_OPERATOR_OUT if step else OPERATOR_OUT
    kind = abi.StepOperatorOut if step else abi.OperatorOut
    zeros = lambda m, t=torch.float64: torch.zeros(m, dtype=t, device="cuda")  # noqa: E731
    out = {k: zeros(n) for k in names}
    out |= {"ppe_values": zeros(slots), "ppe_row_offsets": zeros(n + 1, torch.int32),
            "ppe_col_indices": zeros(slots, torch.int32)}
    cot = {k: normal(gen, n) for k in names} | {"ppe_values": normal(gen, slots)}
    st |= dict(out=out, cot=cot, n=n, bars=[[zeros(n) for _ in range(3)], zeros(n), [zeros(n) for _ in range(3)]],
               f=b.fluid["pressure"])

    def filled(view, tensors):
        view.count = n
        for k, t in tensors.items():
            setattr(view, k, t.data_ptr())
        return view

    def vector(ts):
        return filled(abi.Vector(), dict(zip(XYZ, ts)))

    st["views"] = [b.fluid_view(), b.walls_view(), b.csr_view("fluid"), b.csr_view("wall"), filled(kind(), out),
                   filled(kind(), cot), vector([b.fluid["v" + k] for k in XYZ]), vector(st["bars"][0]),
                   vector(st["bars"][2])]


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].launch()
        state["batch"].synchronize()
        return [(a.flat, b.fluid["surface_type"], b.fluid_neighbors["indices"], b.ppe["values"], b.ppe["rhs"])
                for b, a in state["boxes"]]
    ctx, b, prm = state["ctx"], state["b"], state["prm"]
    if kind == "step":
        ctx.step(b, prm, state["state"])
        return step_outputs(b)
    if kind == "modules":
        ctx.prepare_moments(b, prm, [VELOCITY_A, PRESSURE_A, PRESSURE_B, FLUID_A])
        ctx.provision(b, prm)
        ctx.assemble_ppe(b, prm)
        ctx.solve_ppe(b)
        ctx.pressure_correction(b, prm, b.ppe["pressure"].data_ptr())
        ctx.build_neighbor_lists(b, prm)
        ctx.classify_surface(b, prm)
        return step_outputs(b) | {"solved": b.ppe["pressure"],
                                  "inverse": [b.moments[k]["inverse_matrices"] for k in range(4)]}
    if kind == "solve":
        report = ctx.solve_ppe(b)
        return {"pressure": b.ppe["pressure"], "iterations": int(report.iterations),
                "residual": float(report.final_residual)}
    if kind == "diagnostics":
        ctx.build_neighbor_lists(b, prm)
        ctx.classify_surface(b, prm, state["diag"])
        ctx.virtual_light(b, prm, state["open"][0].data_ptr(), state["open"][1].data_ptr())
        return {"diagnostics": state["out"], "open": state["open"], "label": b.fluid["surface_type"],
                "fluid_rows": b.fluid_neighbors, "wall_rows": b.wall_neighbors, "cells": b.fluid_cells}
    lib, r = pkg.api._lib, ctypes.byref
    fluid, walls, fn, wn, out, cot, vel, u_bar, x_bar = state["views"]
    p_bar = ctypes.c_void_p(state["bars"][1].data_ptr())
    if kind == "operators":
        f = ctypes.c_void_p(state["f"].data_ptr())
        ctx.check(lib.lsmps_operators_forward(ctx.h, r(fluid), r(fn), r(prm), f, r(vel), r(out), None))
        ctx.check(lib.lsmps_operators_backward(ctx.h, r(fluid), r(fn), r(prm), f, r(vel), r(cot), None, p_bar, r(u_bar),
                                               r(x_bar)))
    else:
        ctx.check(lib.lsmps_step_operators_forward(ctx.h, r(fluid), r(walls), r(fn), r(wn), r(prm), r(out)))
        ctx.check(lib.lsmps_step_operators_backward(ctx.h, r(fluid), r(walls), r(fn), r(wn), r(prm), r(cot), r(u_bar),
                                                    p_bar, r(x_bar)))
    return {"out": state["out"], "bars": state["bars"]}


def step_outputs(b):
    return {"fluid": {k: b.fluid[k] for k in FLUID}, "label": b.fluid["surface_type"],
            "fluid_rows": b.fluid_neighbors, "wall_rows": b.wall_neighbors,
            "matrix": {k: b.ppe[k] for k in ("row_offsets", "col_indices", "values")},
            "rhs": b.ppe["rhs"], "divergence": b.ppe["divergence"], "wall_rhs": b.ppe["pressure_laplacian"],
            "laplacian": b.velocity_laplacian, "provisional": b.temporary_velocity, "gradient": b.pressure_gradient,
            "shift": b.ps_displacement, "smoothed": b.smoothed_velocity}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(c, form=case["form"])) for c in boxes_of(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    e = n * PER_ROW
    table = 4 * e + 4 * n
    if kind in ("step", "modules"):
        # particle state in and out, both neighbour tables in and out (the wall table's entries left out), the PPE rows and
        # every per-particle vector out; the plain form also writes its two inverses
        inverses = {"step": 2 if case.get("form") == "plain" else 0, "modules": 4}[kind]
        bytes_, flops = n * (2 * 60 + 18 * 8) + 2 * table + 12 * (e + n) + 648 * n * inverses, 300 * e
        if kind == "modules":
            bytes_, flops = bytes_ + 100 * 12 * e, flops + 200 * e
        return {"bytes": bytes_, "flops": flops}
    if kind == "solve":  # 100 Arnoldi steps that each read the matrix
        return {"bytes": 100 * 12 * (e + n) + 100 * 16 * n, "flops": 200 * e}
    if kind == "diagnostics":
        return {"bytes": n * (24 + 4 + 80 + 12) + table, "flops": 170 * e}
    return {"bytes": n * (7 + 9 + 7) * 8 + table + 8 * 2 * (e + n) + 4 * (e + n), "flops": 700 * e}


# ---------------------------------------------------------------------------
# What the outputs are in 64 bits, in plain torch: the operators over pair lists, written from their formulas.
# ---------------------------------------------------------------------------
def cells_of(x, origin, dims, h):
    c = torch.floor((x - torch.tensor(origin, device="cuda", dtype=torch.float64)) / h).long()
    return torch.minimum(torch.clamp(c, min=0), torch.tensor(dims, device="cuda") - 1)


class Pairs:
    """Neighbour rows in table order: the 27 cells of a particle z, y, x in turn, the members of a cell by index."""

    def __init__(self, x, src, s, same):
        self.x, self.src, self.re, self.same = x, src, RE * s["l0"], same
        origin, self.dims = grid_of(s)
        self.cell = cells_of(x, origin, self.dims, self.re)
        ids = self.flat(cells_of(src, origin, self.dims, self.re))
        self.sorted = torch.sort(ids, stable=True).indices
        count = torch.bincount(ids, minlength=math.prod(self.dims))
        self.begin, self.count = torch.cumsum(count, 0) - count, count

    def flat(self, c):
        return (c[..., 2] * self.dims[1] + c[..., 1]) * self.dims[0] + c[..., 0]

    def rows(self, lo, hi):
        """(i - lo, j) of the entries of particles lo..hi-1."""
        k = torch.arange(-1, 2, device="cuda")
        dz, dy, dx = (a.reshape(-1) for a in torch.meshgrid(k, k, k, indexing="ij"))
        near = self.cell[lo:hi, None, :] + torch.stack([dx, dy, dz], 1)
        inside = ((near >= 0) & (near < torch.tensor(self.dims, device="cuda"))).all(2)
        flat = torch.where(inside, self.flat(near), 0)
        many = torch.where(inside, self.count[flat], 0).reshape(-1)
        total = torch.cumsum(many, 0)
        at = torch.arange(int(total[-1]), device="cuda") - torch.repeat_interleave(total - many, many)
        j = self.sorted[torch.repeat_interleave(self.begin[flat].reshape(-1), many) + at]
        i = torch.repeat_interleave(torch.arange(hi - lo, device="cuda").repeat_interleave(27), many)
        ok = ((self.src[j] - self.x[lo + i]) ** 2).sum(1) < self.re ** 2
        if self.same:
            ok &= j != lo + i
        return i[ok], j[ok]


def basis(v):
    a, b, c = v.unbind(1)
    return torch.stack([a, b, c, a * a, b * b, c * c, a * b, b * c, c * a], 1)


def neumann(v, n):
    a, b, c = v.unbind(1)
    p, q, r = n.unbind(1)
    return torch.stack([p, q, r, 2 * a * p, 2 * b * q, 2 * c * r, b * p + a * q, c * q + b * r, a * r + c * p], 1)


def weight(d, re):
    return torch.clamp(1 - d / re, min=0.0)


def summed(n, i, v):
    return torch.zeros((n, *v.shape[1:]), dtype=v.dtype, device=v.device).index_add(0, i, v)


def inverse(m, lam=1e-8):
    k = m.shape[1]
    tr = torch.diagonal(m, dim1=1, dim2=2).sum(1)
    reg = lam * torch.where(tr > 0, tr / k, torch.ones_like(tr))
    return torch.linalg.inv(m + reg[:, None, None] * torch.eye(k, dtype=m.dtype, device=m.device))


def outer(n, i, w, b):
    return summed(n, i, (w[:, None] * b)[:, :, None] * b[:, None, :])


CHUNK = 12000


def exact_step(s, solve=False, kinds=False, system=False):
    """The outputs of one step of the particle set `s`; `system`: the assembled matrix alone."""
    x, u, wx, wn, n, re, dt = s["x"], s["u"], s["wx"], s["wn"], s["n"], RE * s["l0"], s["dt"]
    g = torch.tensor(GRAVITY, device="cuda", dtype=torch.float64)
    rho, nu = 1000.0, 1e-6
    splash, dirichlet = s["label"] == SPLASH, s["label"] >= SURFACE
    fluid, wall = Pairs(x, x, s, True), Pairs(x, wx, s, False)
    press = torch.clamp(s["p"], min=0.0)
    lap, grows, lrows = (torch.empty(n, k, dtype=torch.float64, device="cuda") for k in (3, 27, 9))
    prows = torch.empty(n, 3, 9, dtype=torch.float64, device="cuda")
    count = torch.empty(n, dtype=torch.int64, device="cuda")
    inverses = [[] for _ in range(4)]
    spans = [(a, min(n, a + CHUNK)) for a in range(0, n, CHUNK)]
    for lo, hi in spans:
        m = hi - lo
        i, j = fluid.rows(lo, hi)
        k, q = wall.rows(lo, hi)
        count[lo:hi] = torch.bincount(i, minlength=m)
        d, dw = x[j] - x[lo + i], wx[q] - x[lo + k]
        w, ww = weight(d.norm(dim=1), re), weight(dw.norm(dim=1), re)
        b, bw, qw = basis(d / re), basis(dw / re), neumann(dw / re, wn[q])
        base = outer(m, i, w, b)
        xv, xp = inverse(base + outer(m, k, ww, bw)), inverse(base + outer(m, k, ww, qw))
        if kinds:
            one = torch.ones(len(i), 1, dtype=torch.float64, device="cuda")
            full = outer(m, i, w, torch.cat([one, b], 1)) + outer(m, k, ww, torch.cat([torch.zeros_like(qw[:, :1]), qw], 1))
            for store, v in zip(inverses, (xv, xp, inverse(full), inverse(base))):
                store.append(v.reshape(-1))
        rhs = summed(m, i, (w[:, None] * b)[:, :, None] * (u[j] - u[lo + i])[:, None, :])
        rhs += summed(m, k, (ww[:, None] * bw)[:, :, None] * (-u[lo + k])[:, None, :])
        lap[lo:hi] = 2 / re ** 2 * torch.einsum("nrc,ncd->nd", xv[:, 3:6, :], rhs)
        grows[lo:hi], lrows[lo:hi], prows[lo:hi] = xv[:, :3, :].reshape(m, 27), xp[:, 3:6, :].sum(1), xp[:, :3, :]
    us = u + dt * (torch.where(splash, 0.0, nu)[:, None] * lap + g)
    uw = (dt * g).expand(len(wx), 3)
    start = torch.cumsum(count, 0) - count + torch.arange(n, device="cuda")
    entries = int(count.sum())
    values = torch.zeros(n + 256 * n, dtype=torch.float64, device="cuda")
    columns = torch.zeros(n + entries, dtype=torch.int64, device="cuda") if solve or system else None
    div, wall_rhs = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
    for lo, hi in spans:
        m = hi - lo
        i, j = fluid.rows(lo, hi)
        k, q = wall.rows(lo, hi)
        d, dw = x[j] - x[lo + i], wx[q] - x[lo + k]
        w, ww = weight(d.norm(dim=1), re), weight(dw.norm(dim=1), re)
        b, bw, qw = basis(d / re), basis(dw / re), neumann(dw / re, wn[q])
        G, L = grows[lo:hi].reshape(m, 3, 9), lrows[lo:hi]
        acc = summed(m, i, w * (torch.einsum("nrc,nc->nr", G[i], b) * (us[j] - us[lo + i])).sum(1))
        acc += summed(m, k, ww * (torch.einsum("nrc,nc->nr", G[k], bw) * (uw[q] - us[lo + k])).sum(1))
        keep = ~dirichlet[lo:hi]
        a = torch.where(keep[i], 2 / (re ** 2 * rho) * w * (L[i] * b).sum(1), 0.0)
        first = torch.searchsorted(i, torch.arange(m, device="cuda"))
        slot = start[lo + i] + 1 + torch.arange(len(i), device="cuda") - first[i]
        values[slot] = a
        values[start[lo:hi]] = torch.where(keep, -summed(m, i, a), 1.0)
        if columns is not None:
            columns[slot], columns[start[lo:hi]] = j, torch.arange(lo, hi, device="cuda")
        div[lo:hi] = torch.where(keep, acc / re, 0.0)
        wall_rhs[lo:hi] = torch.where(keep, summed(m, k, 2 * ww * (wn[q] @ g) * (L[k] * qw).sum(1) / re), 0.0)
    rhs = torch.where(dirichlet, 0.0, div / dt - wall_rhs)
    if solve or system:
        edges = torch.cat([start, torch.tensor([n + entries], device="cuda")])
        matrix = torch.sparse_csr_tensor(edges, columns, values[:n + entries], size=(n, n))
        solved, its, res = gmres(matrix, rhs)
        if system:
            return solved, its, res
        press = solved
    xn, un = torch.empty_like(x), torch.empty_like(u)
    grad, shift = torch.empty_like(x), torch.empty_like(x)
    dmin, smax, clear = 0.85 * s["l0"], 0.2 * s["l0"], 0.25 * s["l0"]
    for lo, hi in spans:
        m = hi - lo
        i, j = fluid.rows(lo, hi)
        k, q = wall.rows(lo, hi)
        d, dw = x[j] - x[lo + i], wx[q] - x[lo + k]
        r, rw = d.norm(dim=1), dw.norm(dim=1)
        w, ww = weight(r, re) * (r > 0), weight(rw, re) * (rw > 0)
        acc = summed(m, i, (w * (press[j] - press[lo + i]))[:, None] * basis(d / re))
        acc += summed(m, k, (ww * re * rho * (wn[q] @ g))[:, None] * neumann(dw / re, wn[q]))
        live = ~splash[lo:hi, None]
        gr = torch.where(live, torch.einsum("nrc,nc->nr", prows[lo:hi], acc) / re, 0.0)
        close, closew = (r > 0) & (r < dmin), (rw > 0) & (rw < dmin)
        e = -d[close] / r[close, None]
        sh = summed(m, i[close], 0.05 * (dmin - r[close])[:, None] * e)
        sh += summed(m, k[closew], 0.05 * (dmin - rw[closew])[:, None] * wn[q[closew]])
        nn = summed(m, i[close], e)
        size = nn.norm(dim=1, keepdim=True)
        nn = torch.where(size > 0, nn / torch.where(size > 0, size, 1.0), 0.0)
        sh = torch.where(dirichlet[lo:hi, None], sh - (sh * nn).sum(1, keepdim=True) * nn, sh)
        size = sh.norm(dim=1, keepdim=True)
        sh = torch.where(size > smax, sh * smax / torch.where(size > 0, size, 1.0), sh) * live
        grad[lo:hi], shift[lo:hi] = gr, sh
        v = us[lo:hi] - dt / rho * gr
        at = x[lo:hi] + 0.5 * dt * (u[lo:hi] + v) + sh
        first = torch.searchsorted(k, torch.arange(m, device="cuda"))
        many = torch.bincount(k, minlength=m)
        for c in range(int(many.max()) if len(k) else 0):  # wall by wall, in row order
            has = many > c
            wq = q[torch.where(has, first + c, 0)]
            sd = ((at - wx[wq]) * wn[wq]).sum(1)
            hit = (has & (sd < clear))[:, None]
            at = torch.where(hit, at + (clear - sd)[:, None] * wn[wq], at)
            nv = (v * wn[wq]).sum(1, keepdim=True)
            v = torch.where(hit & (nv < 0), v - nv * wn[wq], v)
        xn[lo:hi], un[lo:hi] = at, v
    smooth = torch.empty_like(u)
    for lo, hi in spans:
        i, j = fluid.rows(lo, hi)
        r = (xn[j] - xn[lo + i]).norm(dim=1)
        w = weight(r, re) * (r > 0) * ~splash[j]
        total = summed(hi - lo, i, w)
        mean = summed(hi - lo, i, w[:, None] * un[j]) / torch.where(total > 0, total, 1.0)[:, None]
        moved = (~splash[lo:hi] & (total > 0))[:, None]
        smooth[lo:hi] = torch.where(moved, 0.9 * un[lo:hi] + 0.1 * mean, un[lo:hi])
    columns3 = lambda v: {k: v[:, c].contiguous() for c, k in enumerate(XYZ)}  # noqa: E731
    out = {"fluid": columns3(xn) | {"v" + k: t for k, t in columns3(smooth).items()} | {"pressure": press}, "label": None,
           "fluid_rows": None, "wall_rows": None, "matrix": {"row_offsets": None, "col_indices": None, "values": values},
           "rhs": rhs, "divergence": div, "wall_rhs": wall_rhs, "laplacian": columns3(lap),
           "provisional": {"v" + k: t for k, t in columns3(us).items()}, "gradient": columns3(grad), "shift": columns3(shift),
           "smoothed": columns3(smooth)}
    if kinds:
        out |= {"solved": press, "inverse": [torch.cat(v) for v in inverses]}
    return out


def gmres(a, b, restart=20, most=100, tolerance=1e-6):
    """Restarted GMRES from zero, negative values of the result clamped; also the iterations and the last residual."""
    x = torch.zeros_like(b)
    r = b.clone()
    beta = first = float(r.norm())
    its = 0
    while beta > tolerance * first and its < most:
        v, h = [r / beta], np.zeros((restart + 1, restart))
        for j in range(restart):
            w = a @ v[j]
            basis_ = torch.stack(v)
            for _ in range(2):
                c = basis_ @ w
                w = w - c @ basis_
                h[:j + 1, j] += c.cpu().numpy()
            h[j + 1, j] = float(w.norm())
            its += 1
            e1 = np.zeros(j + 2)
            e1[0] = beta
            y = np.linalg.lstsq(h[:j + 2, :j + 1], e1, rcond=None)[0]
            if np.linalg.norm(e1 - h[:j + 2, :j + 1] @ y) <= tolerance * first or its == most:
                break
            v.append(w / h[j + 1, j])
        x = x + torch.tensor(y, device="cuda") @ torch.stack(v[:len(y)])
        r = b - a @ x
        beta = float(r.norm())
    return torch.clamp(x, min=0.0), its, beta


def exact_operators(case, s, seed):
    """Forward outputs and gradients by autograd, a block of particles at a time (a row's terms depend on its own row only)."""
    step = case["kind"] == "step_operators"
    n, re, dt, rho = s["n"], RE * s["l0"], s["dt"], 1000.0
    g = torch.tensor(GRAVITY, device="cuda", dtype=torch.float64)
    x, u, p, wx, wn = s["x"], s["u"], s["p"], s["wx"], s["wn"]
    fluid, wall = Pairs(x, x, s, True), Pairs(x, wx, s, False)
    spans = [(a, min(n, a + 4000)) for a in range(0, n, 4000)]
    count = torch.cat([torch.bincount(fluid.rows(lo, hi)[0], minlength=hi - lo) for lo, hi in spans])
    start = torch.cumsum(count, 0) - count + torch.arange(n, device="cuda")
    slots = n + 256 * n
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    names = STEP_OPERATOR_OUT if step else OPERATOR_OUT
    cot = {k: normal(gen, n) for k in names} | {"ppe_values": normal(gen, slots)}
    out = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k in names}
    out |= {"ppe_values": torch.zeros(slots, dtype=torch.float64, device="cuda"), "ppe_row_offsets": None,
            "ppe_col_indices": None}
    bars = [torch.zeros_like(u), torch.zeros_like(p), torch.zeros_like(x)]
    dirichlet, splash = (s["label"] >= SURFACE, s["label"] == SPLASH) if step else (torch.zeros(n, dtype=torch.bool, device="cuda"),) * 2
    for lo, hi in spans:
        m = hi - lo
        i, j = fluid.rows(lo, hi)
        xr, ur, pr = (t.detach().clone().requires_grad_(True) for t in (x, u, p))
        d = xr[j] - xr[lo + i]
        w = weight(d.norm(dim=1), re)
        b = basis(d / re)
        base = outer(m, i, w, b)
        ru = summed(m, i, (w[:, None] * b)[:, :, None] * (ur[j] - ur[lo + i])[:, None, :])
        rp = summed(m, i, (w * (pr[j] - pr[lo + i]))[:, None] * b)
        mv, mp = base, base
        if step:
            k, q = wall.rows(lo, hi)
            dw = wx[q] - xr[lo + k]
            ww = weight(dw.norm(dim=1), re)
            bw, qw = basis(dw / re), neumann(dw / re, wn[q])
            mv, mp = base + outer(m, k, ww, bw), base + outer(m, k, ww, qw)
            ru = ru + summed(m, k, (ww[:, None] * bw)[:, :, None] * (-ur[lo + k])[:, None, :])
            rp = rp + summed(m, k, (ww * re * rho * (wn[q] @ g))[:, None] * qw)
        xv, xp = inverse(mv), inverse(mp)
        yu, yp = torch.einsum("nrc,ncd->nrd", xv, ru), torch.einsum("nrc,nc->nr", xp, rp)
        keep, live = ~dirichlet[lo:hi], ~splash[lo:hi]
        div = (yu[:, 0, 0] + yu[:, 1, 1] + yu[:, 2, 2]) / re * keep
        L = xp[:, 3:6].sum(1)
        a = 2 / (re ** 2 * rho) * w * (L[i] * b).sum(1) * keep[i]
        got = {"divergence": div}
        for c, name in enumerate(XYZ):
            got["grad_" + name] = yp[:, c] / re * live
        if step:
            wall_rhs = summed(m, k, 2 * ww * (wn[q] @ g) * (L[k] * qw).sum(1) / re) * keep
            got |= {"wall_rhs": wall_rhs, "ppe_rhs": (div / dt - wall_rhs) * keep}
            got |= {"lap_" + name: 2 / re ** 2 * yu[:, 3:6, c].sum(1) for c, name in enumerate(XYZ)}
        else:
            got |= {"laplacian": 2 / re ** 2 * yp[:, 3:6].sum(1), "ppe_rhs": div / dt}
        first = torch.searchsorted(i, torch.arange(m, device="cuda"))
        slot = start[lo + i] + 1 + torch.arange(len(i), device="cuda") - first[i]
        diag = torch.where(keep, -summed(m, i, a), 1.0)
        loss = (cot["ppe_values"][slot] * a).sum() + (cot["ppe_values"][start[lo:hi]] * diag).sum()
        for name, v in got.items():
            loss = loss + (cot[name][lo:hi] * v).sum()
            out[name][lo:hi] = v.detach()
        out["ppe_values"][slot], out["ppe_values"][start[lo:hi]] = a.detach(), diag.detach()
        for store, v in zip(bars, torch.autograd.grad(loss, (ur, pr, xr))):
            store += v
    return {"out": out, "bars": [list(bars[0].unbind(1)), bars[1], list(bars[2].unbind(1))]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for k, c in enumerate(boxes_of(case)):
            s = particles(c, 1000 * seed + k)
            e = exact_step(s)
            pad = -(-s["n"] // 32) * 32
            flat = torch.zeros(7 * pad, dtype=torch.float64, device="cuda")
            for f, name in enumerate(FLUID):
                flat[f * pad:f * pad + s["n"]] = e["fluid"][name]
            out.append((flat, None, None, e["matrix"]["values"], e["rhs"]))
        return out
    s = particles(case, seed)
    if kind == "step":
        return exact_step(s)
    if kind == "modules":
        return exact_step(s, solve=True, kinds=True)
    if kind == "solve":
        solved, _, residual = exact_step(s, system=True)
        return {"pressure": solved, "iterations": None, "residual": residual}
    if kind == "diagnostics":  # counts and thresholds of them: whole values, or sums in the reference's own order
        return None
    return exact_operators(case, s, seed)
