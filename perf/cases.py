"""Performance cases of the framework, through its public entry points.

Each case is a solve that a user's program has the framework do: grids are
made and filled once, stencil functions are mapped once, and a pass is one
PSStencilRun (or one batch, or one burst of served requests) with the
reduction or the residuals that such a program reads afterwards. The grids
stay on the GPU between passes, so a pass continues from the state that the
one before it left; outputs are the grids themselves, seen as tensors.

`bytes` of work() counts each input read once and each output written once
per pass, not once per time step: what a pass of any number of steps cannot
do without. `flops` counts every multiply and add of every step.
"""
import functools
import os
import random
import tempfile
import types

import numpy as np
import torch

import physis_b200 as ps
from physis_b200 import dsl
from physis_b200.workloads import DIFFUSION7_DSL, box27_terms

# Coefficients ce, cw, cn, cs, ct, cb, cc of the diffusion benchmark.
COEF7 = (0.1, 0.1, 0.1, 0.1, 0.1, 0.1, 0.4)
OMEGA = 0.8
NEIGHBOURS6 = ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))


def listed():
    return [
        # The smallest benchmark configuration: a 64^3 diffusion solve of 100
        # steps and its PSReduce sum. Everything stays in L2; launches count.
        dict(name="diffusion_64", kind="diffusion", nx=64, ny=64, nz=64, steps=100, dtype="f32",
             periodic=False, fma=False, reduce=True),
        # The headline configuration: single precision, exact arithmetic (the
        # default), grids far larger than L2.
        dict(name="diffusion_512", kind="diffusion", nx=512, ny=512, nz=512, steps=20,
             dtype="f32", periodic=False, fma=False, reduce=False),
        # The double-precision benchmark configuration, with the sum that
        # checks conservation.
        dict(name="diffusion_256_f64", kind="diffusion", nx=256, ny=256, nz=256, steps=40,
             dtype="f64", periodic=False, fma=False, reduce=True),
        # A periodic domain of no particular size in the contracted (FMA)
        # arithmetic that the headline benchmark times.
        dict(name="periodic_fma", kind="diffusion", nx=250, ny=187, nz=131, steps=50,
             dtype="f32", periodic=True, fma=True, reduce=False),
        # The Himeno benchmark's grid, with the residual of every sweep.
        dict(name="himeno_257", kind="himeno", nx=257, ny=257, nz=513, steps=20),
        # Himeno's small grid: L2-resident, short sweeps.
        dict(name="himeno_65", kind="himeno", nx=65, ny=65, nz=129, steps=40),
        # A user stencil as a table of terms: the 27-point box average.
        dict(name="box27_512", kind="box27", nx=512, ny=512, nz=512, steps=4, dtype="f32",
             fma=False),
        # Red-black Gauss-Seidel relaxation of a Poisson problem, in place.
        dict(name="redblack_256", kind="redblack", nx=256, ny=256, nz=256, steps=10,
             dtype="f32"),
        # A two-dimensional heat equation on a large odd-sized plate.
        dict(name="heat2d_4001", kind="heat2d", nx=4001, ny=2003, steps=20, dtype="f32"),
        # The diffusion kernel as a user writes it in the C DSL (neighbours
        # under face tests), compiled by the front end.
        dict(name="dsl_diffusion", kind="dsl", nx=300, ny=260, nz=220, steps=20),
        # Many small independent solves of uneven sizes in one batch: half
        # periodic diffusion, half Himeno.
        dict(name="batch_24", kind="batch", members=24, lo=32, hi=160, min_steps=20,
             max_steps=60, mix=7),
        # A burst of requests to the solve server, each run until it
        # converges or has done its steps.
        dict(name="serve_16", kind="serve", requests=16, lo=32, hi=160, steps=150, mix=11),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _steps(rng, points, most, lo=2, hi=100):
    """An even number of steps whose point updates stay within `most`."""
    n = _log_int(rng, lo, hi)
    return max(2, min(n, int(most // points)) // 2 * 2)


def draw(rng):
    kind = rng.choice(["diffusion", "diffusion", "diffusion", "diffusion", "himeno", "himeno",
                       "box27", "redblack", "heat2d", "dsl", "batch", "serve"])
    if kind == "heat2d":
        nx, ny = _log_int(rng, 64, 4096), _log_int(rng, 64, 4096)
        return dict(kind=kind, nx=nx, ny=ny, steps=_steps(rng, nx * ny, 3e8, hi=40),
                    dtype=rng.choice(["f32", "f64"]))
    if kind == "batch":
        lo = _log_int(rng, 24, 64)
        return dict(kind=kind, members=rng.randint(8, 30), lo=lo, hi=_log_int(rng, lo, 160),
                    min_steps=20, max_steps=rng.randint(20, 60), mix=rng.randint(0, 9999))
    if kind == "serve":
        lo = _log_int(rng, 24, 64)
        return dict(kind=kind, requests=rng.randint(4, 16), lo=lo, hi=_log_int(rng, lo, 160),
                    steps=rng.randint(3, 15) * 10, mix=rng.randint(0, 9999))
    hi = {"diffusion": 512, "himeno": 400, "box27": 512, "redblack": 256, "dsl": 320}[kind]
    nx, ny, nz = (_log_int(rng, 32, hi) for _ in range(3))
    points = nx * ny * nz
    if kind == "himeno":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, points, 6e8, hi=60))
    if kind == "box27":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, points, 5e8, hi=40),
                    dtype=rng.choice(["f32", "f32", "f64"]), fma=rng.random() < 0.3)
    if kind == "redblack":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, points, 1.5e8, hi=20),
                    dtype=rng.choice(["f32", "f64"]))
    if kind == "dsl":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_steps(rng, points, 5e8, hi=40))
    dtype = rng.choice(["f32", "f32", "f32", "f64"])
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype,
                steps=_steps(rng, points, 2.6e9 if dtype == "f32" else 1e9),
                periodic=rng.random() < 0.35, fma=rng.random() < 0.3,
                reduce=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
TORCH = {"f32": torch.float32, "f64": torch.float64}
GRID = {"f32": ps.PS_FLOAT, "f64": ps.PS_DOUBLE}


def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 7919 * k + 1)


def _uniform(shape, lo, hi, dtype, g):
    return torch.rand(shape, generator=g, device="cuda", dtype=dtype) * (hi - lo) + lo


def _profile(shape, dtype, g):
    """Cosine-product profile plus noise: the benchmark's initial field."""
    f = torch.ones((), device="cuda", dtype=torch.float64)
    for k, n in enumerate(shape):
        x = torch.arange(n, device="cuda", dtype=torch.float64)
        v = 1 - torch.cos(2 * torch.pi * x / n)
        f = f * (0.5 * v).reshape([n if i == k else 1 for i in range(len(shape))])
    return f.to(dtype) + _uniform(shape, 0.0, 1e-3, dtype, g)


def _himeno_fields(shape, g):
    """p and the twelve coefficient fields a0-a3, b0-b2, c0-c2, bnd, wrk1."""
    u = lambda lo, hi: _uniform(shape, lo, hi, torch.float32, g)  # noqa: E731
    coef = [u(0.9, 1.1) for _ in range(3)] + [u(0.95 / 6, 1.05 / 6)]
    coef += [u(-0.01, 0.01) for _ in range(3)] + [u(0.9, 1.1) for _ in range(3)]
    bnd = torch.zeros(shape, device="cuda")
    bnd[1:-1, 1:-1, 1:-1] = 1
    z = torch.arange(shape[0], device="cuda", dtype=torch.float32) / (shape[0] - 1)
    p = (z * z)[:, None, None].expand(shape).contiguous()
    return p, coef + [bnd, torch.zeros(shape, device="cuda")]


def _shape(case):
    return (case["nz"], case["ny"], case["nx"]) if "nz" in case else (case["ny"], case["nx"])


def _members(case):
    """(is Himeno, extents, steps) of each member of a batch case."""
    r = random.Random(case["mix"])
    return [(i % 2 == 1, tuple(_log_int(r, case["lo"], case["hi"]) for _ in range(3)),
             r.randint(case["min_steps"], case["max_steps"])) for i in range(case["members"])]


def _requests(case):
    """(is Himeno, cube side) of each request of a served case."""
    r = random.Random(case["mix"])
    return [(r.random() >= 0.6, _log_int(r, case["lo"], case["hi"]))
            for _ in range(case["requests"])]


# ---------------------------------------------------------------------------
# What a user's program keeps: grids, maps, batches, servers
# ---------------------------------------------------------------------------
class Owned:
    """One grid, freed with the last state or output tensor that uses it."""

    def __init__(self, type_, dims):
        self.grid = ps.grid_new(type_, dims)

    def tensor(self):
        """The grid's device memory as a tensor (which keeps the grid)."""
        g, lay = self.grid, self.grid.layout()
        e = np.dtype(g.dtype).itemsize
        strides = (lay["stride_z"] * e, lay["stride_y"] * e, e)[3 - len(g.dims):]
        p0 = ps.PSGridStruct.from_address(g.ptr.value).p0
        memory = types.SimpleNamespace(owner=self)
        memory.__cuda_array_interface__ = {"shape": g.shape, "strides": strides, "version": 2,
                                           "typestr": np.dtype(g.dtype).str, "data": (p0, False)}
        return torch.as_tensor(memory, device="cuda")

    def __del__(self):
        if hasattr(self, "grid"):
            ps.PSGridFree(self.grid)


class State:
    """The grids and handles of one prepared case."""

    def __init__(self, case):
        self.case, self.owned, self.maps, self.outputs = case, [], [], []
        self.batch = self.server = None
        self.requests = []

    def grid(self, type_, dims, values=None):
        o = Owned(type_, dims)
        self.owned.append(o)
        if values is not None:
            ps.PSGridCopyin(o.grid, values.cpu().numpy())
        return o.grid

    def __del__(self):
        if self.batch is not None:
            self.batch.free()
        if self.server is not None:
            self.server.destroy()


@functools.lru_cache(maxsize=None)
def _table(form, dtype):
    """A registered term table (once per process, as a user's program does)."""
    t = GRID[dtype]
    if form == "box27":
        return ps.GenericStencil(3, [(t, (0, 1, 2))] * 2, 1, t, box27_terms(t)).kernel_id
    if form == "redblack":
        sixth = float(np.float32(1.0 / 6.0))
        terms = [(ps.const(sixth), ps.get(0, o)) for o in NEIGHBOURS6]
        terms.append((ps.const(sixth), ps.get(1)))
        return ps.GenericStencil(3, [(t, (0, 1, 2))] * 2, 0, t, terms).kernel_id
    c = float(np.float32(0.2))
    terms = [(ps.const(c), ps.get(0))]
    terms += [(ps.const(c), ps.get(0, o)) for o in ((1, 0), (-1, 0), (0, 1), (0, -1))]
    return ps.GenericStencil(2, [(t, (0, 1))] * 2, 1, t, terms).kernel_id


@functools.lru_cache(maxsize=None)
def _dsl_kernel():
    cache = os.path.join(tempfile.gettempdir(), "physis_b200_perf_dsl_%d" % os.getuid())
    return dsl.compile_stencils(DIFFUSION7_DSL, cache)["diffusion7"].kernel_id


def prepare(case, seed):
    ps.PSInit()
    ps.set_fp_mode(ps.FP_FMA if case.get("fma") else ps.FP_EXACT)
    s = State(case)
    kind, g = case["kind"], _gen(seed)
    if kind == "batch":
        s.batch = ps.Batch()
        for i, (him, dims, steps) in enumerate(_members(case)):
            shape, gi = tuple(reversed(dims)), _gen(seed, i + 1)
            if him:
                p, coef = _himeno_fields(shape, gi)
                gs = [s.grid(ps.PS_FLOAT, dims, v) for v in [p, p] + coef]
                s.batch.add(ps.HIMENO19, gs, [OMEGA], steps)
            else:
                gs = [s.grid(ps.PS_FLOAT, dims, _profile(shape, torch.float32, gi)),
                      s.grid(ps.PS_FLOAT, dims)]
                s.batch.add(ps.DIFFUSION7_PERIODIC, gs, COEF7, steps)
            s.outputs.append(s.owned[-len(gs) + steps % 2].tensor())
        return s
    if kind == "serve":
        s.server = ps.Server(8 << 30)
        for i, (him, side) in enumerate(_requests(case)):
            shape = (side,) * 3
            out = torch.empty(shape, pin_memory=True).numpy()
            init = None if him else _profile(shape, torch.float32, _gen(seed, i + 1)).cpu()
            s.requests.append((him, side, None if him else init.pin_memory().numpy(), out,
                               1000 * int(seed) + i))
        return s
    dims, shape = tuple(reversed(_shape(case))), _shape(case)
    whole = [v for n in dims for v in (0, n)]
    inside = [v for n in dims for v in (1, n - 1)]
    if kind == "diffusion":
        t = GRID[case["dtype"]]
        a, b = s.grid(t, dims, _profile(shape, TORCH[case["dtype"]], g)), s.grid(t, dims)
        k = ps.DIFFUSION7_PERIODIC if case["periodic"] else ps.DIFFUSION7
        d = ps.PSDomain3DNew(*whole)
        s.maps = [ps.PSStencilMap(k, d, a, b, *COEF7), ps.PSStencilMap(k, d, b, a, *COEF7)]
    elif kind == "himeno":
        p, coef = _himeno_fields(shape, g)
        gs = [s.grid(ps.PS_FLOAT, dims, v) for v in [p, p] + coef]
        d = ps.PSDomain3DNew(*inside)
        s.maps = [ps.PSStencilMap(ps.HIMENO19, d, *gs, OMEGA),
                  ps.PSStencilMap(ps.HIMENO19, d, gs[1], gs[0], *gs[2:], OMEGA)]
        for m in s.maps:
            ps.himeno_residual_enable(m, case["steps"] // 2)
    elif kind == "dsl":
        u = _profile(shape, torch.float32, g)
        a, b = s.grid(ps.PS_FLOAT, dims, u), s.grid(ps.PS_FLOAT, dims)
        d, k = ps.PSDomain3DNew(*whole), _dsl_kernel()
        s.maps = [ps.PSStencilMap(k, d, a, b, *COEF7), ps.PSStencilMap(k, d, b, a, *COEF7)]
    elif kind == "redblack":
        t, dt = GRID[case["dtype"]], TORCH[case["dtype"]]
        a = s.grid(t, dims, _profile(shape, dt, g))
        b = s.grid(t, dims, _uniform(shape, -1e-2, 1e-2, dt, g))
        s.maps = [ps.PSStencilMapRedBlack(_table(kind, case["dtype"]),
                                          ps.PSDomain3DNew(*inside), a, b)]
    else:  # box27, heat2d: the rim keeps its values in both grids
        t = GRID[case["dtype"]]
        u = _profile(shape, TORCH[case["dtype"]], g)
        a, b = s.grid(t, dims, u), s.grid(t, dims, u)
        d = (ps.PSDomain2DNew if kind == "heat2d" else ps.PSDomain3DNew)(*inside)
        k = _table(kind, case["dtype"])
        s.maps = [ps.PSStencilMap(k, d, a, b), ps.PSStencilMap(k, d, b, a)]
    s.outputs = [o.tensor() for o in s.owned[:1 if kind == "redblack" else 2]]
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "batch":
        s.batch.run()
        return s.outputs
    if kind == "serve":
        ids = [s.server.submit(ps.HIMENO19 if him else ps.DIFFUSION7, (side,) * 3,
                               [OMEGA] if him else COEF7, case["steps"], tol=1e-5,
                               check_every=10, init=init, out=out, seed=seed)
               for him, side, init, out, seed in s.requests]
        done = [s.server.wait(i) for i in ids]
        return {"steps": [r["steps_done"] for r in done], "u": [q[3] for q in s.requests]}
    if kind == "redblack":
        ps.PSStencilRun(*s.maps, case["steps"])
        return s.outputs
    ps.PSStencilRun(*s.maps, case["steps"] // 2)
    if kind == "himeno":
        return s.outputs + [np.array(ps.himeno_residual_history(m, case["steps"] // 2))
                            for m in s.maps]
    if case.get("reduce"):
        return s.outputs + [ps.PSReduce(ps.PS_SUM, s.owned[0].grid)]
    return s.outputs


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _shift(u, axis, by, periodic):
    """u at the neighbour `by` along axis (clamped at the faces, or wrapped)."""
    if periodic:
        return u.roll(-by, axis)
    n = u.shape[axis]
    inner, edge = u.narrow(axis, max(by, 0), n - 1), u.narrow(axis, n - 1 if by > 0 else 0, 1)
    return torch.cat([inner, edge] if by > 0 else [edge, inner], axis)


def _diffuse(u, steps, coef, periodic):
    """The fields after the last step and after the one before it."""
    ce, cw, cn, cs, ct, cb, cc = coef
    last = u
    for _ in range(steps):
        v = cc * u
        for c, axis, by in ((cw, 2, -1), (ce, 2, 1), (cs, 1, 1), (cn, 1, -1), (cb, 0, -1),
                            (ct, 0, 1)):
            v += c * _shift(u, axis, by, periodic)
        last, u = u, v
    return u, last


def _jacobi(p, coef, sweeps):
    """Himeno sweeps: the last two fields and the residual of each sweep."""
    a0, a1, a2, a3, b0, b1, b2, c0, c1, c2, bnd, wrk1 = [
        c.double()[1:-1, 1:-1, 1:-1] for c in coef]
    last, gosa = p, []
    n = p.shape

    def at(dx, dy, dz):
        return p[1 + dz:n[0] - 1 + dz, 1 + dy:n[1] - 1 + dy, 1 + dx:n[2] - 1 + dx]

    for _ in range(sweeps):
        s = a0 * at(0, 0, 1) + a1 * at(0, 1, 0) + a2 * at(1, 0, 0)
        s += b0 * (at(0, 1, 1) - at(0, -1, 1) - at(0, 1, -1) + at(0, -1, -1))
        s += b1 * (at(1, 1, 0) - at(1, -1, 0) - at(-1, 1, 0) + at(-1, -1, 0))
        s += b2 * (at(1, 0, 1) - at(-1, 0, 1) - at(1, 0, -1) + at(-1, 0, -1))
        s += c0 * at(0, 0, -1) + c1 * at(0, -1, 0) + c2 * at(-1, 0, 0) + wrk1
        ss = (s * a3 - at(0, 0, 0)) * bnd
        gosa.append(float((ss * ss).sum()))
        q = p.clone()
        q[1:-1, 1:-1, 1:-1] += OMEGA * ss
        last, p = p, q
    return p, last, gosa


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "serve":  # stops where the residual in its own precision says so
        return None
    if kind == "batch":
        out = []
        for i, (him, dims, steps) in enumerate(_members(case)):
            shape, gi = tuple(reversed(dims)), _gen(seed, i + 1)
            if him:
                p, coef = _himeno_fields(shape, gi)
                out.append(_jacobi(p.double(), coef, steps)[0])
            else:
                out.append(_diffuse(_profile(shape, torch.float32, gi).double(), steps,
                                    np.float64(np.float32(COEF7)), True)[0])
        return out
    shape = _shape(case)
    if kind == "himeno":
        p, coef = _himeno_fields(shape, g)
        p, last, gosa = _jacobi(p.double(), coef, case["steps"])
        return [p, last, np.array(gosa[0::2]), np.array(gosa[1::2])]
    dt = TORCH[case.get("dtype", "f32")]
    u = _profile(shape, dt, g)
    if kind in ("diffusion", "dsl"):
        coef = COEF7 if dt == torch.float64 else np.float64(np.float32(COEF7))
        u, last = _diffuse(u.double(), case["steps"], coef, case.get("periodic", False))
        return [u, last] + ([float(u.sum())] if case.get("reduce") else [])
    if kind == "redblack":
        f, u = _uniform(shape, -1e-2, 1e-2, dt, g).double(), u.double()
        c = float(np.float32(1.0 / 6.0))
        inner = tuple(slice(1, -1) for _ in shape)
        index = sum(torch.arange(n, device="cuda").reshape([n if i == k else 1 for i in range(3)])
                    for k, n in enumerate(shape))[inner]
        for _ in range(case["steps"]):
            for colour in (0, 1):
                v = c * f
                for axis in range(3):
                    v += c * (u.roll(1, axis) + u.roll(-1, axis))
                u[inner] = torch.where(index % 2 == colour, v[inner], u[inner])
        return [u]
    u = u.double()
    last = u
    c = float(np.float32(1.0 / 27.0 if kind == "box27" else 0.2))
    inner = tuple(slice(1, -1) for _ in shape)
    for _ in range(case["steps"]):
        if kind == "box27":
            v = u
            for axis in range(3):
                v = v + v.roll(1, axis) + v.roll(-1, axis)
        else:
            v = u + u.roll(1, 0) + u.roll(-1, 0) + u.roll(1, 1) + u.roll(-1, 1)
        w = u.clone()
        w[inner] = c * v[inner]
        last, u = u, w
    return [u, last]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _himeno_work(dims, sweeps, grids=2):
    inner = 1
    for n in dims:
        inner *= n - 2
    return (13 + grids) * 4 * inner, 34 * inner * sweeps


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for him, dims, steps in _members(case):
            n = dims[0] * dims[1] * dims[2]
            wb, wf = _himeno_work(dims, steps, 1) if him else (8 * n, 13 * n * steps)
            b, f = b + wb, f + wf
        return {"bytes": b, "flops": f}
    if kind == "serve":
        b = f = 0
        for him, side in _requests(case):
            wb, wf = _himeno_work((side,) * 3, case["steps"], 1) if him else (
                8 * side ** 3, 13 * side ** 3 * case["steps"])
            b, f = b + wb, f + wf
        return {"bytes": b, "flops": f}
    shape = _shape(case)
    points = inner = 1
    for n in shape:
        points, inner = points * n, inner * (n - 2)
    if kind == "himeno":
        b, f = _himeno_work(shape, case["steps"])
        return {"bytes": b, "flops": f}
    e = 8 if case.get("dtype") == "f64" else 4
    per = {"diffusion": 13, "dsl": 13, "box27": 53, "redblack": 13, "heat2d": 9}[kind]
    n = points if kind in ("diffusion", "dsl") else inner
    return {"bytes": 3 * e * n, "flops": per * n * case["steps"]}
