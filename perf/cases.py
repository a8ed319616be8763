"""Timed cases of the structured-grid library: the calls a solver or time-stepping program makes.

Every case goes through the public Python binding (or, where it has no wrapper, the C entry point).
Kinds and what they stand for:

  apply      Stencil::apply of a StencilLib Laplacian on one box, from the 64^3 box with one ghost
             layer of the smallest workload to 256^3, odd boxes, several components, FP64 and FP32
  transfer   grid transfer written by a caller: AvgDown restriction of a fine field, then the
             piecewise-constant prolongation of a coarse correction added to a copy of a fine field
  algebra    one stage of a time integrator on boxes with ghost cells: out = a x + b y, out += k,
             out *= s, then the square sum and the max norm that a step-size control reads
  boxop      the 4th-order flux-form Laplacian operator evaluated on a box
  partial    one explicit step on a refined level that covers part of its domain: ghost exchange,
             then the 13-point Euler update of every patch
  steps      many explicit steps on a periodic level tiled by patches of uneven sizes, tiles
             autotuned, then the ghost exchange that makes its ghost cells current
  multigrid  a whole solve to tolerance, FP64 or mixed precision, Poisson or Helmholtz
  fas        a whole full-approximation-scheme solve with the 4th-order operator
  serve      a burst of requests of mixed sizes and forms through the serving engine, from host
             right-hand sides to host solutions
"""
import ctypes
import math

import numpy as np
import torch

import proto_b200 as pb
from proto_b200 import workloads as W

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest call: one 64^3 box with one ghost layer
        dict(name="apply_lap7_64", kind="apply", stencil="lap7", nx=64, ny=64, nz=64, ghost=1, ncomp=1, dtype="f64"),
        # the headline stencil call
        dict(name="apply_lap7_256", kind="apply", stencil="lap7", nx=256, ny=256, nz=256, ghost=1, ncomp=1, dtype="f64"),
        # a full 27-point operator on a box of odd sizes, two components
        dict(name="apply_lap27_odd", kind="apply", stencil="lap27", nx=193, ny=161, nz=127, ghost=1, ncomp=2, dtype="f64"),
        # the transfers around a user's own coarse solve
        dict(name="transfer_192", kind="transfer", nx=192, ny=192, nz=192),
        # a Runge-Kutta stage and its norms
        dict(name="algebra_160", kind="algebra", nx=160, ny=160, nz=160, ghost=2),
        # the 4th-order operator as a caller's explicit scheme evaluates it
        dict(name="boxop_160", kind="boxop", nx=160, ny=160, nz=160),
        # a refined level: about 60 % of a 6^3 tiling of uneven patches, not periodic
        dict(name="partial_level", kind="partial", per_axis=6, layout=5, cover=0.6, periodic=False),
        # the 512-patch uneven level
        dict(name="steps_512", kind="steps", per_axis=8, layout=2, steps=20),
        # the headline solve
        dict(name="mg_fp64_256", kind="multigrid", n=256, levels=6, form="poisson", precision="fp64"),
        # the largest solve: 384^3, Helmholtz with alpha per cell, mixed precision, exact coarsest solve
        dict(name="mg_mixed_384", kind="multigrid", n=384, levels=7, form="helmholtz", precision="mixed"),
        # the FAS solver
        dict(name="fas_128", kind="fas", n=128, levels=6),
        # a burst of requests
        dict(name="serve_48", kind="serve", count=48, lo=32, hi=192, layout=4, precision="mixed"),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "transfer", "algebra", "boxop", "partial", "steps", "multigrid", "multigrid",
                       "fas", "serve"])
    if kind == "apply":
        return dict(kind=kind, stencil=rng.choice(["lap7", "lap13", "lap19", "lap27"]), nx=_edge(rng, 32, 280),
                    ny=_edge(rng, 32, 280), nz=_edge(rng, 32, 280), ghost=rng.choice([2, 3]), ncomp=rng.choice([1, 1, 2, 3]),
                    dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "transfer":
        return dict(kind=kind, nx=2 * _edge(rng, 16, 128), ny=2 * _edge(rng, 16, 128), nz=2 * _edge(rng, 16, 128))
    if kind == "algebra":
        return dict(kind=kind, nx=_edge(rng, 32, 256), ny=_edge(rng, 32, 256), nz=_edge(rng, 32, 256),
                    ghost=rng.choice([1, 2, 3]))
    if kind == "boxop":
        return dict(kind=kind, nx=_edge(rng, 32, 256), ny=_edge(rng, 32, 256), nz=_edge(rng, 32, 256))
    if kind == "partial":
        return dict(kind=kind, per_axis=rng.randint(3, 8), layout=rng.randint(10, 1000),
                    cover=round(rng.uniform(0.3, 0.9), 2), periodic=rng.choice([False, True]))
    if kind == "steps":
        return dict(kind=kind, per_axis=rng.randint(3, 8), layout=rng.randint(10, 1000), steps=_edge(rng, 4, 40))
    if kind == "multigrid":
        n, levels = rng.choice([(32, 3), (48, 4), (64, 4), (80, 4), (96, 5), (112, 4), (128, 5), (160, 5), (192, 6), (256, 6)])
        return dict(kind=kind, n=n, levels=levels, form=rng.choice(["poisson", "helmholtz"]),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "fas":
        n, levels = rng.choice([(32, 4), (48, 4), (64, 5), (80, 5), (96, 5), (128, 6), (160, 6), (192, 6), (256, 7)])
        return dict(kind=kind, n=n, levels=levels)
    return dict(kind=kind, count=_edge(rng, 4, 48), lo=32, hi=rng.choice([96, 128, 192]), layout=rng.randint(10, 1000),
                precision=rng.choice(["mixed", "fp64"]))


# ---- stencils (StencilLib's insertion order) --------------------------------------------------------
def _laplacian(name):
    """(coefficients, offsets) of a unit-spacing Laplacian."""
    if name == "lap7":
        return ([-6.0] + [1.0] * 6,
                [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)])
    if name == "lap13":
        c, o = [4 / 3, -7.5, 4 / 3, -1 / 12, -1 / 12], [(1, 0, 0), (0, 0, 0), (-1, 0, 0), (2, 0, 0), (-2, 0, 0)]
        for d in (1, 2):
            for s, v in ((1, 4 / 3), (-1, 4 / 3), (2, -1 / 12), (-2, -1 / 12)):
                c.append(v)
                o.append(tuple(s if k == d else 0 for k in range(3)))
        return c, o
    centre, weight = {"lap19": (-4.0, {1: 1 / 3, 2: 1 / 6, 3: 0.0}),
                      "lap27": (-64 / 15, {1: 7 / 15, 2: 1 / 10, 3: 1 / 30})}[name]
    c, o = [centre], [(0, 0, 0)]
    for z in (-1, 0, 1):
        for y in (-1, 0, 1):
            for x in (-1, 0, 1):
                w = weight.get(abs(x) + abs(y) + abs(z), 0.0)
                if w:
                    c.append(w)
                    o.append((x, y, z))
    return c, o


_CHILDREN = [(i & 1, (i >> 1) & 1, i >> 2) for i in range(8)]


# ---- inputs -----------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(shape, g, lo=-1.0, hi=1.0, dtype=torch.float64):
    return torch.rand(shape, generator=g, device=DEV, dtype=dtype) * (hi - lo) + lo


def _box(case, grow=0):
    return pb.Box((0, 0, 0), (case["nx"] - 1, case["ny"] - 1, case["nz"] - 1)).grow(grow)


def _shape(case, grow=0):
    return (case["nz"] + 2 * grow, case["ny"] + 2 * grow, case["nx"] + 2 * grow)


def _layout(case):
    """Boxes (lo, hi) of the level's patches and the domain's extents."""
    boxes, ext = W.amr_patches(W.amr_widths(seed=case["layout"], per_axis=case["per_axis"]))
    if case["kind"] == "partial":
        keep = np.random.default_rng(case["layout"]).random(len(boxes)) < case["cover"]
        keep[0], keep[-1] = True, False
        boxes = [b for b, k in zip(boxes, keep) if k]
    return boxes, ext


def _apply_inputs(case, seed):
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    return _uniform((case["ncomp"],) + _shape(case, case["ghost"]), _gen(seed), dtype=dt)


def _transfer_inputs(case, seed):
    g = _gen(seed)
    nz, ny, nx = _shape(case)
    return _uniform((nz, ny, nx), g), _uniform((nz, ny, nx), g), _uniform((nz // 2, ny // 2, nx // 2), g)


def _algebra_inputs(case, seed):
    g = _gen(seed)
    return _uniform(_shape(case, case["ghost"]), g), _uniform(_shape(case), g), _uniform(_shape(case, 1), g)


def _level_inputs(case, seed):
    """The slab's initial values: a patch's grown box after another, padding and all."""
    lv = _Slab(_layout(case)[0])
    return lv, _uniform((lv.elems,), _gen(seed))


def _mg_inputs(case, seed):
    f = W.sine_modes_rhs_device(case["n"], seed, modes=8, device=DEV)
    if case["form"] == "poisson":
        return -f, None
    return f, _uniform((case["n"],) * 3, _gen(seed), 0.1, 1.0)


def _serve_requests(case, seed):
    """(edge, helmholtz, alpha, right-hand side on the GPU) of each request."""
    r = np.random.default_rng(case["layout"])
    out = []
    for k in range(case["count"]):
        n = int(np.clip(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))) / 16) * 16, case["lo"], case["hi"]))
        helm, alpha = bool(r.random() < 0.5), float(r.uniform(0.0, 1.0))
        f = W.sine_modes_rhs_device(n, seed * 1000 + k, modes=4, device=DEV)
        out.append((n, helm, alpha, f if helm else -f))
    return out


class _Slab:
    """Offsets of the patches (two ghost cells, each patch 32-element aligned) in a level's slab."""

    def __init__(self, boxes, ghost=2):
        self.ghost, self.boxes, self.offsets, off = ghost, boxes, [], 0
        for lo, hi in boxes:
            self.offsets.append(off)
            off += math.prod(hi[d] - lo[d] + 1 + 2 * ghost for d in range(3))
            off = (off + 31) // 32 * 32
        self.elems = off

    def patch(self, slab, i):
        """View of patch i's grown box, (z, y, x)."""
        lo, hi = self.boxes[i]
        shape = [hi[d] - lo[d] + 1 + 2 * self.ghost for d in (2, 1, 0)]
        return slab[self.offsets[i]:self.offsets[i] + math.prod(shape)].view(shape)


# ---- a user's program: what it keeps, and one pass --------------------------------------------------
def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind == "apply":
        c, o = _laplacian(case["stencil"])
        s.update(S=pb.Stencil(c, o), src=_apply_inputs(case, seed), scale=float(case["nx"]) ** 2)
        s["dst"] = torch.zeros((case["ncomp"],) + _shape(case), dtype=s["src"].dtype, device=DEV)
        s.update(sb=_box(case, case["ghost"]), db=_box(case))
    elif kind == "transfer":
        fine, base, corr = _transfer_inputs(case, seed)
        s.update(avg=pb.Stencil([0.125] * 8, _CHILDREN, src_ratio=(2, 2, 2)), fine=fine, base=base, corr=corr)
        s.update(down=torch.zeros_like(corr), up=torch.zeros_like(fine), fb=_box(case),
                 cb=pb.Box((0, 0, 0), (case["nx"] // 2 - 1, case["ny"] // 2 - 1, case["nz"] // 2 - 1)))
    elif kind == "algebra":
        x, y, k = _algebra_inputs(case, seed)
        s.update(x=x, y=y, k=k, out=torch.zeros_like(y), total=torch.zeros(1, dtype=torch.float64, device=DEV))
        s.update(xb=_box(case, case["ghost"]), yb=_box(case), kb=_box(case, 1))
    elif kind == "boxop":
        s.update(u=_uniform(_shape(case, 2), _gen(seed)), out=torch.zeros(_shape(case), dtype=torch.float64, device=DEV))
        s.update(ub=_box(case, 2), ob=_box(case))
    elif kind in ("partial", "steps"):
        boxes, ext = _layout(case)
        c, o = _laplacian("lap13")
        per = (1, 1, 1) if case.get("periodic", True) else (0, 0, 0)
        lv = pb.Level([pb.Box(*b) for b in boxes], 2, pb.Box((0, 0, 0), [e - 1 for e in ext]), per)
        u0 = _level_inputs(case, seed)[1]
        assert lv.slab_elems == u0.numel()
        s.update(lv=lv, S=pb.Stencil(c, o), u0=u0, u=u0.clone(), tmp=torch.zeros_like(u0))
        s.update(scale=float(ext[0]) ** 2, dt=0.1 / float(ext[0]) ** 2)
        if kind == "steps":
            lv.autotune(s["S"], s["u"], s["tmp"], scale=s["scale"])
            s["tmp"].zero_()
    elif kind == "multigrid":
        helm = case["form"] == "helmholtz"
        s["rhs"], alpha = _mg_inputs(case, seed)
        s["mg"] = pb.Multigrid(pb.MGParams(case["n"], case["levels"], nu1=4, nu2=4, nu_bottom=10, tol=1e-10, max_iter=60,
                                           form=pb.MG_HELMHOLTZ if helm else pb.MG_POISSON, bottom=int(helm),
                                           precision=pb.MG_FP64 if case["precision"] == "fp64" else pb.MG_MIXED))
        if helm:
            s["mg"].set_alpha(alpha)
        s["phi"] = torch.zeros_like(s["rhs"])
    elif kind == "fas":
        s.update(fas=pb.FAS(case["n"], case["levels"]), force=W.sine_modes_rhs_device(case["n"], seed, modes=8, device=DEV))
        s["phi"] = torch.zeros_like(s["force"])
    else:
        s["engine"] = pb.Serve(8 << 30, max_active=64, tol=1e-8,
                               precision=pb.MG_FP64 if case["precision"] == "fp64" else pb.MG_MIXED)
        s["requests"] = []
        for n, helm, alpha, f in _serve_requests(case, seed):
            rhs = torch.empty(n ** 3, dtype=torch.float64, pin_memory=torch.cuda.is_available())
            rhs.copy_(f.reshape(-1))
            out = torch.zeros(n ** 3, dtype=torch.float64, pin_memory=torch.cuda.is_available())
            s["requests"].append((n, helm, alpha, rhs.numpy(), out.numpy()))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "apply":
        s["S"].apply(s["src"], s["sb"], s["dst"], s["db"], scale=s["scale"], ncomp=case["ncomp"])
        return s["dst"]
    if kind == "transfer":
        s["avg"].apply(s["fine"], s["fb"], s["down"], s["cb"])
        pb.boxdata_copy(s["base"], s["fb"], s["up"], s["fb"])
        pb.interp_constant(2, s["corr"], s["cb"], s["up"], s["fb"])
        return s["down"], s["up"]
    if kind == "algebra":
        pb.forall_axpby(s["out"], s["yb"], s["x"], s["xb"], s["y"], s["yb"], 0.5, 2.0)
        pb.boxdata_op(pb.OP_ADD, s["out"], s["yb"], s["k"], s["kb"])
        pb.boxdata_scalar(pb.OP_MUL, s["out"], s["yb"], 0.75)
        pb.reduce_async(pb.RED_SUMSQ, s["out"], s["yb"], s["total"])
        return s["out"], s["total"], pb.reduce(pb.RED_ABS, s["out"], s["yb"])
    if kind == "boxop":
        vp, dbl = ctypes.c_void_p, ctypes.c_double
        status = pb.lib().pb_boxop_laplace_f64(vp(s["u"].data_ptr()), s["ub"].c(), vp(s["out"].data_ptr()), s["ob"].c(),
                                               s["ob"].c(), dbl(1.0 / case["nx"]), dbl(1.0), dbl(1.0),
                                               vp(torch.cuda.current_stream().cuda_stream))
        if status != 0:
            raise pb.ProtoError(status, "pb_boxop_laplace_f64")
        return s["out"]
    if kind == "partial":
        s["lv"].exchange(s["u"])
        s["lv"].stencil(s["S"], pb.EPI_EULER, s["u"], s["tmp"], scale=s["scale"], a=s["dt"])
        return s["u"], s["tmp"]
    if kind == "steps":
        s["u"].copy_(s["u0"])      # a new initial state, as each run of a stepping program has
        s["lv"].steps(s["S"], pb.EPI_EULER, s["u"], s["tmp"], case["steps"], scale=s["scale"], a=s["dt"])
        s["lv"].exchange(s["u"])
        # the tail of each patch's aligned slot belongs to no patch; the slab is returned with it
        return s["u"]
    if kind == "multigrid":
        s["phi"].zero_()
        s["mg"].solve(s["rhs"], s["phi"])
        return s["phi"]
    if kind == "fas":
        s["phi"].zero_()
        s["fas"].solve(s["force"], s["phi"], max_iter=20, tol=1e-10)
        return s["phi"]
    for n, helm, alpha, rhs, out in s["requests"]:
        s["engine"].submit(n, rhs, out, form=pb.MG_HELMHOLTZ if helm else pb.MG_POISSON, alpha=alpha)
    s["engine"].run_until_idle()
    s["engine"].poll()
    return [q[4] for q in s["requests"]]


def work(case):
    """Bytes and operations of one pass: inputs once, outputs once; for a solve, per cycle one read of the
    state and the right-hand side and one write of the state on every level (each cycle ends in a norm
    of the whole grid), and the sweeps' arithmetic."""
    kind = case["kind"]
    if "nx" in case:
        cells = case["nx"] * case["ny"] * case["nz"]
        grown = lambda g: math.prod(case[k] + 2 * g for k in ("nx", "ny", "nz"))
    if kind == "apply":
        item = 8 if case["dtype"] == "f64" else 4
        return {"bytes": item * case["ncomp"] * (grown(2 if case["stencil"] == "lap13" else 1) + cells),
                "flops": 2 * len(_laplacian(case["stencil"])[0]) * cells * case["ncomp"]}
    if kind == "transfer":     # down: read fine, write coarse; up: read fine and coarse, write fine
        return {"bytes": 8 * cells * (1 + 1 / 8 + 1 + 1 / 8 + 1), "flops": 4 * cells}
    if kind == "algebra":      # x, y, k in, out; the norms can be taken as the result is made
        return {"bytes": 8 * 4 * cells, "flops": 8 * cells}
    if kind == "boxop":        # three fluxes of 7 operations, their divergences and the scale
        return {"bytes": 8 * (grown(2) + cells), "flops": 34 * cells}
    if kind in ("partial", "steps"):
        valid = sum(math.prod(hi[d] - lo[d] + 1 for d in range(3)) for lo, hi in _layout(case)[0])
        ghost = sum(math.prod(hi[d] - lo[d] + 5 for d in range(3)) for lo, hi in _layout(case)[0]) - valid
        n = case.get("steps", 1)
        return {"bytes": 16 * valid * n + 16 * ghost, "flops": 28 * valid * n}
    if kind == "multigrid":
        helm = case["form"] == "helmholtz"
        cycles = 15
        cells = case["n"] ** 3 * 8 / 7
        item = 4 if case["precision"] == "mixed" else 8
        return {"bytes": cycles * cells * item * (4 if helm else 3), "flops": cycles * cells * 9 * (22 if helm else 16)}
    if kind == "fas":
        cells = case["n"] ** 3 * 8 / 7
        return {"bytes": 10 * cells * 24, "flops": 10 * cells * 13 * 40}
    cells = sum(n ** 3 for n in _serve_edges(case)) * 8 / 7
    item = 4 if case["precision"] == "mixed" else 8
    return {"bytes": 12 * cells * 3 * item, "flops": 12 * cells * 9 * 16}


def _serve_edges(case):
    r = np.random.default_rng(case["layout"])
    out = []
    for _ in range(case["count"]):
        out.append(int(np.clip(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))) / 16) * 16, case["lo"], case["hi"])))
        r.random(), r.uniform(0.0, 1.0)
    return out


def tolerance(case):
    """About four times the largest distance from exact() seen over these ranges: FP64 sums differ by their
    order, a solve adds its cycles' rounding, and a mixed-precision solve stops at a residual (the Poisson
    form's constant is fixed by FP32 rounding alone)."""
    kind = case["kind"]
    fp64 = case.get("precision") == "fp64"
    if kind == "apply":
        return {"rel": 1.5e-15} if case["dtype"] == "f64" else {"rel": 4e-7}
    if kind == "multigrid":
        return {"rel": 1.5e-13} if fp64 else {"rel": 1e-12 if case["form"] == "helmholtz" else 4e-7}
    if kind == "serve":
        return {"rel": 1.5e-13} if fp64 else {"rel": 1e-6}
    return {"rel": {"transfer": 5e-16, "algebra": 1e-15, "boxop": 1e-15, "partial": 2e-15, "steps": 4e-15,
                    "fas": 3e-15}[kind]}


# ---- the same results in plain 64-bit torch ---------------------------------------------------------
def _taps(u, coefs, offsets, grow, shape):
    """sum_j c_j u(p + o_j) over the box of `shape`, u stored on it grown by `grow`."""
    nz, ny, nx = shape
    out = torch.zeros(u.shape[:-3] + tuple(shape), dtype=u.dtype, device=u.device)
    for c, (x, y, z) in zip(coefs, offsets):
        out += c * u[..., grow + z:grow + z + nz, grow + y:grow + y + ny, grow + x:grow + x + nx]
    return out


def _lap4(u, grow, shape, h):
    """4th-order flux-form Laplacian: differences of the face gradients."""
    out = 0
    for d in range(3):
        e = lambda k: tuple(k if q == d else 0 for q in range(3))
        face = lambda s: _taps(u, [1 / 12, -15 / 12, 15 / 12, -1 / 12], [e(s - 2), e(s - 1), e(s), e(s + 1)], grow, shape) / h
        out = out + (face(1) - face(0)) / h
    return out


def _wrap(u, g):
    for d in range(3):
        u = torch.cat([u.narrow(d, u.shape[d] - g, g), u, u.narrow(d, 0, g)], d)
    return u


def _down(u):
    nz, ny, nx = (v // 2 for v in u.shape)
    return u.view(nz, 2, ny, 2, nx, 2).mean((1, 3, 5))


def _up(u):
    for d in range(3):
        u = u.repeat_interleave(2, d)
    return u


def _lap2(u):
    out = -6.0 * u
    for d in range(3):
        out += torch.roll(u, 1, d)
        out += torch.roll(u, -1, d)
    return out


class _VCycle:
    """Correction-scheme V(4,4) cycles of point Jacobi (omega = 2/3) on periodic cubes; alpha a field or None."""

    def __init__(self, n, levels, alpha, direct, beta=1.0, omega=2.0 / 3.0, nu=4, nu_bottom=10):
        self.n, self.levels, self.direct, self.beta, self.omega, self.nu, self.nu_bottom = n, levels, direct, beta, omega, nu, nu_bottom
        self.alpha = [alpha]
        for _ in range(levels):
            self.alpha.append(None if alpha is None else _down(self.alpha[-1]))

    def op(self, l, u):
        v = _lap2(u) * float(self.n >> l) ** 2
        return v if self.alpha[l] is None else self.alpha[l] * u - self.beta * v

    def relax(self, l, u, f, sweeps):
        h2 = float(self.n >> l) ** -2
        for _ in range(sweeps):
            if self.alpha[l] is None:
                u = u + self.omega / 6 * (_lap2(u) - h2 * f)
            else:
                u = u + self.omega * (f - self.op(l, u)) / (self.alpha[l] + 6 * self.beta / h2)
        return u

    def bottom(self, l, f):
        if not self.direct:
            return self.relax(l, torch.zeros_like(f), f, self.nu_bottom)
        m = f.numel()
        eye = torch.eye(m, dtype=f.dtype, device=f.device)
        a = torch.stack([self.op(l, eye[k].view_as(f)).reshape(-1) for k in range(m)], 1)
        if self.alpha[l] is None:
            a += 6 * float(self.n >> l) ** 2 / m
        return torch.linalg.solve(a, f.reshape(-1)).view_as(f)

    def cycle(self, l, u, f):
        if l == self.levels:
            return self.bottom(l, f)
        u = self.relax(l, u, f, self.nu)
        r = _down(f - self.op(l, u))
        u = u + _up(self.cycle(l + 1, torch.zeros_like(r), r))
        return self.relax(l, u, f, self.nu)

    def solve(self, f, tol, max_iter):
        u = torch.zeros_like(f)
        first = (f - self.op(0, u)).abs().max().item()
        for _ in range(max_iter):
            u = self.cycle(0, u, f)
            if (f - self.op(0, u)).abs().max().item() < tol * first:
                break
        return u


class _FAS:
    """FAS V(6,6) cycles with the 4th-order operator op(u) = -_lap4(u), lambda = 0.5 / (6 / h^2), 10 bottom sweeps."""

    def __init__(self, n, levels):
        self.n, self.last = n, levels - 1

    def op(self, l, u):
        return -_lap4(_wrap(u, 2), 2, u.shape, 1.0 / (self.n >> l))

    def relax(self, l, u, f, sweeps):
        lam = 0.5 / (6.0 * float(self.n >> l) ** 2)
        for _ in range(sweeps):
            u = u - lam * (self.op(l, u) + f)
        return u

    def cycle(self, l, u, f):
        if l == self.last:
            return self.relax(l, u, f, 10)
        u = self.relax(l, u, f, 6)
        c = _down(u)
        fc = _down(self.op(l, u) + f) - self.op(l + 1, c)
        u = u + _up(self.cycle(l + 1, c, fc) - c)
        return self.relax(l, u, f, 6)

    def solve(self, f, tol, max_iter):
        u = torch.zeros_like(f)
        first = (self.op(0, u) + f).abs().max().item()
        for _ in range(max_iter):
            u = self.cycle(0, u, f)
            if (self.op(0, u) + f).abs().max().item() < tol * first:
                break
        return u


def _fill_ghosts(lv, slab, field, mask, periodic):
    """Every patch's cells that the patches cover (images included, on a periodic domain) set to the field."""
    g = lv.ghost
    if periodic:
        field, mask = _wrap(field, g), _wrap(mask, g)
    else:
        field, mask = (torch.nn.functional.pad(v, (g,) * 6) for v in (field, mask))
    for i, (lo, hi) in enumerate(lv.boxes):
        at = tuple(slice(lo[d], hi[d] + 1 + 2 * g) for d in (2, 1, 0))
        p = lv.patch(slab, i)
        p.copy_(torch.where(mask[at] > 0, field[at], p))


def exact(case, seed):
    kind = case["kind"]
    if kind == "apply":
        c, o = _laplacian(case["stencil"])
        return _taps(_apply_inputs(case, seed).double(), c, o, case["ghost"], _shape(case)) * float(case["nx"]) ** 2
    if kind == "transfer":
        fine, base, corr = _transfer_inputs(case, seed)
        return _down(fine), base + _up(corr)
    if kind == "algebra":
        x, y, k = _algebra_inputs(case, seed)
        at = lambda v, g: _taps(v, [1.0], [(0, 0, 0)], g, _shape(case))
        out = 0.75 * (0.5 * at(x, case["ghost"]) + 2.0 * y + at(k, 1))
        return out, out.square().sum().reshape(1), out.abs().max().item()
    if kind == "boxop":
        return _lap4(_uniform(_shape(case, 2), _gen(seed)), 2, _shape(case), 1.0 / case["nx"])
    if kind in ("partial", "steps"):
        lv, slab = _level_inputs(case, seed)
        ext = _layout(case)[1]
        field = torch.zeros((ext[2], ext[1], ext[0]), dtype=torch.float64, device=DEV)
        mask = torch.zeros_like(field)
        for i, (lo, hi) in enumerate(lv.boxes):
            at = tuple(slice(lo[d], hi[d] + 1) for d in (2, 1, 0))
            field[at] = lv.patch(slab, i)[2:-2, 2:-2, 2:-2]
            mask[at] = 1.0
        c, o = _laplacian("lap13")
        if kind == "steps":
            for _ in range(case["steps"]):
                field = field + 0.1 * _taps(_wrap(field, 2), c, o, 2, field.shape)
            if case["steps"] % 2:       # an odd count ends in the scratch slab, whose padding is zero
                slab = torch.zeros_like(slab)
            _fill_ghosts(lv, slab, field, mask, True)
            return slab
        _fill_ghosts(lv, slab, field, mask, case["periodic"])
        new = torch.zeros_like(slab)
        for i in range(len(lv.boxes)):
            p = lv.patch(slab, i)
            v = p[2:-2, 2:-2, 2:-2]
            lv.patch(new, i)[2:-2, 2:-2, 2:-2] = v + 0.1 * _taps(p, c, o, 2, v.shape)
        return slab, new
    if kind == "multigrid":
        rhs, alpha = _mg_inputs(case, seed)
        return _VCycle(case["n"], case["levels"], alpha, alpha is not None).solve(rhs, 1e-10, 60)
    if kind == "fas":
        force = W.sine_modes_rhs_device(case["n"], seed, modes=8, device=DEV)
        return _FAS(case["n"], case["levels"]).solve(force, 1e-10, 20)
    out = []
    for n, helm, alpha, f in _serve_requests(case, seed):
        levels = (n & -n).bit_length() - 1
        a = torch.full_like(f, alpha) if helm else None
        out.append(_VCycle(n, levels, a, False).solve(f, 1e-8, 100).reshape(-1).cpu().numpy())
    return out
