"""Workloads whose time matters to a user of batsrus_b200, with their inputs,
their outputs in 64 bits where plain torch can give them, and the work that
they cannot do without.

Each case runs a whole call sequence of the Python mirror of the reference's
interface: the host ``State_VGB`` (page-locked, as a driver that exchanges
state with the device keeps it) goes in, a number of time steps or solves
runs, and the result comes back in the reference's layout.  The library
keeps one context per process, so the solver of the current grid and scheme
is kept between passes, as a program that runs many sessions on one grid
does; a pass starts from its own state, time 0 and step 0.
"""
import json
import math

import numpy as np
import torch

from batsrus_b200.configs import _blast_refine
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.grid import BlockGrid
from batsrus_b200.heat import HeatSolver
from batsrus_b200.heat_params import HeatParams
from batsrus_b200.implicit import ImplicitSolver
from batsrus_b200.implicit_params import ImplicitParams
from batsrus_b200.learned import LearnedPreconditioner
from batsrus_b200.param import Scheme


def listed():
    E = dict(kind="explicit", order=2, stages=2, precision="fp64", bc="periodic")
    return [
        # the reference's own GPU test: a 1D shock tube, 16 blocks of 64
        # cells, first order, one stage, fixed step, 512 steps (launch latency)
        dict(E, name="shocktube_1d", dim=1, cells=64, nx=16, ny=1, nz=1, flux="Rusanov", limiter="minmod", order=1,
             stages=1, state="shock", bc="float", steps=512),
        # 2D blocks of 8 x 8: an ordinary 2D run
        dict(E, name="orszag_tang_2d", dim=2, cells=8, nx=48, ny=48, nz=1, flux="Linde", limiter="mc3", state="ot",
             steps=50),
        # the smallest 3D grid: the size of the parity tests and the smoke run
        dict(E, name="orszag_tang_16", dim=3, cells=8, nx=2, ny=2, nz=2, flux="Linde", limiter="mc3", state="ot",
             steps=60),
        # ordinary sizes and odd block counts
        dict(E, name="orszag_tang_64", dim=3, cells=8, nx=8, ny=8, nz=8, flux="Linde", limiter="mc3", state="ot",
             steps=50),
        dict(E, name="blast_ragged", dim=3, cells=8, nx=13, ny=9, nz=11, flux="HLLD", limiter="mc", state="blast",
             bc="float", steps=30),
        # blocks of 4^3, the other 3D block size
        dict(E, name="blocks_of_4", dim=3, cells=4, nx=17, ny=16, nz=15, flux="Rusanov", limiter="minmod",
             state="ot", steps=40),
        # the headline workload's scheme on a state larger than L2, in both
        # arithmetic modes
        dict(E, name="orszag_tang_160", dim=3, cells=8, nx=20, ny=20, nz=20, flux="Linde", limiter="mc3", state="ot",
             steps=40),
        dict(E, name="orszag_tang_160_fp32", dim=3, cells=8, nx=20, ny=20, nz=20, flux="Linde", limiter="mc3",
             state="ot", steps=40, precision="fp32"),
        # the block-adaptive blast on a static refined grid, then the
        # criteria that the next regrid would use
        dict(kind="adaptive", name="adaptive_blast", root=12, level=2, flux="HLLD", limiter="mc", precision="fp32",
             steps=30),
        # implicit JFNK steps (backward Euler, then BDF2) at CFL 20
        dict(kind="implicit", name="implicit_96", nx=12, ny=12, nz=12, precond="BILU", factors="bf16", steps=2),
        # semi-implicit heat conduction: set-up and two solves
        dict(kind="heat", name="heat_128", nx=16, ny=16, nz=16, precond="BILU", sweeps="fp32", operator="fp32",
             solves=2),
        # training of the learned preconditioner on stored pairs
        dict(kind="learned", name="learned_training", samples=1024, epochs=8),
    ]


def _roots(rng, lo, hi):
    """three block counts whose product lies between lo and hi, spread over its logarithm"""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    s = n ** (1.0 / 3.0)
    r = [max(1, round(s * a)), max(1, round(s * b)), max(1, round(s / (a * b)))]
    while r[0] * r[1] * r[2] > hi:
        r[r.index(max(r))] -= 1
    rng.shuffle(r)
    return r


def draw(rng):
    kind = rng.choice(["3d", "3d", "3d", "4", "2d", "1d", "adaptive", "implicit", "heat", "learned"])
    flux = rng.choice(["Rusanov", "Linde", "HLLD"])
    limiter = rng.choice(["minmod", "mc", "mc3"])
    bc = rng.choice(["periodic", "float"])
    precision = rng.choice(["fp64", "fp32"])
    E = dict(kind="explicit", order=2, stages=2, precision="fp64", bc=bc, flux=flux, limiter=limiter,
             state=rng.choice(["ot", "blast"]))
    if kind == "3d":
        nx, ny, nz = _roots(rng, 8, 8000)
        return dict(E, dim=3, cells=8, nx=nx, ny=ny, nz=nz, steps=rng.randint(10, 40), precision=precision)
    if kind == "4":
        nx, ny, nz = _roots(rng, 8, 8000)
        return dict(E, dim=3, cells=4, nx=nx, ny=ny, nz=nz, steps=rng.randint(10, 40), precision=precision)
    if kind == "2d":
        return dict(E, dim=2, cells=8, nx=rng.randint(3, 60), ny=rng.randint(3, 60), nz=1, state="ot", bc="periodic",
                    steps=rng.randint(10, 50))
    if kind == "1d":
        return dict(E, dim=1, cells=rng.choice([8, 64]), nx=rng.randint(3, 60), ny=1, nz=1, state="shock", bc="float",
                    steps=rng.randint(50, 500), order=rng.choice([1, 2]))
    if kind == "adaptive":
        return dict(kind="adaptive", root=rng.randint(6, 14), level=rng.randint(1, 2), flux=flux, limiter=limiter,
                    precision=precision, steps=rng.randint(10, 30))
    if kind == "implicit":
        nx, ny, nz = _roots(rng, 27, 1728)
        return dict(kind="implicit", nx=nx, ny=ny, nz=nz, precond=rng.choice(["BILU", "NONE"]),
                    factors=rng.choice(["fp32", "bf16"]), steps=rng.randint(1, 2))
    if kind == "heat":
        nx, ny, nz = _roots(rng, 64, 4096)
        p = rng.choice(["fp64", "fp32"])
        return dict(kind="heat", nx=nx, ny=ny, nz=nz, precond=rng.choice(["BILU", "NONE"]), sweeps=p, operator=p,
                    solves=rng.randint(1, 2))
    return dict(kind="learned", samples=rng.randint(64, 1024), epochs=rng.randint(2, 8))


# ---- grids, schemes and the solver that a program keeps ---------------------
def _key(case):
    return json.dumps({k: v for k, v in case.items() if k not in ("name", "steps", "solves", "epochs")},
                      sort_keys=True)


def _grid(case):
    n = (case.get("nx"), case.get("ny"), case.get("nz"))
    if case["kind"] == "adaptive":
        r = case["root"]
        return BlockGrid.adaptive(3, (8, 8, 8), (r,) * 3, (-0.5,) * 3, (0.5,) * 3, ("periodic",) * 6, case["level"],
                                  _blast_refine(r))
    if case["kind"] == "heat":
        return BlockGrid.uniform(3, (8, 8, 8), n, (-0.5,) * 3, (0.5,) * 3, ("float",) * 6)
    if case["kind"] == "implicit":
        return BlockGrid.uniform(3, (8, 8, 8), n, (0.0,) * 3, (1.0,) * 3, ("periodic",) * 6)
    c, bc = case["cells"], (case["bc"],) * 6
    if case["dim"] == 1:
        h = 0.125 * case["nx"] * c  # cells of 0.25, as in the reference's shock tube
        return BlockGrid.uniform(1, (c, 1, 1), n, (-h, -0.125, -0.125), (h, 0.125, 0.125), bc)
    if case["dim"] == 2:
        return BlockGrid.uniform(2, (c, c, 1), n, (0.0,) * 3, (1.0,) * 3, bc)
    lo = -0.5 if case["state"] == "blast" else 0.0
    return BlockGrid.uniform(3, (c, c, c), n, (lo,) * 3, (lo + 1.0,) * 3, bc)


def _scheme(case):
    if case["kind"] in ("implicit", "heat"):
        return Scheme(nOrder=2, nStage=2, typeFlux="Linde", typeLimiter="mc3", limiterBeta=1.2, cfl=0.8,
                      gamma=5.0 / 3.0, useDivbSource=True, useHalfStep=True)
    if case.get("dim") == 1:
        one = case["stages"] == 1  # the reference's test: a fixed step
        return Scheme(nOrder=case["order"], nStage=case["stages"], typeFlux=case["flux"], typeLimiter=case["limiter"],
                      limiterBeta=_beta(case), cfl=1.0 if one else 0.8, gamma=2.0, useDivbSource=False,
                      useDtFixed=one, dtFixed=0.05, useHalfStep=True)
    return Scheme(nOrder=2, nStage=2, typeFlux=case["flux"], typeLimiter=case["limiter"], limiterBeta=_beta(case),
                  cfl=0.8, gamma=5.0 / 3.0, useDivbSource=True, useHalfStep=True, precision=case["precision"])


def _beta(case):
    return 1.2 if case["limiter"] == "mc3" else 1.5


_kept = {}


def _solver(case):
    """the solver of this case's grid and scheme: one per process, like the library's context"""
    if _kept.get("key") != _key(case):
        _kept.clear()
        g = _grid(case)
        _kept.update(grid=g, solver=ExplicitSolver(g, _scheme(case)))
        if case["kind"] == "implicit":
            p = ImplicitParams(cflImpl=20.0, useBdf2=True, nKrylovVector=30, maxMatvec=100, errorMax=1e-3,
                               typePrecond=case["precond"], precondPrecision=case["factors"])
            _kept["implicit"] = ImplicitSolver(_kept["solver"], p)
        _kept["key"] = _key(case)
    return _kept


# ---- inputs -----------------------------------------------------------------
def _centers(g, ghost=True):
    """cell-centre coordinates of every block on the GPU, ghost cells included"""
    corner, size = (torch.from_numpy(a).cuda() for a in g.block_geometry())
    out = []
    for d, (n, ng) in enumerate(((g.nI, 2), (g.nJ, 2 if g.nDim > 1 else 0), (g.nK, 2 if g.nDim > 2 else 0))):
        ng = ng if ghost else 0
        i = torch.arange(n + 2 * ng, device="cuda", dtype=torch.float64) - ng + 0.5
        shape = [g.nBlock, 1, 1, 1]
        shape[3 - d] = n + 2 * ng
        x = corner[:, d, None] + i[None, :] * size[:, d, None]
        if d >= g.nDim:
            x = torch.full_like(x, 0.5 * (g.xyzMin[d] + g.xyzMax[d]))
        out.append(x.reshape(shape))
    return out


def _waves(X, rng, kmax, count):
    """a smooth random field of unit variance, periodic on the unit cube: `count` random Fourier modes"""
    f = 0.0
    for _ in range(count):
        k = rng.integers(-kmax, kmax + 1, 3)
        ph, a = rng.uniform(0, 2 * math.pi), rng.normal()
        e = [torch.polar(torch.ones_like(x), 2 * math.pi * float(k[d]) * x) for d, x in enumerate(X)]
        f = f + a * (e[0] * e[1] * e[2] * complex(math.cos(ph), math.sin(ph))).real
    return f / max(float(f.std()), 1e-300)


def _state(case, g, seed):
    """State_VGB on the GPU: the workload's initial state with seeded perturbations"""
    rng = np.random.default_rng(seed)
    X = _centers(g)
    shape = g.state_shape_fortran()
    prim = torch.empty((8,) + shape[:4], dtype=torch.float64, device="cuda")
    x, y, z = X
    if case.get("state") == "shock":
        left, right = [1, 0, 0, 0, 0.75, 1, 0, 1], [0.125, 0, 0, 0, 0.75, -1, 0, 0.1]
        inside = x < 0.0
        for v in range(8):
            s = 1.0 + 0.05 * rng.uniform(-1, 1, 2) if v in (0, 5, 7) else (1.0, 1.0)
            prim[v] = torch.where(inside, left[v] * s[0], right[v] * s[1])
    elif case["kind"] == "adaptive" or case.get("state") == "blast":
        r0 = 0.1 * (1.0 + 0.05 * rng.uniform(-1, 1))
        prim[0] = 1.0 + 0.01 * _waves(X, rng, 3, 4)
        for v in (1, 2, 3):
            prim[v] = 0.01 * _waves(X, rng, 3, 4)
        prim[4], prim[5], prim[6] = 1 / math.sqrt(2), 1 / math.sqrt(2), 0.0
        prim[7] = torch.where(x * x + y * y + z * z < r0 * r0, 10.0, 0.1) * (1.0 + 0.01 * _waves(X, rng, 3, 4))
    else:
        t = 2 * math.pi
        b0 = 1.0 / math.sqrt(4 * math.pi)
        prim[0], prim[7] = 25.0 / (36.0 * math.pi), 5.0 / (12.0 * math.pi)
        prim[1], prim[2], prim[3] = -torch.sin(t * y), torch.sin(t * x), 0.01 * torch.sin(t * z)
        prim[4], prim[5], prim[6] = -b0 * torch.sin(t * y), b0 * torch.sin(2 * t * x), 0.0
        for v in range(8):
            f = 1e-2 * _waves(X, rng, 4, 6)
            if v in (0, 7):
                prim[v] *= 1.0 + f
            else:
                prim[v] += f
    prim[1:4] *= prim[0]
    return prim.permute(1, 2, 3, 4, 0).contiguous()


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _heat_fields(case, g, seed):
    rng = np.random.default_rng(seed)
    X = _centers(g, ghost=False)
    Te = 1.0 + torch.exp(0.3 * _waves(X, rng, 8, 24))
    x, y, z = torch.broadcast_tensors(*X)
    r = torch.sqrt(x * x + y * y + z * z)
    rs = torch.clamp(r, min=1e-12)
    mr = z / rs
    B = torch.stack([3 * mr * x / rs, 3 * mr * y / rs, 3 * mr * z / rs - 1.0], dim=-1)
    b = B / torch.clamp(B.norm(dim=-1, keepdim=True), min=1e-300)
    return Te, b.contiguous(), (r >= 0.2).to(torch.uint8)


def _heat_params(case):
    return HeatParams(typePrecond=case["precond"], precondPrecision=case["sweeps"],
                      operatorPrecision=case["operator"])


_SHAPES = ((27, 16, 32), (32,), (27, 32, 32), (32,), (27, 32, 8), (8,))
_LR = 5e-4


def _learned_inputs(case, seed):
    """network inputs (smooth block vectors of unit RMS), targets (a smoothing
    of them, what an ILU correction looks like) and initial parameters"""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n = case["samples"]
    v = torch.randn((n, 8, 8, 8, 8), generator=gen, device="cuda")
    s = torch.nn.functional.avg_pool3d(v, 3, 1, 1)
    v = 0.5 * v + 2.0 * s
    v /= v.square().mean(dim=(1, 2, 3, 4), keepdim=True).sqrt()
    t = 0.6 * v + 0.8 * torch.nn.functional.avg_pool3d(v, 3, 1, 1)
    in16 = torch.zeros((n, 512, 16), device="cuda")
    in16[..., :8] = v.reshape(n, 8, 512).transpose(1, 2).bfloat16().float()
    tgt = t.reshape(n, 8, 512).transpose(1, 2).contiguous()
    p = []
    for q, s in enumerate(_SHAPES):
        w = torch.zeros(s, device="cuda")
        if len(s) == 3:
            w = torch.randn(s, generator=gen, device="cuda") * ((0.1 if q == 4 else 1.0) / math.sqrt(27 * s[1]))
            if q == 0:
                w[:, 8:] = 0.0
        p.append(w.reshape(-1))
    return in16, tgt, torch.cat(p)


def prepare(case, seed):
    if case["kind"] == "learned":
        return {"case": case, "in": [_pinned(t) for t in _learned_inputs(case, seed)]}
    kept = _solver(case)
    g = kept["grid"]
    st = {"case": case, "grid": g}
    if case["kind"] == "heat":
        st["in"] = [_pinned(t) for t in _heat_fields(case, g, seed)]
        return st
    st["in"] = _pinned(_state(case, g, seed))
    st["out"] = torch.empty(g.state_shape_fortran(), dtype=torch.float64, pin_memory=True).numpy()
    return st


# ---- one pass -----------------------------------------------------------------
def run(st):
    case = st["case"]
    if case["kind"] == "learned":
        in16, tgt, p = st["in"]
        net = LearnedPreconditioner(nSampleMax=case["samples"], seed=1)
        net.set_samples(in16, tgt)
        net.set_params(p)
        first, last = net.train(nEpoch=case["epochs"], batch=case["samples"], lr=_LR)
        return {"first": first, "last": last, "params": net.params()}
    kept = _solver(case)
    x = kept["solver"]
    if case["kind"] == "heat":
        h = HeatSolver(x, _heat_params(case), *st["in"])
        for _ in range(case["solves"]):
            h.advance_semi_impl()
        return {"Te": h.te()}
    x.set_state(st["in"])
    x.set_time(0.0, 0)
    if case["kind"] == "implicit":
        for _ in range(1 + case["steps"]):  # the first time-accurate step has Dt = 0
            kept["implicit"].advance_part_impl()
        return {"state": x.get_state(st["out"]), "time": x.time()[0]}
    x.advance(case["steps"])
    out = {"state": x.get_state(st["out"]), "time": x.time()[0]}
    if case["kind"] == "adaptive":
        out["criteria"] = x.amr_criteria(["gradlogp", "pjumpratio"])
    return out


# ---- what a pass cannot do without ----------------------------------------------
def _cells(case):
    if case["kind"] == "adaptive":  # about: the ball of finest blocks inside the root grid
        return 512 * (case["root"] ** 3 + 600 * case["level"])
    return case["nx"] * case["ny"] * case["nz"] * case.get("cells", 8) ** case.get("dim", 3)


def work(case):
    """Bytes and floating point operations of one pass.

    Explicit: a two-stage step reads U, writes U*, reads both and writes U
    (320 B per cell in FP64, 256 B with an FP32 U*); a one-stage step reads
    and writes U; the state crosses to the device once and comes back once.
    About 1300 additions and multiplications per cell and stage (the counted
    instructions of the 3D Linde / mc3 scheme), a third of them per dimension.
    Implicit and heat: the bytes of a solve with the usual number of Krylov
    iterations (30 matrix-vector products per implicit step, 40 per heat
    solve): operator, factors and the Gram-Schmidt reads of half a basis."""
    if case["kind"] == "learned":
        n = case["samples"]
        return {"bytes": n * 512 * (16 * 2 + 8 * 4) * case["epochs"], "flops": 3 * 57e6 * n * case["epochs"]}
    c = _cells(case)
    if case["kind"] == "implicit":
        per = 64 * 3 + (128 + (800 if case["precond"] == "BILU" else 0)) + 15 * 64
        return {"bytes": c * (128 + case["steps"] * 30 * per), "flops": c * case["steps"] * 30 * 2000}
    if case["kind"] == "heat":
        per = 17 + (41 if case["operator"] == "fp32" else 81) + (56 if case["precond"] == "BILU" else 0) + 15 * 8
        return {"bytes": c * (41 + case["solves"] * 40 * per), "flops": c * case["solves"] * 40 * 150}
    step = {"fp64": 320, "fp32": 256}[case["precision"]] if case.get("stages", 2) == 2 else 128
    ops = 1300 * case.get("dim", 3) / 3 * case.get("stages", 2)
    return {"bytes": c * (128 + case["steps"] * step), "flops": c * case["steps"] * ops}


def tolerance(case):
    """About four times what was measured between two correct ways to the same
    result.  Explicit FP64: 5e-16 (largest 4e-15) from exact(); FP32-bulk 9e-8
    (9e-7); the adaptive grid 6e-8 (8e-7) between FP32-bulk and FP64.
    Implicit: 2e-10 (5e-8) between one and four Gram-Schmidt steps a pass,
    with a margin for a residual rounded differently.  Heat: 1.8e-7 (1.4e-5)
    from exact(), what the solver's tolerance of 1e-6 leaves.  Training:
    1.2e-3 from exact(), the BF16 operands."""
    if case["kind"] == "learned":
        return {"rel": 5e-3, "max": 0.2}
    if case["kind"] == "heat":
        return {"rel": 7e-7, "max": 6e-5}
    if case["kind"] == "implicit":
        return {"rel": 2e-9, "max": 5e-7}
    if case["precision"] == "fp32":
        return {"rel": 4e-7, "max": 4e-6}
    return {"rel": 1e-14, "max": 2e-13}


# ---- the same in 64 bits, in plain torch ------------------------------------------
def exact(case, seed):
    if case["kind"] == "learned":
        return _exact_learned(case, seed)
    if case["kind"] == "heat":
        return _exact_heat(case, seed)
    if case["kind"] == "explicit":
        return _exact_explicit(case, seed)
    return None  # refined grids and Krylov iterates of a loose tolerance have no short plain form


def _to_global(a, g, n):
    """(block, k, j, i, ...) in x-fastest block order -> (nz, ny, nx, ...)"""
    r = list(g.nRoot)
    rest = a.shape[4:]
    a = a.reshape([r[2], r[1], r[0], g.nK, g.nJ, g.nI] + list(rest))
    a = a.permute([0, 3, 1, 4, 2, 5] + list(range(6, a.dim())))
    return a.reshape([n[2], n[1], n[0]] + list(rest))


def _from_global(a, g, ghost):
    """global cells -> blocks, ghost cells by wrapping (periodic) or copying the boundary cell (float)"""
    out = a
    for d, nc in enumerate((g.nI, g.nJ, g.nK)):
        n = g.nRoot[d] * nc
        ng = 2 if ghost and d < g.nDim else 0
        i = torch.arange(-ng, nc + ng, device=a.device)[None, :] + nc * torch.arange(g.nRoot[d], device=a.device)[:, None]
        i = i % n if g.typeBc[2 * d] == "periodic" else i.clamp(0, n - 1)
        dim = 2 - d if d < 2 else 0
        out = out.index_select(dim, i.reshape(-1))
    r = g.nRoot
    e = [(g.nI, g.nJ, g.nK)[d] + (4 if ghost and d < g.nDim else 0) for d in range(3)]
    rest = list(out.shape[3:])
    out = out.reshape([r[2], e[2], r[1], e[1], r[0], e[0]] + rest)
    out = out.permute([0, 2, 4, 1, 3, 5] + list(range(6, out.dim())))
    return out.reshape([r[0] * r[1] * r[2], e[2], e[1], e[0]] + rest)


def _limited(lim, beta, q0, q1, q2, q3):
    a, b, c = q1 - q0, q2 - q1, q3 - q2
    sab, sbc = 0.5 * (torch.sign(a) + torch.sign(b)), 0.5 * (torch.sign(b) + torch.sign(c))
    A, B, C = a.abs(), b.abs(), c.abs()
    if lim == "minmod":
        return q1 + 0.5 * sab * torch.minimum(A, B), q2 - 0.5 * sbc * torch.minimum(B, C)
    dl, dr = beta * torch.minimum(A, B), beta * torch.minimum(B, C)
    if lim == "mc":
        dl, dr = torch.minimum(dl, 0.5 * (a + b).abs()), torch.minimum(dr, 0.5 * (b + c).abs())
    else:
        dl, dr = torch.minimum(dl, (a + 2 * b).abs() / 3), torch.minimum(dr, (2 * b + c).abs() / 3)
    return q1 + 0.5 * sab * dl, q2 - 0.5 * sbc * dr


def _speed(S, D, gamma):
    rho, bn = S[0], S[4 + D]
    a2 = gamma * S[7] / rho
    f2 = a2 + (S[4] ** 2 + S[5] ** 2 + S[6] ** 2) / rho
    disc = torch.clamp(f2 * f2 - 4 * a2 * bn * bn / rho, min=0).sqrt()
    return (0.5 * (f2 + disc)).sqrt()


def _conserved(S, D, ig):
    """conserved variables (energy last) and their physical flux normal to D"""
    rho, u, B, p = S[0], S[1:4], S[4:7], S[7]
    un, bn = u[D], B[D]
    pt = 0.5 * (B * B).sum(0)
    e = ig * p + 0.5 * rho * (u * u).sum(0)
    U = torch.cat([rho[None], rho * u, B, (e + pt)[None]])
    m = rho * un
    F = torch.empty_like(U)
    F[0] = m
    F[1:4] = m * u - bn * B
    F[1 + D] += p + pt
    F[4:7] = un * B - u * bn
    F[7] = un * (e + p) + (F[4:7] * B).sum(0)
    return U, F


def _star(S, D, s, Un, Ptot12, Bn, ig):
    """the outer star state of HLLD on one side: density, tangential velocity and field, energy, u.B"""
    t1, t2 = (D + 1) % 3, (D + 2) % 3
    rho, un = S[0], S[1 + D]
    ut = torch.stack([S[1 + t1], S[1 + t2]])
    bt = torch.stack([S[4 + t1], S[4 + t2]])
    Ds = s - un
    pb = 0.5 * (Bn * Bn + (bt * bt).sum(0))
    ptot = S[7] + pb
    rs = Ds * rho / (s - Un)
    den = Ds * rho * (s - Un) - Bn * Bn
    plain = den < 1e-6
    inv = 1.0 / torch.where(plain, torch.ones_like(den), den)
    uts = torch.where(plain, ut, ut - Bn * bt * (Un - un) * inv)
    bts = torch.where(plain, bt, bt * (Ds * rho * Ds - Bn * Bn) * inv)
    e = ig * S[7] + pb + 0.5 * rho * (un * un + (ut * ut).sum(0))
    ub = un * Bn + (ut * bt).sum(0)
    ubs = Un * Bn + (uts * bts).sum(0)
    es = (Ds * e - ptot * un + Ptot12 * Un + Bn * (ub - ubs)) / (s - Un)
    return rs, uts, bts, es, ubs


def _hlld(L, R, D, gamma, ig):
    t1, t2 = (D + 1) % 3, (D + 2) % 3
    fl, fr = _speed(L, D, gamma), _speed(R, D, gamma)
    sL = torch.minimum(L[1 + D] - fl, R[1 + D] - fr)
    sR = torch.maximum(L[1 + D] + fl, R[1 + D] + fr)
    cmax = torch.maximum(sR, -sL)
    Bn = 0.5 * (L[4 + D] + R[4 + D])
    sg = torch.where(Bn < 0, -1.0, 1.0)
    pt = [S[7] + 0.5 * (Bn * Bn + S[4 + t1] ** 2 + S[4 + t2] ** 2) for S in (L, R)]
    dl, dr = (sL - L[1 + D]) * L[0], (sR - R[1 + D]) * R[0]
    Un = (dr * R[1 + D] - dl * L[1 + D] - pt[1] + pt[0]) / (dr - dl)
    P = (dr * pt[0] - dl * pt[1] + dr * dl * (R[1 + D] - L[1 + D])) / (dr - dl)
    a, b = _star(L, D, sL, Un, P, Bn, ig), _star(R, D, sR, Un, P, Bn, ig)
    ra, rb = a[0].abs().sqrt(), b[0].abs().sqrt()
    left = Un >= 0
    # inner star states
    w = 1.0 / (ra + rb)
    uti = (ra * a[1] + rb * b[1] + (b[2] - a[2]) * sg) * w
    bti = (ra * b[2] + rb * a[2] + (b[1] - a[1]) * ra * rb * sg) * w
    ubi = Un * Bn + (uti * bti).sum(0)
    outer = torch.where(left, Un - Bn.abs() / ra >= 0, Un + Bn.abs() / rb <= 0)
    pick = lambda q: torch.where(left, a[q], b[q])  # noqa: E731
    rho = pick(0)
    ut, bt = torch.where(outer, pick(1), uti), torch.where(outer, pick(2), bti)
    ub = torch.where(outer, pick(4), ubi)
    ei = torch.where(left, a[3] - ra * (a[4] - ubi) * sg, b[3] + rb * (b[4] - ubi) * sg)
    e = torch.where(outer, pick(3), ei)
    F = torch.zeros_like(L)
    F[0] = rho * Un
    F[1 + D] = rho * Un * Un - Bn * Bn + P
    for q, t in enumerate((t1, t2)):
        F[1 + t] = rho * Un * ut[q] - Bn * bt[q]
        F[4 + t] = Un * bt[q] - ut[q] * Bn
    F[7] = Un * (e + P) - Bn * ub
    F = torch.where(sL >= 0, _conserved(L, D, ig)[1], F)
    return torch.where((sL < 0) & (sR <= 0), _conserved(R, D, ig)[1], F), cmax


def _face_flux(L, R, D, flux, gamma, ig):
    if flux == "Rusanov":
        UL, FL = _conserved(L, D, ig)
        UR, FR = _conserved(R, D, ig)
        S = 0.5 * (L + R)
        cmax = S[1 + D].abs() + _speed(S, D, gamma)
        return 0.5 * (FL + FR - cmax * (UR - UL)), cmax
    L, R = L.clone(), R.clone()
    dB = 0.5 * (R[4 + D] - L[4 + D])
    L[4 + D] += dB
    R[4 + D] -= dB
    dE = 0.5 * (R[4 + D] + L[4 + D]) * dB
    if flux == "HLLD":
        F, cmax = _hlld(L, R, D, gamma, ig)
    else:
        UL, FL = _conserved(L, D, ig)
        UR, FR = _conserved(R, D, ig)
        S = 0.5 * (L + R)
        fs, u = _speed(S, D, gamma), S[1 + D]
        cmax = u.abs() + fs
        cl = torch.clamp(torch.minimum(L[1 + D] - _speed(L, D, gamma), u - fs), max=0)
        cr = torch.clamp(torch.maximum(R[1 + D] + _speed(R, D, gamma), u + fs), min=0)
        wL = cr / (cr - cl)
        F = (1 - wL) * FR + wL * FL - cr * (1 - wL) * (UR - UL)
    F[4 + D] -= cmax * dB
    F[7] -= cmax * dE
    return F, cmax


def _exact_stage(U, old, dt, case, g, n, sch):
    """one stage: U* from the stage input U (pressure form) and the step's
    first state; returns it and the smallest cell time step"""
    gamma, ig = sch.gamma, 1.0 / (sch.gamma - 1.0)
    W = U.clone()
    W[1:4] /= U[0]
    h = [(g.xyzMax[d] - g.xyzMin[d]) / (n[d] if d < g.nDim else 1) for d in range(3)]
    chg, vdt = torch.zeros_like(U), 0.0
    divb = 0.0
    for D in range(g.nDim):
        ax = 3 - D
        i = torch.arange(-2, n[D] + 2, device=U.device)
        i = i % n[D] if g.typeBc[2 * D] == "periodic" else i.clamp(0, n[D] - 1)
        q = W.index_select(ax, i)
        s = [q.narrow(ax, m, n[D] + 1) for m in range(4)]
        if sch.nOrder == 1:
            L, R = s[1], s[2]
        else:
            L, R = _limited(case["limiter"], sch.limiterBeta, *s)
        F, cmax = _face_flux(L, R, D, case["flux"], gamma, ig)
        chg += (F.narrow(ax, 0, n[D]) - F.narrow(ax, 1, n[D])) / h[D]
        bn = (L[4 + D] + R[4 + D]) * 0.5
        divb = divb + (bn.narrow(ax - 1, 1, n[D]) - bn.narrow(ax - 1, 0, n[D])) / h[D]
        vdt = vdt + torch.maximum(cmax.narrow(ax - 1, 0, n[D]), cmax.narrow(ax - 1, 1, n[D])) / h[D]
    if sch.useDivbSource:
        u, B = W[1:4], W[4:7]
        chg[1:4] -= divb * B
        chg[4:7] -= divb * u
        chg[7] -= divb * (u * B).sum(0)
    low = float((1.0 / vdt).min())
    if dt == 0.0:
        return old.clone(), low
    e = ig * old[7] + 0.5 * (old[1:4] ** 2).sum(0) / old[0] + 0.5 * (old[4:7] ** 2).sum(0)
    new = old + dt * chg
    e = e + dt * chg[7]
    new[7] = (sch.gamma - 1.0) * (e - 0.5 * (new[4:7] ** 2).sum(0) - 0.5 * (new[1:4] ** 2).sum(0) / new[0])
    return new, low


def _exact_explicit(case, seed):
    g, sch = _grid(case), _scheme(case)
    n = [(g.nI, g.nJ, g.nK)[d] * g.nRoot[d] for d in range(3)]
    st = _state(case, g, seed)
    U = _to_global(st[g.interior_slices()], g, n).permute(3, 0, 1, 2).contiguous()
    t, low = 0.0, 0.0
    for step in range(case["steps"]):
        dt = sch.dtFixed if sch.useDtFixed else (0.0 if step == 0 else low)
        old = U
        for s in range(1, sch.nStage + 1):
            f = sch.cfl * s / sch.nStage if sch.useHalfStep else sch.cfl
            U, low = _exact_stage(U, old, f * dt, case, g, n, sch)
        for _ in range(sch.nStage):
            t += sch.cfl * dt / sch.nStage
    return {"state": _from_global(U.permute(1, 2, 3, 0), g, True).cpu().numpy(), "time": t}


def _exact_heat(case, seed):
    g, p = _grid(case), _heat_params(case)
    n = [8 * r for r in g.nRoot]
    Te, b, used = _heat_fields(case, g, seed)
    Te = _to_global(Te, g, n)
    b = _to_global(b, g, n).permute(3, 0, 1, 2)
    used = _to_global(used, g, n).bool()
    dx = [1.0 / m for m in n]
    V = dx[0] * dx[1] * dx[2]
    pad = lambda a: torch.nn.functional.pad(a[None, None], (1,) * 6, mode="replicate")[0, 0]  # noqa: E731
    pb = torch.stack([pad(b[d]) for d in range(3)])

    def faces(a, D):  # the cells on the two sides of every face normal to D, one transverse ghost layer kept
        ax = 2 - D
        return a.narrow(ax, 0, n[D] + 1), a.narrow(ax, 1, n[D] + 1)

    def inner(a, D, off=None):  # drop the transverse ghost layers, shifted by one cell along `off`
        for e in range(3):
            if e != D:
                a = a.narrow(2 - e, 1 + (off[1] if off and off[0] == e else 0), n[e])
        return a

    def tensor(T):
        hc = pad(p.heatCondPar * T ** 2.5)
        K = []
        for D in range(3):
            l, r = faces(hc, D)
            c = V / dx[D] * 0.5 * inner(l + r, D)
            row = []
            for e in range(3):
                bb = p.fieldAligned * pb[D] * pb[e] + ((1.0 - p.fieldAligned) if e == D else 0.0)
                l, r = faces(bb, D)
                row.append(c * 0.5 * inner(l + r, D))
            K.append(row)
        return K

    def residual(K, S):
        S = pad(S)
        res = 0.0
        for D in range(3):
            l, r = faces(S, D)
            f = K[D][D] * inner(r - l, D) / dx[D]
            for e in range(3):
                if e != D:
                    f = f + K[D][e] * 0.25 / dx[e] * (inner(l + r, D, (e, 1)) - inner(l + r, D, (e, -1)))
            res = res + (f.narrow(2 - D, 1, n[D]) - f.narrow(2 - D, 0, n[D])) / V
        return res

    zero = torch.zeros_like(Te)
    for _ in range(case["solves"]):
        K = tensor(Te)
        A = lambda x: torch.where(used, V * (x * p.cv / p.dt - p.semiImplCoeff * residual(K, torch.where(used, x, zero))),  # noqa: E731
                                  V * x * p.cv / p.dt)
        rhs = torch.where(used, V * residual(K, Te), zero)
        dg = V * p.cv / p.dt + sum((K[d][d].narrow(2 - d, 0, n[d]) + K[d][d].narrow(2 - d, 1, n[d])) / dx[d]
                                   for d in range(3)) * p.semiImplCoeff
        # BiCGStab with the diagonal as preconditioner
        x, r = zero.clone(), rhs.clone()
        r0, rho, al, om, v, q = r.clone(), 1.0, 1.0, 1.0, zero, zero
        for _ in range(2000):
            rn = float((r0 * r).sum())
            q = r + (rn / rho) * (al / om) * (q - om * v)
            rho = rn
            z = q / dg
            v = A(z)
            al = rho / float((r0 * v).sum())
            s = r - al * v
            zs = s / dg
            t = A(zs)
            om = float((t * s).sum() / (t * t).sum())
            x = x + al * z + om * zs
            r = s - om * t
            if float(r.norm()) <= 1e-11 * float(rhs.norm()):
                break
        Te = torch.where(used, Te + x, Te)
    return {"Te": _from_global(Te, g, False).cpu().numpy()}


def _exact_learned(case, seed):
    in16, tgt, flat = _learned_inputs(case, seed)
    n = case["samples"]
    x = in16.double().reshape(n, 8, 8, 8, 16).permute(0, 4, 1, 2, 3)[:, :8]
    y = tgt.double().reshape(n, 8, 8, 8, 8).permute(0, 4, 1, 2, 3)
    y = y / y.square().mean().sqrt()
    w, o = [], 0
    for s in _SHAPES:
        m = int(np.prod(s))
        if len(s) == 3:
            w.append(flat[o:o + m].double().reshape(s))
        o += m
    mom = [(torch.zeros_like(a), torch.zeros_like(a)) for a in w]
    losses = []
    conv = lambda a, k: torch.nn.functional.conv3d(a, k, padding=1)  # noqa: E731
    for e in range(1, case["epochs"] + 1):
        grads, loss = [torch.zeros_like(a) for a in w], 0.0
        for c in range(0, n, 128):
            ws = [a.clone().requires_grad_(True) for a in w]
            k = [a.reshape(3, 3, 3, a.shape[1], a.shape[2]).permute(4, 3, 0, 1, 2) for a in ws]
            d = conv(conv(conv(x[c:c + 128], k[0][:, :8]), k[1]), k[2]) - y[c:c + 128]
            part = d.square().sum() / y.numel()
            for q, gq in enumerate(torch.autograd.grad(part, ws)):
                grads[q] += gq
            loss += float(part)
        losses.append(loss)
        for q, a in enumerate(w):
            m, v = mom[q]
            m.mul_(0.9).add_(grads[q], alpha=0.1)
            v.mul_(0.999).addcmul_(grads[q], grads[q], value=0.001)
            a -= _LR * (m / (1 - 0.9 ** e)) / ((v / (1 - 0.999 ** e)).sqrt() + 1e-8)
    out = []
    for s, a in zip(_SHAPES[::2], w):
        out += [a.reshape(-1), torch.zeros(s[2], dtype=torch.float64, device=a.device)]
    return {"first": losses[0], "last": losses[-1], "params": torch.cat(out).cpu().numpy()}
