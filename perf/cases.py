"""Workloads that stand for what this framework is used for, with their inputs,
their float64 reference values and the work they cannot do without.

Each case is a dict of plain values whose ``kind`` names the user program:

  tube     a whole small 1D run: upload, ``evolve`` to the final time, read back
  blast    the same in 2D (Sedov blast between reflecting walls)
  plane    ``evolve`` of a device-resident 2D grid, ``steps`` steps a pass
  box      ``evolve`` of a device-resident 3D grid, ``steps`` steps a pass
  batch    ``Batch.run_steps`` over many boxes, every state read back
  adjoint  forward run and reverse sweep of a Kelvin-Helmholtz box
  muscl    the unsplit MUSCL scheme on a 3D grid with periodic ghost zones
  gravity  ``evolve`` of a self-gravitating periodic cube (a solve per step)
  amr      ``evolve`` of a composite mesh refined around a blast
  faces    ``compute_face_fluxes`` on host arrays, the batched flux drop-in

The grids that stay on the device march on from pass to pass, as a program that
steps a simulation does; the first pass starts from the inputs themselves.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "vespa.jl_b200"))
import vespa_b200 as vb  # noqa: E402
from vespa_b200 import amr, flux, gravity, muscl  # noqa: E402

BCS = {"p": vb.Periodic, "o": vb.Outflow, "r": vb.Reflecting}
DEV = "cuda"
L2_BYTES = 126e6
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the shock-tube run at the problem's own default size: latency of many
        # tiny steps, from upload to read-back
        dict(name="tube_128", kind="tube", nx=128),
        # the 2D blast at the problem's default size, walls on every side
        dict(name="blast_64", kind="blast", nx=64),
        # 2D throughput grid of the benchmark, mixed precision
        dict(name="plane_4096_mixed", kind="plane", nx=4096, ny=4096, prec="mixed", bc="pp", steps=8),
        # the headline 3D periodic cube in both precisions
        dict(name="box_256_mixed", kind="box", nx=256, ny=256, nz=256, prec="mixed", bc="ppp", steps=8),
        dict(name="box_256_fp64", kind="box", nx=256, ny=256, nz=256, prec="fp64", bc="ppp", steps=4),
        # an everyday 3D box with sides that fit no tile and every kind of wall
        dict(name="box_ragged_fp64", kind="box", nx=150, ny=90, nz=75, prec="fp64", bc="pro", steps=8),
        # many small independent boxes, stepped together and read back
        dict(name="batch_12_mixed", kind="batch", sides="32,32,32,48,48,48,64,64,64,96,96,96",
             prec="mixed", steps=32),
        # gradient of a Kelvin-Helmholtz run through its checkpoints
        dict(name="adjoint_512", kind="adjoint", nx=512, steps=40, every=20),
        # the second scheme on a 3D grid
        dict(name="muscl_192", kind="muscl", nx=192, ny=192, nz=192, ng=3, steps=4),
        # self-gravity with the multigrid-preconditioned solve
        dict(name="gravity_256_fp64", kind="gravity", nx=256, prec="fp64", precond="mg", steps=2),
        # the refined mesh around a blast, single rate
        dict(name="amr_48", kind="amr", nx=48, levels=4, steps=64),
        # one stage's faces of a 40^3 box handed over by a host program
        dict(name="faces_200k", kind="faces", nf=200000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bc(rng, nd):
    if rng.random() < 0.5:
        return "p" * nd
    return "".join(rng.choice("por") for _ in range(nd))


def draw(rng):
    kind = rng.choice(["tube", "blast", "plane", "plane", "box", "box", "box", "batch", "adjoint",
                       "muscl", "gravity", "amr", "faces"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "tube":
        return dict(kind=kind, nx=_log(rng, 64, 1024))
    if kind == "blast":
        return dict(kind=kind, nx=_log(rng, 32, 112))
    if kind == "plane":
        nx, ny = _log(rng, 200, 4096), _log(rng, 200, 4096)
        if rng.random() < 0.5:
            nx = min(4096, -(-nx // 256) * 256)
        return dict(kind=kind, nx=nx, ny=ny, prec=prec, bc=_bc(rng, 2), steps=8)
    if kind == "box":
        side = _log(rng, 24, 224)
        n = [max(17, int(side * rng.uniform(0.7, 1.15))) for _ in range(3)]
        if rng.random() < 0.5:
            n = [-(-v // 16) * 16 for v in n]
        n = [min(256, v) for v in n]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], prec=prec, bc=_bc(rng, 3), steps=4)
    if kind == "batch":
        k = rng.randint(4, 12)
        sides = ",".join(str(rng.choice((32, 48, 64, 96))) for _ in range(k))
        return dict(kind=kind, sides=sides, prec=prec, steps=32)
    if kind == "adjoint":
        return dict(kind=kind, nx=_log(rng, 64, 512), steps=rng.choice((20, 40)), every=rng.choice((1, 10, 20)))
    if kind == "muscl":
        n = [_log(rng, 40, 192) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], ng=rng.choice((2, 3)), steps=4)
    if kind == "gravity":
        if rng.random() < 0.25:
            return dict(kind=kind, nx=_log(rng, 24, 96), prec=prec, precond="none", steps=2)
        return dict(kind=kind, nx=2 * _log(rng, 16, 128), prec=prec, precond="mg", steps=2)
    if kind == "amr":
        return dict(kind=kind, nx=rng.randint(32, 56), levels=rng.randint(2, 4), steps=64)
    return dict(kind="faces", nf=_log(rng, 1000, 1000000))


# ----------------------------------------------------------------- the inputs
def _dims(c):
    if c["kind"] in ("tube",):
        return (c["nx"],)
    if c["kind"] in ("blast", "adjoint"):
        return (c["nx"], c["nx"])
    if c["kind"] == "plane":
        return (c["nx"], c["ny"])
    if c["kind"] == "gravity":
        return (c["nx"],) * 3
    return (c["nx"], c["ny"], c["nz"])


def _bcstr(c):
    k = c["kind"]
    return {"tube": "o", "blast": "rr", "adjoint": "pp", "gravity": "ppp"}.get(k) or c["bc"]


def _gamma(c):
    return {"tube": 1.4, "blast": 1.4, "adjoint": 1.4, "amr": 1.4, "batch": 1.4, "faces": 1.4}.get(
        c["kind"], 5.0 / 3.0)


def _cfl(c):
    return 0.3 if c["kind"] in ("blast", "amr") else 0.4


def _tfinal(c):
    return {"tube": 0.2, "blast": 0.05}.get(c["kind"], math.inf)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _u(g, n, lo, hi):
    return torch.rand(n, generator=g, device=DEV, dtype=F64) * (hi - lo) + lo


def _centres(dims):
    """Cell-centre coordinates on the unit box, flat, x fastest."""
    ax = [(torch.arange(n, device=DEV, dtype=F64) + 0.5) / n for n in dims]
    grids = torch.meshgrid(*reversed(ax), indexing="ij")
    return [g.reshape(-1) for g in reversed(grids)]


def _prim2cons(W, gamma):
    r, u, v, w, p = W
    return torch.stack([r, r * u, r * v, r * w, p / (gamma - 1.0) + 0.5 * r * (u * u + v * v + w * w)])


def _smooth_random(dims, seed, gamma, amp=0.5):
    """Smooth density modes with cell-by-cell random velocity and pressure: the
    framework's own throughput state."""
    g, r = _gen(seed), random.Random(seed)
    x = _centres(dims)
    n = x[0].numel()
    rho = torch.zeros(n, device=DEV, dtype=F64)
    for _ in range(8):
        k = [r.randint(-4, 4) for _ in dims]
        ph = r.uniform(0, 2 * math.pi)
        rho += torch.sin(2 * math.pi * sum(a * b for a, b in zip(k, x)) + ph)
    zero = torch.zeros(n, device=DEV, dtype=F64)
    vel = [_u(g, n, -amp, amp) if d < len(dims) else zero for d in range(3)]
    return _prim2cons(torch.stack([1.0 + 0.3 * rho / 8, *vel, _u(g, n, 0.8, 1.2)]), gamma)


def _two_states(dims, seed, index, gamma):
    """A random plane between two gas states (a Riemann problem in a box)."""
    r = random.Random(seed * 1000 + index)
    x = _centres(dims)
    nrm = [r.uniform(-1, 1) for _ in range(3)]
    left = sum(a * (b - 0.5) for a, b in zip(nrm, x)) < r.uniform(-0.1, 0.1)
    st = [[r.uniform(0.3, 3), *(r.uniform(-0.4, 0.4) for _ in range(3)), r.uniform(0.5, 3)] for _ in range(2)]
    return _prim2cons(torch.stack([torch.where(left, a, b).to(F64) for a, b in zip(*st)]), gamma)


def _tube(c, seed):
    r = random.Random(seed)
    (x,) = _centres(_dims(c))
    one, left = torch.ones_like(x), x < 0.5
    rho = torch.where(left, 1.0 * one, 0.125 * r.uniform(0.9, 1.1) * one)
    p = torch.where(left, 1.0 * one, 0.1 * r.uniform(0.9, 1.1) * one)
    return _prim2cons(torch.stack([rho, 0 * x, 0 * x, 0 * x, p]), _gamma(c))


def _blast(c, seed):
    x, y = _centres(_dims(c))
    one = torch.ones_like(x)
    r0 = 2.0 / c["nx"]
    p = torch.where(torch.hypot(x - 0.5, y - 0.5) <= r0, 0.4 / (math.pi * r0 * r0) * one, 1e-5 * one)
    rho = 1 + 1e-2 * _u(_gen(seed), x.numel(), -1, 1)
    return _prim2cons(torch.stack([rho, 0 * x, 0 * x, 0 * x, p]), _gamma(c))


def _kelvin_helmholtz(c, seed):
    """The two-band shear layer with a seeded texture (a generic state: no
    limiter sits exactly on a tie)."""
    x, y = _centres(_dims(c))
    g, n = _gen(seed), x.numel()
    band = ((y - 0.5).abs() < 0.25).to(F64)
    t = 1e-2
    rho = (1 + band) * (1 + t * _u(g, n, -1, 1))
    ux = band - 0.5 + t * _u(g, n, -1, 1)
    uy = 0.01 * torch.sin(4 * math.pi * x) + 1e-3 * _u(g, n, -1, 1)
    return _prim2cons(torch.stack([rho, ux, uy, 0 * x, 2.5 * (1 + t * _u(g, n, -1, 1))]), _gamma(c))


def _state(c, seed):
    k = c["kind"]
    if k == "tube":
        return _tube(c, seed)
    if k == "blast":
        return _blast(c, seed)
    if k == "adjoint":
        return _kelvin_helmholtz(c, seed)
    return _smooth_random(_dims(c), seed, _gamma(c), 0.2 if k == "gravity" else 0.5)


class _Device:
    """The library's device buffer as a CUDA array; keeps its owner alive."""

    def __init__(self, ptr, shape, owner):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3, "strides": None}
        self.owner = owner


def _view(ptr, shape, owner):
    return torch.as_tensor(_Device(ptr, shape, owner), device=DEV)


def _problem(c, dims, bcs):
    return vb.Problem(name=c["kind"], dims=dims, domain=((0.0, 1.0),) * len(dims), gamma=_gamma(c),
                      bcs=tuple((BCS[b], BCS[b]) for b in bcs), init=lambda x, y, z: (1.0, 0.0, 0.0, 0.0, 1.0),
                      tfinal=_tfinal(c), cfl=_cfl(c))


def _simulation(c, dims, bcs, U, prec):
    prob = _problem(c, dims, bcs)
    return vb.Simulation(vb.B200Mesh(prob.dims, prob.domain), prob, precision=prec, initial=U.cpu().numpy())


def _pinned(shape):
    return torch.empty(shape, dtype=F64, pin_memory=True).numpy()


GRAV_G = 0.1  # well inside the Jeans-stable range of the inputs
MUSCL = dict(gamma=5.0 / 3.0, theta=1.5, small_rho=1e-10, bc="periodic")


def _muscl_state(c, seed):
    """Conserved D, S, Tau of the smooth random state, ghost zones included."""
    return _smooth_random(_dims(c), seed, MUSCL["gamma"])


def _muscl_dx(c):
    return 1.0 / max(_dims(c))


def _muscl_dt(c):
    return 0.2 * _muscl_dx(c) / 3.0


AMR_RADII = (0.38, 0.28, 0.18, 0.10)


def _amr_state(x, y, seed, gamma):
    g = _gen(seed)
    r2 = (x - 0.5) ** 2 + (y - 0.5) ** 2
    n = x.numel()
    rho = 1 + 0.2 * torch.sin(6 * x + 4 * y) + 1e-2 * _u(g, n, -1, 1)
    p = 0.1 + 3 * torch.exp(-r2 / 0.01) + 1e-3 * _u(g, n, -1, 1)
    return _prim2cons(torch.stack([rho, 0.1 * torch.sin(5 * y), 0.1 * torch.cos(5 * x), 0 * x, p]), gamma)


def _face_states(c, seed):
    g, n = _gen(seed), c["nf"]

    def side():
        return torch.stack([_u(g, n, 0.2, 2), _u(g, n, -2, 2), _u(g, n, -2, 2), _u(g, n, -2, 2),
                            _u(g, n, 0.1, 2)], dim=1).contiguous()
    ax = torch.randint(1, 4, (n,), generator=g, device=DEV, dtype=torch.int32)
    return side(), side(), ax


def prepare(case, seed):
    c, k = case, case["kind"]
    if k in ("tube", "blast"):
        U0 = _state(c, seed)
        sim = _simulation(c, _dims(c), _bcstr(c), U0, "fp64")
        return dict(c=c, sim=sim, U0=U0.cpu().numpy())
    if k in ("plane", "box", "gravity"):
        sim = _simulation(c, _dims(c), _bcstr(c), _state(c, seed), c["prec"])
        if k == "gravity":
            gravity.enable_gravity(sim, G=GRAV_G, tol=1e-8, precond=c["precond"])
        return dict(c=c, sim=sim, U=_view(sim.device_state_ptr(), (5, sim.ncell), sim))
    if k == "batch":
        sides = [int(s) for s in c["sides"].split(",")]
        probs = [_problem(c, (s, s, s), "ooo") for s in sides]
        U = [_two_states((s, s, s), seed, i, _gamma(c)).cpu().numpy() for i, s in enumerate(sides)]
        return dict(c=c, batch=vb.Batch(probs, precision=c["prec"], initial=U),
                    out=[_pinned((5, s ** 3)) for s in sides])
    if k == "adjoint":
        sim = _simulation(c, _dims(c), _bcstr(c), _state(c, seed), "fp64")
        adj = vb.Adjoint(sim, c["steps"], c["every"])
        lam = _u(_gen(seed + 77), 5 * sim.ncell, -1, 1).reshape(5, -1).cpu().numpy()
        return dict(c=c, sim=sim, adj=adj, lam=lam, U=_view(sim.device_state_ptr(), (5, sim.ncell), sim))
    if k == "muscl":
        g = muscl.MusclGrid(_dims(c), c["ng"])
        g.upload(_muscl_state(c, seed).cpu().numpy())
        return dict(c=c, grid=g, U=_view(g.device_state_ptr(), (5, g.N), g))
    if k == "amr":
        n = c["nx"]
        prob = _problem(c, (n, n), "rr")
        sim = amr.AmrSimulation(amr.AmrMesh(prob.dims, prob.domain), prob)
        for lev in range(c["levels"]):
            x, y = sim.cell_centers()
            at, _ = sim.leaves()
            sim.refine(np.flatnonzero((at == lev) & ((x - 0.5) ** 2 + (y - 0.5) ** 2 < AMR_RADII[lev] ** 2)))
        x, y = (torch.from_numpy(v).to(DEV) for v in sim.cell_centers())
        sim.upload(_amr_state(x, y, seed, _gamma(c)).cpu().numpy())
        return dict(c=c, sim=sim)
    WL, WR, ax = (t.cpu().numpy() for t in _face_states(c, seed))
    return dict(c=c, backend=flux.B200Flux(), WL=WL, WR=WR, ax=ax, F=np.empty_like(WL))


# ------------------------------------------------------------------- one pass
def run(state):
    c = state["c"]
    k = c["kind"]
    if k in ("tube", "blast"):
        sim = state["sim"]
        sim.upload(state["U0"])
        sim.set_time(0.0, 0)
        vb.evolve(sim)
        return sim.state()
    if k in ("plane", "box", "gravity"):
        vb.evolve(state["sim"], max_steps=c["steps"])
        return state["U"]
    if k == "batch":
        b = state["batch"]
        b.run_steps(c["steps"])
        return [b.state(i, out) for i, out in enumerate(state["out"])]
    if k == "adjoint":
        adj = state["adj"]
        adj.forward(max_steps=c["steps"])
        return {"state": state["U"], "gradient": adj.backward(state["lam"])}
    if k == "muscl":
        state["grid"].run_async(c["steps"], dt=_muscl_dt(c), dx=_muscl_dx(c), **MUSCL)
        return state["U"]
    if k == "amr":
        amr.evolve(state["sim"], max_steps=c["steps"])
        return state["sim"].state()
    return flux.compute_face_fluxes(state["backend"], _gamma(c), state["F"], state["WL"], state["WR"], state["ax"])


# ------------------------------------------------- work, tolerance, reference
def _amr_leaves(c):
    n, cells = c["nx"], 1.0 * c["nx"] ** 2
    for lev in range(c["levels"]):
        cells += 3 * math.pi * (AMR_RADII[lev] * n * 2 ** lev) ** 2
    return cells


def work(case):
    """Bytes: five float64 fields read once and written once, per step where the
    state is larger than L2 (each step's dt depends on the whole of the last
    one) and per pass where it is not.  Flops: PLM, HLLC and the update of both
    stages, per axis."""
    c, k = case, case["kind"]
    if k == "faces":
        return {"bytes": c["nf"] * 124.0, "flops": c["nf"] * 75.0}
    if k == "batch":
        cells = float(sum(int(s) ** 3 for s in c["sides"].split(",")))
        nd = 3
    elif k == "amr":
        cells, nd = _amr_leaves(c), 2
    else:
        cells, nd = float(np.prod(_dims(c))), len(_dims(c))
    steps = c.get("steps") or {"tube": 1.1, "blast": 9.0}[k] * c["nx"]
    passes = steps if cells * 40 > L2_BYTES else 1
    flops = cells * steps * 2 * (120.0 * nd + 50.0)
    bytes_ = cells * 80.0 * passes
    if k == "adjoint":
        flops, bytes_ = 4 * flops, 2 * bytes_
    if k == "gravity":  # a preconditioned iteration at the least: phi and its residual
        flops, bytes_ = flops + cells * steps * 100, bytes_ + cells * steps * 16
    return {"bytes": bytes_, "flops": flops}


# Relative errors against exact(), about four times what was measured.  float64:
# 1e-16 to 1e-15 (rounding of a few to a few hundred steps; a gravity step adds
# the solver's 1e-8 of an acceleration times dt, at most 1e-12).  Mixed: 4e-8 to
# 1e-7 on smooth states from float32 reconstruction and fluxes, and up to 3e-6 in
# the batch's strong jumps, where a limiter's choice near a tie travels on.
TOL = {"tube": 4e-15, "blast": 1e-14, "plane": 2e-15, "box": 2e-15, "batch": 1e-14, "adjoint": 1e-14,
       "muscl": 1e-15, "amr": 4e-15, "faces": 1e-15, "gravity": 4e-12}


def tolerance(case):
    if case.get("prec") == "mixed":
        return {"rel": 1.2e-5 if case["kind"] == "batch" else 4e-7}
    return {"rel": TOL[case["kind"]]}


def _c2p(U, gamma):
    r = U[0]
    v = U[1:4] / r
    ke = 0.5 * r * (v * v).sum(0)
    return torch.cat([r[None], v, torch.maximum((gamma - 1) * (U[4] - ke), 1e-12 * ke)[None]])


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _hllc(L, R, d, g):
    """HLLC flux normal to axis d with Davis speeds; states (rho, v, p)."""
    def side(W):
        un = W[1 + d]
        E = W[4] / (g - 1) + 0.5 * W[0] * (W[1:4] * W[1:4]).sum(0)
        U = [W[0], W[0] * W[1], W[0] * W[2], W[0] * W[3], E]
        F = [u * un for u in U]
        F[1 + d] = F[1 + d] + W[4]
        F[4] = F[4] + W[4] * un
        return un, torch.sqrt(g * W[4] / W[0]), E, U, F
    uL, cL, EL, UL, FL = side(L)
    uR, cR, ER, UR, FR = side(R)
    SL, SR = torch.minimum(uL - cL, uR - cR), torch.maximum(uL + cL, uR + cR)
    aL, aR = L[0] * (SL - uL), R[0] * (SR - uR)
    Ss = (R[4] - L[4] + uL * aL - uR * aR) / (aL - aR)

    def star(W, S, un, E, U, F):
        f = W[0] * (S - un) / (S - Ss)
        V = [W[1], W[2], W[3]]
        V[d] = Ss
        Us = [f, f * V[0], f * V[1], f * V[2], f * (E / W[0] + (Ss - un) * (Ss + W[4] / (W[0] * (S - un))))]
        return [a + S * (b - e) for a, b, e in zip(F, Us, U)]
    sl, sr = star(L, SL, uL, EL, UL, FL), star(R, SR, uR, ER, UR, FR)
    return torch.stack([torch.where(SL >= 0, a, torch.where(SR <= 0, b, torch.where(Ss >= 0, x, y)))
                        for a, b, x, y in zip(FL, FR, sl, sr)])


def _pad(W, ax, d, bc):
    """Two ghost cells on each side along tensor axis `ax` (space axis d)."""
    n = W.shape[ax]
    if bc == "p":
        lo, hi = W.narrow(ax, n - 2, 2), W.narrow(ax, 0, 2)
    else:
        lo, hi = W.narrow(ax, 0, 2).flip(ax), W.narrow(ax, n - 2, 2).flip(ax)
        if bc == "r":
            s = torch.ones(5, device=W.device, dtype=F64)
            s[1 + d] = -1
            s = s.reshape(5, *([1] * (W.dim() - 1)))
            lo, hi = lo * s, hi * s
    return torch.cat([lo, W, hi], dim=ax)


def _rate(U, g, bcs, w):
    """-div F of a uniform grid, U as (5, nz, ny, nx)."""
    W = _c2p(U, g)
    out = torch.zeros_like(U)
    for d in range(U.dim() - 1):
        ax = U.dim() - 1 - d
        P = _pad(W, ax, d, bcs[d])
        n = U.shape[ax]
        D = P.narrow(ax, 1, n + 3) - P.narrow(ax, 0, n + 3)
        s = 0.5 * _minmod(D.narrow(ax, 0, n + 2), D.narrow(ax, 1, n + 2))
        M = P.narrow(ax, 1, n + 2)
        F = _hllc((M + s).narrow(ax, 0, n + 1), (M - s).narrow(ax, 1, n + 1), d, g)
        out = out - (F.narrow(ax, 1, n) - F.narrow(ax, 0, n)) / w[d]
    return out


def _fastest(U, g, w):
    W = _c2p(U, g)
    c = torch.sqrt(g * W[4] / W[0])
    return max(float(((W[1 + d].abs() + c) / w[d]).max()) for d in range(U.dim() - 1))


def _march(U, c, bcs, steps=None, tfinal=math.inf, source=None, free_fall=0.0, keep=None):
    """CFL-limited SSP-RK2 steps; `source(U)` is evaluated once per step."""
    g, w = _gamma(c), [1.0 / n for n in reversed(U.shape[1:])]
    t, done = 0.0, 0
    while (steps is None or done < steps) and t < tfinal * (1 - 1e-12):
        rate = _fastest(U, g, w)
        if free_fall:
            rate = max(rate, math.sqrt(4 * math.pi * free_fall * float(U[0].max())) / 0.5)
        dt = min(_cfl(c) / rate, tfinal - t)
        acc = source(U) if source else None
        if keep is not None:
            keep.append((U, dt))
        U = _step(U, dt, g, bcs, w, acc)
        t, done = t + dt, done + 1
    return U


def _step(U, dt, g, bcs, w, acc=None):
    def rate(V):
        r = _rate(V, g, bcs, w)
        if acc is not None:
            z = torch.zeros_like(V[:1])
            r = r + torch.cat([z, V[:1] * acc, (V[1:4] * acc).sum(0, keepdim=True)])
        return r
    V = U + dt * rate(U)
    return 0.5 * U + 0.5 * (V + dt * rate(V))


def _grid(U, dims):
    return U.reshape(5, *reversed(dims))


def _poisson_accel(n, G):
    """g = -grad phi of the seven-point periodic Poisson problem, by FFT."""
    h = 1.0 / n
    k = (2 * torch.cos(2 * math.pi * torch.arange(n, device=DEV, dtype=F64) / n) - 2) / (h * h)
    lam = k[:, None, None] + k[None, :, None] + k[None, None, :n // 2 + 1]
    lam[0, 0, 0] = 1.0

    def accel(U):
        f = torch.fft.rfftn(4 * math.pi * G * (U[0] - U[0].mean())) / lam
        f[0, 0, 0] = 0
        phi = torch.fft.irfftn(f, s=(n, n, n))
        return torch.stack([-(phi.roll(-1, a) - phi.roll(1, a)) / (2 * h) for a in (2, 1, 0)])
    return accel


def _exact_adjoint(c, seed):
    dims = _dims(c)
    lam = _u(_gen(seed + 77), 5 * dims[0] * dims[1], -1, 1).reshape(5, *dims)
    tape, w = [], [1.0 / n for n in dims]
    UT = _march(_grid(_state(c, seed), dims), c, "pp", steps=c["steps"], keep=tape)
    for U, dt in reversed(tape):
        U = U.detach().requires_grad_(True)
        (lam,) = torch.autograd.grad(_step(U, dt, _gamma(c), "pp", w), U, lam)
    return {"state": UT.reshape(5, -1), "gradient": lam.reshape(5, -1).cpu().numpy()}


def _exact_muscl(c, seed):
    g, th, floor, ng = MUSCL["gamma"], MUSCL["theta"], MUSCL["small_rho"], c["ng"]
    dims, dtdx = _dims(c), _muscl_dt(c) / _muscl_dx(c)
    U = _grid(_muscl_state(c, seed), dims).clone()

    def fill(U):
        for a in (3, 2, 1):
            n = U.shape[a]
            act = n - 2 * ng
            U.narrow(a, 0, ng).copy_(U.narrow(a, act, ng).clone())
            U.narrow(a, ng + act, ng).copy_(U.narrow(a, ng, ng).clone())

    def minmod3(a, b, q):
        s = [torch.where(v > 0, 1.0, -1.0).to(F64) for v in (a, b, q)]
        return 0.25 * (s[0] + s[1]) * (s[0] + s[2]).abs() * torch.minimum(a.abs(), torch.minimum(b.abs(), q.abs()))

    def plm(m, v, p):
        return v + 0.5 * minmod3((v - m) * th, (p - v) * th, 0.5 * (p - m))

    def parts(W, d):
        r, e, un = W[0], W[1], W[2 + d]
        p = (g - 1) * r * e
        c_ = torch.sqrt(g * p / r)
        E = r * (e + 0.5 * (W[2:5] * W[2:5]).sum(0))
        Uc = torch.stack([r, r * W[2], r * W[3], r * W[4], E])
        F = Uc * un
        F[1 + d] += p
        F[4] += p * un
        return Uc, F, un + c_, un - c_

    def rate(U):
        D = U[0]
        v = U[1:4] / D
        e = torch.clamp(U[4] / D - 0.5 * (v * v).sum(0), min=floor)
        W = torch.cat([D[None], e[None], v])
        dU = torch.zeros_like(U)
        for d in range(3):
            a, n = 3 - d, dims[d]
            nf = n - 2 * ng + 1
            cells = [W.narrow(a, ng - 2 + j, nf) for j in range(4)]
            L, R = plm(*cells[:3]), plm(cells[3], cells[2], cells[1])
            L[0].clamp_(min=floor)
            R[0].clamp_(min=floor)
            Ul, Fl, pl, ml = parts(L, d)
            Ur, Fr, pr, mr = parts(R, d)
            ap = torch.clamp(torch.maximum(pl, pr), min=0)
            am = torch.clamp(torch.maximum(-ml, -mr), min=0)
            F = (ap * Fl + am * Fr - ap * am * (Ur - Ul)) / (ap + am)
            dU.narrow(a, ng, n - 2 * ng).sub_((F.narrow(a, 1, nf - 1) - F.narrow(a, 0, nf - 1)) * dtdx)
        return dU
    for _ in range(c["steps"]):
        U0 = U.clone()
        fill(U)
        U = U0 + rate(U)
        fill(U)
        U = 0.5 * (U0 + U + rate(U))
    return U.reshape(5, -1)


def _amr_mesh(c):
    """Leaves (level, x, y) of the refined mesh in order: roots column-major,
    then depth first with the children's x fastest."""
    n, L = c["nx"], c["levels"]
    y, x = np.divmod(np.arange(n * n), n)
    lev = np.zeros(n * n, dtype=np.int64)
    for r in range(L):
        w = 1.0 / (n * 2.0 ** lev)
        cut = (lev == r) & (((x + 0.5) * w - 0.5) ** 2 + ((y + 0.5) * w - 0.5) ** 2 < AMR_RADII[r] ** 2)
        rep = np.where(cut, 4, 1)
        at = np.repeat(np.arange(len(lev)), rep)
        child = np.arange(len(at)) - np.repeat(np.cumsum(rep) - rep, rep)
        m = cut[at]
        lev, x, y = lev[at] + m, np.where(m, 2 * x[at] + child % 2, x[at]), np.where(m, 2 * y[at] + child // 2, y[at])
    return lev, x, y


def _exact_amr(c, seed):
    n, L, g = c["nx"], c["levels"], _gamma(c)
    lev, x, y = _amr_mesh(c)
    num = len(lev)
    maps = []
    for r in range(L + 1):
        m = np.full((n << r, n << r), -1, dtype=np.int64)
        at = lev == r
        m[y[at], x[at]] = np.flatnonzero(at)
        maps.append(m)

    def look(r, xx, yy):
        """Leaf at level-r cell (xx, yy): the leaf itself or the coarser one over it, else -1."""
        out = np.full(len(xx), -1, dtype=np.int64)
        for s in range(L + 1):
            at = (r == s) & (xx >= 0) & (yy >= 0) & (xx < (n << s)) & (yy < (n << s))
            out[at] = maps[s][yy[at], xx[at]]
        return out
    rep, faces = {}, {0: [], 1: []}
    ids = np.arange(num)
    for d in (0, 1):
        for hi in (0, 1):
            dx, dy = (2 * hi - 1, 0) if d == 0 else (0, 2 * hi - 1)
            xx, yy = x + dx, y + dy
            wall = (xx < 0) | (yy < 0) | (xx >= (n << lev)) | (yy >= (n << lev))
            same = look(lev, xx, yy)
            over = np.where((same < 0) & ~wall & (lev > 0), look(np.maximum(lev - 1, 0), xx >> 1, yy >> 1), -1)
            cx, cy = 2 * xx, 2 * yy
            if d == 0:
                cx = cx + (0 if hi else 1)
            else:
                cy = cy + (0 if hi else 1)
            fine = np.where((same < 0) & (over < 0) & ~wall, look(lev + 1, cx, cy), -1)
            rep[d, hi] = np.where(same >= 0, same, np.where(over >= 0, over, fine))
            own = wall | (over >= 0) | ((same >= 0) & bool(hi))
            other = np.where(wall, -1, rep[d, hi])[own]
            pair = (ids[own], other) if hi else (other, ids[own])
            faces[d].append((*pair, lev[own]))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    w = dev(1.0 / (n * 2.0 ** lev))
    U = _amr_state((dev(x) + 0.5) * w, (dev(y) + 0.5) * w, seed, g)
    nb = {k: dev(v) for k, v in rep.items()}
    fl = {d: tuple(dev(np.concatenate([f[j] for f in faces[d]])) for j in range(3)) for d in faces}
    flip = {d: torch.tensor([-1.0 if j == 1 + d else 1.0 for j in range(5)], device=DEV, dtype=F64)[:, None]
            for d in (0, 1)}

    def rate(U):
        W = _c2p(U, g)
        acc = torch.zeros_like(U)
        for d in (0, 1):
            l, r = (torch.where(nb[d, h] >= 0, W[:, nb[d, h].clamp(min=0)], W * flip[d]) for h in (0, 1))
            s = 0.5 * _minmod(W - l, r - W)
            left, right, fv = fl[d]
            a, b = (W + s)[:, left.clamp(min=0)], (W - s)[:, right.clamp(min=0)]
            WL, WR = torch.where(left >= 0, a, b * flip[d]), torch.where(right >= 0, b, a * flip[d])
            F = _hllc(WL, WR, d, g) / (n * 2.0 ** fv.to(F64))
            acc.index_add_(1, left[left >= 0], -F[:, left >= 0])
            acc.index_add_(1, right[right >= 0], F[:, right >= 0])
        return acc / (w * w)
    for _ in range(c["steps"]):
        W = _c2p(U, g)
        cs = torch.sqrt(g * W[4] / W[0])
        dt = _cfl(c) / max(float(((W[1 + d].abs() + cs) / w).max()) for d in (0, 1))
        V = U + dt * rate(U)
        U = 0.5 * U + 0.5 * (V + dt * rate(V))
    return U.cpu().numpy()


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("tube", "blast"):
        U = _march(_grid(_state(c, seed), _dims(c)), c, _bcstr(c), tfinal=_tfinal(c))
        return U.reshape(5, -1).cpu().numpy()
    if k in ("plane", "box"):
        return _march(_grid(_state(c, seed), _dims(c)), c, c["bc"], steps=c["steps"]).reshape(5, -1)
    if k == "gravity":
        return _march(_grid(_state(c, seed), _dims(c)), c, "ppp", steps=c["steps"],
                      source=_poisson_accel(c["nx"], GRAV_G), free_fall=GRAV_G).reshape(5, -1)
    if k == "batch":
        out = []
        for i, s in enumerate(int(v) for v in c["sides"].split(",")):
            U = _grid(_two_states((s, s, s), seed, i, _gamma(c)), (s, s, s))
            out.append(_march(U, c, "ooo", steps=c["steps"]).reshape(5, -1).cpu().numpy())
        return out
    if k == "adjoint":
        return _exact_adjoint(c, seed)
    if k == "muscl":
        return _exact_muscl(c, seed)
    if k == "amr":
        return _exact_amr(c, seed)
    WL, WR, ax = _face_states(c, seed)
    F = torch.zeros_like(WL)
    for d in range(3):
        m = ax == d + 1
        F[m] = _hllc(WL[m].T, WR[m].T, d, _gamma(c)).T
    return F.cpu().numpy()
