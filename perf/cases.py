"""The performance cases: what users of this package have it do, through its public entry
points, over the range of sizes, layouts, limiters and arithmetic modes it serves.

Kinds of case:

* ``interval`` -- one output interval of the solver, as the command line and a parameter
  study run it: the state goes up from host memory (or is loaded from a restart payload),
  the ghosts are filled, ``Solver.steps`` advances it by a number of Heun steps with the CFL
  control, and the ten output fields of every block come back to page-locked memory.
  ``mode`` is "exact" (the default: bit for bit the reference) or "fast".
* ``batch`` -- many small independent cases advanced together by ``BatchSolver``.
* ``adjoint`` -- ``Sensitivity``: a forward run and its reverse sweep, with the gradient of
  the functional with respect to the initial state and the Knudsen number.
* ``stage`` -- both Heun stages on device buffers that the caller owns
  (``mbm_stage_noalloc``), as a host framework with a memory pool of its own calls them.

Layouts: ``square`` (the 2 x 2 tiling of [-1,1]^2 of the benchmark, open edges), ``square4``
(the reference's four unequal blocks with walls between two of them), ``step28`` (28 blocks
around a forward-facing step, Dirichlet inflow, walls, an outflow), ``lshape`` (three blocks,
a concave corner, every kind of edge) and ``strips`` (one to four strips, for batches).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from multiblockmomentsfv_b200 import _abi
from multiblockmomentsfv_b200 import adjoint as adj
from multiblockmomentsfv_b200 import blockfile as bf
from multiblockmomentsfv_b200 import scenario as sc
from multiblockmomentsfv_b200 import solver as sv

NG, NV = bf.NG, bf.NV


def listed():
    return [
        # a quick look or a unit test of a user's own set-up: 400 cells, where launch latency is all
        {"name": "square4-tiny-exact", "kind": "interval", "layout": "square4", "n": 10, "limiter": "harmonic",
         "mode": "exact", "Kn": 0.001, "F": 0.0, "state": "disk", "steps": 19, "single": False, "restart": False},
        # the step deck as shipped: many small blocks, its own unlimited slopes, an inflow and walls
        {"name": "step28-exact", "kind": "interval", "layout": "step28", "n": 60, "limiter": "average",
         "mode": "exact", "Kn": 0.001, "F": 0.0, "state": "stream", "steps": 40, "single": True, "restart": False},
        # the square4 deck as shipped, restarted from a result file's payload, with a body force
        {"name": "square4-restart-exact", "kind": "interval", "layout": "square4", "n": 75, "limiter": "minmod",
         "mode": "exact", "Kn": 0.001, "F": 0.2, "state": "quadrant", "steps": 50, "single": False, "restart": True},
        # an ordinary production grid in the default mode
        {"name": "square-256-exact", "kind": "interval", "layout": "square", "n": 256, "limiter": "harmonic",
         "mode": "exact", "Kn": 0.01, "F": 0.0, "state": "quadrant", "steps": 60, "single": True, "restart": False},
        # the benchmark's grid in the default mode
        {"name": "square-1024-exact", "kind": "interval", "layout": "square", "n": 1024, "limiter": "harmonic",
         "mode": "exact", "Kn": 0.01, "F": 0.0, "state": "quadrant", "steps": 30, "single": True, "restart": False},
        # a coarse study in fast arithmetic: odd sizes, latency and launches still count
        {"name": "square-61-fast", "kind": "interval", "layout": "square", "n": 61, "limiter": "minmod",
         "mode": "fast", "Kn": 0.05, "F": 0.0, "state": "quadrant", "steps": 60, "single": True, "restart": False},
        # an ordinary grid in fast arithmetic
        {"name": "square-256-fast", "kind": "interval", "layout": "square", "n": 256, "limiter": "harmonic",
         "mode": "fast", "Kn": 0.01, "F": 0.0, "state": "quadrant", "steps": 100, "single": True, "restart": False},
        # ragged blocks, a concave corner, every kind of edge
        {"name": "lshape-331-fast", "kind": "interval", "layout": "lshape", "n": 331, "limiter": "superbee",
         "mode": "fast", "Kn": 0.005, "F": 0.0, "state": "quadrant", "steps": 60, "single": False, "restart": False},
        # the benchmark's workload
        {"name": "square-1024-fast", "kind": "interval", "layout": "square", "n": 1024, "limiter": "harmonic",
         "mode": "fast", "Kn": 0.01, "F": 0.0, "state": "quadrant", "steps": 100, "single": True, "restart": False},
        # a parameter study: a dozen small cases of all limiters in one context
        {"name": "batch-12-fast", "kind": "batch", "cases": 12, "layout": "strips", "nmin": 64, "nmax": 320,
         "plan": 7, "mode": "fast", "steps": 40},
        # sensitivities, on the grid of the benchmark's adjoint figures
        {"name": "adjoint-256-fast", "kind": "adjoint", "layout": "square", "n": 256, "limiter": "harmonic",
         "mode": "fast", "Kn": 0.01, "F": 0.0, "steps": 60, "every": 20, "functional": "heat_flux"},
        # the stages alone on a caller's buffers, ragged sizes
        {"name": "stage-777x391", "kind": "stage", "nx": 777, "ny": 391, "limiter": "harmonic", "Kn": 0.01,
         "F": 0.0, "dt": 2e-4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["interval"] * 5 + ["batch", "adjoint", "stage"])
    mode = rng.choice(["exact", "fast"])
    Kn = round(10 ** rng.uniform(-3, -1), 5)
    F = rng.choice([0.0, 0.0, 0.25])
    # the limited slopes; unlimited ones stop being finite at shocks on fine grids
    limiter = rng.choice(["none", "minmod", "superbee", "harmonic", "harmonic"])
    if kind == "stage":
        return {"kind": kind, "nx": _log(rng, 5, 1100), "ny": _log(rng, 5, 1100), "limiter": limiter, "Kn": Kn, "F": F,
                "dt": 1e-4}
    if kind == "adjoint":
        n = _log(rng, 24, 256)
        return {"kind": kind, "layout": "square", "n": n, "limiter": rng.choice(["harmonic", "minmod", "average"]),
                "mode": mode, "Kn": Kn, "F": F, "steps": rng.randint(20, 60), "every": rng.randint(7, 25),
                "functional": rng.choice(["heat_flux", "temperature", "deviatoric"])}
    if kind == "batch":
        lo = _log(rng, 24, 128)
        return {"kind": kind, "cases": rng.randint(3, 16), "layout": "strips", "nmin": lo,
                "nmax": lo + _log(rng, 8, 192), "plan": rng.randrange(10000), "mode": mode, "steps": rng.randint(15, 40)}
    layout = rng.choice(["square", "square", "square4", "step28", "lshape"])
    n = _log(rng, *{"square": (9, 700), "square4": (10, 800), "step28": (60, 480), "lshape": (12, 600)}[layout])
    cells = sum(b.nx * b.ny for b in _blocks(layout, n))
    steps = max(15, min(rng.randint(20, 100), int(8e7 / cells)))
    return {"kind": kind, "layout": layout, "n": n, "limiter": limiter, "mode": mode, "Kn": Kn, "F": F,
            "state": "stream" if layout == "step28" else rng.choice(["quadrant", "disk"]), "steps": steps,
            "single": rng.random() < 0.5, "restart": rng.random() < 0.3}


# ---------------------------------------------------------------- layouts and states --

def _blocks(layout, n):
    """The block table; n cells per unit length (square: per block side)."""
    B = bf.Block
    if layout == "square":
        return bf.quadrant_deck(n).blocks
    r = lambda length: max(4, int(round(length * n)))
    if layout == "square4":
        a, b, c, d = r(1.5), r(0.5), r(1.2), r(0.8)
        return [B(1, -1.0, 0.5, -1.0, 0.2, a, c, (0, 2, -1, 4)), B(2, 0.5, 1.0, -1.0, 0.2, b, c, (1, 0, -1, 3)),
                B(3, 0.5, 1.0, 0.2, 1.0, b, d, (4, 0, 2, -1)), B(4, -1.0, 0.5, 0.2, 1.0, a, d, (0, 3, 1, -1))]
    if layout == "lshape":
        a, b, c, d = r(1.5), r(0.5), r(1.2), r(0.8)
        return [B(1, -1.0, 0.5, -1.0, 0.2, a, c, (-2, -1, 0, 2)), B(2, -1.0, 0.5, 0.2, 1.0, a, d, (-2, 3, 1, -1)),
                B(3, 0.5, 1.0, 0.2, 1.0, b, d, (2, 0, -1, -1))]
    # step28: blocks of 1/2 x 1/6 around a step at x = 1; row by row from the bottom, two
    # blocks per row below the step's height (2/6), six above
    nx, ny = r(0.5), r(1.0 / 6)
    where = {}
    for j in range(6):
        for i in range(2 if j < 2 else 6):
            where[(i, j)] = len(where) + 1
    out = []
    for (i, j), b in where.items():
        left = where[(i - 1, j)] if i > 0 else -2
        right = where.get((i + 1, j), 0 if i == 5 else -1)
        bottom = where.get((i, j - 1), -1)
        top = where.get((i, j + 1), -1)
        out.append(B(b, 0.5 * i, 0.5 * (i + 1), j / 6.0, (j + 1) / 6.0, nx, ny, (left, right, bottom, top)))
    return out


def _deck(case):
    d = bf.Deck(Kn=case["Kn"], R13=1.0, F=case["F"], CFL=0.95, limiter=bf.limiter_code(case["limiter"]))
    d.blocks = _blocks(case["layout"], case["n"])
    return d


def _scenario(case, seed):
    """What SetInitial gives on Dirichlet edges, and the initial state but for the disk."""
    if case["state"] == "stream":
        mach = np.random.default_rng(seed).uniform(1.8, 2.2)
        return sc.Scenario(sc.KIND_UNIFORM, [(1.0, float(mach * math.sqrt(5.0 / 3.0)), 0.0, 1.0)] * 4)
    if case["state"] == "disk":
        return sc.Scenario(sc.KIND_UNIFORM, [(1.0, 0.0, 0.0, 1.0)] * 4)
    return sc.Scenario.seeded_quadrant(seed)


def _initial(case, seed, deck, scn):
    """Padded layers of the initial state, ghosts zero: the scenario's, with a dense disk at
    rest (the reference goldens' state) for state "disk"."""
    layers = [sc.initial_block(scn, b) for b in deck.blocks]
    if case["state"] == "disk":
        rng = np.random.default_rng(seed)
        rho, rad = rng.uniform(3.0, 6.0), rng.uniform(0.3, 0.5)
        for b, U in zip(deck.blocks, layers):
            x, y = b.centres()
            inner = np.zeros(x.shape, dtype=bool)
            inner[NG:-NG, NG:-NG] = True
            U[inner & (x * x + y * y < rad * rad)] = sc.moments(rho, 0.0, 0.0, 1.0)
    return layers


def _payload(deck, layers, single):
    """The zones of a result file of this state, as Output writes them (interior and a ring
    of ghosts, x outer): what a restart reads."""
    out = []
    for b, U in zip(deck.blocks, layers):
        V = U.copy()
        V[:, :NG] = V[:, NG:NG + 1]
        V[:, -NG:] = V[:, -NG - 1:-NG]
        V[:NG] = V[NG]
        V[-NG:] = V[-NG - 1]
        V = V[2:-2, 2:-2]
        r = V[..., 0]
        u, v = V[..., 1] / r, V[..., 2] / r
        th = (2 * V[..., 3] / r - u * u - v * v) / 3
        f = [r, u, v, th, r * th, r * th, 0 * r, r * th, 0 * r, 0 * r]      # q = 0, T_ij = theta delta_ij
        out.append(np.stack(f, axis=-1).transpose(1, 0, 2).reshape(-1, 10).astype(np.float32 if single else np.float64))
    return out


def _batch_cases(case, seed):
    """Seeded cases of one to four strips; the plan (sizes, limiters) belongs to the case, the
    states to the seed."""
    rng = np.random.default_rng(case["plan"])
    out = []
    for k in range(case["cases"]):
        nb, n = int(rng.integers(1, 4)), int(rng.integers(case["nmin"], case["nmax"] + 1))
        h = 2.0 / nb
        d = bf.Deck(Kn=float(10 ** rng.uniform(-3, -1)), R13=1.0, limiter=k % 5, CFL=0.95)
        d.blocks = [bf.Block(j + 1, -1.0, 1.0, -1.0 + j * h, -1.0 + (j + 1) * h, n, n,
                             (0, 0, j if j > 0 else 0, j + 2 if j < nb - 1 else 0)) for j in range(nb)]
        out.append((d, sc.Scenario.seeded_quadrant(seed * 1000 + k)))
    return out


def _pinned(a):
    """Page-locked host memory holding a."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _pinned_out(deck, single):
    dt = torch.float32 if single else torch.float64
    return [torch.empty(((b.nx + 2) * (b.ny + 2), 10), dtype=dt, pin_memory=True).numpy() for b in deck.blocks]


# --------------------------------------------------------------------- the measured calls --

class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    if case["kind"] == "interval":
        d = _deck(case)
        scn = _scenario(case, seed)
        layers = _initial(case, seed, d, scn)
        st.restart = case["restart"]
        src = _payload(d, layers, case["single"]) if st.restart else layers
        st.src = [_pinned(a) for a in src]
        st.out = _pinned_out(d, case["single"])
        st.solver = sv.Solver(d, scn, mode=case["mode"], show_every=20)
    elif case["kind"] == "batch":
        cases = _batch_cases(case, seed)
        st.src = [[_pinned(sc.initial_block(scn, b)) for b in d.blocks] for d, scn in cases]
        st.out = [a for d, _ in cases for a in _pinned_out(d, True)]
        st.solver = sv.BatchSolver(cases, mode=case["mode"])
    elif case["kind"] == "adjoint":
        d, base, th = _adjoint_problem(case, seed)
        st.layers = adj.state_from_theta(d, base, th)
        st.sens = adj.Sensitivity(d, base, mode=case["mode"], functional=case["functional"])
    else:
        blk, U, D0 = _stage_problem(case, seed)
        st.descs = _abi.block_descs([blk])
        pitch = (blk.nxp + 1 + 3) & ~3
        plane = (pitch * blk.nyp + 31) & ~31
        st.view = (NV, blk.nyp, blk.nxp), (plane, pitch, 1), 1

        def planes(A):
            buf = torch.zeros(NV * plane, dtype=torch.float64, device="cuda")
            torch.as_strided(buf, *st.view).copy_(torch.from_numpy(A).permute(2, 0, 1))
            return buf

        st.u, st.d0 = planes(U), planes(D0)
        st.o1, st.o2 = torch.zeros_like(st.u), torch.zeros_like(st.u)
        st.cfl = np.zeros(2)
        st.L = _abi.lib()
        st.stream = torch.cuda.current_stream().cuda_stream
    return st


def run(st):
    case = st.case
    if case["kind"] == "interval":
        s = st.solver
        for b, a in enumerate(st.src):
            if st.restart:
                s.load_fields(b, a, faithful=True)
            else:
                s.upload(sv.L_DATA, b, a)
        s.set_boundary(sv.L_DATA, 0.0)
        t, n, rej = s.steps(0.0, 1e3, max_steps=case["steps"])
        for b, a in enumerate(st.out):
            s.output_fields_async(b, a, case["single"])
        s.output_wait()
        return {"t": t, "steps": n, "rejected": rej, "fields": st.out}
    if case["kind"] == "batch":
        s = st.solver
        for k, blocks in enumerate(st.src):
            for b, a in enumerate(blocks):
                s.upload(sv.L_DATA, k, b, a)
        _abi.check(s.L.mbm_set_boundary(s.ctx, sv.L_DATA, 0.0), s.ctx)
        t, n, rej = s.steps(0.0, 1e3, max_steps=case["steps"], check=False)
        for g, a in enumerate(st.out):
            _abi.check(s.L.mbm_output_fields_async(s.ctx, g, 1, a.ctypes.data), s.ctx)
        _abi.check(s.L.mbm_output_wait(s.ctx), s.ctx)
        return {"t": t, "steps": n, "rejected": rej, "fields": st.out}
    if case["kind"] == "adjoint":
        st.sens.load(st.layers)
        J, grad, gK, dts, _ = st.sens.run(case["steps"], case["every"])
        return {"J": J, "grad": grad, "grad_Kn": gK, "dts": dts}
    lim = bf.limiter_code(case["limiter"])
    cfl = st.cfl.ctypes.data_as(C.POINTER(C.c_double))
    for heun, x, o in ((0, st.d0, st.o1), (1, st.u, st.o2)):
        at = C.cast(C.byref(cfl.contents, 8 * heun), C.POINTER(C.c_double))
        _abi.check(st.L.mbm_stage_noalloc(st.descs, 1, x.data_ptr(), st.d0.data_ptr(), o.data_ptr(), case["Kn"],
                                          case["F"], lim, case["dt"], heun, at, st.stream))
    return {"stage1": torch.as_strided(st.o1, *st.view), "stage2": torch.as_strided(st.o2, *st.view), "cfl": st.cfl}


# FP64 operations of one Heun stage of one cell, counted from the formulas with one cell's
# share of the faces: the primitives, the relaxations, two slopes and two fluxes of nine
# components, the update
STAGE_FLOPS = 1050


def work(case):
    if case["kind"] == "stage":
        cells = case["nx"] * case["ny"]
        return {"bytes": 8.0 * NV * cells * (2 + 3), "flops": 2.0 * STAGE_FLOPS * cells}
    if case["kind"] == "batch":
        cells = sum(d.full_grid_size for d, _ in _batch_cases(case, 0))
        io = cells * (72 + 40)
    else:
        cells = sum(b.nx * b.ny for b in _blocks(case["layout"], case["n"]))
        io = cells * (72 + (72 if case["kind"] == "adjoint" else 40 if case["single"] else 80))
    steps = case["steps"]
    # a step reads its state and writes the next one; the reverse sweep reads the states back
    # and carries an adjoint state, at about twice the forward operations
    k = 3 if case["kind"] == "adjoint" else 1
    return {"bytes": float(io + k * 2 * 8 * NV * cells * steps), "flops": 2.0 * k * STAGE_FLOPS * cells * steps}


# ------------------------------------------------- the same in plain torch, 64 bits --
# Layers are (9, rows, columns) tensors of the padded grid.

def _adjoint_problem(case, seed):
    d = _deck(case)
    base = adj.smooth_base(d, seed)
    rng = np.random.default_rng(seed + 1)
    k, ph = rng.uniform(1, 4, size=(4, 2)), rng.uniform(0, 2 * np.pi, size=4)
    th = []
    for b in d.blocks:
        x, y = (a[NG:-NG, NG:-NG] for a in b.centres())
        th.append(1.0 + 0.1 * sum(np.sin(k[m, 0] * x + k[m, 1] * y + ph[m]) for m in range(4)) / 4)
    return d, base, th


def _stage_problem(case, seed):
    """A block and two padded states on it: smooth waves with a little noise, and a heat flux
    and stresses as the moments carry them."""
    blk = bf.Block(1, -1.0, 1.0, -1.0, 1.0, case["nx"], case["ny"], (0, 0, 0, 0))
    rng = np.random.default_rng(seed)
    x, y = blk.centres()

    def field(amp):
        k, ph = rng.uniform(1, 6, size=(3, 2)), rng.uniform(0, 2 * np.pi, size=3)
        f = sum(np.sin(k[m, 0] * x + k[m, 1] * y + ph[m]) for m in range(3)) / 3
        return amp * (f + 0.02 * rng.standard_normal(x.shape))

    def state():
        r, th = 1.2 + field(0.3), 1.1 + field(0.2)
        P = np.stack([r, field(0.3), field(0.3), th, th + field(0.05), field(0.05), th + field(0.05), field(0.05),
                      field(0.05)])
        return _cons(torch.from_numpy(P)).numpy().transpose(1, 2, 0).copy()

    return blk, state(), state()


def _prim(U):
    r, E = U[0], U[3]
    u, v = U[1] / r, U[2] / r
    T11, T12, T22 = U[4] / r - u * u, U[5] / r - u * v, U[6] / r - v * v
    return torch.stack([r, u, v, (2 * E / r - (u * u + v * v)) / 3, T11, T12, T22,
                        U[7] - E * u - r * (T11 * u + T12 * v), U[8] - E * v - r * (T12 * u + T22 * v)])


def _cons(P):
    r, u, v, th, T11, T12, T22, q1, q2 = P.unbind(0)
    E = 0.5 * r * (u * u + v * v) + 1.5 * r * th
    return torch.stack([r, r * u, r * v, E, r * (T11 + u * u), r * (T12 + u * v), r * (T22 + v * v),
                        q1 + E * u + r * (T11 * u + T12 * v), q2 + E * v + r * (T12 * u + T22 * v)])


def _damp(z, flag):
    if flag in (-1, 0):
        return (1 + 0.5 * z - 0.25 * z * z) / (1 + z + 0.25 * z * z)
    if flag == 1:
        return (1 + z) / (1 + z + 0.25 * z * z)
    return torch.ones_like(z) if flag == 2 else 1 / (1 + 0.5 * z)


def _relax(P, dt, Kn, F, flag):
    """The relaxed state in primitive form, and the damping factor of the heat flux."""
    th = P[3]
    z = P[0] * torch.sqrt(th) / Kn * dt
    d1, d2 = _damp(z, flag), _damp(2.0 / 3 * z, flag)
    push = dt * F if flag in (0, 2) else 0.0
    return torch.stack([P[0], P[1] + push, P[2], th, d1 * (P[4] - th) + th, d1 * P[5], d1 * (P[6] - th) + th,
                        d2 * P[7], d2 * P[8]]), d2


def _limit(lim, d1, d2):
    if lim == 0:
        return torch.zeros_like(d1)
    if lim == 1:
        return 0.5 * (d1 + d2)
    if lim == 2:
        s1, s2 = torch.sign(d1).detach(), torch.sign(d2).detach()
        return 0.5 * (s1 + s2) * torch.where(d1.abs() < d2.abs(), d1 * s1, d2 * s2)
    if lim == 3:
        th = d2 / torch.where(d1 == 0, torch.ones_like(d1), d1)
        phi = torch.where(th < 0, 0 * th, torch.where(th < 0.5, 2 * th, torch.where(th < 1, th * 0 + 1, torch.where(
            th < 2, th, th * 0 + 2))))
        return torch.where(d1 == 0, torch.zeros_like(d1), d1 * phi)
    one = torch.ones_like(d1)
    w1 = d1 * torch.where(d1 < 0, -one, one) + 1e-10
    w2 = d2 * torch.where(d2 < 0, -one, one) + 1e-10
    return (w1 * d2 + w2 * d1) / (w1 + w2)


_SWAP = [0, 2, 1, 3, 6, 5, 4, 8, 7]


def _flux_x(P):
    r, u, v, th, T11, T12, T22, q1, q2 = P.unbind(0)
    vs = u * u + v * v
    E = 0.5 * r * vs + 1.5 * r * th
    A = T11 * u + T12 * v
    return torch.stack([
        r * u, r * (T11 + u * u), r * (T12 + u * v), E * u + r * A + q1, 1.2 * q1 + r * (3 * T11 * u + u * u * u),
        0.4 * q2 + r * (T11 * v + 2 * T12 * u + u * u * v), 0.4 * q1 + r * (T22 * u + 2 * T12 * v + v * v * u),
        2 * (q1 + r * A) * u + E * u * u + 1.2 * q1 * u + 0.4 * q2 * v
        + 0.5 * r * (T11 * vs + 5 * th * th + 7 * th * (T11 - th)),
        q2 * u + q1 * v + r * (u * v * (T11 + T22) + 1.5 * T12 * vs) + E * u * v + 0.4 * q2 * u + 0.4 * q1 * v
        + 3.5 * r * th * T12])


def _hll_x(L, R):
    """The HLL flux along x between the states L and R, and the largest wave speed."""
    both = torch.stack([L, R], dim=1)
    U, f = _cons(both), _flux_x(both)
    cL, cR = 2 * torch.sqrt(5.0 / 3 * L[3]), 2 * torch.sqrt(5.0 / 3 * R[3])
    zero = torch.zeros_like(cL)
    lamL, lamR = torch.minimum(L[1] - cL, zero), torch.maximum(R[1] + cR, zero)
    F = (lamR * f[:, 0] - lamL * f[:, 1] + lamL * lamR * (U[:, 1] - U[:, 0])) / (lamR - lamL)
    return F, (0.5 * (L[1] + R[1])).abs() + torch.maximum(cL, cR)


def _stage(blk, U, D0, dt, Kn, F, lim, heun):
    """One Heun stage of a block: the new interior (9, ny, nx) and its CFL number."""
    P = _prim(U)
    Q, _ = _relax(P, dt, Kn, F, 2 * heun + 1)
    Pr = P.clone()
    Pr[:, 1:-1, 1:-1] = Q[:, 1:-1, 1:-1]
    Sx = _limit(lim, Pr[:, :, 1:-1] - Pr[:, :, :-2], Pr[:, :, 2:] - Pr[:, :, 1:-1])        # columns 1 .. nxp-2
    Sy = _limit(lim, Pr[:, 1:-1] - Pr[:, :-2], Pr[:, 2:] - Pr[:, 1:-1])
    Mx, My = Pr[:, 1:-2, 1:-1], Pr[:, 1:-1, 1:-2]
    Sx, Sy = Sx[:, 1:-2], Sy[:, :, 1:-2]
    Gx, lx = _hll_x((Mx + 0.5 * Sx)[:, :, :-1], (Mx - 0.5 * Sx)[:, :, 1:])                   # faces c | c+1, c = 1 .. nxp-3
    Gy, ly = _hll_x((My + 0.5 * Sy)[_SWAP][:, :-1], (My - 0.5 * Sy)[_SWAP][:, 1:])
    Gy = Gy[_SWAP]
    R, d2 = _relax(P, dt, Kn, F, 2 * heun)
    prod = (0.5 * (1 - d2[1:-1, 1:-1])).max().clamp_min(0)
    cfl = dt * lx.max() / blk.dx + dt * ly.max() / blk.dy + prod
    inner = (slice(None), slice(NG, -NG), slice(NG, -NG))
    new = _cons(R[inner])
    if heun:
        new = new + _cons(_relax(_prim(D0[inner]), dt, Kn, F, -1)[0])
    ny, nx = blk.ny, blk.nx
    new = new + dt / blk.dx * (Gx[:, 2:2 + ny, 1:1 + nx] - Gx[:, 2:2 + ny, 2:2 + nx])
    new = new + dt / blk.dy * (Gy[:, 1:1 + ny, 2:2 + nx] - Gy[:, 2:2 + ny, 2:2 + nx])
    return (0.5 * new if heun else new), cfl


def _fill(deck, scn, interiors):
    """Padded layers from the interiors: both sweeps of the ghost fill, edge by edge."""
    S = [torch.nn.functional.pad(u, (NG, NG, NG, NG)) for u in interiors]
    flip = [torch.ones(NV, 1, 1, dtype=torch.float64, device=S[0].device) for _ in range(2)]
    flip[0][[1, 5, 7]], flip[1][[2, 5, 8]] = -1.0, -1.0

    def edge(b, side, s):
        code = deck.blocks[b].bc[side]
        d = 1 if side % 2 else -1                     # outward
        ax = 2 if side < 2 else 1
        n = S[b].shape[ax]
        at = lambda t, i: t.select(ax, i)
        for k in range(1, NG + 1):
            g = NG - k if d < 0 else n - 1 - NG + k
            m = NG - 1 + k if d < 0 else n - NG - k      # the k-th interior layer of this side
            if code > 0:
                ns = S[s].shape[ax]
                v = at(S[s], ns - NG - k if d < 0 else NG - 1 + k)
            elif code == 0:
                v = at(S[b], NG if d < 0 else n - 1 - NG)
            elif code == -1:
                v = at(S[b], m) * flip[ax == 1].squeeze(-1)
            else:
                v = scn[(b, side)][:, k - 1].T
            idx = torch.tensor([g], device=v.device)
            S[b] = S[b].index_copy(ax, idx, v.unsqueeze(ax))

    for again in (False, True):
        for b, blk in enumerate(deck.blocks):
            for side in range(4):
                if not again or blk.bc[side] > 0:
                    edge(b, side, blk.bc[side] - 1)
    return S


def _dirichlet(deck, scn, dev):
    return {(b, side): torch.from_numpy(sc.dirichlet_edge(scn, blk, side)).to(dev)
            for b, blk in enumerate(deck.blocks) for side in range(4) if blk.bc[side] <= -2}


def _heun_step(deck, diri, data, dt):
    out, cfl = [], 0.0
    tmp = []
    for blk, U in zip(deck.blocks, data):
        new, c = _stage(blk, U, U, dt, deck.Kn, deck.F, deck.limiter, 0)
        tmp.append(new)
        cfl = max(cfl, float(c.detach()))
    for blk, U, D0 in zip(deck.blocks, _fill(deck, diri, tmp), data):
        new, c = _stage(blk, U, D0, dt, deck.Kn, deck.F, deck.limiter, 1)
        out.append(new)
        cfl = max(cfl, float(c.detach()))
    return _fill(deck, diri, out), cfl


def _advance(deck, diri, data, steps):
    """Steps with its CFL control (limit 1): the data, t, accepted, rejected, the step sizes."""
    t, dt, n, rej, dts = 0.0, 1e-4, 0, 0, []
    while n < steps:
        new, cfl = _heun_step(deck, diri, data, dt)
        if not math.isfinite(cfl) or not all(bool(torch.isfinite(x).all()) for x in new):
            return data, t, n, rej, dts
        if cfl > 1.0:
            rej += 1
        else:
            data, t, n = new, t + dt, n + 1
            dts.append(dt)
        dt = dt * deck.CFL / cfl
    return data, t, n, rej, dts


def _fields(deck, data, single):
    out = []
    for U in data:
        P = _prim(U[:, 2:-2, 2:-2])
        f = torch.stack([P[0], P[1], P[2], P[3], P[0] * P[3], P[0] * P[4], P[0] * P[5], P[0] * P[6], P[7], P[8]])
        out.append(f.permute(2, 1, 0).reshape(-1, 10).cpu().numpy())
    return out


def _inner(layers, dev):
    return [torch.from_numpy(np.ascontiguousarray(U[NG:-NG, NG:-NG].transpose(2, 0, 1))).to(dev) for U in layers]


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "stage":
        blk, U, D0 = _stage_problem(case, seed)
        u, d0 = (torch.from_numpy(a.transpose(2, 0, 1).copy()).to(dev) for a in (U, D0))
        lim, got, cfl = bf.limiter_code(case["limiter"]), [], []
        for heun, x in ((0, d0), (1, u)):
            new, c = _stage(blk, x, d0, case["dt"], case["Kn"], case["F"], lim, heun)
            got.append(torch.nn.functional.pad(new, (NG, NG, NG, NG)))
            cfl.append(float(c))
        return {"stage1": got[0], "stage2": got[1], "cfl": np.array(cfl)}
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, dev)
    if case["kind"] == "batch":
        t, n, rej, fields = [], [], [], []
        for d, scn in _batch_cases(case, seed):
            data = _fill(d, {}, _inner([sc.initial_block(scn, b) for b in d.blocks], dev))
            data, tt, nn, rr, _ = _advance(d, {}, data, case["steps"])
            t.append(tt), n.append(nn), rej.append(rr)
            fields += _fields(d, data, True)
        return {"t": np.array(t), "steps": np.array(n), "rejected": np.array(rej), "fields": fields}
    d, scn = _deck(case), _scenario(case, seed)
    layers = _initial(case, seed, d, scn)
    if case["restart"]:                    # the fields as the payload stores them
        got = []
        for b, p in zip(d.blocks, _payload(d, layers, case["single"])):
            f = torch.from_numpy(p.astype(np.float64)).reshape(b.nx + 2, b.ny + 2, 10).permute(2, 1, 0)
            P = torch.stack([f[0], f[1], f[2], f[3], f[5] / f[0], f[6] / f[0], f[7] / f[0], f[8], f[9]])
            got.append(_cons(P)[:, 1:-1, 1:-1].to(dev))
    else:
        got = _inner(layers, dev)
    diri = _dirichlet(d, scn, dev)
    data, t, n, rej, _ = _advance(d, diri, _fill(d, diri, got), case["steps"])
    return {"t": t, "steps": n, "rejected": rej, "fields": _fields(d, data, case["single"])}


def _exact_adjoint(case, seed, dev):
    from torch.utils.checkpoint import checkpoint
    d, base, th = _adjoint_problem(case, seed)
    u0 = _inner(adj.state_from_theta(d, base, th), dev)
    with torch.no_grad():
        dts = _advance(d, {}, _fill(d, {}, u0), case["steps"])[4]
    u0 = [u.requires_grad_(True) for u in u0]
    Kn = torch.tensor(d.Kn, dtype=torch.float64, device=dev, requires_grad=True)

    def step(dt, K, *data):
        d.Kn = K
        return tuple(_heun_step(d, {}, list(data), dt)[0])

    data = tuple(_fill(d, {}, u0))
    for dt in dts:
        data = checkpoint(step, dt, Kn, *data, use_reentrant=False)
    J = 0.0
    for U in data:
        P = _prim(U[:, NG:-NG, NG:-NG])
        if case["functional"] == "temperature":
            f = P[3]
        elif case["functional"] == "deviatoric":
            f = (P[4] - P[3]) ** 2 + 2 * P[5] ** 2 + (P[6] - P[3]) ** 2
        else:
            f = P[7] ** 2 + P[8] ** 2
        J = J + f.sum()
    J.backward()
    grad = [torch.nn.functional.pad(u.grad, (NG, NG, NG, NG)).permute(1, 2, 0).contiguous().cpu().numpy() for u in u0]
    return {"J": float(J.detach()), "grad": grad, "grad_Kn": float(Kn.grad), "dts": np.array(dts)}
