"""The work that programs built on this package have it do, as cases to time and compare.

Four kinds, each through a public entry point:

* ``launch``: one call of the drop-in launcher (`launcher2d` / `launcher3d`), the step that
  the reference's unchanged host program makes once per iteration, from one state into
  another;
* ``loop``: iterations of the reference's host time loop (`BlastRun.step`): step, Dt back
  to the host, swap;
* ``batch``: steps of the batched engine (`Batch.run`) over blasts of uneven sizes, then
  every instance's status, as the serving loop does each tick;
* ``csv``: a state written as the reference's CSV file (`write_csv`), bytes read back.

A loop's and a batch's state advances with each pass, as in a program that uses them.
"""
import ctypes
import importlib
import math
import os
import random
import tempfile

import numpy as np
import torch

H = importlib.import_module("scalable-fpga-hydrodynamics_b200")
B = importlib.import_module("scalable-fpga-hydrodynamics_b200.batch")

NP = {"f64": np.float64, "f32": np.float32}
TORCH = {"f64": torch.float64, "f32": torch.float32}
GAMMA, K = 1.4, 1.1


def listed():
    return [
        # the reference's default timing grid: one call, where launch and wait dominate
        dict(name="launch 2d f64 60x60", kind="launch", dtype="f64", arith="strict", nx=60, ny=60),
        # an odd row length in FP32: rows whose pitch no tensor map takes
        dict(name="launch 2d f32 1500x1001", kind="launch", dtype="f32", arith="strict", nx=1500, ny=1001),
        # an ordinary 2D run in the reference's precision and operation order
        dict(name="loop 2d f64 1024x1024", kind="loop", dtype="f64", arith="strict", nx=1024, ny=1024, steps=20),
        # the grid of the reference's published single-device 2D run
        dict(name="loop 2d f64 20000x20000", kind="loop", dtype="f64", arith="strict", nx=20000, ny=20000, steps=4),
        # a large 2D run in the fast arithmetic
        dict(name="loop 2d f32 fused 8000x4000", kind="loop", dtype="f32", arith="fused", nx=8000, ny=4000, steps=10),
        # the small 3D grid of the reference's tests: one call
        dict(name="launch 3d f64 60x60x60", kind="launch", dtype="f64", arith="strict", nx=60, ny=60, nz=60),
        # the grid of the reference's published 3D run
        dict(name="loop 3d f64 170x170x170", kind="loop", dtype="f64", arith="strict", nx=170, ny=170, nz=170, steps=10),
        # the largest 3D grid of the benchmark
        dict(name="loop 3d f64 512x512x512", kind="loop", dtype="f64", arith="strict", nx=512, ny=512, nz=512, steps=4),
        # a ragged 3D grid in FP32 and fused arithmetic
        dict(name="loop 3d f32 fused 321x255x259", kind="loop", dtype="f32", arith="fused", nx=321, ny=255, nz=259,
             steps=10),
        # the batched workload's sizes: many uneven 2D blasts in FP32
        dict(name="batch 2d f32 fused 24", kind="batch", dtype="f32", arith="fused", dim=2, count=24, lo=64, hi=2048,
             sizes=5, steps=10),
        # the serving workload's 3D requests in FP64, one tick of its server
        dict(name="batch 3d f64 12", kind="batch", dtype="f64", arith="strict", dim=3, count=12, lo=32, hi=256,
             sizes=3, steps=8),
        # the output file of an ordinary 2D run
        dict(name="csv 2d f64 1200x800", kind="csv", dtype="f64", nx=1200, ny=800),
    ]


def _log(rng, lo, hi):
    return max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["launch"] * 4 + ["loop"] * 4 + ["batch"] * 3 + ["csv"])
    dtype, arith = rng.choice(["f64", "f32"]), rng.choice(["strict", "fused"])
    dim = rng.choice([2, 3])
    if kind == "batch":
        return dict(kind=kind, dtype=dtype, arith=arith, dim=dim, count=rng.randint(2, 24),
                    lo=64 if dim == 2 else 32, hi=2048 if dim == 2 else 192, sizes=rng.randint(10, 10 ** 6),
                    steps=2 * rng.randint(2, 5))
    if kind == "csv":
        c = dict(kind=kind, dtype=dtype, nx=_log(rng, 20, 1000), ny=_log(rng, 20, 1000))
        if dim == 3:
            c.update(nx=_log(rng, 10, 100), ny=_log(rng, 10, 100), nz=_log(rng, 10, 100))
        return c
    c = dict(kind=kind, dtype=dtype, arith=arith)
    if dim == 2:
        n = [_log(rng, 40, 10000), _log(rng, 40, 10000)]
        c.update(nx=n[0], ny=n[1])
    else:
        n = [_log(rng, 24, 400), _log(rng, 24, 400), _log(rng, 24, 400)]
        c.update(nx=n[0], ny=n[1], nz=n[2])
    if kind == "loop":
        c["steps"] = rng.randint(4, 12)
    return c


def _nb(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if "nz" in case else ())


def _sizes(case):
    """The grids of a batch case: they belong to the case, not to the seed."""
    rng = random.Random(case["sizes"])
    out = []
    for _ in range(case["count"]):
        if case["dim"] == 2:
            n = _log(rng, case["lo"], case["hi"])
            side = [n, max(2, int(round(n / rng.uniform(1.0, 2.0))))]
            rng.shuffle(side)
        else:
            side = [_log(rng, case["lo"], case["hi"]) for _ in range(3)]
        out.append(tuple(side))
    return out


def _blast(rng, nb):
    """A blast of the seeded workloads: gas at rest, density 1, a hot circle or sphere."""
    return B.Blast(nb=nb, centre=tuple(1.0 + (n - 1) * rng.uniform(0.25, 0.75) for n in nb),
                   radius=rng.uniform(0.05, 0.2) * min(nb), rho_in=1.0, rho_out=1.0,
                   p_in=0.1 * math.exp(rng.uniform(math.log(10.0), math.log(1000.0))), p_out=0.1, gamma=GAMMA, K=K)


def _shaped(a, nb):
    """A state array as (rows..., components)."""
    return a.view(tuple(n + 2 for n in nb) + (-1,))


def _inner(nb):
    return tuple(slice(1, n + 1) for n in nb)


def _wave_state(nb, dtype, seed):
    """(rhoE, uvx) of an expanding blast wave (dense shell, radial flow, ripples) in gas at rest."""
    rng = random.Random(seed)
    d = len(nb)
    centre = [n * rng.uniform(0.35, 0.65) for n in nb]
    radius = min(nb) * rng.uniform(0.2, 0.35)
    p_in, vmax = rng.uniform(2.0, 10.0), rng.uniform(0.5, 1.5)
    phase = [rng.uniform(0, 6.28) for _ in nb]
    rhoE, uvx = H.alloc_state(nb, NP[dtype])
    R, U = _shaped(rhoE, nb), _shaped(uvx, nb)
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") for n in nb]
    rows = max(1, 2 ** 25 // math.prod(nb[1:]))
    for a in range(0, nb[0], rows):
        b = min(nb[0], a + rows)
        x = [ax[0][a:b]] + ax[1:]
        x = [v.view((1,) * i + (-1,) + (1,) * (d - 1 - i)) for i, v in enumerate(x)]
        off = [(v - c) / radius for v, c in zip(x, centre)]
        r2 = sum(o * o for o in off)
        hot = torch.exp(-4.0 * r2)
        rip = 1.0 + 0.02 * sum(torch.sin(0.05 * v + f) for v, f in zip(x, phase)) / d
        inside = (r2 < 1.0).double()
        rho = (1.0 + inside * (r2 * r2 - 0.5 * hot)) * rip
        p = 0.1 + inside * (p_in * hot + 1.0 * r2) * rip
        vel = [vmax * inside * o * rip for o in off]
        at = (slice(a + 1, b + 1),) + _inner(nb)[1:]
        R[at + (0,)] = rho.to(rhoE.dtype)
        R[at + (1,)] = (p / (GAMMA - 1.0) + 0.5 * rho * sum(v * v for v in vel)).to(rhoE.dtype)
        for i, v in enumerate(vel):
            U[at + (i,)] = (rho * v).to(rhoE.dtype)
    return rhoE, uvx


class _Device:
    """A device array of another owner, for torch.as_tensor; the tensor keeps its owner alive."""

    def __init__(self, owner, ptr, shape, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=np.dtype(dtype).str, data=(ptr, False), version=2)


def prepare(case, seed):
    kind, T = case["kind"], NP[case["dtype"]]
    if kind == "batch":
        b = B.Batch(case["dim"], T, capacity=case["count"], arith=case["arith"])
        rng = random.Random(seed)
        slots = [(b.add(_blast(rng, nb)), nb) for nb in _sizes(case)]
        b.prepare(case["steps"])
        b.L.hydro_batch_state.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_void_p),
                                          ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_longlong)]
        return dict(case=case, batch=b, slots=slots, views={})
    nb = _nb(case)
    if kind == "loop":
        return dict(case=case, run=H.BlastRun(nb, T, blast=_blast(random.Random(seed), nb), arith=case["arith"]))
    state = _wave_state(nb, case["dtype"], seed)
    if kind == "csv":
        f = tempfile.NamedTemporaryFile(suffix=".csv", delete=False)
        f.close()
        room = np.zeros(64 + 112 * math.prod(nb), dtype=np.uint8)
        return dict(case=case, state=state, nb=nb, file=_File(f.name), room=room)
    phys = H.Physics(T, nb, gamma=GAMMA, K=K)
    dt = float(phys.C_min) / _max_speed(state, nb)
    return dict(case=case, state=state, out=H.alloc_state(nb, T), dt=torch.zeros(1, dtype=TORCH[case["dtype"]], device="cuda"),
                phys=phys, dtd=phys.dtd(dt), nb=nb)


class _File:
    """A temporary file that goes with its state."""

    def __init__(self, path):
        self.path = path

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def _views(s, slot, nb):
    """The instance's current state on the device, where the engine holds it."""
    b = s["batch"]
    r, u, ys = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_longlong()
    H._check(b.L.hydro_batch_state(b.h, slot, ctypes.byref(r), ctypes.byref(u), ctypes.byref(ys)))
    key = (slot, r.value)
    if key not in s["views"]:
        full = tuple(n + 2 for n in nb[:-1]) + ((ys.value,) if len(nb) == 2 else (nb[-1] + 2,))
        s["views"][key] = tuple(torch.as_tensor(_Device(b, p, full + (c,), b.T), device="cuda")[_inner(nb)]
                                for p, c in ((r.value, 2), (u.value, len(nb))))
    return s["views"][key]


def run(s):
    case = s["case"]
    if case["kind"] == "launch":
        p, (r, u), (rn, un), nb = s["phys"], s["state"], s["out"], s["nb"]
        f = H.launcher2d if len(nb) == 2 else H.launcher3d
        us = f(r, u, rn, un, s["dt"], p.C_min, p.g, p.gm1, p.divgamma, p.k, *nb, *s["dtd"], arith=case["arith"])
        if us < 0:
            raise RuntimeError(H.last_error()[1])
        return rn, un, s["dt"]
    if case["kind"] == "loop":
        r = s["run"]
        for _ in range(case["steps"]):
            r.step()
        return r.cur[0], r.cur[1], np.array([r.t, float(r.dt)]).astype(r.T)
    if case["kind"] == "batch":
        b = s["batch"]
        b.run(case["steps"])
        st = [b.status(slot) for slot, _ in s["slots"]]
        told = np.array([[x["t"], x["dt"], x["mass"], x["energy"], x["max_speed"]] for x in st]).astype(b.T)
        return [_views(s, slot, nb) for slot, nb in s["slots"]], told
    H.write_csv(s["state"], s["nb"], s["file"].path)
    with open(s["file"].path, "rb") as f:
        n = f.readinto(s["room"])
    return s["room"], n


def work(case):
    grids = _sizes(case) if case["kind"] == "batch" else [_nb(case)]
    cells = sum(math.prod(nb) for nb in grids)
    d = len(grids[0])
    b = 8 if case["dtype"] == "f64" else 4
    if case["kind"] == "csv":
        return dict(bytes=cells * ((2 + d) * b + 30), flops=0)
    steps = case.get("steps", 1)
    # each conserved value read once and written once per step; operations of the update
    # with every face once and every cell's primitives once
    return dict(bytes=2 * (2 + d) * b * cells * steps, flops=(130 if d == 2 else 220) * cells * steps)


# ------------------------------------------------------------- the same in plain torch ---
def _prim(U):
    """(rho, [velocities], p, E) of conserved values given as a list rho, E, momenta..."""
    r, E, m = U[0], U[1], U[2:]
    v = [x / r for x in m]
    p = (GAMMA - 1.0) * (E - 0.5 * r * sum(x * x for x in v))
    return r, v, p, E


def _flux(L, R, d):
    """The upwind face flux along axis d between two sides of primitives."""
    a = K * torch.maximum(torch.sqrt(GAMMA * L[2] * L[0]), torch.sqrt(GAMMA * R[2] * R[0]))
    us = 0.5 * (L[1][d] + R[1][d] - (R[2] - L[2]) / a)
    ps = 0.5 * (L[2] + R[2] - a * (R[1][d] - L[1][d]))
    up = us >= 0
    m = torch.where(up, L[0], R[0]) * us
    mom = [m * torch.where(up, x, y) for x, y in zip(L[1], R[1])]
    mom[d] = mom[d] + ps
    return [m, us * torch.where(up, L[3], R[3]) + ps * us] + mom


def _cut(P, axis, sl):
    at = (slice(None),) * axis + (sl,)
    return P[0][at], [v[at] for v in P[1]], P[2][at], P[3][at]


def _wall(P, axis, sl):
    """The wall cells mirrored: normal velocity negated."""
    r, v, p, E = _cut(P, axis, sl)
    return r, [-x if i == axis else x for i, x in enumerate(v)], p, E


def _join(Ps, axis):
    cat = lambda xs: torch.cat(xs, axis)
    return cat([P[0] for P in Ps]), [cat([P[1][i] for P in Ps]) for i in range(len(Ps[0][1]))], cat([P[2] for P in Ps]), cat(
        [P[3] for P in Ps])


def _speed(P):
    return float((torch.sqrt(GAMMA * P[2] / P[0]) + torch.sqrt(sum(x * x for x in P[1]))).max())


def _slab(nb):
    return max(1, 2 ** 25 // math.prod(nb[1:]))


def _max_speed(state, nb):
    R, U = (_shaped(a, nb) for a in state)
    best = 0.0
    for a in range(1, nb[0] + 1, _slab(nb)):
        at = (slice(a, min(nb[0] + 1, a + _slab(nb))),) + _inner(nb)[1:]
        cols = [R[at + (0,)], R[at + (1,)]] + [U[at + (i,)] for i in range(len(nb))]
        best = max(best, _speed(_prim([x.double() for x in cols])))
    return best


def _advance(U, nb, dtd):
    """One step of interior conserved values (a list of tensors), periodic in axis 0,
    reflecting walls in the others; returns the new values and their largest signal speed."""
    new = [torch.empty_like(x) for x in U]
    best, n = 0.0, nb[0]
    for a in range(0, n, _slab(nb)):
        b = min(n, a + _slab(nb))
        rows = torch.arange(a - 1, b + 1, device="cuda") % n
        P = _prim([x.index_select(0, rows) for x in U])
        F = _flux(_cut(P, 0, slice(None, -1)), _cut(P, 0, slice(1, None)), 0)
        upd = [x[a:b] + dtd[0] * (f[:-1] - f[1:]) for x, f in zip(U, F)]
        P = _cut(P, 0, slice(1, -1))
        for d in range(1, len(nb)):
            L = _join([_wall(P, d, slice(0, 1)), P], d)
            R = _join([P, _wall(P, d, slice(-1, None))], d)
            F = _flux(L, R, d)
            lo, hi = (slice(None),) * d + (slice(None, -1),), (slice(None),) * d + (slice(1, None),)
            upd = [x + dtd[d] * (f[lo] - f[hi]) for x, f in zip(upd, F)]
        for x, y in zip(new, upd):
            x[a:b] = y
        best = max(best, _speed(_prim(upd)))
    return new, best


def _evolve(nb, blast, steps, dtype):
    """A blast after `steps` iterations: conserved values, t, Dt and the largest speed."""
    at = [torch.arange(1, n + 1, dtype=torch.float64, device="cuda") for n in nb]
    r2 = sum(((v - c) ** 2).view((1,) * i + (-1,) + (1,) * (len(nb) - 1 - i)) for i, (v, c) in enumerate(zip(at, blast.centre)))
    T = NP[dtype]
    E = [float(T(T(p) / T(T(GAMMA) - T(1)))) for p in (blast.p_in, blast.p_out)]
    U = [torch.ones(nb, dtype=torch.float64, device="cuda"),
         torch.where(torch.sqrt(r2) <= blast.radius, *(r2.new_tensor(e) for e in E))] + [
             torch.zeros(nb, dtype=torch.float64, device="cuda") for _ in nb]
    D = [1.0 / (n + 1) for n in nb]
    C = (0.4 if len(nb) == 3 else 0.5) * min(D)
    dt, t, best = C / _speed(_prim(U)), 0.0, 0.0
    for _ in range(steps):
        U, best = _advance(U, nb, [dt / x for x in D])
        dt = C / best
        t += dt
    return U, t, dt, best


def _laid_out(U, nb, dtype):
    """(rhoE, uvx) in 64 bits, ghost cells at zero, laid out as the state arrays."""
    shape = tuple(n + 2 for n in nb)
    rhoE = torch.zeros(shape + (2,), dtype=torch.float64, device="cuda")
    uvx = torch.zeros(shape + (len(nb),), dtype=torch.float64, device="cuda")
    for i, x in enumerate(U):
        (rhoE if i < 2 else uvx)[_inner(nb) + (i if i < 2 else i - 2,)] = x
    return rhoE.view(-1), uvx.view(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "csv":
        return None
    if kind == "launch":
        nb = _nb(case)
        s = prepare(case, seed)
        R, V = (_shaped(a, nb) for a in s["state"])
        U = [R[_inner(nb) + (i,)].double() for i in range(2)] + [V[_inner(nb) + (i,)].double() for i in range(len(nb))]
        U, best = _advance(U, nb, [float(x) for x in s["dtd"]])
        dt = torch.tensor([float(s["phys"].C_min) / best], dtype=torch.float64)
        return _laid_out(U, nb, case["dtype"]) + (dt,)
    if kind == "loop":
        nb = _nb(case)
        U, t, dt, _ = _evolve(nb, _blast(random.Random(seed), nb), case["steps"], case["dtype"])
        return _laid_out(U, nb, case["dtype"]) + (np.array([t, dt]),)
    rng = random.Random(seed)
    states, told = [], []
    for nb in _sizes(case):
        U, t, dt, best = _evolve(nb, _blast(rng, nb), case["steps"], case["dtype"])
        states.append((torch.stack(U[:2], -1), torch.stack(U[2:], -1)))
        told.append([t, dt, float(U[0].sum()), float(U[1].sum()), best])
    return states, np.array(told)
