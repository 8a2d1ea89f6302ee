"""Strict steps of states at the ends of the type's range against the oracle, bit for bit:
pressures and momenta down to subnormal numbers, fluxes that overflow, cells of every size next
to one another (those inside and outside of the conversion's straight-line range in one warp),
and a negative K."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_pkg

hb = load_pkg()
pytestmark = pytest.mark.gpu

SHAPES = [(40, 130), (12, 21, 62)]
KINDS = ["tiny", "tiny mixed", "tiny pressure", "huge", "huge mixed", "mixed", "edges", "slow"]


def state(nb, T, seed, kind):
    """(rhoE, uvx) in the reference layout and a bound of its signal speeds."""
    rng = np.random.default_rng(seed)
    n, d = int(np.prod([k + 2 for k in nb])), len(nb)
    end = 36 if T is np.float32 else 306
    rho, p, vel = rng.uniform(0.5, 2.0, n), rng.uniform(0.05, 10.0, n), rng.uniform(-0.5, 0.5, (n, d))
    f = np.ones(n)  # of the pressure, and squared of the velocity
    if kind == "tiny":
        f *= 10.0 ** -end
    elif kind == "tiny mixed":
        f = 10.0 ** rng.uniform(-end - 2, -end / 2, n)
    elif kind == "tiny pressure":
        p *= 10.0 ** rng.uniform(-end - 1, 0, n)
    elif kind == "huge":
        f *= 10.0 ** end
    elif kind == "huge mixed":
        f = 10.0 ** rng.uniform(0, end + 1, n)
    elif kind == "mixed":
        rho, p = rho * 10.0 ** rng.uniform(-9, 9, n), p * 10.0 ** rng.uniform(-9, 9, n)
    elif kind == "edges":  # densities next to 2^20 and 2^-20 (FP64 2^+-200), impedances to match
        e = 20 if T is np.float32 else 200
        rho = np.ldexp(rng.uniform(0.9, 1.1, n), rng.choice([-e, 0, e], n))
        p = np.ldexp(rng.uniform(0.6, 0.8, n), rng.choice([-e, 0, e], n))
        vel *= np.sqrt(p / rho)[:, None]
    elif kind == "slow":
        vel *= 10.0 ** rng.uniform(-end - 1, -end + 3, (n, d))
    p, vel = p * f, vel * np.sqrt(f)[:, None]
    with np.errstate(over="ignore"):
        E = p / 0.4 + 0.5 * rho * (vel ** 2).sum(1)
        speed = float(np.sqrt((1.4 * p / rho).max()) + np.abs(vel).max())
        return (np.stack([rho, E], 1).reshape(-1).astype(T), (vel * rho[:, None]).reshape(-1).astype(T)), speed


def same(a, b):
    """Equal bits, any NaN for any NaN."""
    u = np.uint32 if a.dtype == np.float32 else np.uint64
    return bool(((a.view(u) == b.view(u)) | (np.isnan(a) & np.isnan(b))).all())


@pytest.mark.parametrize("K", [1.1, -1.1, 3e6])
@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("nb", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_states_at_the_ends_of_the_range(cuda, oracle, kind, nb, T, K):
    for seed in range(3):
        phys = hb.Physics(T, nb, K=K)
        st, speed = state(nb, T, seed, kind)
        oracle.ghost_x(st, nb)
        ref = tuple(np.zeros_like(a) for a in st)
        dtd = phys.dtd(T(0.1 * float(phys.min_spacing) / min(max(speed, 1e-30), 1e30)))
        dref = oracle.step(st, ref, phys, dtd)
        for kernel in (hb.KERNEL_STRIP, hb.KERNEL_DIRECT):
            cur = tuple(cuda.from_numpy(a.copy()).cuda() for a in st)
            nxt = tuple(cuda.zeros_like(a) for a in cur)
            dt = cuda.zeros(1, dtype=cur[0].dtype, device="cuda")
            rc, _ = hb.step(cur, nxt, dt, phys, dtd, kernel=kernel, arith="strict", check=False)
            for a, b in zip(nxt, ref):
                assert same(a.cpu().numpy(), b), (seed, kernel)
            if rc == hb.HYDRO_OK:  # (with a NaN among them the reference's max depends on their order)
                assert phys.dtype(dt.item()).tobytes() == dref.tobytes()


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("nb", [(8, 40), (6, 9, 40)])
def test_impedance_of_the_largest_significand(cuda, oracle, nb, T, sign):
    """K = +-(1 - 2^-53) and cells with gamma p rho = 1: K a has the one significand whose reciprocal
    lies next to a rounding midpoint."""
    phys = hb.Physics(T, nb, gamma=2.0, K=sign * float(T(1) - np.finfo(T).epsneg))
    rng = np.random.default_rng(11)
    n = int(np.prod([k + 2 for k in nb]))
    E = np.where(rng.random(n) < 0.5, 0.5, rng.uniform(0.01, 0.49, n)) # p = E, gas at rest of density 1
    st = (np.stack([np.ones(n), E], 1).reshape(-1).astype(T), np.zeros(n * len(nb), T))
    oracle.ghost_x(st, nb)
    ref = tuple(np.zeros_like(a) for a in st)
    dtd = phys.dtd(T(0.1) * phys.min_spacing)
    dref = oracle.step(st, ref, phys, dtd)
    for kernel in (hb.KERNEL_STRIP, hb.KERNEL_DIRECT):
        cur = tuple(cuda.from_numpy(a.copy()).cuda() for a in st)
        nxt = tuple(cuda.zeros_like(a) for a in cur)
        dt = cuda.zeros(1, dtype=cur[0].dtype, device="cuda")
        rc, _ = hb.step(cur, nxt, dt, phys, dtd, kernel=kernel, arith="strict", check=False)
        assert all(same(a.cpu().numpy(), b) for a, b in zip(nxt, ref)), kernel
        # (K < 0 adds to the differences it should even out: some new pressures are negative)
        assert rc == hb.HYDRO_ERR_NONPHYSICAL or phys.dtype(dt.item()).tobytes() == dref.tobytes()
