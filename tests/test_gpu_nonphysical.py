"""A new state with a negative pressure (positive density, energy below the kinetic energy) is
reported by every call, wherever the cell lies, whatever history the signal-speed skip has and
whichever of the launch's blocks have finished by then."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_pkg

hb = load_pkg()
pytestmark = pytest.mark.gpu

# three cells along X in gas at rest (density 1, pressure 1), which with Dt / DX = 0.081 leave a
# cell behind whose energy is 0.06 of its kinetic energy and whose speed bound is 1.9
PATCH = [(0.05177534, 0.00885609, 7.23058716, 1.97188887), (0.05436528, 0.05401418, -0.50276884, -8.16626605),
         (2.16991578, 0.00284897, -2.61052343, 0.40176438)]
DTD = 0.3 / 3.7


def make(nb, T, row, patch=True):
    """Gas at rest, hot (speed 5.3) in two columns, with the patch around X row `row`."""
    d = len(nb)
    W = np.zeros(tuple(n + 2 for n in nb) + (2 + d,))
    W[..., 0], W[..., 1] = 1.0, 1.0
    W[:, 1:3, ..., 1] = 20.0
    if patch:
        for i, (r, p, u, v) in enumerate(PATCH):
            W[row - 1 + i, nb[1] // 2, ..., :4] = (r, p, u, v)
    E = W[..., 1] / 0.4 + 0.5 * W[..., 0] * (W[..., 2:] ** 2).sum(-1)
    rhoE = np.stack([W[..., 0], E], -1).reshape(-1).astype(T)
    return rhoE, (W[..., 2:] * W[..., :1]).reshape(-1).astype(T)


@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("small, big, chunk", [((9, 12), (3000, 700), 2), ((9, 12, 5), (400, 60, 70), 1)])
@pytest.mark.parametrize("arith", ["strict", "fused"])
def test_negative_pressure_is_reported(cuda, oracle, orc, small, big, chunk, T, arith):
    phys = hb.Physics(T, small)
    st = make(small, T, 5)
    ref = tuple(np.zeros_like(a) for a in st)
    dtd = [T(DTD)] * len(small)
    oracle.step(st, ref, phys, dtd)
    rhoE, m = (a.astype(np.float64) for a in orc.interior(ref, small))
    over = (m ** 2).sum(-1) / (2 * rhoE[..., 0] * rhoE[..., 1])
    assert (rhoE > 1e-3).all() and (over[4, 5] > 2).all() and np.sort(over.ravel())[:-over[4, 5].size].max() < 0.99

    phys = hb.Physics(T, big)
    try:
        hb.set_launch_shape(len(big), T, 0, chunk, 0)  # more blocks than the GPU holds at a time
        for row in (3, big[0] // 2, big[0] - 3):
            states = [tuple(cuda.from_numpy(a).cuda() for a in make(big, T, row, patch)) for patch in (False, True)]
            nxt = tuple(cuda.zeros_like(a) for a in states[0])
            keep = []
            for with_history in (False, False, True):
                dt = cuda.zeros(1, dtype=nxt[0].dtype, device="cuda")
                keep.append(dt)  # (the history goes by the address of Dt)
                if with_history:
                    assert hb.step(states[0], nxt, dt, phys, dtd, arith=arith, check=False)[0] == hb.HYDRO_OK
                rc, info = hb.step(states[1], nxt, dt, phys, dtd, arith=arith, check=False)
                assert rc == hb.HYDRO_ERR_NONPHYSICAL and info.err & 1, (row, with_history)
    finally:
        hb.set_launch_shape(len(big), T, 0, 0, 0)
