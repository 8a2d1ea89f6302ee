"""The 3D march's staging against the oracle, bit for bit: rows of momenta that start at every
place within 16 bytes (NB_Z mod 4, odd and even numbers of rows per plane), tiles that end at a
wall with one to all of their rows and columns, X ghost planes from memory, arrays aligned to
their values only, and chunks that start and end at the periodic planes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_pkg
from test_oracle import cfl_dt, seeded_state

hb = load_pkg()
pytestmark = pytest.mark.gpu

GRIDS = [(5, 8, 29), (5, 8, 30), (5, 9, 31), (6, 7, 32), (4, 15, 61), (4, 22, 62), (7, 16, 63), (3, 9, 91), (1, 1, 1),
         (2, 14, 33)]


def _run(cuda, oracle, nb, T, offset, x_ghosts):
    phys = hb.Physics(T, nb)
    st = seeded_state(nb, T, 5)
    if x_ghosts:
        other = seeded_state(nb, T, 6)
        for a, b in zip(st, other):
            k = a.size // (nb[0] + 2)
            a[:k], a[-k:] = b[k:2 * k], b[-2 * k:-k]
    else:
        oracle.ghost_x(st, nb)
    ref = tuple(np.zeros_like(a) for a in st)
    dtd = phys.dtd(cfl_dt(phys, 5))
    dref = oracle.step(st, ref, phys, dtd)

    def dev(a):
        v = cuda.zeros(a.size + offset, dtype=cuda.from_numpy(a[:1]).dtype, device="cuda")[offset:]
        v.copy_(cuda.from_numpy(a))
        return v

    cur, nxt = tuple(dev(a) for a in st), tuple(dev(np.zeros_like(a)) for a in st)
    dt = cuda.zeros(1, dtype=cur[0].dtype, device="cuda")
    _, info = hb.step(cur, nxt, dt, phys, dtd, kernel=hb.KERNEL_STRIP, x_ghosts=x_ghosts, arith="strict")
    assert info.kernel == hb.KERNEL_STRIP
    assert phys.dtype(dt.item()).tobytes() == dref.tobytes()
    for a, b in zip(nxt, ref):
        assert a.cpu().numpy().tobytes() == b.tobytes()


@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("x_ghosts", [False, True])
@pytest.mark.parametrize("nb", GRIDS)
def test_staging(cuda, oracle, nb, T, x_ghosts):
    _run(cuda, oracle, nb, T, 0, x_ghosts)


@pytest.mark.parametrize("T, offset", [(np.float64, 1), (np.float32, 1), (np.float32, 2), (np.float32, 3)])
@pytest.mark.parametrize("nb", [(5, 8, 30), (4, 15, 61)])
def test_arrays_aligned_to_their_values(cuda, oracle, nb, T, offset):
    _run(cuda, oracle, nb, T, offset, False)


@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("chunk", [1, 2, 5])
def test_chunks(cuda, oracle, T, chunk):
    try:
        hb.set_launch_shape(3, T, 0, chunk, 0)
        _run(cuda, oracle, (7, 9, 35), T, 0, False)
        assert hb.last_launch_shape()["chunk"] <= chunk
    finally:
        hb.set_launch_shape(3, T, 0, 0, 0)


@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("nb, chunk", [((150, 150, 150), 48), ((151, 151, 149), None), ((3001, 13, 59), None)])
def test_long_and_short_chunks(cuda, oracle, nb, T, chunk):
    """Columns split in two lengths of chunk, with a ragged last one."""
    _run(cuda, oracle, nb, T, 0, False)
    if chunk and T is np.float64:
        assert hb.last_launch_shape()["chunk"] == chunk


@pytest.mark.parametrize("T, nb", [(np.float32, (203, 197, 199)), (np.float32, (221, 150, 148)),
                                   (np.float64, (170, 170, 170)), (np.float64, (203, 151, 149))])
def test_two_lengths_and_a_ragged_end(cuda, oracle, T, nb):
    """Grids whose columns are split in long and short chunks with a shorter last one, by tensor maps
    and by row copies, in both precisions."""
    from test_march_host import march_chunks

    tiles = -(-nb[1] // 7) * -(-nb[2] // 30)
    c = march_chunks(nb[0], tiles, 2 if T is np.float64 else 3)
    assert c.longs > 0 and 0 < nb[0] - c.begin(c.count - 1) + 1 < c.rest
    _run(cuda, oracle, nb, T, 0, False)
    shape = hb.last_launch_shape()
    assert shape["chunk"] == c.len and shape["tma"] == (T is np.float64 and nb[2] % 2 == 0)
