"""The strict arithmetic's straight-line reciprocal and square root (csrc/hydro_math.cuh, Ex)
are correctly rounded: equal to IEEE division and square root on the host, bit for bit.

FP32: every significand, at exponents of both parities over the range the kernels use.
FP64: random significands, and the inputs that a correction step of this kind could round
the wrong way, those whose exact result lies within about 2^-46 ulp of a rounding midpoint:
* reciprocal: n q = 2^106 - k with n of 53 bits, q odd of 54 bits; k = 1 has the single
  solution n = 2^53 - 1 (2^106 - 1 = (2^53 - 1)(2^53 + 1)); the divisors of 2^106 - 2 too;
* square root: s - (q/2)^2 = c in units of 2^-106, q odd: q^2 = -c mod 2^54 (s in [1, 2)) or
  mod 2^55 (s in [2, 4)), solved by lifting, for |c| <= 2048.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from conftest import load_pkg

hb = load_pkg()
pytestmark = pytest.mark.gpu


def _device(cuda, x):
    L = hb.lib()
    fn = L.hydro_strict_math_f64 if x.dtype == np.float64 else L.hydro_strict_math_f32
    fn.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    d = cuda.from_numpy(x).cuda()
    r, s = cuda.zeros_like(d), cuda.zeros_like(d)
    assert fn(hb._ptr(d), x.size, hb._ptr(r), hb._ptr(s), hb._stream_handle()) == 0, hb.last_error()
    return r.cpu().numpy(), s.cpu().numpy()


def _check(cuda, x):
    r, s = _device(cuda, x)
    one = x.dtype.type(1)
    bad = np.flatnonzero((one / x) != r)
    assert bad.size == 0, ("rcp", bad.size, [float(v).hex() for v in x[bad[:4]]])
    pos = x > 0
    bad = np.flatnonzero(np.sqrt(x[pos]) != s[pos])
    assert bad.size == 0, ("sqrt", bad.size, [float(v).hex() for v in x[pos][bad[:4]]])


@pytest.mark.parametrize("e", [-60, -31, -2, -1, 0, 1, 2, 30, 59])
def test_fp32_every_significand(cuda, e):
    x = ((np.arange(2 ** 23, dtype=np.uint32)) | np.uint32((127 + e) << 23)).view(np.float32)
    _check(cuda, x)
    r, _ = _device(cuda, -x)
    assert np.array_equal(np.float32(1) / -x, r)


def _sqrt_hard():
    """Significands s in [1, 4) near the square of a midpoint."""
    out = []
    for bits, lo, hi in ((54, 2 ** 53, math.isqrt(2 ** 107)), (55, math.isqrt(2 ** 107) + 1, 2 ** 54)):
        for c in range(-2048, 2049):
            if (-c) % 8 != 1:
                continue
            q = 1
            for k in range(3, bits):  # q^2 = -c mod 2^k -> mod 2^(k+1)
                if (q * q + c) % 2 ** (k + 1):
                    q += 2 ** (k - 1)
            assert (q * q + c) % 2 ** bits == 0
            for root in {q, -q, q + 2 ** (bits - 1), -q + 2 ** (bits - 1)}:
                root %= 2 ** bits
                for cand in (root, root + 2 ** bits):
                    if lo <= cand < hi:
                        n = (cand * cand + c) >> bits
                        if n < 2 ** 53:
                            out.append(math.ldexp(n, -52 if bits == 54 else -51))
    return out


def _rcp_hard():
    divs = {1}
    for f in (152041, 106681, 122921, 29191, 337, 151, 71, 7, 7, 31, 127, 2):  # 2^106 - 2
        divs |= {d * f for d in divs}
    return [math.ldexp(n, -52) for n in sorted(divs) if 2 ** 52 < n < 2 ** 53] + [math.ldexp(2 ** 53 - 1, -52)]


def test_fp64_hard_cases(cuda):
    hard = _sqrt_hard()
    assert len(hard) > 300 and all(1 <= v < 4 for v in hard)
    hard = np.array(hard + _rcp_hard() + [1.0, 2.0, 1.0 + 2 ** -52, 2.0 - 2 ** -52, 4.0 - 2 ** -51])
    for e in range(-398, 398, 2):  # even: the square root keeps its significand
        _check(cuda, hard * 2.0 ** e)


def test_fp64_random(cuda):
    rng = np.random.default_rng(7)
    x = np.ldexp(rng.uniform(1.0, 2.0, 4_000_000), rng.integers(-400, 400, 4_000_000))
    _check(cuda, x)
    near = 1.0 + rng.integers(0, 2 ** 20, 500_000) * 2.0 ** -52  # next to 1, 2 and 4
    _check(cuda, np.concatenate([near, 2.0 / near, 4.0 / near]))


def test_fp64_hard_cases_negative(cuda):
    """The reciprocals of negative arguments, which the impedances of K < 0 are."""
    x = -np.array(_rcp_hard() + [1.0, 2.0, 1.0 + 2 ** -52, 1.5 - 2 ** -52, 4.0 - 2 ** -51])
    for e in range(-399, 399, 3):
        r, _ = _device(cuda, x * 2.0 ** e)
        assert np.array_equal(1.0 / (x * 2.0 ** e), r)
    rng = np.random.default_rng(8)
    x = -np.ldexp(rng.uniform(1.0, 2.0, 4_000_000), rng.integers(-400, 400, 4_000_000))
    assert np.array_equal(1.0 / x, _device(cuda, x)[0])
