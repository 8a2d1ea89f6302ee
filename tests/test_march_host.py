"""Host-side parts of the steps, without a GPU: what a step returns for its error bits, and the
bookkeeping of the 3D march's ring of stages, and the split of its planes."""
from __future__ import annotations

import ctypes
import random
import subprocess

import pytest

from conftest import ROOT, load_pkg

hb = load_pkg()


@pytest.fixture(scope="module", autouse=True)
def built():
    hb.build()


def test_result_of_a_step_by_its_error_bits():
    """A step that reports a wait that gave up (bit 1) returns HYDRO_ERR_TIMEOUT, also where the
    state is non-physical (bit 0) too, and leaves its scratch words to be zeroed. The synchronous 2D
    and 3D steps and hydro_last_step_info share this mapping."""
    fn = hb.lib()["_ZN5hydro11step_resultEjPKcPb"]
    fn.argtypes = [ctypes.c_uint, ctypes.c_char_p, ctypes.POINTER(ctypes.c_bool)]
    for bits, rc, word in ((0, hb.HYDRO_OK, None), (1, hb.HYDRO_ERR_NONPHYSICAL, "non-physical"),
                           (2, hb.HYDRO_ERR_TIMEOUT, "timed out"), (3, hb.HYDRO_ERR_TIMEOUT, "timed out")):
        hb.lib().hydro_clear_error()
        dirty = ctypes.c_bool(False)
        assert fn(bits, b"step3d", ctypes.byref(dirty)) == rc
        assert dirty.value == (rc == hb.HYDRO_ERR_TIMEOUT)
        code, msg = hb.last_error()
        assert (code, bool(word) and word in msg and "step3d" in msg) == (rc, bool(word))
        assert fn(bits, None, ctypes.byref(dirty)) == rc


RING = r"""
#include <cstdio>
#include <vector>
#include "ring.h"

// A barrier that one arrival and its bytes complete.
struct Barrier {
    int completed = 0;
    bool pending = false;
    bool over(uint32_t parity) const { return (uint32_t)(completed & 1) != parity; }
    void land() { if (pending) { pending = false; ++completed; } }
};

// Marches of `planes` planes through one ring, as thread 0 runs them; plane `lost` of march `which`
// never lands while it is waited for. Returns the number of rules broken.
template <int NS> int run(const std::vector<int> &planes, int which, int lost)
{
    hydro::Ring<NS> ring;
    Barrier bar[NS];
    int bad = 0;
    for (int k = 0; k < (int)planes.size(); ++k) {
        const int n = planes[k];
        int loads = 0;
        auto issue = [&](int m, int s) {
            if (m < n && !ring.dead) {
                bad += bar[s].pending; // a second arrival within a phase
                bar[s].pending = true;
                ++loads;
            }
        };
        for (int m = 0, s = ring.st; m < NS - 1; ++m, s = s + 1 == NS ? 0 : s + 1) issue(m, s);
        for (int m = 0; m < n; ++m) {
            issue(m + NS - 1, ring.st == 0 ? NS - 1 : ring.st - 1);
            if (!ring.dead) {
                bad += bar[ring.st].over(ring.phase); // the phase of plane m is this one
                if (k == which && m == lost) {
                    ring.dead = n - m;
                } else {
                    bar[ring.st].land();
                    bad += !bar[ring.st].over(ring.phase);
                }
            }
            ring.advance();
        }
        std::vector<bool> drained(NS, false);
        ring.drain([&](int s, uint32_t parity) {
            bad += s < 0 || s >= NS || drained[s] || !bar[s].pending || bar[s].over(parity);
            drained[s] = true;
            bar[s].land();
            bad += !bar[s].over(parity);
        });
        for (const Barrier &b : bar) bad += b.pending; // a load in flight behind the march
        bad += k > which && loads > 0;
        bad += (ring.dead != 0) != (k >= which);
    }
    return bad;
}

int main()
{
    int cases = 0;
    for (int n0 = 3; n0 < 12; ++n0)
        for (int n1 = 3; n1 < 12; ++n1)
            for (int which = 0; which < 4; ++which)
                for (int lost = 0; lost < (which == 0 ? n0 : which == 1 ? n1 : which == 2 ? 5 : 1); ++lost, ++cases)
                    if (run<3>({n0, n1, 5}, which, lost) || run<4>({n0, n1, 5}, which, lost)) {
                        printf("%d %d march %d plane %d\n", n0, n1, which, lost);
                        return 1;
                    }
    printf("%d cases\n", cases);
    return 0;
}
"""


def test_ring_after_a_wait_that_gave_up(tmp_path):
    """A march whose wait for a plane gave up issues no further load (a second arrival within a
    phase, a load that nothing waits for) and drains exactly those in flight, at every plane, number
    of planes and place in the ring."""
    (tmp_path / "ring.cpp").write_text(RING)
    exe = tmp_path / "ring"
    csrc = ROOT / "scalable-fpga-hydrodynamics_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(csrc), "-o", str(exe), str(tmp_path / "ring.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


class Chunks(ctypes.Structure):
    _fields_ = [("longs", ctypes.c_int), ("len", ctypes.c_int), ("rest", ctypes.c_int), ("count", ctypes.c_int)]

    def begin(self, k):
        return 1 + (k * self.len if k < self.longs else self.longs * self.len + (k - self.longs) * self.rest)


def march_chunks(rows, tiles, per_sm, cap=0, least=3):
    """How the 3D step splits `rows` planes over `tiles` columns of blocks (csrc/context.cu)."""
    fn = hb.lib()["_ZN5hydro12march_chunksEmmiii"]
    fn.argtypes = [ctypes.c_size_t, ctypes.c_size_t] + [ctypes.c_int] * 3
    fn.restype = Chunks
    return fn(rows, tiles, per_sm, cap, least)


def test_chunks_cover_every_plane_once():
    """Long chunks and short ones, any numbers: each plane belongs to one chunk, none is empty, at most
    65535 of them, and an asked-for chunk length is not exceeded."""
    two = ragged = 0
    rng = random.Random(3)
    for _ in range(4000):
        rows = max(1, int(10 ** rng.uniform(0, 4.5)))
        tiles = max(1, int(10 ** rng.uniform(0, 4)))
        cap = rng.choice([0, 0, 0, 1, 2, 7, 64, 300])
        # (without a GPU the model sees one SM: the resident blocks of 148 asked for in its place)
        c = march_chunks(rows, tiles, rng.choice([1, 2, 3, 222, 296, 444]), cap, rng.choice([2, 3]))
        ends = [min(c.begin(k + 1) - 1, rows) for k in range(c.count)]
        assert 1 <= c.count <= 65535 and c.begin(0) == 1 and ends[-1] == rows, (rows, tiles, cap)
        assert all(c.begin(k) <= ends[k] for k in range(c.count)), (rows, tiles, cap)
        assert all(ends[k] + 1 == c.begin(k + 1) for k in range(c.count - 1)), (rows, tiles, cap)
        assert cap == 0 or (c.longs == 0 and c.rest <= cap)
        two += c.longs > 0
        ragged += c.longs > 0 and rows - c.begin(c.count - 1) + 1 < c.rest
    assert two > 100 and ragged > 50
