// The bookkeeping of a ring of shared-memory stages that one thread fills and every thread waits
// for (strip3d_march.cuh), apart from the barriers themselves: no CUDA in here, so that it can be
// run on the host.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define HYDRO_HD __host__ __device__ __forceinline__
#else
#define HYDRO_HD inline
#endif

namespace hydro {

// A thread's place in the ring, the same in every thread, and what it gave up on.
template <int NS> struct Ring {
    int st = 0;         // the stage of the plane at hand
    uint32_t phase = 0; // the parity of its barrier's phase
    // 0: every wait so far ended. n > 0: a bounded wait gave up on a plane n planes before the end
    // of its march; this thread waits no more, and issues no more. -1: the same in an earlier march.
    int dead = 0;

    HYDRO_HD void advance()
    {
        if (++st == NS) {
            st = 0;
            phase ^= 1u;
        }
    }
    // Behind the last plane: the loads that may be in flight still, those of the plane that was given
    // up on and of the planes issued ahead of it (its own place among the NS stages and the next
    // ones; a plane is issued NS - 1 ahead, no further than the last one). wait(stage, parity) for
    // each.
    template <class F> HYDRO_HD void drain(F &&wait)
    {
        for (int back = dead, n = 0; back > 0 && n < NS; --back, ++n) {
            const int turns = back > st ? (back - st + NS - 1) / NS : 0; // from that plane's place to here
            wait(st - back + turns * NS, phase ^ (uint32_t)(turns & 1));
        }
        if (dead > 0) dead = -1;
    }
};

} // namespace hydro
