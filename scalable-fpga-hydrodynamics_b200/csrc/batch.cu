// Batched step: many independent 2D or 3D blast instances of uneven sizes advanced by
// one persistent kernel per step, each instance with its own time step, boundaries and
// simulated time (the layered "batching" change of the plain path; no counterpart in the
// reference, whose host loop advances one domain, hydro2d/main.cxx:689-815).
//
// Each instance keeps the plain path's arithmetic: the same strip march
// (strip2d_march.cuh / strip3d_march.cuh), so an instance's state after n batched steps
// is bit-identical to n plain steps in the same precision. 2D instances keep the pair
// layout with rows padded to 16 bytes; 3D instances keep the reference's
// pair/triple layout (row copies). Work is a flat list of items, rows or planes of a strip or
// tile of an instance, long ones first and short ones last; persistent blocks take one item each by
// their number and more from an atomic counter. Every item writes its max signal speed and error
// bits to its own slot; the item that completes an instance's step (ticket per instance) merges
// that instance's slots -- the result depends neither on which block ran which item nor on how
// the rows were cut nor on the other instances in the batch -- and advances
// the instance on the device:
//   Dt = min(1e20, C_min / max_speed)   (hydro2d/kernel.cxx:318, main.cxx:706-781)
//   t += Dt (FP64 accumulator), DtDx = Dt / DX ... (main.cxx:703-704, in T)
//   active while t < t_end and steps < max_steps (main.cxx:689)
// so a step needs no host round trip and n steps are captured as one CUDA graph. The
// graph ends with one pass over the final state that forms each instance's compensated
// FP64 conservation sums (mass, momenta, energy) over items of its own, merged per
// instance in a fixed order (the step kernels carry no sums: fewer registers, more
// resident blocks). The signal speed uses the plain path's exact skip (see
// batch_threshold).
#include <algorithm>
#include <stdio.h>
#include <string.h>
#include <utility>
#include <vector>

#include "../../include/hydro_b200.h"
#include "hydro_host.h"
#include "strip2d_march.cuh"
#include "strip3d_march.cuh"

namespace hydro {

constexpr int kSums = 5; // rho, rho u, rho v, rho w (0 in 2D), E

template <class T> struct alignas(128) Inst2 {
    T *rhoE[2], *uv[2];
    Phys<T> ph;
    T DX, DY, dt, DtDx, DtDy;
    double t, t_end;
    double vmax_prev; // exact max signal speed of the previous step (0 before the first)
    float ggm1;       // gamma * (gamma - 1), for the signal-speed skip test
    long long exact_passes;
    unsigned sum_items; // items of the end-of-run conservation sums done
    long long ys;
    long long steps, max_steps;
    int nb_x, nb_y;
    int parity, active;
    unsigned done_items, err;
};

template <class T> struct alignas(128) Inst3 {
    T *rhoE[2], *uvw[2];
    Phys<T> ph;
    T DX, DY, DZ, dt, DtDx, DtDy, DtDz;
    double t, t_end;
    double vmax_prev; // exact max signal speed of the previous step (0 before the first)
    float ggm1;       // gamma * (gamma - 1), for the signal-speed skip test
    long long exact_passes;
    unsigned sum_items; // items of the end-of-run conservation sums done
    long long zs, zy;
    long long steps, max_steps;
    int nb_x, nb_y, nb_z;
    int parity, active;
    unsigned done_items, err;
};

// A step item: rows (planes) i0 to i1 of one strip (tx) or tile (tx along Z, ty along Y) of an
// instance; its slot of the parts, and the slots of all of the instance's items.
struct __align__(16) Item {
    int inst, part, tx, ty, i0, i1, first, count;
};

// An item of the end-of-run sums: share k of `count` of an instance, the first of which has the
// slot `first` of the parts.
struct __align__(16) SumItem {
    int inst, k, first, count;
};

struct ItemPart {
    double s[kSums], c[kSums];
    unsigned long long maxbits;
    unsigned err, pad;
};

// per-slot status, host-mapped, written by the finalising item
struct SlotStatus {
    double t, dt, sums[kSums], max_speed;
    long long steps, exact_passes;
    int active;
    unsigned err;
};

// The end-of-run conservation sums of one item (compensated FP64), merged per instance.
struct BatchAcc {
    double s[kSums] = {0, 0, 0, 0, 0}, c[kSums] = {0, 0, 0, 0, 0};
    double vmax = 0.0;
    unsigned err = 0;

    __device__ __forceinline__ void kahan(int q, double x)
    {
        const double y = __dadd_rn(x, c[q]);
        const double tt = __dadd_rn(s[q], y);
        c[q] = __dsub_rn(y, __dsub_rn(tt, s[q]));
        s[q] = tt;
    }
    // conservation sums of one updated cell (the rho w sum stays 0 in 2D)
    template <int D, class T> __device__ __forceinline__ void add_sums(T r, T mu, T mv, T mw, T E)
    {
        kahan(0, (double)r);
        kahan(1, (double)mu);
        kahan(2, (double)mv);
        if (D == 3) kahan(3, (double)mw);
        kahan(4, (double)E);
        if (!(r > T(0))) err |= kErrNonPhysical;
    }
};

// What a step accumulates per cell: the max exact signal speed and error bits.
struct MaxAcc {
    double vmax = 0.0;
    unsigned err = 0;
    // a cell that the skip test does not pass (it passes positive densities only)
    template <class T> __device__ __forceinline__ void add_speed(T rho, double sp)
    {
        if (!(rho > T(0))) err |= kErrNonPhysical;
        vmax = (sp > vmax) ? sp : vmax;
        if (!(sp <= 1.0e300)) err |= kErrNonPhysical;
    }
};

// deterministic merge of (s, c) pairs: the lower lane's value first
__device__ __forceinline__ void merge_pair(double &s, double &c, double s2, double c2, bool upper)
{
    if (upper) {
        double a = s2, b = c2;
        neumaier_merge(a, b, s, c);
        s = a;
        c = b;
    } else {
        neumaier_merge(s, c, s2, c2);
    }
}

// Block-wide reduction of a BatchAcc; the result is valid in thread 0.
template <int NT> __device__ __forceinline__ void block_reduce(BatchAcc &a)
{
    constexpr int NW = NT / 32;
    __shared__ double r_s[NW][kSums], r_c[NW][kSums];
    __shared__ unsigned long long r_m[NW];
    __shared__ unsigned r_e[NW];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned long long mb = __double_as_longlong(a.vmax);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < kSums; ++q) {
            const double s2 = __shfl_xor_sync(0xffffffffu, a.s[q], o);
            const double c2 = __shfl_xor_sync(0xffffffffu, a.c[q], o);
            merge_pair(a.s[q], a.c[q], s2, c2, up);
        }
        const unsigned long long om = __shfl_xor_sync(0xffffffffu, mb, o);
        mb = om > mb ? om : mb;
        a.err |= __shfl_xor_sync(0xffffffffu, a.err, o);
    }
    if (lane == 0) {
        for (int q = 0; q < kSums; ++q) {
            r_s[warp][q] = a.s[q];
            r_c[warp][q] = a.c[q];
        }
        r_m[warp] = mb;
        r_e[warp] = a.err;
    }
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < NW; ++w) {
            for (int q = 0; q < kSums; ++q) neumaier_merge(a.s[q], a.c[q], r_s[w][q], r_c[w][q]);
            mb = r_m[w] > mb ? r_m[w] : mb;
            a.err |= r_e[w];
        }
        a.vmax = __longlong_as_double((long long)mb);
    }
    __syncthreads();
}

// The signal-speed skip of the plain path, per instance: a cell computes its exact
// speed only when its FP32 upper bound reaches kSkipFrac x the previous step's max.
// skip_frac is kSkipFrac unless a caller set another fraction (0 turns the skip off;
// above 1 every cell skips and every step takes the exact pass).
template <class I> __device__ __forceinline__ float batch_threshold(const I *in, double skip_frac)
{
    return __double2float_rd(skip_frac * in->vmax_prev);
}

// Exact max signal speed over an instance's new state (the buffer the step wrote),
// whole block; valid in thread 0. Runs only when every cell skipped the exact speed.
template <int NT> __device__ __forceinline__ double block_max(double v, unsigned &err)
{
    __shared__ unsigned long long s_max[NT / 32];
    const unsigned long long mb = block_max_bits<NT>((unsigned long long)__double_as_longlong(v), s_max);
    if (__syncthreads_or(err != 0)) err = kErrNonPhysical;
    return __longlong_as_double((long long)mb);
}
template <int NT, class T, bool kF> __device__ double exact_max(const Inst2<T> *in, unsigned &err)
{
    const int b = in->parity ^ 1;
    const T *r = in->rhoE[b], *u = in->uv[b];
    const long long ny = in->nb_y, n = (long long)in->nb_x * ny;
    double vmax = 0.0;
    for (long long q = threadIdx.x; q < n; q += NT) {
        const long long c = (1 + q / ny) * in->ys + 1 + q % ny;
        const double sp = (double)speed2<T, kF>(__ldcg(r + 2 * c), __ldcg(u + 2 * c), __ldcg(u + 2 * c + 1),
                                                __ldcg(r + 2 * c + 1), in->ph);
        vmax = (sp > vmax) ? sp : vmax;
        if (!(sp <= 1.0e300)) err = kErrNonPhysical;
    }
    return block_max<NT>(vmax, err);
}
template <int NT, class T, bool kF> __device__ double exact_max(const Inst3<T> *in, unsigned &err)
{
    const int b = in->parity ^ 1;
    const T *r = in->rhoE[b], *u = in->uvw[b];
    const long long ncol = (long long)in->nb_y * in->nb_z, n = (long long)in->nb_x * ncol;
    double vmax = 0.0;
    for (long long q = threadIdx.x; q < n; q += NT) {
        const long long rr = q % ncol;
        const long long c = (1 + q / ncol) * in->zy + (1 + rr / in->nb_z) * in->zs + 1 + rr % in->nb_z;
        const double sp = (double)speed3<T, kF>(__ldcg(r + 2 * c), __ldcg(u + 3 * c), __ldcg(u + 3 * c + 1),
                                                __ldcg(u + 3 * c + 2), __ldcg(r + 2 * c + 1), in->ph);
        vmax = (sp > vmax) ? sp : vmax;
        if (!(sp <= 1.0e300)) err = kErrNonPhysical;
    }
    return block_max<NT>(vmax, err);
}

template <class T> __device__ __forceinline__ void set_dtdz(Inst2<T> *, T) {}
template <class T> __device__ __forceinline__ void set_dtdz(Inst3<T> *in, T Dt) { in->DtDz = Ar<T>::div(Dt, in->DZ); }

// Time-step bookkeeping of one instance after its step (thread 0 of the finalising block).
template <class T, class I> __device__ __forceinline__ void advance(I *in, double vmax, unsigned err, SlotStatus *st)
{
    using A = Ar<T>;
    const T big = T(1e20);
    const T dtn = A::div(in->ph.C_min, static_cast<T>(vmax));
    const T Dt = (dtn < big) ? dtn : big;
    in->steps += 1;
    in->t = __dadd_rn(in->t, (double)Dt);
    in->dt = Dt;
    in->DtDx = A::div(Dt, in->DX);
    in->DtDy = A::div(Dt, in->DY);
    set_dtdz<T>(in, Dt);
    in->parity ^= 1;
    in->vmax_prev = vmax;
    in->err |= err;
    in->active = (in->t < in->t_end) && (in->steps < in->max_steps) && !(in->err & kErrNonPhysical);
    if (st) {
        st->t = in->t;
        st->dt = (double)Dt;
        st->max_speed = vmax;
        st->steps = in->steps;
        st->exact_passes = in->exact_passes;
        st->active = in->active;
        st->err = in->err;
    }
    __threadfence();
    in->done_items = 0;
}

// Block-wide max of a non-negative double and OR of error bits; valid in thread 0.
template <int NT> __device__ __forceinline__ double block_max_err(double v, unsigned &err)
{
    __shared__ unsigned long long s_max[NT / 32];
    __shared__ unsigned s_err;
    if (threadIdx.x == 0) s_err = 0u;
    __syncthreads();
    if (err) atomicOr(&s_err, err);
    const unsigned long long mb = block_max_bits<NT>((unsigned long long)__double_as_longlong(v), s_max);
    err = s_err;
    __syncthreads(); // s_err / s_max free for the next use
    return __longlong_as_double((long long)mb);
}

// Merge an instance's item maxima, take the exact pass if no cell reached the skip
// threshold, and advance the instance (whole block).
template <int NT, class T, bool kF, class I>
__device__ void finalize_step(I *in, const ItemPart *parts, int nitems, SlotStatus *st, double skip_frac)
{
    unsigned long long mb = 0ull;
    unsigned err = 0;
    for (int i = threadIdx.x; i < nitems; i += NT) {
        const unsigned long long m = __ldcg(&parts[i].maxbits);
        mb = m > mb ? m : mb;
        err |= __ldcg(&parts[i].err);
    }
    double vmax = block_max_err<NT>(__longlong_as_double((long long)mb), err);
    // cells whose speed bound was under the threshold skipped the exact speed; if no
    // cell reached the threshold the skipped cells may hold the max: all cells again
    __shared__ int s_redo;
    if (threadIdx.x == 0) s_redo = (vmax < (double)batch_threshold(in, skip_frac)) ? 1 : 0;
    __syncthreads();
    if (s_redo) {
        unsigned e2 = 0;
        const double m = exact_max<NT, T, kF>(in, e2);
        if (threadIdx.x == 0) {
            vmax = m;
            err |= e2;
            in->exact_passes += 1;
        }
    }
    if (threadIdx.x == 0) advance<T>(in, vmax, err, st);
}

// Merge an instance's conservation-sum slots (fixed thread and lane order: the result
// depends only on the instance) and publish them (whole block).
template <int NT, class I>
__device__ void finalize_sums(I *in, const ItemPart *parts, int nitems, SlotStatus *st)
{
    BatchAcc a;
    for (int i = threadIdx.x; i < nitems; i += NT) {
        const ItemPart &p = parts[i];
        for (int q = 0; q < kSums; ++q) neumaier_merge(a.s[q], a.c[q], __ldcg(&p.s[q]), __ldcg(&p.c[q]));
        a.err |= __ldcg(&p.err);
    }
    block_reduce<NT>(a);
    if (threadIdx.x == 0) {
        if (st)
            for (int q = 0; q < kSums; ++q) st->sums[q] = __dadd_rn(a.s[q], a.c[q]);
        __threadfence();
        in->sum_items = 0;
    }
}

// A step item's max and error bits into its slot; returns (in every thread) whether this
// item completed its instance's step.
template <int NT>
__device__ __forceinline__ bool publish_step(const MaxAcc &acc, ItemPart *parts, int w, unsigned *done, int nitems,
                                             int *s_last)
{
    unsigned err = acc.err;
    const double vmax = block_max_err<NT>(acc.vmax, err);
    if (threadIdx.x == 0) {
        ItemPart &p = parts[w];
        p.maxbits = (unsigned long long)__double_as_longlong(vmax);
        p.err = err;
        __threadfence();
        *s_last = (atomicAdd(done, 1u) == (unsigned)nitems - 1u);
    }
    __syncthreads();
    const bool last = *s_last != 0;
    if (last) __threadfence();
    return last;
}

// The item's partial sums into its slot; returns (in every thread) whether this item
// completed its instance's step.
template <int NT>
__device__ __forceinline__ bool publish_item(BatchAcc &acc, ItemPart *parts, int w, unsigned *done, int nitems,
                                             int *s_last)
{
    block_reduce<NT>(acc);
    if (threadIdx.x == 0) {
        ItemPart &p = parts[w];
        for (int q = 0; q < kSums; ++q) {
            p.s[q] = acc.s[q];
            p.c[q] = acc.c[q];
        }
        p.maxbits = (unsigned long long)__double_as_longlong(acc.vmax);
        p.err = acc.err;
        __threadfence();
        *s_last = (atomicAdd(done, 1u) == (unsigned)nitems - 1u);
    }
    __syncthreads();
    const bool last = *s_last != 0;
    if (last) __threadfence();
    return last;
}

// The item at hand, its instance's grid and constants, in shared memory: read again where they
// are needed. Held in registers through the march they cost about 30 of its 128 in 3D FP64, and
// it spilled: 8 steps of 15.8 M cells took 6.6 ms, so 4.2 ms (5.2 ms with the former march).
template <class T, class Grid> struct Now {
    int w;   // index of the item
    Item it;
    Grid grid;
    StepConsts<T> c;
};

// Thread 0: the block's next item. Taken when the one before is done: taken ahead, at its start, a
// block with a long item held back the one after it (10 steps of 24 2D instances 1145 against
// 1070 us).
__device__ __forceinline__ void next_item(int &next, unsigned *counter)
{
    if (threadIdx.x == 0) next = (int)(gridDim.x + atomicAdd(counter, 1u));
}

// resident blocks per SM the register budget of the 2D step aims at
template <class T> struct Batch2dOcc { static constexpr int value = sizeof(T) == 4 ? 6 : 4; };

// kF: fused arithmetic (hydro_math.cuh)
template <class T, bool kF>
__global__ void __launch_bounds__(kStripNT, Batch2dOcc<T>::value) batch2d(Inst2<T> *insts, const Item *items, int nitems,
                                                                             unsigned *counter, ItemPart *parts,
                                                                             SlotStatus *status, double skip_frac)
{
    __shared__ Smem2<T> S;
    __shared__ Now<T, Grid2> s_now;
    __shared__ int s_last;
    const volatile Now<T, Grid2> &now = s_now;
    int next = (int)blockIdx.x; // thread 0: the item to take
    for (;;) {
        __syncthreads(); // everyone is done with the previous item
        if (threadIdx.x == 0) {
            const int w = next;
            s_now.w = w;
            if (w < nitems) {
                const Item it = items[w];
                const Inst2<T> *I = insts + it.inst;
                s_now.it = it;
                s_now.grid = Grid2{I->nb_x, I->nb_y, 1, I->ys};
                s_now.c = StepConsts<T>(I->ph, I->DtDx, I->DtDy, T(0), (T)I->ggm1,
                                        (T)skip_tlo2(batch_threshold(I, skip_frac)));
                s_now.c.odd = I->ph.odd && !kF;
            }
        }
        __syncthreads();
        if (now.w >= nitems) break;
        MaxAcc acc;
        {
            const Inst2<T> *I = insts + now.it.inst;
            if (!I->active) {
                next_item(next, counter);
                continue;
            }
            const int par = I->parity;
            // (the constants stay in shared memory, the grid is copied: 24 instances of 10.4 M cells,
            // 10 steps FP32 1183 us fused and 1184 strict, FP64 1734 strict; all in shared memory
            // 1228 fused, constants copied 1230 FP32 strict and 1739 FP64)
            const volatile StepConsts<T> &ph = s_now.c;
            const Grid2 grid = s_now.grid;
            const March2 geo{kStripW * now.it.tx, now.it.i0, now.it.i1};
            march2d<T, kF>(S, I->rhoE[par], I->uv[par], I->rhoE[par ^ 1], I->uv[par ^ 1], geo, grid, ph,
                           [&](const Upd2<T> &o) {
                               if (!state_below(o, ph.ggm1, ph.tlo2))
                                   acc.add_speed(o.r, (double)speed2<T, kF>(o.r, o.u, o.v, o.E, ph));
                           });
        }
        next_item(next, counter); // (in flight while the item's result is published)
        Inst2<T> *I = insts + now.it.inst;
        const int first = now.it.first, count = now.it.count;
        if (publish_step<kStripNT>(acc, parts, now.it.part, &I->done_items, count, &s_last))
            finalize_step<kStripNT, T, kF>(I, parts + first, count, status ? status + now.it.inst : nullptr, skip_frac);
    }
}

// The tile of the 3D batch: 9 rows on 8 warps, planes by row copies (any NB_Z).
template <class T> using Tile3 = Smem3<T, 8, true, Stage3::Rows>;
template <class T> constexpr int k3NT = 32 * Tile3<T>::W;
template <class T> constexpr int k3TY = Tile3<T>::R - 2; // interior rows per tile

template <class T, bool kF>
__global__ void __launch_bounds__(k3NT<T>, min_blocks3<T>(8)) batch3d(Inst3<T> *insts, const Item *items, int nitems,
                                                                      unsigned *counter, ItemPart *parts,
                                                                      SlotStatus *status, double skip_frac)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Tile3<T> &S = *reinterpret_cast<Tile3<T> *>(smem_raw);
    __shared__ Now<T, Grid3> s_now;
    __shared__ int s_last;
    const volatile Now<T, Grid3> &now = s_now;
    const volatile StepConsts<T> &ph = s_now.c;
    const volatile Grid3 &grid = s_now.grid;
    march3d_init(S);
    Ring<Tile3<T>::NS> ring;
    int next = (int)blockIdx.x; // thread 0: the item to take
    for (;;) {
        __syncthreads(); // everyone is done with the previous item
        if (threadIdx.x == 0) {
            const int w = next;
            s_now.w = w;
            if (w < nitems) {
                const Item it = items[w];
                const Inst3<T> *I = insts + it.inst;
                s_now.it = it;
                s_now.grid = Grid3(I->nb_x, I->nb_y, I->nb_z, 1);
                s_now.c = StepConsts<T>(I->ph, I->DtDx, I->DtDy, I->DtDz, (T)I->ggm1,
                                        (T)skip_tlo2(batch_threshold(I, skip_frac)));
                s_now.c.odd = I->ph.odd && !kF;
            }
        }
        __syncthreads();
        if (now.w >= nitems) break;
        MaxAcc acc;
        {
            const Inst3<T> *I = insts + now.it.inst;
            if (!I->active) {
                next_item(next, counter);
                continue;
            }
            const int par = I->parity;
            const March3 geo{k3TZ * now.it.tx, k3TY<T> * now.it.ty, now.it.i0, now.it.i1};
            const bool ok = march3d<T, kF>(S, I->rhoE[par], I->uvw[par], I->rhoE[par ^ 1], I->uvw[par ^ 1], geo, grid,
                                           ph, Tmaps3{}, ring, [&](const Upd3<T> &o) {
                                               if (!state_below(o, ph.ggm1, ph.tlo2))
                                                   acc.add_speed(o.r, (double)speed3<T, kF>(o.r, o.u, o.v, o.w, o.E, ph));
                                           });
            if (!ok) acc.err |= kErrWaitTimeout;
        }
        next_item(next, counter); // (in flight while the item's result is published)
        Inst3<T> *I = insts + now.it.inst;
        const int first = now.it.first, count = now.it.count;
        if (publish_step<k3NT<T>>(acc, parts, now.it.part, &I->done_items, count, &s_last))
            finalize_step<k3NT<T>, T, kF>(I, parts + first, count, status ? status + now.it.inst : nullptr, skip_frac);
    }
}

// End-of-run conservation sums (compensated FP64 mass, momenta, energy) of every instance: one
// pass over the current state after the run's last step. An instance's items share its
// interior cells out evenly, kSumCells to each thread, so that their number and what they hold
// depend on the instance alone. kSumLoads cells are loaded at a time ahead of their additions,
// which are chains of four FP64 operations each: with one cell at a time they waited for its
// loads (10.4 M cells FP32 in 68 us, 4 at a time 74, 8 at a time 56; 15.8 M cells 3D FP64 226 us
// one at a time, 8 at a time 140).
constexpr int kSumNT = 128, kSumCells = 64, kSumLoads = 8;

// Where an instance's interior rows lie (3D: the rows (i, j) in order), in registers.
template <class T> struct Rows {
    const typename Vec2<T>::type *r;
    const T *u;
    int len, nj;        // cells of a row, rows per plane (1 in 2D)
    long long n, si, sj; // rows, strides of i and j in cells
    __device__ explicit Rows(const Inst2<T> *I)
        : r(reinterpret_cast<const typename Vec2<T>::type *>(I->rhoE[I->parity])), u(I->uv[I->parity]), len(I->nb_y),
          nj(1), n(I->nb_x), si(I->ys), sj(0)
    {
    }
    __device__ explicit Rows(const Inst3<T> *I)
        : r(reinterpret_cast<const typename Vec2<T>::type *>(I->rhoE[I->parity])), u(I->uvw[I->parity]), len(I->nb_z),
          nj(I->nb_y), n((long long)I->nb_x * I->nb_y), si(I->zy), sj(I->zs)
    {
    }
    // the first interior cell of row q
    __device__ __forceinline__ long long start(unsigned q) const
    {
        const unsigned i = q / (unsigned)nj, j = q - i * (unsigned)nj;
        return (1 + (long long)i) * si + (sj ? (1 + (long long)j) * sj : 0) + 1;
    }
};

template <int NT, int D, class T, class I> __device__ __forceinline__ void sum_item(const I *in, int y, int n, BatchAcc &acc)
{
    using V2 = typename Vec2<T>::type;
    const Rows<T> g(in);
    const long long total = g.n * g.len, q0 = total * y / n;
    int left = (int)(total * (y + 1) / n - q0) - (int)threadIdx.x; // cells from this thread's on
    unsigned row = (unsigned)((q0 + threadIdx.x) / g.len);
    int col = (int)((q0 + threadIdx.x) - (long long)row * g.len);
    long long base = g.start(row);
    while (left > 0) {
        long long c[kSumLoads];
        int got = 0;
#pragma unroll
        for (int e = 0; e < kSumLoads; ++e) {
            c[e] = base + col;
            got += left > 0;
            left -= NT;
            col += NT;
            if (col >= g.len && left > 0) {
                do {
                    col -= g.len;
                    ++row;
                } while (col >= g.len);
                base = g.start(row);
            }
        }
        V2 a[kSumLoads], b[kSumLoads];
        T m2[kSumLoads];
#pragma unroll
        for (int e = 0; e < kSumLoads; ++e) {
            const long long k = e < got ? c[e] : c[0];
            a[e] = __ldg(g.r + k);
            if (D == 2) {
                b[e] = __ldg(reinterpret_cast<const V2 *>(g.u) + k);
            } else {
                b[e].x = __ldg(g.u + 3 * k);
                b[e].y = __ldg(g.u + 3 * k + 1);
                m2[e] = __ldg(g.u + 3 * k + 2);
            }
        }
#pragma unroll
        for (int e = 0; e < kSumLoads; ++e)
            if (e < got) acc.add_sums<D>(a[e].x, b[e].x, b[e].y, D == 3 ? m2[e] : T(0), a[e].y);
    }
}

template <int NT, int D, class T, class I>
__global__ void __launch_bounds__(NT) batch_sums(I *insts, const SumItem *items, int nitems, unsigned *counter,
                                                 ItemPart *parts, SlotStatus *status)
{
    __shared__ int s_item;
    __shared__ int s_last;
    int next = (int)blockIdx.x; // thread 0: the item to take
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s_item = next;
            if (next < nitems) next = (int)(gridDim.x + atomicAdd(counter, 1u));
        }
        __syncthreads();
        const int w = s_item;
        if (w >= nitems) break;
        const SumItem it = items[w];
        I *in = insts + it.inst;
        BatchAcc acc;
        sum_item<NT, D, T>(in, it.k, it.count, acc);
        if (publish_item<NT>(acc, parts, it.first + it.k, &in->sum_items, it.count, &s_last))
            finalize_sums<NT>(in, parts + it.first, it.count, status ? status + it.inst : nullptr);
    }
}

// ----------------------------------------------------------------------- host engine ---
class BatchBase {
  public:
    virtual ~BatchBase() = default;
    virtual int add(const hydro_blast_t &spec) = 0;
    virtual int remove(int slot) = 0;
    virtual int run(int nsteps, bool sync) = 0;
    virtual int status(int slot, hydro_batch_status_t *out) = 0;
    virtual int state(int slot, const void **rhoE, const void **uvx, long long *row_stride) = 0;
    virtual size_t bytes(const hydro_blast_t &spec) const = 0;
    virtual int copy_state(int slot, void *rhoE, void *uvx, bool to_host) = 0;
    virtual int sync() = 0;
    virtual int prepare(int nsteps) = 0;
    virtual int set_skip_fraction(double f) = 0;
    virtual int set_arith(bool fused) = 0;
};

template <class T, int D> class BatchEngine final : public BatchBase {
    using Inst = typename std::conditional<D == 2, Inst2<T>, Inst3<T>>::type;

  public:
    BatchEngine(int chunk, int capacity, cudaStream_t stream, int *rc)
        : chunk_(chunk), cap_(capacity)
    {
        own_stream_ = (stream == nullptr);
        cudaError_t e = cudaSuccess;
        if (own_stream_) e = cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking);
        else stream_ = stream;
        if (e == cudaSuccess) e = cudaMalloc(&insts_, sizeof(Inst) * cap_);
        if (e == cudaSuccess) e = cudaMalloc(&counter_, sizeof(unsigned) * counters_);
        if (e == cudaSuccess) e = cudaMalloc(&scratch_bits_, 64);
        if (e == cudaSuccess) e = cudaMemset(scratch_bits_, 0, 64);
        if (e == cudaSuccess) e = cudaHostAlloc(&status_h_, sizeof(SlotStatus) * cap_, cudaHostAllocMapped);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer(&status_d_, status_h_, 0);
        if (e == cudaSuccess) memset(status_h_, 0, sizeof(SlotStatus) * cap_);
        int dev = 0, nsm = 1, occ = 1;
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        // persistent grid: the resident blocks of the step kernel (the smaller of the
        // strict and fused variants' occupancy)
        int occ_f = 1;
        if constexpr (D == 2) {
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch2d<T, false>, kStripNT, 0);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_f, batch2d<T, true>, kStripNT, 0);
        } else {
            smem_ = (int)sizeof(Tile3<T>);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(batch3d<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(batch3d<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch3d<T, false>, k3NT<T>, smem_);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_f, batch3d<T, true>, k3NT<T>, smem_);
        }
        blocks_ = nsm * std::max(1, std::min(occ, occ_f));
        int occ_s = 0;
        if (e == cudaSuccess) {
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, batch_sums<kSumNT, D, T, Inst>, kSumNT, 0);
        }
        sum_blocks_ = nsm * std::max(1, occ_s);
        slots_.resize(cap_);
        *rc = (e == cudaSuccess) ? kOk : kErrCuda;
        if (e != cudaSuccess) set_error(kErrCuda, "batch create: %s", cudaGetErrorString(e));
    }

    ~BatchEngine() override
    {
        if (graph_) cudaGraphExecDestroy(graph_);
        for (auto &s : slots_)
            if (s.used) free_slot(s);
        cudaStreamSynchronize(stream_);
        cudaFree(insts_);
        cudaFree(counter_);
        cudaFree(scratch_bits_);
        cudaFree(parts_);
        cudaFreeHost(status_h_);
        if (own_stream_) cudaStreamDestroy(stream_);
    }

    // 2D rows are padded to a 16-byte multiple (one spare cell for odd NB_Y in FP32); 3D keeps the
    // reference strides.
    static size_t row_stride(size_t nb_y)
    {
        const size_t per = 16 / (2 * sizeof(T)); // cells per 16 bytes of one pair array
        return (nb_y + 2 + per - 1) / per * per;
    }

    size_t bytes(const hydro_blast_t &s) const override
    {
        if constexpr (D == 2) return 2 * 4 * sizeof(T) * (s.nb[0] + 2) * row_stride(s.nb[1]);
        else return 2 * 5 * sizeof(T) * (s.nb[0] + 2) * (s.nb[1] + 2) * (s.nb[2] + 2);
    }

    int add(const hydro_blast_t &s) override
    {
        const size_t nb_x = s.nb[0], nb_y = s.nb[1], nb_z = (D == 3) ? s.nb[2] : 0;
        const size_t lim = D == 2 ? (1u << 24) : (1u << 14);
        if (nb_x == 0 || nb_y == 0 || nb_x > lim || nb_y > lim || (D == 3 && (nb_z == 0 || nb_z > lim)) ||
            !(s.gamma > 1.0)) {
            set_error(kErrArg, "batch add: invalid %dD blast (grid %zu x %zu x %zu, gamma %g)", D, nb_x, nb_y, nb_z,
                      s.gamma);
            return kErrArg;
        }
        int slot = -1;
        for (int i = 0; i < cap_; ++i)
            if (!slots_[i].used) {
                slot = i;
                break;
            }
        if (slot < 0) {
            set_error(kErrArg, "batch add: all %d slots are in use", cap_);
            return kErrArg;
        }
        Slot &sl = slots_[slot];
        const size_t ys = (D == 2) ? row_stride(nb_y) : nb_y + 2;
        const size_t ncell = (D == 2) ? ys * (nb_x + 2) : (nb_x + 2) * (nb_y + 2) * (nb_z + 2);
        const size_t nv = (D == 2) ? 2 : 3;
        cudaError_t e = cudaSuccess;
        for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
            e = cudaMallocAsync(&sl.rhoE[b], 2 * ncell * sizeof(T), stream_);
            if (e == cudaSuccess) e = cudaMallocAsync(&sl.uvx[b], nv * ncell * sizeof(T), stream_);
            if (e == cudaSuccess) e = cudaMemsetAsync(sl.rhoE[b], 0, 2 * ncell * sizeof(T), stream_);
            if (e == cudaSuccess) e = cudaMemsetAsync(sl.uvx[b], 0, nv * ncell * sizeof(T), stream_);
        }
        if (e != cudaSuccess) {
            set_error(kErrCuda, "batch add: allocation of %zu bytes failed: %s", bytes(s), cudaGetErrorString(e));
            free_slot(sl);
            return kErrCuda;
        }
        Inst I;
        memset(&I, 0, sizeof I);
        const T one = T(1);
        I.DX = one / T(nb_x + 1);
        I.DY = one / T(nb_y + 1);
        T ms = (I.DY < I.DX) ? I.DY : I.DX; // std::min({DX, DY[, DZ]}) (main.cxx:484)
        if constexpr (D == 3) {
            I.DZ = one / T(nb_z + 1);
            ms = (I.DZ < ms) ? I.DZ : ms;
        }
        {
            const T gamma = T(s.gamma), gm1 = T(gamma - one);
            I.ph = Phys<T>::make(T(T(s.C) * ms), gamma, gm1, T(one / gm1), T(s.K));
        }
        I.ggm1 = skip_ggm1(I.ph.gamma, I.ph.gm1);
        T first = 0;
        int rc;
        if constexpr (D == 2)
            rc = init2d_at<T>(sl.rhoE[0], sl.uvx[0], nb_x, nb_y, s.centre[0], s.centre[1], s.radius, T(s.rho_in),
                              T(s.rho_out), T(s.p_in), T(s.p_out), I.ph.C_min, I.ph.gamma, &first, stream_,
                              scratch_bits_, (long long)ys);
        else
            rc = init3d_at<T>(sl.rhoE[0], sl.uvx[0], nb_x, nb_y, nb_z, s.centre[0], s.centre[1], s.centre[2],
                              s.radius, T(s.rho_in), T(s.rho_out), T(s.p_in), T(s.p_out), I.ph.C_min, I.ph.gamma,
                              &first, stream_, scratch_bits_);
        if (rc != kOk) {
            free_slot(sl);
            return rc;
        }
        const T big = T(1e20);
        I.dt = (first < big) ? first : big; // first_Dt = min(1e20, IC min), main.cxx:618-660
        I.DtDx = I.dt / I.DX;
        I.DtDy = I.dt / I.DY;
        I.t = 0.0;
        I.t_end = s.t_end;
        I.max_steps = s.max_steps;
        I.steps = 0;
        I.nb_x = (int)nb_x;
        I.nb_y = (int)nb_y;
        I.parity = 0;
        I.active = (0.0 < s.t_end) && (0 < s.max_steps);
        if constexpr (D == 2) {
            I.ys = (long long)ys;
            for (int b = 0; b < 2; ++b) {
                I.rhoE[b] = sl.rhoE[b];
                I.uv[b] = sl.uvx[b];
            }
            sl.tiles = sl.across = (int)((nb_y + kStripW - 1) / kStripW);
        } else {
            I.DtDz = I.dt / I.DZ;
            I.nb_z = (int)nb_z;
            I.zs = (long long)nb_z + 2;
            I.zy = (long long)(nb_y + 2) * I.zs;
            for (int b = 0; b < 2; ++b) {
                I.rhoE[b] = sl.rhoE[b];
                I.uvw[b] = sl.uvx[b];
            }
            sl.across = (int)((nb_z + k3TZ - 1) / k3TZ);
            sl.tiles = sl.across * (int)((nb_y + k3TY<T> - 1) / k3TY<T>);
        }
        e = cudaMemcpyAsync(insts_ + slot, &I, sizeof I, cudaMemcpyHostToDevice, stream_);
        SlotStatus st0{};
        st0.dt = (double)I.dt;
        st0.active = I.active;
        status_h_[slot] = st0;
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
        if (e != cudaSuccess) {
            free_slot(sl);
            set_error(kErrCuda, "batch add: %s", cudaGetErrorString(e));
            return kErrCuda;
        }
        sl.used = true;
        sl.ys = ys;
        sl.nb[0] = nb_x;
        sl.nb[1] = nb_y;
        sl.nb[2] = nb_z;
        dirty_ = true;
        return slot;
    }

    int remove(int slot) override
    {
        if (slot < 0 || slot >= cap_ || !slots_[slot].used) {
            set_error(kErrArg, "batch remove: no instance in slot %d", slot);
            return kErrArg;
        }
        cudaError_t e = cudaStreamSynchronize(stream_);
        free_slot(slots_[slot]);
        dirty_ = true;
        if (e != cudaSuccess) {
            set_error(kErrCuda, "batch remove: %s", cudaGetErrorString(e));
            return kErrCuda;
        }
        return kOk;
    }

    int run(int nsteps, bool sync) override
    {
        if (nsteps < 0) {
            set_error(kErrArg, "batch run: negative step count");
            return kErrArg;
        }
        int rc = kOk;
        if (dirty_ || nsteps != graph_steps_) rc = rebuild(nsteps);
        if (rc != kOk) return rc;
        cudaError_t e = cudaSuccess;
        if (nitems_ > 0 && nsteps > 0) e = cudaGraphLaunch(graph_, stream_);
        if (e == cudaSuccess && sync) e = cudaStreamSynchronize(stream_);
        if (e != cudaSuccess) {
            set_error(kErrCuda, "batch run: %s", cudaGetErrorString(e));
            return kErrCuda;
        }
        return kOk;
    }

    int status(int slot, hydro_batch_status_t *out) override
    {
        if (slot < 0 || slot >= cap_ || !slots_[slot].used || !out) {
            set_error(kErrArg, "batch status: no instance in slot %d", slot);
            return kErrArg;
        }
        const volatile SlotStatus *v = status_h_ + slot;
        out->t = v->t;
        out->dt = v->dt;
        out->mass = v->sums[0];
        out->mom[0] = v->sums[1];
        out->mom[1] = v->sums[2];
        out->mom[2] = v->sums[3];
        out->energy = v->sums[4];
        out->max_speed = v->max_speed;
        out->steps = v->steps;
        out->active = v->active;
        out->err = v->err;
        out->exact_passes = v->exact_passes;
        return kOk;
    }

    int state(int slot, const void **rhoE, const void **uvx, long long *row_stride) override
    {
        if (slot < 0 || slot >= cap_ || !slots_[slot].used) {
            set_error(kErrArg, "batch state: no instance in slot %d", slot);
            return kErrArg;
        }
        // the current buffer is the one the last completed step wrote: parity of steps
        const int par = (int)(status_h_[slot].steps & 1);
        *rhoE = slots_[slot].rhoE[par];
        *uvx = slots_[slot].uvx[par];
        if (row_stride) *row_stride = (long long)slots_[slot].ys;
        return kOk;
    }

    int copy_state(int slot, void *rhoE, void *uvx, bool to_host) override
    {
        const void *r, *u;
        long long ys;
        int rc = state(slot, &r, &u, &ys);
        if (rc != kOk) return rc;
        const Slot &sl = slots_[slot];
        const cudaMemcpyKind k = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
        cudaError_t e;
        if constexpr (D == 2) {
            const size_t w = 2 * sizeof(T) * (sl.nb[1] + 2), sp = 2 * sizeof(T) * (size_t)ys;
            e = cudaMemcpy2DAsync(rhoE, w, r, sp, w, sl.nb[0] + 2, k, stream_);
            if (e == cudaSuccess) e = cudaMemcpy2DAsync(uvx, w, u, sp, w, sl.nb[0] + 2, k, stream_);
        } else {
            const size_t n = (sl.nb[0] + 2) * (sl.nb[1] + 2) * (sl.nb[2] + 2) * sizeof(T);
            e = cudaMemcpyAsync(rhoE, r, 2 * n, k, stream_);
            if (e == cudaSuccess) e = cudaMemcpyAsync(uvx, u, 3 * n, k, stream_);
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
        if (e != cudaSuccess) {
            set_error(kErrCuda, "batch copy_state: %s", cudaGetErrorString(e));
            return kErrCuda;
        }
        return kOk;
    }

    int set_skip_fraction(double f) override
    {
        if (!(f >= 0.0) || !(f <= 1e300)) {
            set_error(kErrArg, "batch skip fraction: %g is not a finite non-negative number", f);
            return kErrArg;
        }
        skip_frac_ = f;
        dirty_ = true; // the fraction is a kernel argument of the captured graph
        return kOk;
    }

    int set_arith(bool fused) override
    {
        fused_ = fused;
        dirty_ = true; // the step kernel of the captured graph changes
        return kOk;
    }

    int prepare(int nsteps) override
    {
        if (nsteps < 0) {
            set_error(kErrArg, "batch prepare: negative step count");
            return kErrArg;
        }
        return (dirty_ || nsteps != graph_steps_) ? rebuild(nsteps) : kOk;
    }

    int sync() override
    {
        const cudaError_t e = cudaStreamSynchronize(stream_);
        if (e != cudaSuccess) {
            set_error(kErrCuda, "batch sync: %s", cudaGetErrorString(e));
            return kErrCuda;
        }
        return kOk;
    }

  private:
    struct Slot {
        bool used = false;
        T *rhoE[2] = {nullptr, nullptr}, *uvx[2] = {nullptr, nullptr};
        int tiles = 0, across = 1; // strips (2D) or tiles (3D) in all, along the fastest axis
        size_t ys = 0, nb[3] = {0, 0, 0};
    };

    // How the instances' rows (planes) are cut into step items: `tail` of them, at least, in
    // items of at most `rest`, what is before in items of `len`.
    struct Plan {
        double tail = 1.0;
        int len = 1, rest = 1;
    };
    static constexpr double kTail = 0.6; // in items of `len` per block

    void free_slot(Slot &s)
    {
        for (int b = 0; b < 2; ++b) {
            if (s.rhoE[b]) cudaFreeAsync(s.rhoE[b], stream_);
            if (s.uvx[b]) cudaFreeAsync(s.uvx[b], stream_);
            s.rhoE[b] = s.uvx[b] = nullptr;
        }
        s.used = false;
        s.tiles = 0;
    }

    void launch(unsigned *counter)
    {
        if constexpr (D == 2) {
            auto k = fused_ ? batch2d<T, true> : batch2d<T, false>;
            k<<<blocks_, kStripNT, 0, stream_>>>(insts_, items_, nitems_, counter, parts_, status_d_,
                                                 skip_frac_);
        } else {
            auto k = fused_ ? batch3d<T, true> : batch3d<T, false>;
            k<<<blocks_, k3NT<T>, smem_, stream_>>>(insts_, items_, nitems_, counter, parts_, status_d_,
                                                   skip_frac_);
        }
    }

    void launch_sums(unsigned *counter)
    {
        batch_sums<kSumNT, D, T, Inst><<<sum_blocks_, kSumNT, 0, stream_>>>(insts_, sum_list_, nsums_, counter, parts_,
                                                                           status_d_);
    }

    // The rows (planes) of an instance's step items: `longs` items of `len`, then items of `rest`.
    static Chunks split(int rows, const Plan &p)
    {
        const int longs = (int)(rows * (1.0 - p.tail)) / p.len, left = rows - longs * p.len;
        if (left == 0) return Chunks{longs, p.len, 1, longs};
        const int n = (left + p.rest - 1) / p.rest;
        return Chunks{longs, p.len, (left + n - 1) / n, longs + n};
    }

    // Every item costs its rows and about 3 more (halo rows, start and end), and the resident
    // blocks share them out. All items alike (the caller's rows, or the candidate): at the end the
    // blocks wait for half an item on average. Long ones first and short ones last: the blocks
    // end within a part of a short one, as long as the long ones end well before (kTail). Measured
    // per run: 24 2D instances of 10.4 M cells, 10 steps FP32 fused, 1105 us in items of 32, 1070 of 32
    // and 12 rows; 48 instances 1957 and 1893; 12 3D instances of 15.8 M cells, 8 steps FP64, 4480 in
    // items of 32, 4391 of 64 and 32 planes (items of 12 planes lose more than they even out).
    Plan pick_plan() const
    {
        if (chunk_ > 0) return Plan{1.0, chunk_, chunk_};
        double rows = 0.0, most = 0.0;
        for (int i : live_) {
            rows += (double)slots_[i].tiles * (double)slots_[i].nb[0];
            most = std::max(most, (double)slots_[i].nb[0]);
        }
        // The candidates in the order of what they cost at least, with rows cut without a remainder:
        // the set is gone through for the first few, until none left can be the best. (Preparing a run
        // of 256 2D instances took 390 us with all of them and every item sorted, now 205; of two equal
        // ones the one of shorter items.)
        struct Candidate {
            double least;
            Plan p;
        };
        Candidate cand[11 * 6];
        int n = 0;
        for (int len : {8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256})
            for (int rest : {0, 8, 12, 16, 24, 32}) {
                if (2 * rest > len || (D == 3 && rest > 0 && rest < 16)) continue;
                Plan p{1.0, len, rest ? rest : len};
                if (rest) p.tail = std::min(1.0, kTail * blocks_ * (len + 3) / rows);
                const double end = p.tail * most;
                const double least = rows * (1.0 + 3.0 * ((1.0 - p.tail) / len + p.tail / p.rest)) / blocks_ +
                                     0.5 * (p.rest * end / (p.rest + end) + 3);
                cand[n++] = Candidate{std::max(least, rest ? len + 3.0 : 0.0), p};
            }
        std::stable_sort(cand, cand + n, [](const Candidate &a, const Candidate &b) { return a.least < b.least; });
        Plan best;
        double best_cost = 0.0;
        for (int k = 0; k < n && (best_cost == 0.0 || cand[k].least <= best_cost); ++k) {
            const Plan &p = cand[k].p;
            double work = 0.0, first = 0.0;
            int longest = 0;
            for (int i : live_) {
                const Slot &s = slots_[i];
                const Chunks c = split((int)s.nb[0], p);
                work += (double)s.tiles * ((double)s.nb[0] + 3.0 * c.count);
                first += (double)s.tiles * c.longs * (p.len + 3.0);
                longest = std::max(longest, c.rest);
            }
            double cost = work / blocks_ + 0.5 * (longest + 3);
            if (p.rest != p.len) cost = std::max(cost, first / blocks_ + p.len + 3);
            if (best_cost == 0.0 || cost < best_cost ||
                (cost == best_cost && std::make_pair(p.len, p.rest) < std::make_pair(best.len, best.rest))) {
                best = p;
                best_cost = cost;
            }
        }
        return best;
    }

    // Work list and partial slots for the instances in use; the graph of `nsteps` steps
    // followed by the conservation sums.
    int rebuild(int nsteps)
    {
        live_.clear();
        for (int i = 0; i < cap_; ++i)
            if (slots_[i].used) live_.push_back(i);
        // step items, the longest first, so that the last ones to be taken are short: runs of chunks
        // of one instance and one length are put in order, and their items written out
        struct Run {
            int slot, ck, n, rows, part, count; // chunks ck .. ck + n - 1 of `rows` each
        };
        const Plan plan = pick_plan();
        std::vector<Run> runs;
        size_t parts = 0, nsums = 0;
        auto sum_count = [](const Slot &sl) {
            const size_t cells = sl.nb[0] * sl.nb[1] * (D == 3 ? sl.nb[2] : 1), per = (size_t)kSumNT * kSumCells;
            return (cells + per - 1) / per;
        };
        for (int i : live_) {
            const Slot &sl = slots_[i];
            const Chunks c = split((int)sl.nb[0], plan);
            const int count = sl.tiles * c.count, whole = c.count - 1 - c.longs; // (and the last chunk)
            const int last = (int)sl.nb[0] - c.begin(c.count - 1) + 1;
            if (c.longs > 0) runs.push_back(Run{i, 0, std::min(c.longs, c.count), c.len, (int)parts, count});
            if (whole > 0) runs.push_back(Run{i, c.longs, whole, c.rest, (int)parts, count});
            if (c.count > c.longs) runs.push_back(Run{i, c.count - 1, 1, last, (int)parts, count});
            parts += (size_t)count;
            nsums += sum_count(sl);
        }
        std::stable_sort(runs.begin(), runs.end(), [](const Run &a, const Run &b) { return a.rows > b.rows; });
        // the step items and behind them those of the sums, to the device in one copy
        std::vector<unsigned char> lists(parts * sizeof(Item) + nsums * sizeof(SumItem));
        Item *item = reinterpret_cast<Item *>(lists.data());
        for (const Run &r : runs) {
            const Slot &sl = slots_[r.slot];
            const Chunks c = split((int)sl.nb[0], plan);
            for (int k = r.ck; k < r.ck + r.n; ++k)
                for (int t = 0, tx = 0, ty = 0; t < sl.tiles; ++t) {
                    const int i0 = c.begin(k);
                    *item++ = Item{r.slot, r.part + k * sl.tiles + t, tx, ty, i0, i0 + r.rows - 1, r.part, r.count};
                    if (++tx == sl.across) {
                        tx = 0;
                        ++ty;
                    }
                }
        }
        SumItem *sum = reinterpret_cast<SumItem *>(item);
        int first = 0;
        for (int i : live_) {
            const int count = (int)sum_count(slots_[i]);
            for (int k = 0; k < count; ++k) *sum++ = SumItem{i, k, first, count};
            first += count;
        }
        cudaError_t e = cudaStreamSynchronize(stream_);
        // one allocation: the parts (of the items of a step, or of the sums), the lists
        const size_t at = sizeof(ItemPart) * std::max(parts, nsums), need = at + lists.size();
        if (e == cudaSuccess && need > room_) {
            cudaFree(parts_);
            parts_ = nullptr;
            room_ = std::max(need, 2 * room_);
            e = cudaMalloc(&parts_, room_);
            if (e != cudaSuccess) room_ = 0;
        }
        nitems_ = (int)parts;
        nsums_ = (int)nsums;
        if (e == cudaSuccess && nitems_ > 0) {
            items_ = reinterpret_cast<Item *>(reinterpret_cast<unsigned char *>(parts_) + at);
            sum_list_ = reinterpret_cast<SumItem *>(items_ + parts);
            e = cudaMemcpyAsync(items_, lists.data(), lists.size(), cudaMemcpyHostToDevice, stream_);
        }
        if (graph_) {
            cudaGraphExecDestroy(graph_);
            graph_ = nullptr;
        }
        if (e == cudaSuccess && (size_t)nsteps + 1 > counters_) {
            cudaFree(counter_);
            counter_ = nullptr;
            counters_ = std::max<size_t>((size_t)nsteps + 1, 2 * counters_);
            e = cudaMalloc(&counter_, sizeof(unsigned) * counters_);
            if (e != cudaSuccess) counters_ = 0;
        }
        if (e == cudaSuccess && nitems_ > 0 && nsteps > 0) {
            cudaGraph_t g = nullptr;
            e = cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal);
            // a counter per step and one for the sums, cleared together (a clear ahead of every
            // step was a graph node of its own between the kernels)
            if (e == cudaSuccess) e = cudaMemsetAsync(counter_, 0, sizeof(unsigned) * ((size_t)nsteps + 1), stream_);
            for (int k = 0; k < nsteps && e == cudaSuccess; ++k) {
                launch(counter_ + k);
                e = cudaGetLastError();
            }
            // the conservation sums of the state the run ends on
            if (e == cudaSuccess) {
                launch_sums(counter_ + nsteps);
                e = cudaGetLastError();
            }
            const cudaError_t e2 = cudaStreamEndCapture(stream_, &g);
            if (e == cudaSuccess) e = e2;
            if (e == cudaSuccess) e = cudaGraphInstantiate(&graph_, g, 0);
            if (g) cudaGraphDestroy(g);
        }
        // the copy reads the lists: on its way while the graph was made
        const cudaError_t e3 = cudaStreamSynchronize(stream_);
        if (e == cudaSuccess) e = e3;
        if (e != cudaSuccess) {
            set_error(kErrCuda, "batch rebuild: %s", cudaGetErrorString(e));
            return kErrCuda;
        }
        dirty_ = false;
        graph_steps_ = nsteps;
        return kOk;
    }

    int chunk_, cap_;
    double skip_frac_ = kSkipFrac;
    bool fused_ = false; // fused arithmetic of the step kernels (hydro_batch_set_arith)
    bool own_stream_ = false, dirty_ = true;
    cudaStream_t stream_ = nullptr;
    Inst *insts_ = nullptr;
    Item *items_ = nullptr;
    SumItem *sum_list_ = nullptr;
    size_t room_ = 0; // bytes allocated at parts_
    ItemPart *parts_ = nullptr;
    unsigned *counter_ = nullptr; // one per step of the graph and one for the sums
    size_t counters_ = 256;
    unsigned long long *scratch_bits_ = nullptr;
    SlotStatus *status_h_ = nullptr, *status_d_ = nullptr;
    std::vector<Slot> slots_;
    std::vector<int> live_; // the slots in use, as of the last rebuild
    int nitems_ = 0, nsums_ = 0, blocks_ = 1, sum_blocks_ = 1, graph_steps_ = -1, smem_ = 0;
    cudaGraphExec_t graph_ = nullptr;
};

} // namespace hydro

using namespace hydro;

extern "C" {

void *hydro_batch_create(int dim, int precision_bytes, int chunk, int capacity, void *stream)
{
    if ((dim != 2 && dim != 3) || (precision_bytes != 4 && precision_bytes != 8) || capacity <= 0 ||
        capacity > (1 << 20) || chunk < 0) {
        set_error(kErrArg, "hydro_batch_create: unsupported (dim %d, precision %d bytes, capacity %d)", dim,
                  precision_bytes, capacity);
        return nullptr;
    }
    int rc = kOk;
    BatchBase *b = nullptr;
    const cudaStream_t s = (cudaStream_t)stream;
    if (dim == 2 && precision_bytes == 8) b = new BatchEngine<double, 2>(chunk, capacity, s, &rc);
    else if (dim == 2) b = new BatchEngine<float, 2>(chunk, capacity, s, &rc);
    else if (precision_bytes == 8) b = new BatchEngine<double, 3>(chunk, capacity, s, &rc);
    else b = new BatchEngine<float, 3>(chunk, capacity, s, &rc);
    if (rc != kOk) {
        delete b;
        return nullptr;
    }
    return b;
}

int hydro_batch_add(void *b, const hydro_blast_t *spec)
{
    if (!b || !spec) {
        set_error(kErrArg, "hydro_batch_add: null argument");
        return kErrArg;
    }
    return static_cast<BatchBase *>(b)->add(*spec);
}

int hydro_batch_remove(void *b, int slot)
{
    if (!b) return kErrArg;
    return static_cast<BatchBase *>(b)->remove(slot);
}

int hydro_batch_run(void *b, int nsteps, int sync)
{
    if (!b) return kErrArg;
    return static_cast<BatchBase *>(b)->run(nsteps, sync != 0);
}

int hydro_batch_status(void *b, int slot, hydro_batch_status_t *out)
{
    if (!b) return kErrArg;
    return static_cast<BatchBase *>(b)->status(slot, out);
}

int hydro_batch_state(void *b, int slot, const void **rhoE, const void **uvx, long long *row_stride)
{
    if (!b || !rhoE || !uvx) return kErrArg;
    return static_cast<BatchBase *>(b)->state(slot, rhoE, uvx, row_stride);
}

int hydro_batch_copy_state(void *b, int slot, void *rhoE, void *uvx, int to_host)
{
    if (!b || !rhoE || !uvx) return kErrArg;
    return static_cast<BatchBase *>(b)->copy_state(slot, rhoE, uvx, to_host != 0);
}

long long hydro_batch_bytes(void *b, const hydro_blast_t *spec)
{
    if (!b || !spec) return kErrArg;
    return (long long)static_cast<BatchBase *>(b)->bytes(*spec);
}

int hydro_batch_prepare(void *b, int nsteps)
{
    if (!b) return kErrArg;
    return static_cast<BatchBase *>(b)->prepare(nsteps);
}

int hydro_batch_set_arith(void *b, int arith)
{
    if (!b || (arith & ~(HYDRO_ARITH_FUSED | HYDRO_ARITH_STRICT))) {
        set_error(kErrArg, "hydro_batch_set_arith: null batch or unknown bits 0x%x", arith);
        return kErrArg;
    }
    return static_cast<BatchBase *>(b)->set_arith((arith & HYDRO_ARITH_FUSED) && !(arith & HYDRO_ARITH_STRICT));
}

int hydro_batch_set_skip_fraction(void *b, double frac)
{
    if (!b) return kErrArg;
    return static_cast<BatchBase *>(b)->set_skip_fraction(frac);
}

int hydro_batch_sync(void *b)
{
    if (!b) return kErrArg;
    return static_cast<BatchBase *>(b)->sync();
}

void hydro_batch_destroy(void *b) { delete static_cast<BatchBase *>(b); }

int hydro2d_init_blast_at_f64(double *d_rhoE, double *d_uv, size_t NB_X, size_t NB_Y, double cx, double cy,
                              double radius, double rho_in, double rho_out, double p_in, double p_out, double C_min,
                              double gamma, double *min_dt, void *stream)
{
    int err;
    DevCtx *ctx = ctx_current(&err);
    if (!ctx) return err;
    return init2d_at<double>(d_rhoE, d_uv, NB_X, NB_Y, cx, cy, radius, rho_in, rho_out, p_in, p_out, C_min, gamma,
                             min_dt, (cudaStream_t)stream, &ctx->scr->max_bits);
}
int hydro2d_init_blast_at_f32(float *d_rhoE, float *d_uv, size_t NB_X, size_t NB_Y, double cx, double cy,
                              double radius, float rho_in, float rho_out, float p_in, float p_out, float C_min,
                              float gamma, float *min_dt, void *stream)
{
    int err;
    DevCtx *ctx = ctx_current(&err);
    if (!ctx) return err;
    return init2d_at<float>(d_rhoE, d_uv, NB_X, NB_Y, cx, cy, radius, rho_in, rho_out, p_in, p_out, C_min, gamma,
                            min_dt, (cudaStream_t)stream, &ctx->scr->max_bits);
}
int hydro3d_init_blast_at_f64(double *d_rhoE, double *d_uvw, size_t NB_X, size_t NB_Y, size_t NB_Z, double cx,
                              double cy, double cz, double radius, double rho_in, double rho_out, double p_in,
                              double p_out, double C_min, double gamma, double *min_dt, void *stream)
{
    int err;
    DevCtx *ctx = ctx_current(&err);
    if (!ctx) return err;
    return init3d_at<double>(d_rhoE, d_uvw, NB_X, NB_Y, NB_Z, cx, cy, cz, radius, rho_in, rho_out, p_in, p_out,
                             C_min, gamma, min_dt, (cudaStream_t)stream, &ctx->scr->max_bits);
}
int hydro3d_init_blast_at_f32(float *d_rhoE, float *d_uvw, size_t NB_X, size_t NB_Y, size_t NB_Z, double cx,
                              double cy, double cz, double radius, float rho_in, float rho_out, float p_in,
                              float p_out, float C_min, float gamma, float *min_dt, void *stream)
{
    int err;
    DevCtx *ctx = ctx_current(&err);
    if (!ctx) return err;
    return init3d_at<float>(d_rhoE, d_uvw, NB_X, NB_Y, NB_Z, cx, cy, cz, radius, rho_in, rho_out, p_in, p_out,
                            C_min, gamma, min_dt, (cudaStream_t)stream, &ctx->scr->max_bits);
}

} // extern "C"
