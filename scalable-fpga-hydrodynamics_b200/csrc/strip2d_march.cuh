// The row march of the 2D strip kernels, shared by the plain step (strip2d, one
// strip x chunk per block) and the batched step (batch2d, many strips x chunks of many
// instances per persistent block).
//
// One block of kStripNT lanes covers kStripNT consecutive columns starting at `jbase`
// (kStripW interior columns plus a halo column each side) and marches over rows
// i0-1 .. i1+1. Each lane brings its own cell of each row into a kStages-deep ring in shared
// memory by cp.async, so it reads only what it copied and the ring needs no barrier of its own.
// (Rows by TMA tile loads, with a thread that issues them and a wait on an mbarrier per row, took
// 234 instructions per cell-update instead of 218 in FP32 and twice the branches: 8000 x 8000 FP32
// fused 117 against 135 GCell/s, FP64 strict 77.5 against 79.8.) Every updated interior cell is
// handed to `sink`.
//
// Walls: a ghost cell (j = 0 or NB_Y+1) is its wall cell with the normal momentum negated: the
// lane copies the wall cell and flips a sign bit; converting that gives the mirrored cell's
// values exactly, so no face knows of walls and every strip runs the same loop. Lanes further out
// hold copies of the last wall cell, whose values nothing uses.
#pragma once

#include "hydro_rt.cuh"

namespace hydro {

constexpr int kStripNT = 128;
constexpr int kStripW = kStripNT - 2; // interior columns per strip
constexpr int kStages = 4;

__device__ __forceinline__ int wrap_row(int n, int nb_x) { return n == 0 ? nb_x : (n == nb_x + 1 ? 1 : n); }

template <class T> __device__ __forceinline__ typename Vec2<T>::type mk2(T a, T b)
{
    typename Vec2<T>::type v;
    v.x = a;
    v.y = b;
    return v;
}

template <class T> struct Smem2 {
    using V2 = typename Vec2<T>::type;
    __align__(128) V2 sr[kStages][kStripNT]; // (rho, E) rows
    __align__(128) V2 su[kStages][kStripNT]; // (rho u, rho v) rows
    // y-face inputs of every lane's cell (lane t at [t]) and every lane's right face flux
    // (lane t at [t+1]), as pairs so that each lane moves them with 128-bit (FP64) or 64-bit
    // (FP32) shared-memory accesses. Both are double-buffered by row parity, which leaves one
    // barrier per row: a lane may publish row n's inputs while its neighbour still reads row
    // n-1's, and the fluxes of row n-1 are read after row n's barrier.
    __align__(16) V2 xP[2][4][kStripNT + 1];
    __align__(16) V2 xF[2][2][kStripNT + 1];
};

struct March2 {
    int jbase, i0, i1; // columns jbase .. jbase+kStripNT-1, interior rows i0 .. i1
};

// The grid, read where it is needed: in the kernel's parameters for the plain step, in shared
// memory (volatile) for the batched one.
struct Grid2 {
    int nb_x, nb_y;
    int xwrap; // X neighbours of rows 1 and NB_X by periodic wrap (1) or ghost rows (0)
    long long ys;
};

// A warp whose first column is past the last ghost column (NB_Y+1) computes nothing that is
// used: no interior cell, and its lane 0's cell only enters the face (NB_Y+1 | NB_Y+2) of the
// warp before it. It takes part in the row barriers only.
//
// Per row m, the y face (j | j+1) of row m-1 (its neighbour's inputs were published before the
// previous barrier), the conversion of row m and the x face (row m-1 | row m) form one
// straight-line block ahead of the row's barrier, which gives the scheduler three independent
// chains; after the barrier only the update of row m-1 remains. (Converting first and
// evaluating the faces after the barrier measured 77.3 against 80.9 GCell/s at 40000 x 20000
// FP64; columns two to a lane, loaded straight to registers, 59 against 79 at 8000 x 8000; strips
// of one warp, which need no block barrier, 75.)
//
// kF: fused arithmetic (hydro_math.cuh). kUnroll: rows per turn of the loop; two need more than the
// 96 registers of 5 blocks per SM in FP64 (8000 x 8000 fused 1469 us with the spills, 920 one at a
// time; strict 1127 and 848; 738 and 784 with two rows and 4 blocks, the built-in form).
template <class T, bool kF, int kUnroll = 2, class GR, class PH, class Sink>
__device__ __forceinline__ void march2d(Smem2<T> &S, const T *rhoE, const T *uv, T *rhoE_n, T *uv_n, const March2 &geo,
                                        const GR &g, const PH &ph, Sink &&sink)
{
    using V2 = typename Vec2<T>::type;
    const int t = threadIdx.x;
    const int j = geo.jbase + t, nb_y = g.nb_y;
    const int nrows = geo.i1 - geo.i0 + 3; // with one halo row above and below
    const bool interior = (t >= 1) && (t <= kStripW) && (j <= nb_y);
    const int jw = min(max(j, 1), nb_y); // the column of the lane's cell, or of its wall cell
    const unsigned flip = j == jw ? 0u : 0x80000000u;
    if (geo.jbase + (t & ~31) > nb_y + 1) {
        for (int m = 0; m < nrows; ++m) __syncthreads();
        return;
    }
    // this lane's cell of row m into its place of stage m % kStages, one commit group per row
    // (an empty one past the last row)
    auto issue = [&](int m) {
        if (m < nrows) {
            const int row = g.xwrap ? wrap_row(geo.i0 - 1 + m, g.nb_x) : geo.i0 - 1 + m;
            const long long c = (long long)row * g.ys + jw;
            const int s = m % kStages;
            cp_async(&S.sr[s][t], reinterpret_cast<const V2 *>(rhoE) + c, (int)sizeof(V2), true);
            cp_async(&S.su[s][t], reinterpret_cast<const V2 *>(uv) + c, (int)sizeof(V2), true);
        }
        cp_async_commit();
    };
    for (int m = 0; m < kStages - 1; ++m) issue(m);

    Cell2<T> Pm{};
    T Ur = 0, Uu = 0, Uv = 0, UE = 0;
    Flux2<T> fxlo{};
    // row m's conserved values
    auto load = [&](int m, V2 &a, V2 &b) {
        issue(m + kStages - 1);       // into the place this lane read for row m-1
        cp_async_wait<kStages - 1>(); // this lane's copy of row m landed
        a = S.sr[m % kStages][t];
        b = S.su[m % kStages][t];
        b.y = flip_sign(b.y, flip);
    };
    // this lane's y-face inputs of row mm, for the previous lane's y face
    auto publish = [&](int mm, const Cell2<T> &P) {
        const FaceIn<T> me = face_y(P);
        S.xP[mm & 1][0][t] = mk2<T>(me.r, me.un);
        S.xP[mm & 1][1][t] = mk2<T>(me.p, me.Ka);
        S.xP[mm & 1][2][t] = mk2<T>(me.iKa, me.mn);
        S.xP[mm & 1][3][t] = mk2<T>(me.mt, me.eup);
    };
    // y face (j | j+1) of row mm-1, from this lane's cell of that row and the next lane's
    auto yface = [&](int mm) {
        const V2 n0 = S.xP[(mm - 1) & 1][0][t + 1], n1 = S.xP[(mm - 1) & 1][1][t + 1],
                 n2 = S.xP[(mm - 1) & 1][2][t + 1], n3 = S.xP[(mm - 1) & 1][3][t + 1];
        return face_flux<T, kF>(face_y(Pm), FaceIn<T>{n0.x, n0.y, n1.x, n1.y, n2.x, n2.y, n3.x, n3.y});
    };
    int m = 0;
    // row 0 (the halo row below) and row 1: conversion, row 1's y-face inputs and the first
    // x face
#pragma unroll 1
    for (; m < 2; ++m) {
        V2 a, b;
        load(m, a, b);
        const Cell2<T> P = make_cell2<T, kF>(a.x, b.x, b.y, a.y, ph);
        if (m == 1) {
            publish(m, P);
            fxlo = face_flux<T, kF>(face_x(Pm), face_x(P));
        }
        __syncthreads(); // row 1's inputs published
        Pm = P;
        Ur = a.x; Uu = b.x; Uv = b.y; UE = a.y;
    }
#pragma unroll kUnroll
    for (; m < nrows; ++m) {
        V2 a, b;
        load(m, a, b);
        const Flux2<T> fyr = yface(m);
        const Cell2<T> P = make_cell2<T, kF>(a.x, b.x, b.y, a.y, ph);
        const Flux2<T> fxhi = face_flux<T, kF>(face_x(Pm), face_x(P));
        // row m-1's right face for the next lane (its left face), double-buffered by row
        // parity: the buffer of row m-3 was last read before the previous barrier
        S.xF[(m - 1) & 1][0][t + 1] = mk2<T>(fyr.r, fyr.n);
        S.xF[(m - 1) & 1][1][t + 1] = mk2<T>(fyr.t, fyr.E);
        publish(m, P);
        __syncthreads(); // row m's inputs and row m-1's fluxes published
        if (interior) {
            // row m-1's left face is lane t-1's right face of that row
            const V2 f0 = S.xF[(m - 1) & 1][0][t], f1 = S.xF[(m - 1) & 1][1][t];
            const Flux2<T> fyl{f0.x, f0.y, f1.x, f1.y};
            const Upd2<T> o = update2<T, kF>(Ur, Uu, Uv, UE, fxlo, fxhi, fyl, fyr, ph.DtDx, ph.DtDy);
            const long long c = (long long)(geo.i0 + m - 2) * g.ys + j;
            reinterpret_cast<V2 *>(rhoE_n)[c] = mk2<T>(o.r, o.E);
            reinterpret_cast<V2 *>(uv_n)[c] = mk2<T>(o.u, o.v);
            sink(o);
        }
        fxlo = fxhi;
        Pm = P;
        Ur = a.x; Uu = b.x; Uv = b.y; UE = a.y;
    }
    cp_async_wait<0>();
}

} // namespace hydro
