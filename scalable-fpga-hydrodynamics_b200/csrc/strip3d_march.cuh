// The X-march of the 3D strip kernels, shared by the plain step (strip3d, one tile x
// chunk per block) and the batched step (batch3d, tiles of many instances per persistent
// block).
//
// One block of W warps covers a tile of R y rows x 32 z columns starting at (jbase, kbase): the
// interior columns plus a one-cell halo ring. Two tile layouts: R = W + 1 rows on W = 8 warps
// (kPair, the default: warp 0 holds both halo rows, all other warps interior rows), or R = W
// rows on W warps (warps 0 and W-1 hold the halo rows). Each X plane of the tile arrives in a
// shared-memory ring in one of two forms:
//  - tensor maps (kTma): two 3D TMA tile loads per plane (the (rho, E) pairs and the momentum
//    triples of the tile's rows), issued by one thread, completing on the stage's mbarrier;
//    needs a row pitch of a multiple of 16 bytes (FP64 with even NB_Z) and 16-byte aligned
//    arrays;
//  - row copies, every warp its own rows: cp.async of 16 bytes a lane along each row of momenta
//    from the 16-byte boundary at or below its start (the lanes index from the remainder), of one
//    cell a lane along each row of (rho, E): 2 copy instructions per row in FP32 and 3 in FP64,
//    against 5 value by value, the form for arrays that are not all 16-byte aligned. (All rows copied by warp 0: 512^3 FP32 39.7 GCell/s, the other warps wait for it.)
// Each lane converts its cell to primitives once and publishes them as pairs (double-buffered
// by plane parity; one barrier per plane). Per plane a lane computes one x face, one z face
// (the next lane's cell from shared memory, the flux back by shuffles) and one y face (the row
// above's cell, the flux back through shared memory), then updates the plane behind it. Every
// updated interior cell is handed to `sink`.
//
// Walls: a ghost cell (j or k = 0 or NB+1) is its wall cell with the normal momentum negated,
// which a lane gets by reading the wall cell's place with a flipped sign bit; converting that
// gives the mirrored cell's values exactly, so no face knows of walls. Lanes further out hold
// copies of the last wall cell, whose values nothing uses.
//
// What bounds it is issue slots, so the plane loop keeps little: a face loads the upwind cell's
// momenta and energy from the published pairs of whichever cell is upwind (one address select
// instead of eight or ten selects of values in two registers each), which also means that they
// need not be kept in registers from plane to plane; places in the rings are running offsets;
// and a wait that gives up is noted in a flag of its thread, not looked up by every thread
// after every barrier. Per cell-update FP64 strict 490 instructions at 256^3, from 590 (512^3: 39.4 ->
// 42.7 GCell/s strict, 43.1 -> 45.0 fused; 512 x 512 x 511: 34.0 -> 37.7, 36.7 -> 41.1; FP32
// 61.4 -> 62.9, 67.6 -> 71.2). Without a second form of the loop for tiles at the walls it also
// stays in the instruction cache where both kinds of tile run side by side: 256^3 FP32 fused
// 53.4 -> 62.8, 321 x 255 x 259 56.8 -> 65.2, 170^3 FP64 27.5 -> 31.3.
#pragma once

#include "hydro_rt.cuh"
#include "ring.h"

namespace hydro {

// Resident blocks per SM that the registers of a W-warp tile are budgeted for: FP64 two (128
// registers), FP32 three (80) for 8 warps.
template <class T> constexpr int min_blocks3(int W) { return W <= 8 ? (sizeof(T) == 4 ? 3 : 2) : 1; }
constexpr int k3TZ = 30; // interior columns per tile

__device__ __forceinline__ int wrap_plane(int n, int nb_x) { return n == 0 ? nb_x : (n == nb_x + 1 ? 1 : n); }

template <class T> __device__ __forceinline__ typename Vec2<T>::type pair3(T a, T b)
{
    typename Vec2<T>::type v;
    v.x = a;
    v.y = b;
    return v;
}

// How the planes arrive (above): tensor maps, row copies, value by value.
enum class Stage3 { Tma, Rows, Values };

template <class T, int W_, bool kPair_, Stage3 kStage> struct Smem3 {
    using V2 = typename Vec2<T>::type;
    static constexpr int W = W_, R = kPair_ ? W_ + 1 : W_, NR = 32 * R;
    static constexpr bool kPair = kPair_, kTma = kStage == Stage3::Tma, kRows = kStage == Stage3::Rows;
    static constexpr int NS = sizeof(T) == 8 ? 3 : 4;                     // stages
    static constexpr int kU = kRows ? 96 + (int)(16 / sizeof(T)) : 96;     // pitch of a row of momenta
    struct Stage {
        __align__(128) T r[NR][2];  // (rho, E), lane t = 32 row + column
        __align__(128) T u[R * kU]; // (rho u, rho v, rho w), row by row
    } st[NS];
    // by plane parity: each cell as pairs (r,p) (Ka,iKa) (v,w) (mu,mv) (mw,eup_xy) (mw,eup_z),
    // the last one in strict arithmetic only, and the +y face fluxes of the rows below the last
    // interior one
    struct Ex {
        V2 xP[6][NR];
        V2 xF[2][32 * (R - 2)];
        T xFE[32 * (R - 2)];
    } ex[2];
    uint64_t full[NS]; // tensor maps: the stage holds its plane
};

struct March3 {
    int kbase, jbase, i0, i1; // tile corner (halo included) and interior X planes
};

// The grid, read where it is needed: in the kernel's parameters for the plain step, in shared
// memory (volatile) for the batched one.
struct Grid3 {
    int nb_x, nb_y, nb_z;
    int xwrap;        // X neighbours of planes 1 and NB_X by periodic wrap (1) or ghost planes (0)
    long long zs, zy; // strides in cells of a Y row and of an X plane

    Grid3() = default;
    __host__ __device__ Grid3(int x, int y, int z, int wrap)
        : nb_x(x), nb_y(y), nb_z(z), xwrap(wrap), zs((long long)z + 2), zy((long long)(y + 2) * ((long long)z + 2))
    {
    }
};

// Tensor maps of the two input arrays for the kTma form (null otherwise).
struct Tmaps3 {
    const CUtensorMap *r = nullptr, *u = nullptr;
};

// One-time set-up of the stage barriers of the tensor-map form (thread 0), then a block barrier.
template <class SM> __device__ __forceinline__ void march3d_init(SM &S)
{
    if (SM::kTma) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < SM::NS; ++s) mbar_init(&S.full[s], 1);
            fence_mbar_init();
        }
        __syncthreads();
    }
}

// What a face needs of a cell before the upwind side is known.
template <class T> struct Side3 {
    T r, un, p, Ka, iKa;
};

// The flux of a face with normal along axis kAx between two cells, the upwind cell's momenta
// and energy read from its published pairs (`bl`, `br`: those of L and R, NR apart). Same
// operations as face_flux3.
template <int kAx, bool kF, int NR, class T>
__device__ __forceinline__ Flux3<T> face_from(const Side3<T> &L, const Side3<T> &R, const typename Vec2<T>::type *bl,
                                              const typename Vec2<T>::type *br)
{
    using A = Ar<T>;
    const bool right = A::abs(L.Ka) < A::abs(R.Ka);
    const T a = right ? R.Ka : L.Ka;
    const T diva = right ? R.iKa : L.iKa;
    T us, ps;
    if constexpr (kF) {
        us = A::mul(A::half, A::fma(-diva, A::sub(R.p, L.p), A::add(L.un, R.un)));
        ps = A::mul(A::half, A::fma(-a, A::sub(R.un, L.un), A::add(L.p, R.p)));
    } else {
        us = A::mul(A::half, A::sub(A::add(L.un, R.un), A::mul(diva, A::sub(R.p, L.p))));
        ps = A::mul(A::half, A::sub(A::add(L.p, R.p), A::mul(a, A::sub(R.un, L.un))));
    }
    const bool up = us >= T(0);
    const T r = up ? L.r : R.r;
    const typename Vec2<T>::type *b = up ? bl : br;
    const auto q3 = b[3 * NR];
    const auto q4 = b[((kAx == 2 && !kF) ? 5 : 4) * NR];
    const T mn = kAx == 0 ? q3.x : kAx == 1 ? q3.y : q4.x;
    const T m1 = kAx == 0 ? q3.y : kAx == 1 ? q3.x : q3.y;
    const T m2 = kAx == 2 ? q3.x : q4.x;
    const T e = q4.y;
    Flux3<T> F;
    F.r = A::mul(r, us);
    if constexpr (kF) {
        F.n = A::fma(mn, us, ps);
        F.t1 = A::mul(m1, us);
        F.t2 = A::mul(m2, us);
        F.E = A::fma(e, us, A::mul(ps, us));
    } else {
        F.n = A::add(A::mul(mn, us), ps);
        F.t1 = A::add(A::mul(m1, us), T(0));
        F.t2 = A::add(A::mul(m2, us), T(0));
        F.E = A::add(A::mul(e, us), A::mul(ps, us));
    }
    return F;
}

// The plane loop is written once per warp role (interior rows; warp 0: the bottom halo row,
// with kPair the top one too, and the copies; else the top halo row). In the interior rows'
// loop the +y and +z faces of plane m-1 (their neighbours' pairs were published before the
// previous barrier), the conversion of plane m and the x face (m-1 | m) come ahead of the
// plane's barrier: independent chains the scheduler interleaves; after the barrier only the
// update of plane m-1 remains. Not unrolled: two planes of it and warp 0's loop beside them are
// more than the SM's instruction cache keeps. Returns false when a bounded wait gave up (the
// march runs on without waiting; its values are then not the step's).
template <class T, bool kF, class SM, class GR, class PH, class Sink>
__device__ __forceinline__ bool march3d(SM &S, const T *rhoE, const T *uvw, T *rhoE_n, T *uvw_n, const March3 &geo,
                                             const GR &g, const PH &ph, const Tmaps3 &tm, Ring<SM::NS> &ring,
                                             Sink &&sink)
{
    using V2 = typename Vec2<T>::type;
    using Ex = typename SM::Ex;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NR = SM::NR, NS = SM::NS, R = SM::R, kU = SM::kU;
    constexpr int V = (int)(16 / sizeof(T)); // values per 16 bytes
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int k = geo.kbase + lane, j = geo.jbase + w;
    const int nplanes = geo.i1 - geo.i0 + 3;
    auto plane_of = [&](int m) { return g.xwrap ? wrap_plane(geo.i0 - 1 + m, g.nb_x) : geo.i0 - 1 + m; };

    __syncthreads(); // the previous march of this block is done with the stages and exchange buffers

    // Plane m into stage s: tensor maps by one thread; copies by every warp for its own rows (a
    // ghost row's is its wall cell's row), one commit group per plane (an empty one past the last
    // plane). The places of the copies run on from plane to plane: `qr`, this lane's (rho, E) of
    // row w, and `qu`, the row's first momentum; the periodic planes before the first and behind
    // the last are NB_X planes away.
    const bool wrap_first = g.xwrap && geo.i0 == 1, wrap_last = g.xwrap && geo.i1 == g.nb_x;
    const long long c0 = (long long)(wrap_first ? g.nb_x : geo.i0 - 1) * g.zy + (long long)geo.jbase * g.zs + geo.kbase;
    auto source = [&](int r) { return (long long)(min(max(geo.jbase + r, 1), g.nb_y) - geo.jbase) * g.zs; };
    const T *qr = rhoE + 2 * (c0 + source(w) + lane), *qu = uvw + 3 * (c0 + source(w));
    const int cells = min(32, g.nb_z + 1 - geo.kbase); // of a row, up to the last real one
    auto copy_row = [&](const T *pr, const T *pu, int s, int r) {
        const bool in = lane < cells;
        if constexpr (SM::kRows) {
            if (in) cp_async(&S.st[s].r[32 * r + lane][0], pr, (int)(2 * sizeof(T)), true);
            const uintptr_t at = reinterpret_cast<uintptr_t>(pu);
            const char *base = reinterpret_cast<const char *>(at & ~(uintptr_t)15);
            const int end = (int)(at & 15) + 3 * (int)sizeof(T) * cells; // behind the row's last value
#pragma unroll
            for (int q = 0; q < kU / V; q += 32) {
                const int i = q + lane; // 16 bytes each (the last ones reach into the next row)
                if (16 * i < end) cp_async_16(&S.st[s].u[r * kU + V * i], base + 16 * i);
            }
        } else if (in) {
            T *dr = &S.st[s].r[32 * r + lane][0], *du = &S.st[s].u[r * kU + 3 * lane];
            const T *pl = pu + 3 * lane;
            cp_async(dr, pr, sizeof(T), true);
            cp_async(dr + 1, pr + 1, sizeof(T), true);
            cp_async(du, pl, sizeof(T), true);
            cp_async(du + 1, pl + 1, sizeof(T), true);
            cp_async(du + 2, pl + 2, sizeof(T), true);
        }
    };
    auto issue = [&](int m, int s) {
        if constexpr (SM::kTma) {
            if (t == 0 && m < nplanes && !ring.dead) {
                mbar_arrive_expect_tx(&S.full[s], (uint32_t)(5 * NR * sizeof(T)));
                tma_load_3d(&S.st[s].r[0][0], tm.r, 2 * geo.kbase, geo.jbase, plane_of(m), &S.full[s]);
                tma_load_3d(&S.st[s].u[0], tm.u, 3 * geo.kbase, geo.jbase, plane_of(m), &S.full[s]);
            }
        } else {
            if (m < nplanes) {
                copy_row(qr, qu, s, w);
                if (SM::kPair && w == 0) {
                    const long long d = source(R - 1) - source(0);
                    copy_row(qr + 2 * d, qu + 3 * d, s, R - 1);
                }
                const long long zy = g.zy;
                qr += 2 * zy;
                qu += 3 * zy;
                if ((m == 0 && wrap_first) || (m == nplanes - 2 && wrap_last)) {
                    qr -= 2 * zy * g.nb_x;
                    qu -= 3 * zy * g.nb_x;
                }
            }
            cp_async_commit();
        }
    };
    {
        int s = ring.st;
#pragma unroll 1
        for (int m = 0; m < NS - 1; ++m) {
            issue(m, s);
            s = s + 1 == NS ? 0 : s + 1;
        }
    }
    // top of plane m: refill the stage of plane m-1, which every lane read before the previous
    // barrier, and wait for plane m
    auto wait = [&](int m) {
        if (!SM::kTma || w == 0) issue(m + NS - 1, ring.st == 0 ? NS - 1 : ring.st - 1);
        if constexpr (SM::kTma) {
            if (!ring.dead && !mbar_wait_bounded(&S.full[ring.st], ring.phase)) ring.dead = nplanes - m;
        } else {
            cp_async_wait<NS - 1>();
            __syncwarp();
        }
    };
    // Row copies: the place within 16 bytes of the first momentum of tile row 0, which runs on
    // with the planes, and of the row that tile row r reads, relative to it.
    unsigned sh = SM::kRows ? (unsigned)(reinterpret_cast<uintptr_t>(uvw + 3 * c0) & 15) : 0u;
    auto row_shift = [&](int r) {
        return 3u * (unsigned)sizeof(T) * (unsigned)source(r);
    };
    auto next_shift = [&](int m) { // from plane m to m + 1
        if constexpr (SM::kRows) {
            const unsigned d = 3u * (unsigned)sizeof(T) * (unsigned)g.zy;
            sh += d;
            if ((m == 0 && wrap_first) || (m == nplanes - 2 && wrap_last)) sh -= d * (unsigned)g.nb_x;
            sh &= 15u;
        }
    };
    // Where a lane of tile row r reads its cell: its own place, or its wall cell's.
    struct Place {
        int r, u;              // of (rho, E) and of the momenta, in values
        unsigned flip_v, flip_w;
    };
    auto place_of = [&](int r) {
        const int jj = geo.jbase + r, jw = min(max(jj, 1), g.nb_y), kw = min(max(k, 1), g.nb_z);
        const int row = SM::kTma ? jw - geo.jbase : r, col = kw - geo.kbase; // (copies: the wall cell's row, above)
        return Place{2 * (32 * row + col), row * kU + 3 * col, jj == jw ? 0u : 0x80000000u, k == kw ? 0u : 0x80000000u};
    };
    // the cell there; its row's momenta start `shift` bytes into their place
    auto load = [&](const Place &p, unsigned shift, T &ur, T &uE, T &uu, T &uv, T &uw) {
        const auto &st = S.st[ring.st];
        const V2 a = *reinterpret_cast<const V2 *>(&st.r[0][0] + p.r);
        const T *u = reinterpret_cast<const T *>(reinterpret_cast<const char *>(&st.u[p.u]) + shift);
        ur = a.x;
        uE = a.y;
        uu = u[0];
        uv = flip_sign(u[1], p.flip_v);
        uw = flip_sign(u[2], p.flip_w);
    };
    auto publish = [&](Ex *x, int slot, const Cell3<T> &P) {
        V2 *q = &x->xP[0][slot];
        q[0 * NR] = pair3<T>(P.r, P.p);
        q[1 * NR] = pair3<T>(P.Ka, P.iKa);
        q[2 * NR] = pair3<T>(P.v, P.w);
        q[3 * NR] = pair3<T>(P.mu, P.mv);
        q[4 * NR] = pair3<T>(P.mw, P.eup_xy);
        if constexpr (!kF) q[5 * NR] = pair3<T>(P.mw, P.eup_z);
    };
    // what is kept of a cell for the faces of the next plane
    struct Keep {
        T r, u, v, w, p, Ka, iKa;
    };
    auto keep = [](const Cell3<T> &P) { return Keep{P.r, P.u, P.v, P.w, P.p, P.Ka, P.iKa}; };
    // +y face between the cell `me` of a row and the row above's, both published in x
    auto yface = [&](const Ex *x, const Keep &me, int slot) {
        const V2 *own = &x->xP[0][slot], *nb = own + 32;
        const V2 n0 = nb[0 * NR], n1 = nb[1 * NR], n2 = nb[2 * NR];
        return face_from<1, kF, NR>(Side3<T>{me.r, me.v, me.p, me.Ka, me.iKa}, Side3<T>{n0.x, n2.x, n0.y, n1.x, n1.y}, own,
                                    nb);
    };
    auto publish_y = [&](Ex *x, int slot, const Flux3<T> &fy) {
        x->xF[0][slot] = pair3<T>(fy.r, fy.n);
        x->xF[1][slot] = pair3<T>(fy.t1, fy.t2);
        x->xFE[slot] = fy.E;
    };

    Ex *xc = &S.ex[0], *xp = &S.ex[1]; // this plane's exchange buffer, the previous plane's
    auto swap = [&]() {
        Ex *h = xc;
        xc = xp;
        xp = h;
    };
    if (w >= 1 && w <= R - 2) {
        // interior rows (in a tile at the wall some may lie past the grid's last row)
        const Place at = place_of(w);
        sh = SM::kRows ? (sh + row_shift(w)) & 15u : 0u;
        const bool interior = (lane >= 1) && (lane <= k3TZ) && (j <= g.nb_y) && (k <= g.nb_z);
        const bool pub = w <= R - 3; // the row above is interior and reads this +y flux
        Keep Pm{};
        T Uu = 0, Uv = 0, Uw = 0, UE = 0;
        Flux3<T> fxlo{};
        // +z face of (k | k+1): the next lane's cell (lane 31 reads the next row's lane 0, a face
        // no interior lane uses)
        auto zface = [&]() {
            const V2 *own = &xp->xP[0][t], *nb = own + 1;
            const V2 n0 = nb[0 * NR], n1 = nb[1 * NR], n2 = nb[2 * NR];
            return face_from<2, kF, NR>(Side3<T>{Pm.r, Pm.w, Pm.p, Pm.Ka, Pm.iKa}, Side3<T>{n0.x, n2.y, n0.y, n1.x, n1.y},
                                        own, nb);
        };
        auto xface = [&](const Cell3<T> &P) {
            return face_from<0, kF, NR>(Side3<T>{Pm.r, Pm.u, Pm.p, Pm.Ka, Pm.iKa},
                                               Side3<T>{P.r, P.u, P.p, P.Ka, P.iKa}, &xp->xP[0][t], &xc->xP[0][t]);
        };
        T ur, uE, uu, uv, uw;
        // planes 0 and 1: conversion, and plane 1's x face
#pragma unroll 1
        for (int m = 0; m < 2; ++m) {
            wait(m);
            load(at, sh, ur, uE, uu, uv, uw);
            next_shift(m);
            const Cell3<T> P = make_cell3<T, kF>(ur, uu, uv, uw, uE, ph);
            publish(xc, t, P);
            if (m == 1) fxlo = xface(P);
            __syncthreads();
            ring.advance();
            swap();
            Pm = keep(P);
            Uu = uu; Uv = uv; Uw = uw; UE = uE;
        }
        long long c = (long long)geo.i0 * g.zy + (long long)j * g.zs + k;
        T *pr = rhoE_n + 2 * c, *pu = uvw_n + 3 * c;
#pragma unroll 1
        for (int m = 2; m < nplanes; ++m) {
            wait(m);
            load(at, sh, ur, uE, uu, uv, uw);
            next_shift(m);
            const Flux3<T> fy = yface(xp, Pm, t);
            const Flux3<T> fz = zface();
            const Cell3<T> P = make_cell3<T, kF>(ur, uu, uv, uw, uE, ph);
            publish(xc, t, P);
            const Flux3<T> fxhi = xface(P);
            if (pub) publish_y(xc, t, fy);
            __syncthreads(); // plane m's cells and plane m-1's +y faces published
            Flux3<T> fzl;
            fzl.r = __shfl_up_sync(FULL, fz.r, 1);
            fzl.n = __shfl_up_sync(FULL, fz.n, 1);
            fzl.t1 = __shfl_up_sync(FULL, fz.t1, 1);
            fzl.t2 = __shfl_up_sync(FULL, fz.t2, 1);
            fzl.E = __shfl_up_sync(FULL, fz.E, 1);
            if (interior) {
                const V2 a0 = xc->xF[0][t - 32], a1 = xc->xF[1][t - 32];
                const Flux3<T> fyl{a0.x, a0.y, a1.x, a1.y, xc->xFE[t - 32]};
                const Upd3<T> o =
                    update3<T, kF>(Pm.r, Uu, Uv, Uw, UE, fxlo, fxhi, fyl, fy, fzl, fz, ph.DtDx, ph.DtDy, ph.DtDz);
                if (SM::kTma || SM::kRows) {
                    *reinterpret_cast<V2 *>(pr) = pair3<T>(o.r, o.E);
                } else {
                    pr[0] = o.r;
                    pr[1] = o.E;
                }
                pu[0] = o.u;
                pu[1] = o.v;
                pu[2] = o.w;
                sink(o);
            }
            const long long zy = g.zy;
            pr += 2 * zy;
            pu += 3 * zy;
            ring.advance();
            swap();
            fxlo = fxhi;
            Pm = keep(P);
            Uu = uu; Uv = uv; Uw = uw; UE = uE;
        }
    } else if (w == 0) {
        // the bottom halo row: conversion, and from plane 2 on its +y face (the first interior
        // row's -y face); with kPair also the top halo row. The stage of plane m-1, which every
        // lane read before the previous barrier, is refilled.
        const Place at0 = place_of(0), att = place_of(R - 1);
        const unsigned sh0 = row_shift(0), sht = row_shift(R - 1);
        Keep Pm{};
#pragma unroll 1
        for (int m = 0; m < nplanes; ++m) {
            T ur, uE, uu, uv, uw;
            wait(m);
            load(at0, SM::kRows ? (sh + sh0) & 15u : 0u, ur, uE, uu, uv, uw);
            if (m >= 2) publish_y(xc, lane, yface(xp, Pm, lane));
            const Cell3<T> P = make_cell3<T, kF>(ur, uu, uv, uw, uE, ph);
            publish(xc, lane, P);
            if constexpr (SM::kPair) {
                load(att, SM::kRows ? (sh + sht) & 15u : 0u, ur, uE, uu, uv, uw);
                publish(xc, 32 * (R - 1) + lane, make_cell3<T, kF>(ur, uu, uv, uw, uE, ph));
            }
            next_shift(m);
            __syncthreads();
            ring.advance();
            swap();
            Pm = keep(P);
        }
    } else {
        // the top halo row (R = W): conversion only
        const Place at = place_of(w);
        sh = SM::kRows ? (sh + row_shift(w)) & 15u : 0u;
#pragma unroll 1
        for (int m = 0; m < nplanes; ++m) {
            T ur, uE, uu, uv, uw;
            wait(m);
            load(at, sh, ur, uE, uu, uv, uw);
            next_shift(m);
            publish(xc, t, make_cell3<T, kF>(ur, uu, uv, uw, uE, ph));
            __syncthreads();
            ring.advance();
            swap();
        }
    }
    if (!SM::kTma) cp_async_wait<0>();
    if (SM::kTma && t == 0 && ring.dead) {
        // gave up on a plane: wait (bounded) for the loads still in flight before the block's
        // shared memory is used again or released
        ring.drain([&](int s, uint32_t parity) { (void)mbar_wait_bounded(&S.full[s], parity); });
    }
    return !ring.dead;
}

} // namespace hydro
