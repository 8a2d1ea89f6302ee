// Per-device contexts, error latch and TMA descriptor encoding.
#include <algorithm>
#include <atomic>
#include <cudaTypedefs.h>
#include <mutex>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>
#include <vector>

#include "hydro_host.h"

namespace hydro {

namespace {
std::mutex g_mu;
DevCtx *g_ctx[64] = {};
int g_err = 0;
char g_msg[512] = "";
} // namespace

void set_error(int code, const char *fmt, ...)
{
    std::lock_guard<std::mutex> lk(g_mu);
    g_err = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_msg, sizeof g_msg, fmt, ap);
    va_end(ap);
}

int last_error()
{
    std::lock_guard<std::mutex> lk(g_mu);
    return g_err;
}

const char *last_error_string()
{
    std::lock_guard<std::mutex> lk(g_mu);
    return g_msg;
}

void clear_error()
{
    std::lock_guard<std::mutex> lk(g_mu);
    g_err = 0;
    g_msg[0] = 0;
}

DevCtx *ctx_current(int *err)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
        set_error(kErrCuda, "cudaGetDevice failed: %s", cudaGetErrorString(e));
        *err = kErrCuda;
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_ctx[dev]) {
        *err = kOk;
        return g_ctx[dev];
    }
    DevCtx *c = new DevCtx;
    c->device = dev;
    e = cudaMalloc(&c->scr, sizeof(StepScratch));
    if (e == cudaSuccess) e = cudaMemset(c->scr, 0, sizeof(StepScratch));
    if (e == cudaSuccess) e = cudaHostAlloc(&c->status_h, sizeof(StepStatus), cudaHostAllocMapped);
    if (e == cudaSuccess) {
        memset(c->status_h, 0, sizeof(StepStatus));
        e = cudaHostGetDevicePointer(&c->status_d, c->status_h, 0);
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        snprintf(g_msg, sizeof g_msg, "device context set-up failed: %s", cudaGetErrorString(e));
        g_err = kErrCuda;
        *err = kErrCuda;
        if (c->scr) cudaFree(c->scr);
        if (c->status_h) cudaFreeHost(c->status_h);
        delete c;
        return nullptr;
    }
    g_ctx[dev] = c;
    *err = kOk;
    return c;
}

int device_sms()
{
    static std::atomic<int> cache[64];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 1;
    cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

cudaError_t blocks_per_sm(const void *kernel, int threads, int smem, int *blocks)
{
    struct Known {
        const void *kernel;
        int dev, blocks;
    };
    static std::mutex mu;
    static std::vector<Known> known; // one entry per kernel and device
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    for (const Known &k : known)
        if (k.kernel == kernel && k.dev == dev) {
            *blocks = k.blocks;
            return cudaSuccess;
        }
    if (smem > 0) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int n = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    known.push_back(Known{kernel, dev, std::max(1, n)});
    *blocks = known.back().blocks;
    return cudaSuccess;
}

// The time of a launch, in rows of one full SM, for `chunk` rows per block: the busiest SM
// takes m = ceil(blocks / SMs) blocks, per_sm at a time. r of them beside one another march at
// 0.3 + 0.7 r / per_sm of the time of a full SM (3D FP64: 1.03 us a plane alone, 1.65 us two
// beside one another; 3D FP32 0.85, 1.1, 1.65; 2D FP64 0.86 alone, 1.4 four). A block costs 3
// rows beyond its own (two halo rows, start and end), and blocks that end at different times
// about 0.12 of one block's rows. The fastest chunk found by a sweep lies within 3 % of the
// one taken; before (about 24 or 16 blocks per SM, at least 16 or 8 rows) 170^3 FP64 took 11
// planes in 195 us, with 25 177 us; 170^3 FP32 173 against 129 us; 321 x 255 x 259 FP32 393
// against 363 us; 8000 x 4000 FP32 293 against 275 us; 60 x 60 FP64 16 rows in 29 us, 2 in 16.
int march_chunk(size_t rows, size_t tiles, int per_sm, int cap, int least, double *cost_out)
{
    struct Plan {
        size_t rows = 0, tiles = 0;
        int per_sm = 0, cap = 0, least = 0, sms = 0, chunk = 0;
        double cost = 0.0;
    };
    static thread_local Plan last[4];
    static thread_local unsigned next = 0;
    const int sms = device_sms();
    for (const Plan &p : last)
        if (p.rows == rows && p.tiles == tiles && p.per_sm == per_sm && p.cap == cap && p.least == least &&
            p.sms == sms) {
            if (cost_out) *cost_out = p.cost;
            return p.chunk;
        }
    cap = std::max(1, cap);
    least = std::max(1, std::min(least, cap));
    const auto blocks_of = [&](size_t chunk) { return tiles * ((rows + chunk - 1) / chunk); };
    // candidates: for each m the fewest rows per block that keep within m blocks per SM
    const size_t m0 = (blocks_of((size_t)cap) + sms - 1) / sms;
    size_t best = std::min<size_t>(rows, (size_t)cap);
    double best_cost = 0.0;
    for (size_t m = m0; m < m0 + 12 * (size_t)per_sm; ++m) {
        const size_t nchunks = m * sms / tiles;
        if (nchunks == 0) continue;
        size_t chunk = std::max<size_t>((rows + nchunks - 1) / nchunks, (size_t)least);
        chunk = std::min(chunk, (size_t)cap);
        const size_t full = (blocks_of(chunk) + sms - 1) / sms, r = full % per_sm;
        const double rounds = (double)(full / per_sm) + (r ? 0.3 + 0.7 * (double)r / per_sm : 0.0);
        const double cost = rounds * (double)(chunk + 3) + 0.12 * (double)chunk;
        if (best_cost == 0.0 || cost < best_cost) {
            best_cost = cost;
            best = chunk;
        }
        if (chunk <= (size_t)least) break;
    }
    Plan &p = last[next++ % 4];
    p = Plan{rows, tiles, per_sm, cap, least, sms, (int)best, best_cost};
    if (cost_out) *cost_out = best_cost;
    return (int)best;
}

// Long chunks first and short ones last: with all alike, the blocks that start last run while
// other SMs have nothing left. Blocks start in the order of their index, chunks slowest, so the
// short ones fill the SMs up at the end. By the same model, every chunk costs its planes and 3
// more, and the resident blocks share the work evenly, to within 0.3 of a short chunk, if the long
// ones end well before (1.1: 200 x 201 x 203 FP32, whose one long chunk of 96 planes lasted to the
// end, took 164 against 156 us). Taken where that beats the best even split, which 512^3 keeps
// (256 planes are nine full rounds). FP64 strict: 170^3 161.7 -> 153.1 us, 256^3 450 -> 426, 300^3
// 647 -> 627; FP32 fused: 170^3 105 -> 96, 400^3 950 -> 909. From 48 planes per resident block
// on: 128^3 FP64 with 41 lost (82.1 -> 85.7 us). The same sweep in 2D gained 2 % at most and lost
// up to 17 %.
Chunks march_chunks(size_t rows, size_t tiles, int per_sm, int cap, int least)
{
    double cost = 0.0;
    size_t c = (size_t)march_chunk(rows, tiles, per_sm, cap > 0 ? cap : 256, least, &cost);
    c = std::max(c, (rows + 65534) / 65535);
    Chunks best{0, 0, (int)c, (int)((rows + c - 1) / c)};
    const size_t slots = (size_t)device_sms() * per_sm;
    if (cap > 0 || rows > 65535 || rows * tiles < 48 * slots) return best;
    for (int len : {16, 24, 32, 48, 64, 96, 128, 192, 256})
        for (int n = (int)rows / len, longs = n; longs > 0 && longs > n - 3; --longs)
            for (int rest : {8, 12, 16, 24, 32, 48}) {
                const int left = (int)rows - longs * len, shorts = (left + rest - 1) / rest;
                if (2 * rest > len || shorts == 0) continue;
                const double work = (double)tiles * (double)(rows + 3 * (size_t)(longs + shorts)) / slots;
                const double first = (double)((tiles * longs + slots - 1) / slots) * (len + 3);
                const double t = std::max(work, 1.1 * first) + 0.3 * (rest + 3);
                if (t < cost) {
                    cost = t;
                    best = Chunks{longs, len, rest, longs + shorts};
                }
            }
    return best;
}

namespace {
LaunchShape g_shape[2][2]; // [dim - 2][FP64]
} // namespace

LaunchShape launch_shape(int dim, size_t tsize)
{
    std::lock_guard<std::mutex> lk(g_mu);
    return g_shape[dim == 3][tsize == 8];
}

int set_launch_shape(int dim, size_t tsize, int warps, int chunk, int blocks)
{
    const int alt_blocks = tsize == 8 ? 5 : 8;
    if ((dim != 2 && dim != 3) || (tsize != 4 && tsize != 8) || chunk < 0 || chunk > (1 << 20) ||
        (dim == 2 && (warps != 0 || (blocks != 0 && blocks != 4 && blocks != alt_blocks))) ||
        (dim == 3 && (blocks != 0 || (warps != 0 && warps != 8 && warps != 16 &&
                                          !(tsize == 8 && (warps == 9 || warps == 12)))))) {
        set_error(kErrArg,
                  "hydro_set_launch_shape: unsupported shape (dim %d, %zu-byte values, %d warps, chunk %d, %d blocks)",
                  dim, tsize, warps, chunk, blocks);
        return kErrArg;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    g_shape[dim == 3][tsize == 8] = LaunchShape{warps, chunk, blocks};
    return kOk;
}

int step_result(unsigned err, const char *step, bool *dirty)
{
    if (err & kErrWaitTimeout) {
        *dirty = true;
        if (step) set_error(kErrTimeout, "%s: a TMA barrier wait timed out", step);
        return kErrTimeout;
    }
    if (err & kErrNonPhysical) {
        if (step) set_error(kErrPhys, "%s: non-physical state (rho <= 0 or non-finite signal speed)", step);
        return kErrPhys;
    }
    return kOk;
}

int ctx_count()
{
    std::lock_guard<std::mutex> lk(g_mu);
    int n = 0;
    for (DevCtx *c : g_ctx) n += (c != nullptr);
    return n;
}

int ctx_reserve(DevCtx *c, size_t n)
{
    if (n <= c->partial_cap) return kOk;
    size_t cap = c->partial_cap ? c->partial_cap : 1024;
    while (cap < n) cap *= 2;
    cudaError_t e = cudaDeviceSynchronize();
    if (c->partials) cudaFree(c->partials);
    c->partials = nullptr;
    c->partial_cap = 0;
    if (e == cudaSuccess) e = cudaMalloc(&c->partials, cap * sizeof(double2));
    if (e != cudaSuccess) {
        set_error(kErrCuda, "scratch allocation of %zu partials failed: %s", cap, cudaGetErrorString(e));
        return kErrCuda;
    }
    c->partial_cap = cap;
    return kOk;
}

namespace {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}
} // namespace

bool encode_tmap_3d(CUtensorMap *tm, CUtensorMapDataType dt, const void *base, uint64_t dim0, uint64_t dim1,
                    uint64_t dim2, uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t box0, uint32_t box1,
                    uint32_t box2)
{
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {dim0, dim1, dim2};
    cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
    cuuint32_t box[3] = {box0, box1, box2};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = fn(tm, dt, 3, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

} // namespace hydro
