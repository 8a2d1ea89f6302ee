// CSV output of a state, formatted on the GPU, byte-identical to the reference's
// write_results (hydro2d/main.cxx:166-235, hydro3d/main.cxx:172-247): a header, then one
// line "i,j[,k],rho,E,rho_u,rho_v[,rho_w]" per interior cell in row-major order, each value
// as std::ostream writes a double by default, i.e. printf("%g"): 6 significant digits,
// correctly rounded (ties to even) from the exact binary value, fixed notation for decimal
// exponents -4..5 and "d.ddddde+XX" otherwise, trailing zeros removed. FP32 states are
// formatted through their exact double value, as the stream does.
//
// Decimal conversion (every double, subnormals included): an estimate of the decimal
// exponent X and of the 6-digit integer N with |v| ~ N * 10^(X-5), from log10/exp10 in
// double (N off by at most one), then exact comparisons of |v| = m * 2^q with the rounding
// midpoints (N +- 1/2) * 10^(X-5) in fixed-size integer arithmetic (m * 5^k or
// (2N+1) * 5^k, shifted by powers of two; 5^k from a table built once per device), which
// move N to the correctly rounded value.
//
// Pipeline, per chunk of rows: one thread formats one cell's line into a fixed-size slot,
// a device scan of the line lengths gives each line's offset, and a compaction writes the
// lines back to back; while the next chunk is formatted, this one goes to the host in pieces
// through two pinned buffers, each copied while the host writes the other to the file.
//
// The kernels of a 1200 x 800 FP64 file (28.6 MB) take 0.6 ms together; what bounds the call is
// the host: the write itself (about 8 ms into the page cache) and the allocations. Pinned memory
// is the expensive one (1.5 to 4 ms per MB to allocate and free), so only two pieces of 384 KB are
// pinned. That file took 121 to 220 ms with whole chunks pinned (4 M cells, 112 bytes a line);
// with these pieces it takes 10 to 20, of which 2 are left when written to /dev/null (pieces of
// 1 MB: 5.5; 2 MB: 8.5). A chunk of 64 K cells keeps the device's share at 22 MB and its kernels
// behind the writing of the chunk before; 16 K cells leave 4 ms, 256 K no less than 2.
#include <cub/device/device_scan.cuh>

#include <math.h>
#include <mutex>
#include <stdio.h>
#include <stdlib.h>

#include "../../include/hydro_b200.h"
#include "hydro_host.h"

namespace hydro {
namespace {

constexpr int kLimbs = 14;     // 896-bit integers: enough for m*5^330*2^s and (2N+1)*5^310
constexpr int kPow5Max = 340;  // 5^k for the decimal exponents of every finite double
constexpr int kSlot = 112;     // bytes reserved per line (longest 3D line: 103)

__device__ unsigned long long g_pow5[kPow5Max + 1][kLimbs];

// 5^k, k = 0..kPow5Max, by repeated multiplication (one thread, once per device)
__global__ void pow5_init_kernel()
{
    unsigned long long p[kLimbs] = {1ull};
    for (int k = 0; k <= kPow5Max; ++k) {
        for (int l = 0; l < kLimbs; ++l) g_pow5[k][l] = p[l];
        unsigned long long carry = 0;
        for (int l = 0; l < kLimbs; ++l) {
            const unsigned long long lo = p[l] * 5ull, hi = __umul64hi(p[l], 5ull);
            const unsigned long long s = lo + carry;
            carry = hi + (s < lo ? 1ull : 0ull);
            p[l] = s;
        }
    }
}

struct Big {
    unsigned long long w[kLimbs];
};

// r = a * m (a a table entry, m < 2^64)
__device__ __forceinline__ void big_mul_small(Big &r, const unsigned long long *a, unsigned long long m)
{
    unsigned long long carry = 0;
#pragma unroll
    for (int l = 0; l < kLimbs; ++l) {
        const unsigned long long lo = a[l] * m, hi = __umul64hi(a[l], m);
        const unsigned long long s = lo + carry;
        carry = hi + (s < lo ? 1ull : 0ull);
        r.w[l] = s;
    }
}
__device__ __forceinline__ void big_set(Big &r, unsigned long long v)
{
    r.w[0] = v;
#pragma unroll
    for (int l = 1; l < kLimbs; ++l) r.w[l] = 0;
}
// r <<= s (the operands here never lose bits: sizes checked in the header comment)
__device__ __forceinline__ void big_shl(Big &r, int s)
{
    const int q = s >> 6, b = s & 63;
    for (int l = kLimbs - 1; l >= 0; --l) {
        const int src = l - q;
        unsigned long long v = src >= 0 ? r.w[src] << b : 0ull;
        if (b && src - 1 >= 0) v |= r.w[src - 1] >> (64 - b);
        r.w[l] = v;
    }
}
__device__ __forceinline__ int big_cmp(const Big &a, const Big &b)
{
    for (int l = kLimbs - 1; l >= 0; --l)
        if (a.w[l] != b.w[l]) return a.w[l] < b.w[l] ? -1 : 1;
    return 0;
}

// sign of m*2^q - (2N+1) * 10^t / 2, exactly
__device__ int cmp_midpoint(unsigned long long m, int q, unsigned long long n2p1, int t)
{
    Big A, B;
    int ea, eb;
    if (t >= 0) {
        big_set(A, m);
        ea = q;
        big_mul_small(B, g_pow5[t], n2p1);
        eb = t - 1;
    } else {
        big_mul_small(A, g_pow5[-t], m);
        ea = q;
        big_set(B, n2p1);
        eb = t - 1;
    }
    const int d = ea - eb;
    if (d >= 0)
        big_shl(A, d);
    else
        big_shl(B, -d);
    return big_cmp(A, B);
}

__device__ __forceinline__ int put_uint(char *s, unsigned long long v)
{
    char tmp[20];
    int n = 0;
    do {
        tmp[n++] = char('0' + v % 10);
        v /= 10;
    } while (v);
    for (int i = 0; i < n; ++i) s[i] = tmp[n - 1 - i];
    return n;
}

// printf("%g", v); returns the length (at most 13)
__device__ int format_g(double v, char *s)
{
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const bool neg = bits >> 63;
    const int bexp = (int)((bits >> 52) & 0x7ff);
    const unsigned long long frac = bits & ((1ull << 52) - 1);
    int n = 0;
    if (neg) s[n++] = '-';
    if (bexp == 0x7ff) {
        const char *w = frac ? "nan" : "inf";
        for (int i = 0; i < 3; ++i) s[n++] = w[i];
        return n;
    }
    if (bexp == 0 && frac == 0) {
        s[n++] = '0';
        return n;
    }
    const unsigned long long m = bexp ? (frac | (1ull << 52)) : frac;
    const int q = bexp ? bexp - 1075 : -1074;
    const double a = fabs(v);
    // estimate: X = floor(log10 a), N = round(a * 10^(5-X)) within one unit
    const double lg = log10(a);
    int X = (int)floor(lg);
    long long N = llrint(exp10(lg - (double)X + 5.0));
    for (int guard = 0; guard < 8; ++guard) {
        const int t = X - 5;
        if (N < 99999) N = 99999;
        if (N > 1000000) N = 1000000;
        // move N until a lies within [N - 1/2, N + 1/2] * 10^t, ties to even
        bool moved = true;
        for (int it = 0; it < 4 && moved; ++it) {
            moved = false;
            const int hi = cmp_midpoint(m, q, 2ull * (unsigned long long)N + 1ull, t);
            if (hi > 0 || (hi == 0 && (N & 1))) {
                ++N;
                moved = true;
                continue;
            }
            const int lo = cmp_midpoint(m, q, 2ull * (unsigned long long)N - 1ull, t);
            if (lo < 0 || (lo == 0 && (N & 1))) {
                --N;
                moved = true;
            }
        }
        if (N >= 1000000) { // rounds up to the next decade
            ++X;
            N = 100000;
            break;
        }
        if (N < 100000) { // the decade was overestimated
            --X;
            N = llrint(exp10(lg - (double)X + 5.0));
            continue;
        }
        break;
    }
    char d[6];
    for (int i = 5; i >= 0; --i) {
        d[i] = char('0' + N % 10);
        N /= 10;
    }
    int last = 5; // last significant digit kept after removing trailing zeros
    while (last > 0 && d[last] == '0') --last;
    if (X < -4 || X >= 6) {
        s[n++] = d[0];
        if (last > 0) {
            s[n++] = '.';
            for (int i = 1; i <= last; ++i) s[n++] = d[i];
        }
        s[n++] = 'e';
        s[n++] = X < 0 ? '-' : '+';
        const int ax = X < 0 ? -X : X;
        if (ax < 10) s[n++] = '0';
        n += put_uint(s + n, (unsigned long long)ax);
    } else if (X >= 0) {
        for (int i = 0; i <= X; ++i) s[n++] = d[i];
        if (last > X) {
            s[n++] = '.';
            for (int i = X + 1; i <= last; ++i) s[n++] = d[i];
        }
    } else {
        s[n++] = '0';
        s[n++] = '.';
        for (int i = 0; i < -X - 1; ++i) s[n++] = '0';
        for (int i = 0; i <= last; ++i) s[n++] = d[i];
    }
    return n;
}

// One line per cell of rows [row0, row0 + rows) (interior rows, 1-based) into fixed slots.
template <class T, int D>
__global__ void format_lines(const T *rhoE, const T *uvx, int nb_y, int nb_z, long long row0, int rows,
                             long long i_offset, char *slots, unsigned *lens)
{
    const long long per_row = (long long)nb_y * (D == 3 ? nb_z : 1);
    const long long ncell = per_row * rows;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < ncell;
         q += (long long)gridDim.x * blockDim.x) {
        const long long r = q / per_row, rem = q % per_row;
        const long long i = row0 + r; // 1-based interior row
        long long j, k = 0, c;
        if (D == 2) {
            j = rem;
            c = i * (nb_y + 2) + j + 1;
        } else {
            j = rem / nb_z;
            k = rem % nb_z;
            c = (i * (long long)(nb_y + 2) + j + 1) * (nb_z + 2) + k + 1;
        }
        uint4 buf[kSlot / 16];
        char *s = reinterpret_cast<char *>(buf);
        int n = put_uint(s, (unsigned long long)(i_offset + i - 1));
        s[n++] = ',';
        n += put_uint(s + n, (unsigned long long)j);
        s[n++] = ',';
        if (D == 3) {
            n += put_uint(s + n, (unsigned long long)k);
            s[n++] = ',';
        }
        n += format_g((double)rhoE[2 * c], s + n);
        s[n++] = ',';
        n += format_g((double)rhoE[2 * c + 1], s + n);
        for (int v = 0; v < D; ++v) {
            s[n++] = ',';
            n += format_g((double)uvx[D * c + v], s + n);
        }
        s[n++] = '\n';
        uint4 *dst = reinterpret_cast<uint4 *>(slots + q * kSlot);
#pragma unroll
        for (int w = 0; w < kSlot / 16; ++w)
            if (16 * w < n) dst[w] = buf[w];
        lens[q] = (unsigned)n;
    }
}

// Lines back to back at their scanned offsets.
__global__ void compact_lines(const char *slots, const unsigned *lens, const unsigned long long *offs, long long n,
                              char *out)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const char *src = slots + q * kSlot;
        char *dst = out + offs[q];
        const unsigned len = lens[q];
        for (unsigned b = 0; b < len; ++b) dst[b] = src[b];
    }
}

// g_values formatted as %g into 16-byte records (for tests)
__global__ void format_values(const double *v, long long n, char *out)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        char s[16];
        const int len = format_g(v[q], s);
        for (int b = 0; b < 16; ++b) out[q * 16 + b] = b < len ? s[b] : '\0';
    }
}

std::mutex g_pow5_mu;
bool g_pow5_done[64];

int ensure_pow5(cudaStream_t st)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        set_error(kErrCuda, "csv: no current device");
        return kErrCuda;
    }
    std::lock_guard<std::mutex> lk(g_pow5_mu);
    if (g_pow5_done[dev]) return kOk;
    pow5_init_kernel<<<1, 1, 0, st>>>();
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        set_error(kErrCuda, "csv: power table: %s", cudaGetErrorString(e));
        return kErrCuda;
    }
    g_pow5_done[dev] = true;
    return kOk;
}

template <class T, int D>
long long write_csv(const T *rhoE, const T *uvx, size_t nb_x, size_t nb_y, size_t nb_z, size_t i_offset,
                    const char *path, cudaStream_t st)
{
    if (!rhoE || !uvx || !path) {
        set_error(kErrArg, "write_csv: null argument");
        return kErrArg;
    }
    if (nb_x > (1u << 30) || nb_y > (1u << 30) || (D == 3 && nb_z > (1u << 30)) || i_offset > (1ull << 40)) {
        set_error(kErrArg, "write_csv: grid or row offset too large");
        return kErrArg;
    }
    int rc = ensure_pow5(st);
    if (rc != kOk) return rc;
    FILE *f = fopen(path, "wb");
    if (!f) {
        set_error(kErrArg, "write_csv: cannot open %s", path);
        return kErrArg;
    }
    const char *header = D == 2 ? "x,y,rho,p,u,v\n" : "x,y,z,rho,p,u,v,w\n";
    long long total = (long long)fwrite(header, 1, strlen(header), f);
    const long long per_row = (long long)nb_y * (D == 3 ? (long long)nb_z : 1);
    if (nb_x == 0 || per_row == 0) {
        fclose(f);
        return total;
    }
    // cells per chunk (HYDRO_B200_CSV_CHUNK_CELLS overrides, e.g. to exercise many chunks)
    long long target = 1ll << 16;
    if (const char *env = getenv("HYDRO_B200_CSV_CHUNK_CELLS")) {
        const long long v = atoll(env);
        if (v > 0) target = v;
    }
    const int rows = (int)std::max<long long>(1, std::min<long long>((long long)nb_x, target / per_row));
    const long long cap = per_row * rows;
    const size_t line_bytes = (size_t)cap * kSlot;
    const size_t piece = std::min<size_t>(line_bytes, (size_t)384 << 10);
    // device: the slots, two buffers of lines back to back, lengths, offsets, the scan's scratch
    size_t tmp_bytes = 0;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, (unsigned *)nullptr, (unsigned long long *)nullptr,
                                                  (int)cap, st);
    const auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    const bool many = rows < (int)nb_x; // more than one chunk
    char *dev = nullptr, *out[2] = {nullptr, nullptr}, *host[2] = {nullptr, nullptr};
    unsigned long long *h_tot = nullptr; // per chunk parity: the last line's offset and length
    cudaEvent_t ready[2] = {nullptr, nullptr}, copied[2] = {nullptr, nullptr};
    cudaStream_t copies = nullptr;
    if (e == cudaSuccess)
        e = cudaMalloc(&dev, up(line_bytes) * (many ? 3 : 2) + up(cap * sizeof(unsigned)) +
                                 up(cap * sizeof(unsigned long long)) + tmp_bytes);
    char *const slots = dev;
    unsigned *lens = nullptr;
    unsigned long long *offs = nullptr;
    void *tmp = nullptr;
    if (e == cudaSuccess) {
        char *q = dev + up(line_bytes);
        out[0] = q;
        if (many) q += up(line_bytes);
        out[1] = q;
        q += up(line_bytes);
        lens = reinterpret_cast<unsigned *>(q);
        q += up(cap * sizeof(unsigned));
        offs = reinterpret_cast<unsigned long long *>(q);
        tmp = q + up(cap * sizeof(unsigned long long));
        char *pinned = nullptr;
        e = cudaMallocHost(&pinned, 2 * up(piece) + 4 * sizeof(unsigned long long));
        if (e == cudaSuccess) {
            host[0] = pinned;
            host[1] = pinned + up(piece);
            h_tot = reinterpret_cast<unsigned long long *>(pinned + 2 * up(piece));
        }
    }
    for (int b = 0; b < 2; ++b) {
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ready[b], cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&copied[b], cudaEventDisableTiming);
    }
    // (one chunk is copied behind its kernels: creating the stream took a quarter of the 0.3 ms of a
    // 60 x 60 file)
    if (e == cudaSuccess && many) e = cudaStreamCreateWithFlags(&copies, cudaStreamNonBlocking);
    const cudaStream_t from = many ? copies : st;

    // the lines of chunk c, whose kernels have been launched, to the file
    auto write_chunk = [&](int c) {
        const int b = c & 1;
        e = cudaEventSynchronize(ready[b]);
        if (e != cudaSuccess) return;
        const size_t bytes = (size_t)h_tot[2 * b] + (unsigned)h_tot[2 * b + 1];
        auto fetch = [&](size_t at, int h) {
            e = cudaMemcpyAsync(host[h], out[b] + at, std::min(piece, bytes - at), cudaMemcpyDeviceToHost, from);
            if (e == cudaSuccess) e = cudaEventRecord(copied[h], from);
        };
        int h = 0;
        fetch(0, h);
        for (size_t at = 0; e == cudaSuccess && at < bytes; at += piece, h ^= 1) {
            if (at + piece < bytes) fetch(at + piece, h ^ 1); // while this piece is written
            if (e == cudaSuccess) e = cudaEventSynchronize(copied[h]);
            if (e != cudaSuccess) return;
            const size_t n = std::min(piece, bytes - at);
            if (fwrite(host[h], 1, n, f) != n) {
                set_error(kErrArg, "write_csv: short write to %s", path);
                rc = kErrArg;
                return;
            }
            total += (long long)n;
        }
    };
    int chunk = 0;
    for (long long row0 = 1; e == cudaSuccess && rc == kOk && row0 <= (long long)nb_x; row0 += rows, ++chunk) {
        const int nr = (int)std::min<long long>(rows, (long long)nb_x - row0 + 1);
        const long long n = per_row * nr;
        const int b = chunk & 1;
        const int blocks = (int)std::min<long long>((n + 255) / 256, (long long)device_sms() * 16);
        format_lines<T, D><<<blocks, 256, 0, st>>>(rhoE, uvx, (int)nb_y, (int)nb_z, row0, nr, (long long)i_offset,
                                                    slots, lens);
        e = cudaGetLastError();
        // offsets of the n lines
        if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, lens, offs, (int)n, st);
        if (e == cudaSuccess) {
            compact_lines<<<blocks, 256, 0, st>>>(slots, lens, offs, n, out[b]);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) h_tot[2 * b + 1] = 0; // (a 4-byte length in an 8-byte word)
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&h_tot[2 * b], offs + (n - 1), sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&h_tot[2 * b + 1], lens + (n - 1), sizeof(unsigned), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ready[b], st);
        // the previous chunk, whose buffer the next one takes over
        if (e == cudaSuccess && chunk > 0) write_chunk(chunk - 1);
    }
    if (e == cudaSuccess && rc == kOk && chunk > 0) write_chunk(chunk - 1);
    cudaStreamSynchronize(st); // (after an error work may still be in flight)
    if (copies) {
        cudaStreamSynchronize(copies);
        cudaStreamDestroy(copies);
    }
    cudaFree(dev);
    if (host[0]) cudaFreeHost(host[0]);
    for (int b = 0; b < 2; ++b) {
        if (ready[b]) cudaEventDestroy(ready[b]);
        if (copied[b]) cudaEventDestroy(copied[b]);
    }
    if (fclose(f) != 0 && rc == kOk) {
        set_error(kErrArg, "write_csv: closing %s failed", path);
        rc = kErrArg;
    }
    if (e != cudaSuccess) {
        set_error(kErrCuda, "write_csv: %s", cudaGetErrorString(e));
        return kErrCuda;
    }
    return rc == kOk ? total : rc;
}

} // namespace
} // namespace hydro

using namespace hydro;

extern "C" {

long long hydro2d_write_csv_f64(const double *d_rhoE, const double *d_uv, size_t NB_X, size_t NB_Y, size_t i_offset,
                                const char *path, void *stream)
{
    return write_csv<double, 2>(d_rhoE, d_uv, NB_X, NB_Y, 0, i_offset, path, (cudaStream_t)stream);
}
long long hydro2d_write_csv_f32(const float *d_rhoE, const float *d_uv, size_t NB_X, size_t NB_Y, size_t i_offset,
                                const char *path, void *stream)
{
    return write_csv<float, 2>(d_rhoE, d_uv, NB_X, NB_Y, 0, i_offset, path, (cudaStream_t)stream);
}
long long hydro3d_write_csv_f64(const double *d_rhoE, const double *d_uvw, size_t NB_X, size_t NB_Y, size_t NB_Z,
                                size_t i_offset, const char *path, void *stream)
{
    return write_csv<double, 3>(d_rhoE, d_uvw, NB_X, NB_Y, NB_Z, i_offset, path, (cudaStream_t)stream);
}
long long hydro3d_write_csv_f32(const float *d_rhoE, const float *d_uvw, size_t NB_X, size_t NB_Y, size_t NB_Z,
                                size_t i_offset, const char *path, void *stream)
{
    return write_csv<float, 3>(d_rhoE, d_uvw, NB_X, NB_Y, NB_Z, i_offset, path, (cudaStream_t)stream);
}

int hydro_format_g(const double *d_values, size_t n, char *d_out, void *stream)
{
    if (!d_values || !d_out) {
        set_error(kErrArg, "hydro_format_g: null argument");
        return kErrArg;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int rc = ensure_pow5(st);
    if (rc != kOk) return rc;
    if (n == 0) return kOk;
    format_values<<<(int)std::min<size_t>((n + 255) / 256, (size_t)device_sms() * 16), 256, 0, st>>>(d_values, (long long)n, d_out);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        set_error(kErrCuda, "hydro_format_g: %s", cudaGetErrorString(e));
        return kErrCuda;
    }
    return kOk;
}

} // extern "C"
