// sliced_gemm.cuh -- FP64 products C = A B on the bf16 tensor cores, by exact slices.
//
// GB300's FP64 MMA runs on the FP64 pipe at 1.1 TFLOP/s; its bf16 tensor cores are three orders
// faster.  Ozaki, Ogita, Oishi and Rump's error-free splitting (Numer. Algorithms 59, 2012) writes each
// operand as a short sum of matrices whose products the fast unit computes without rounding:
//   * each row i of A is scaled by a power of two, 2^-ea_i, so that its entries lie in (-1, 1), and
//     written in S = 9 balanced base-128 digits |d_s| <= 64: a = 2^ea sum_s d_s 2^(-6-7s) up to 2^(ea-63);
//     the columns of B likewise;
//   * the products of digit planes s and t with s + t = l < S ("level" l) are summed in FP32: integers below
//     (l + 1) Kc 2^12 <= 2^23 over a chunk of Kc of the inner dimension, so every operation is exact;
//   * each chunk's sums go to 64-bit integers, levels S-1 .. 5 to one, 4 .. 0 to another, still exactly,
//     and those two to FP64 at the end: two roundings in all.  (FP64 sums per chunk cost 128 instructions a
//     thread at the FP64 pipe's two lanes a clock, 16k cycles; as integers it is 512.)
// What is dropped (digits past 2^-63, levels past S - 1) is at most 10 n 2^-63 of the row's maximum times the
// column's, and about sqrt(n) 2^-63 of them where the digits' signs are mixed, whatever the entries that
// meet.  FP64 rounds each term by 2^-53 of its own size: its error is on the scale of 2^-53 sum |a_k| |b_k|, and
// that sum is far below n max max where the large entries of one operand meet small ones or zeros of the other.
// So the sum is measured: one more plane holds the leading digit of each magnitude, floor(64 |a| 2^-ea), and the
// product of the leading planes, L, bounds it from below, sum |a_k| |b_k| >= 2^(ea + eb - 12) L.  With
//   L >= kLeadFactor sqrt(n),  kLeadFactor = 4,
// sqrt(n) 2^-63 max max is below 2^-53 sum |a_k| |b_k|, and 10 n 2^-63 max max below FP64's bound
// n 2^-53 sum |a_k| |b_k| (n >= 100).  The caller asks that of every entry of the first product, and of the
// second one summed over a row with the weights its entries enter the gradient with.  Errors of the gradient's
// entries over 2^-53 times their FP64 scale, against longer arithmetic, FP64 -> sliced: Toeplitz eigenvectors n = 256 .. 1100
// (L from 130 sqrt(n)) 0.6-1.5 -> 0.2-0.35; Gaussian orthogonal Q, n = 600 (10.8) 4.8 -> 1.1; a gradient of one
// eigenvector (0.7) 15 -> 5; localized eigenvectors (random diagonal as large as the couplings, 0.05)
// 12 -> 14: equal at about a hundredth of the line.  Without the question two uncoupled chains with spectra 1e-10 apart
// (L = 0: 1 / gap of a pair from both chains meets a zero of Q) gave 1e5 where FP64 gives 1.
// Localized Q is turned away before that, from its rows' and columns' norms (kMaxOverRms): it would mostly fail.
// A localized operand, an L too small, an infinity or a NaN sets the matrix's flag word: the sliced
// kernels return at once for it and the caller's FP64 MMA kernels, launched behind them
// with the opposite test, do the work.
//
// The product kernel: 128 x 128 tiles by tcgen05.mma (bf16, FP32 sums in TMEM), one CTA per tile.  Operands lie
// in memory as the tensor core wants them, 128 x 64 tiles of 16 KB with the 128-byte swizzle, so one
// bulk copy brings each.  Four levels at a time have a 128-column accumulator each, so that a plane's
// tile is read once for all of them, 37 bytes a clock and SM at the tensor core's rate (one product at a
// time would take 128).  Two products at n = 2047 take 1.85 ms with everything (mma.sync with 128 x 128 tiles of
// the same operands: 5.4), at n = 4096 10.6 ms.  At
// n = 2047 256 tiles on 152 SMs are two waves, 84 % full; a tile's own time is the products (256 cycles
// each, 1440 of them), the sums' way out of TMEM (18 times, between which the tensor core waits) and the
// epilogue's FP64 division.
#pragma once
#include <cuda_bf16.h>

#include "launch_after.cuh"
#include <cstdint>

namespace symeig {
namespace sliced {

constexpr int S = 9;                      // digit planes
constexpr int BM = 128, BN = 128, BK = 64;
constexpr int kTileValues = BM * BK, kTileBytes = kTileValues * 2;   // one operand tile
constexpr int kSlots = 13;                                // operand tiles in shared memory
constexpr int kSmem = kSlots * kTileBytes + 1024;         // the tiles on a 1 KB boundary
constexpr int kEpiThreads = 256;                          // warps 0-7: TMEM -> integers -> result
constexpr int kThreads = kEpiThreads + 64;                // warp 8 copies, warp 9 issues the MMAs
constexpr int kSmallLevels = 5;                           // levels from this one on are small
static_assert(BM == 128 && BN == 128, "a tile is one tcgen05 shape");

inline int64_t pad_rows(int64_t n) { return (n + BM - 1) / BM * BM; }
inline int64_t pad_k(int64_t n) { return (n + BK - 1) / BK * BK; }
// bf16 values of one operand's planes: the digits and, plane S, the magnitudes' leading digits
constexpr int kPlanes = S + 1;
inline int64_t plane_values(int64_t rows, int64_t k) { return kPlanes * pad_rows(rows) * pad_k(k); }
constexpr double kLeadFactor = 4.0;

// A magnitude's exponent e with |x| < 2^e, or kNoScale for infinity and NaN, kZeroScale for 0.
constexpr int kNoScale = 1 << 20, kZeroScale = -1075;
__device__ __forceinline__ int magnitude_exponent(uint64_t abs_bits)
{
    if (abs_bits >= 0x7FF0000000000000ull) return kNoScale;
    const int ef = (int)(abs_bits >> 52);
    if (ef > 0) return ef - 1022;
    return abs_bits == 0 ? kZeroScale : -1010 - (__clzll((long long)abs_bits));   // subnormal: 2^-1074 * 2^(64 - clz)
}

constexpr int kFixedBits = 6 + 7 * (S - 1);

// x 2^(kFixedBits - e) rounded to an integer (|x| < 2^e, so below 2^62), from the bits: in FP64 the
// scaling and the conversion kept the slicing kernels on the 2-lane FP64 pipe (80 % busy; 0.2 ms of the whole
// adjoint of n = 2047).
__device__ __forceinline__ long long fixed_point(double x, int e)
{
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int ef = (int)(b >> 52) & 0x7FF;
    uint64_t m = b & 0x000FFFFFFFFFFFFFull;
    if (ef) m |= 0x0010000000000000ull;
    const int sh = max(ef, 1) - 1075 + kFixedBits - e;   // |x| = m 2^(max(ef, 1) - 1075); m << sh < 2^62
    const int down = min(-sh, 60);                       // m < 2^53: from 55 on the result is 0
    m = sh >= 0 ? m << sh : (m + (1ull << (down - 1))) >> down;
    return (long long)b < 0 ? -(long long)m : (long long)m;
}

// the S balanced digits of v, plane s at d[s], and |v|'s leading digit
__device__ __forceinline__ void digits(long long v, int (&d)[kPlanes])
{
    d[S] = (int)(llabs(v) >> 7 * (S - 1));
#pragma unroll
    for (int s = S - 1; s > 0; --s) {
        const int t = (int)((v + 64) & 127) - 64;
        d[s] = t;
        v = (v - t) >> 7;
    }
    d[0] = (int)v;
}

__device__ __forceinline__ uint32_t pack(int lo, int hi)
{
    const __nv_bfloat162 p = __floats2bfloat162_rn((float)lo, (float)hi);   // exact: |d| <= 64
    return *reinterpret_cast<const uint32_t*>(&p);
}

// `spread` operands: n max^2 <= kMaxOverRms^2 sum x^2 per row or column (entries of an eigenvector of
// a Toeplitz matrix reach 1.4 times their rms, Gaussian ones 4 to 5, a localized one's about sqrt(n), 16 for
// the smallest order).  Where the squares leave the FP64 range the answer is no.  This spares a
// localized Q the slicing; what the slices are good for, L decides.
constexpr double kMaxOverRms = 6.0;
__device__ __forceinline__ bool spread(double mx, double sum, int64_t n)
{
    return mx == 0.0 || (mx > 1e-140 && mx < 1e140 && mx * mx * (double)n <= kMaxOverRms * kMaxOverRms * sum);
}

// The weight |x| 2^-e of |x| < 2^e in FP32, -2^-60 for one below 2^-60 (but not 0).
__device__ __forceinline__ float weight(double x, int e)
{
    const int hi = __double2hiint(x) & 0x7FFFFFFF, lo = __double2loint(x);
    const int d = (hi >> 20) - 1022 - e;   // |x| in [2^(d-1), 2^d) 2^e
    const float w = d <= -60 ? -0x1p-60f : __int_as_float((d + 126) << 23 | (hi & 0xFFFFF) << 3 | (int)((uint32_t)lo >> 29));
    return (hi | lo) == 0 ? 0.0f : w;
}
// weight times v, never more: a weight below 2^-60 counts as 2^-60 where v is negative and as 0 where it is not
__device__ __forceinline__ float weighted(float w, float v) { return fabsf(w) * (w < 0.0f ? fminf(v, 0.0f) : v); }

// Two operands of one launch (blockIdx.z, or its part beyond the matrices, picks one): a launch saved
// where Q is localized and the FP64 MMA does the work after all.
struct Operand {
    const double* x;
    int* exps;
    __nv_bfloat16* planes;
    bool must_spread;
};

// exps[i] of the columns of X (n x n): one warp per column, blockIdx.y = matrix.  (A block per column, and one per
// row in slice_columns_kernel, were mostly idle in batches of small orders: 25 of n = 300 844 us, 757 this way.)
constexpr int kExpWarps = 8;
static __global__ void __launch_bounds__(32 * kExpWarps)
column_exponents_kernel(Operand o0, Operand o1, int64_t n, int* __restrict__ flag)
{
    wait_previous_launch();
    const int64_t i = (int64_t)blockIdx.x * kExpWarps + (threadIdx.x >> 5);
    if (i >= n || __any_sync(0xffffffffu, flag[blockIdx.y])) return;
    const Operand& o = blockIdx.z == 0 ? o0 : o1;
    const double* x = o.x + (blockIdx.y * n + i) * n;
    unsigned long long m = 0;
    double s[4] = {};
    int64_t k = threadIdx.x & 31;
    for (; k + 96 < n; k += 128) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = x[k + 32 * u];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            m = max(m, (unsigned long long)__double_as_longlong(v[u]) & 0x7FFFFFFFFFFFFFFFull);
            if (o.must_spread) s[u] = fma(v[u], v[u], s[u]);
        }
    }
    for (; k < n; k += 32) {
        const double v = x[k];
        m = max(m, (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull);
        if (o.must_spread) s[0] = fma(v, v, s[0]);
    }
    double sum = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        if (o.must_spread) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    }
    if ((threadIdx.x & 31) == 0) {
        const int e = magnitude_exponent(m);
        o.exps[blockIdx.y * n + i] = e;
        if (e == kNoScale || (o.must_spread && !spread(__longlong_as_double((long long)m), sum, n))) flag[blockIdx.y] = 1;
    }
}

// exps[i] of the rows of X (n x n), which must spread: 32 rows per block, its 32 warps take every 32nd column.
static __global__ void __launch_bounds__(1024)
row_exponents_kernel(const double* __restrict__ X, int64_t n, int* __restrict__ exps, int* __restrict__ flag)
{
    wait_previous_launch();
    if (__syncthreads_or(flag[blockIdx.y])) return;
    __shared__ unsigned long long sh[32][33];
    __shared__ double ss[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i = (int64_t)blockIdx.x * 32 + lane;
    const double* x = X + blockIdx.y * n * n;
    unsigned long long m = 0;
    double sum = 0.0;
    if (i < n)
        for (int64_t k = w; k < n; k += 32) {
            const double v = x[i + k * n];
            m = max(m, (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull);
            sum = fma(v, v, sum);
        }
    sh[w][lane] = m;
    ss[w][lane] = sum;
    __syncthreads();
    // warp w sums row w
    m = sh[lane][w];
    sum = ss[lane][w];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        sum += __shfl_xor_sync(0xffffffffu, sum, d);
    }
    const int64_t r = (int64_t)blockIdx.x * 32 + w;
    if (lane == 0 && r < n) {
        const int e = magnitude_exponent(m);
        exps[blockIdx.y * n + r] = e;
        if (e == kNoScale || !spread(__longlong_as_double((long long)m), sum, n)) flag[blockIdx.y] = 1;
    }
}

// Where 8 inner indices from k0 on of row i of plane s lie: 128 x 64 tiles, 16-byte pieces of a row
// rotated by the row (the 128-byte swizzle).
__device__ __forceinline__ int64_t plane_offset(int s, int64_t i, int64_t k0, int64_t rows, int64_t kp)
{
    const int r = (int)(i & (BM - 1)), c = (int)(k0 & (BK - 1)) >> 3;
    return ((s * (rows / BM) + i / BM) * (kp / BK) + k0 / BK) * kTileValues + r * BK + ((c ^ (r & 7)) << 3);
}

// Planes of the columns of X (rows, kp padded; zeros outside).  One thread per 8 inner indices, a column's
// beside each other; blockIdx.y = matrix, from `count` on the second operand's.
static __global__ void __launch_bounds__(256)
slice_columns_kernel(Operand o0, Operand o1, int count, int64_t n, int64_t rows, int64_t kp, int64_t pstride,
                     const int* flag)
{
    wait_previous_launch();
    const Operand& o = (int)blockIdx.y < count ? o0 : o1;
    const int64_t z = (int)blockIdx.y < count ? blockIdx.y : blockIdx.y - count;
    if (flag[z]) return;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t i = t / (kp / 8), k0 = t % (kp / 8) * 8;
    if (i >= rows) return;
    const double* x = o.x + (z * n + i) * n;
    const int e = i < n ? o.exps[z * n + i] : 0;
    uint32_t out[kPlanes][4];
    int d0[kPlanes], d1[kPlanes];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int64_t k = k0 + 2 * q;
        digits(i < n && k < n ? fixed_point(x[k], e) : 0, d0);
        digits(i < n && k + 1 < n ? fixed_point(x[k + 1], e) : 0, d1);
#pragma unroll
        for (int s = 0; s < kPlanes; ++s) out[s][q] = pack(d0[s], d1[s]);
    }
    __nv_bfloat16* p = o.planes + z * pstride + plane_offset(0, i, k0, rows, kp);
#pragma unroll
    for (int s = 0; s < kPlanes; ++s)
        *reinterpret_cast<uint4*>(p + s * rows * kp) = make_uint4(out[s][0], out[s][1], out[s][2], out[s][3]);
}

// Planes of the rows of X (n x n): as slice_columns_kernel on the transpose, through a 32 x 64
// shared tile.
static __global__ void __launch_bounds__(256)
slice_rows_kernel(const double* __restrict__ X, int64_t n, const int* exps, int64_t rows, int64_t kp,
                  __nv_bfloat16* __restrict__ planes, int64_t pstride,
                  const int* flag)
{
    wait_previous_launch();
    if (flag[blockIdx.z]) return;
    __shared__ double tile[64][33];   // [inner][row]
    const int64_t i0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * 64;
    const double* x = X + blockIdx.z * n * n;
    for (int t = threadIdx.x; t < 64 * 32; t += blockDim.x) {
        const int r = t & 31, c = t >> 5;
        tile[c][r] = i0 + r < n && k0 + c < n ? x[i0 + r + (k0 + c) * n] : 0.0;
    }
    __syncthreads();
    const int r = threadIdx.x >> 3, c = (threadIdx.x & 7) * 8;
    const int64_t i = i0 + r;
    if (i >= rows || k0 + c >= kp) return;
    const int e = i < n ? exps[blockIdx.z * n + i] : 0;
    uint32_t out[kPlanes][4];
    int d0[kPlanes], d1[kPlanes];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        digits(i < n ? fixed_point(tile[c + 2 * q][r], e) : 0, d0);
        digits(i < n ? fixed_point(tile[c + 2 * q + 1][r], e) : 0, d1);
#pragma unroll
        for (int s = 0; s < kPlanes; ++s) out[s][q] = pack(d0[s], d1[s]);
    }
    __nv_bfloat16* p = planes + blockIdx.z * pstride + plane_offset(0, i, k0 + c, rows, kp);
#pragma unroll
    for (int s = 0; s < kPlanes; ++s)
        *reinterpret_cast<uint4*>(p + s * rows * kp) = make_uint4(out[s][0], out[s][1], out[s][2], out[s][3]);
}

// ---- the product ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* b, uint32_t bytes)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(smem_addr(b)),
                 "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_addr(b)), "r"(parity) : "memory");
    return ok != 0;
}

// The levels lo .. hi are summed in one pass over the inner dimension.  For each 64 of it (a block)
// and each plane s of A, in order, the tiles that come in and the products done are:
//   s = 0: A_0, B_hi .. B_lo;  s >= 1: A_s, and B_(lo - s) while that exists
//   A_s B_t for max(0, lo - s) <= t <= hi - s; then A_s and B_(hi - s) are done with
// so each tile comes in once a block, and at most hi - lo + 3 of them are held.
struct Pass {
    int lo, hi;
    __device__ __forceinline__ int loads() const { return 2 * (hi + 1); }
    __device__ __forceinline__ int index_a(int s) const
    {
        return s == 0 ? 0 : hi - lo + 2 + (s <= lo ? 2 * (s - 1) : lo + s - 1);
    }
    __device__ __forceinline__ int index_b(int t) const { return t >= lo ? 1 + hi - t : hi - lo + 2 + 2 * (lo - t - 1) + 1; }
    // blocks whose sums stay below 2^23: (hi + 1) 64 2^12 each
    __device__ __forceinline__ int chunk_blocks() const { return 32 / (hi + 1); }
};
// The last pass alone, on the planes S, gives the leading digits' product L (LEAD).
constexpr int kPasses = 3;
__device__ __forceinline__ Pass pass_of(int p)
{
    return p == 0 ? Pass{kSmallLevels, S - 1} : p == 1 ? Pass{1, kSmallLevels - 1} : Pass{0, 0};
}
static_assert(S - kSmallLevels <= 4 && kSmallLevels - 1 <= 4, "four accumulators of 128 columns");

struct Control {
    uint64_t full[kSlots], empty[kSlots], sums_full, sums_empty, drained;
    uint32_t tmem;
    int failed;
};

// Where a wait that ran out is reported (the handle's error word) and the test hook.
struct Report {
    int* err;
    uint32_t stall;   // tiles copied before the copies stop
    // the FP64 MMA takes the matrix
    __device__ __forceinline__ void timeout(int& fallback) const
    {
        fallback = 1;
        atomicOr(err, 1);
    }
};

// Waits for the phase of `parity`, for about a second at most (failure: false, for every warp).
__device__ __forceinline__ bool wait(Control& c, uint64_t* b, uint32_t parity)
{
    if (mbar_try(b, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(b, parity)) {
        if (*(volatile int*)&c.failed) return false;
        if (clock64() - t0 > 2000000000ll) {
            *(volatile int*)&c.failed = 1;
            return false;
        }
    }
    return true;
}

// A K-major operand tile with the 128-byte swizzle: 8 rows are 1024 bytes.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}

// The copying thread: all tiles of the passes, in order.  Returns once what it started has landed.  `stall`
// (the test hook): tiles from that one on are not copied, so that the waits for them run out.
template <bool LEAD>
__device__ __forceinline__ void copy_tiles(Control& c, uint32_t tiles, const __nv_bfloat16* A, const __nv_bfloat16* B,
                                           int64_t plane, int blocks, uint32_t stall)
{
    uint32_t g = 0;
    bool ok = true;
    auto load = [&](const __nv_bfloat16* src) {
        const uint32_t slot = g % kSlots, turn = g / kSlots;
        if (g >= stall) ok = false;
        else if (turn > 0) ok = wait(c, &c.empty[slot], (turn - 1) & 1);
        if (!ok) return;
        mbar_expect(&c.full[slot], kTileBytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         tiles + slot * kTileBytes),
                     "l"(src), "r"(kTileBytes), "r"(smem_addr(&c.full[slot])) : "memory");
        ++g;
    };
    for (int p = LEAD ? kPasses - 1 : 0; p < kPasses && ok; ++p) {
        const Pass q = pass_of(p);
        for (int kb = 0; kb < blocks && ok; ++kb) {
            const int64_t o = (int64_t)kb * kTileValues;
            for (int s = 0; s <= q.hi && ok; ++s) {
                load(A + s * plane + o);
                if (s == 0) {
                    for (int t = q.hi; t >= q.lo && ok; --t) load(B + t * plane + o);
                } else if (q.lo - s >= 0 && ok) {
                    load(B + (q.lo - s) * plane + o);
                }
            }
        }
    }
    // the last tile of each slot (on failure too: none may land after the block has gone)
    for (uint32_t k = 0; k < kSlots && k < g; ++k) {
        const uint32_t last = g - 1 - k;
        const long long t0 = clock64();
        while (!mbar_try(&c.full[last % kSlots], (last / kSlots) & 1))
            if (clock64() - t0 > 2000000000ll) break;
    }
}

// The issuing thread, a pass unrolled: what it computes per product has to stay below the 256 cycles
// that the tensor core takes for it.  (With the loops rolled and a wait per operand a product took 640.)
__device__ __forceinline__ void commit(uint64_t* b)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(b)) : "memory");
}

struct Ring {
    uint32_t slot, turn;   // of the block's first tile
    __device__ __forceinline__ Ring at(uint32_t index) const
    {
        Ring r{slot + index, turn};
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (r.slot >= kSlots) {
                r.slot -= kSlots;
                ++r.turn;
            }
        return r;
    }
};
static_assert(2 * S + kSlots - 1 < 3 * kSlots, "two wraps");

template <int LO, int HI>
__device__ __forceinline__ bool issue_pass(Control& c, uint64_t desc0, uint32_t tmem, int blocks, Ring& ring, uint32_t& chunk)
{
    constexpr uint32_t idesc = 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(BN >> 3) << 17 | (uint32_t)(BM >> 4) << 24;
    const Pass q{LO, HI};
    const int step = q.chunk_blocks();
    for (int k0 = 0; k0 < blocks; k0 += step, ++chunk) {
        if (chunk > 0 && !wait(c, &c.sums_empty, (chunk - 1) & 1)) return false;
        const int k1 = min(k0 + step, blocks);
        for (int kb = k0; kb < k1; ++kb, ring = ring.at(q.loads())) {
#pragma unroll
            for (int s = 0; s <= HI; ++s) {
                const Ring ra = ring.at(q.index_a(s));
                bool ok = wait(c, &c.full[ra.slot], ra.turn & 1);
#pragma unroll
                for (int t = HI; t >= 0; --t)   // the tiles of B that came in with A_s
                    if (s == 0 ? t >= LO : t == LO - s) {
                        const Ring rb = ring.at(q.index_b(t));
                        ok = ok && wait(c, &c.full[rb.slot], rb.turn & 1);
                    }
                if (!ok) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t da = desc0 + ra.slot * (kTileBytes >> 4);
#pragma unroll
                for (int t = HI - s; t >= (s < LO ? LO - s : 0); --t) {
                    const uint64_t db = desc0 + ring.at(q.index_b(t)).slot * (kTileBytes >> 4);
                    const uint32_t d = tmem + (uint32_t)(s + t - LO) * BN;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) {
                        const uint32_t add = s > 0 || kk > 0 || kb > k0;
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                                     "l"(da + 2 * kk), "l"(db + 2 * kk), "r"(idesc), "r"(add) : "memory");
                    }
                }
                commit(&c.empty[ra.slot]);
                commit(&c.empty[ring.at(q.index_b(HI - s)).slot]);
            }
        }
        commit(&c.sums_full);
    }
    return true;
}

template <bool LEAD>
__device__ __forceinline__ void issue_products(Control& c, uint32_t tiles, uint32_t tmem, int blocks)
{
    Ring ring{0, 0};
    uint32_t chunk = 0;
    const uint64_t desc0 = operand_desc(tiles);
    bool ok = true;
    if constexpr (!LEAD)
        ok = issue_pass<kSmallLevels, S - 1>(c, desc0, tmem, blocks, ring, chunk) &&
             issue_pass<1, kSmallLevels - 1>(c, desc0, tmem, blocks, ring, chunk);
    if (ok) issue_pass<0, 0>(c, desc0, tmem, blocks, ring, chunk);
    // nothing may be in flight when the accumulators are given back
    commit(&c.drained);
    const long long t0 = clock64();
    while (!mbar_try(&c.drained, 0))
        if (clock64() - t0 > 2000000000ll) break;
}

// One 128 x 128 tile of sum_{s+t<S} 2^(-12-7(s+t)) A_s B_t^T, rows i0 .. of A's planes by rows j0 .. of B's; with
// LEAD of the leading digits' product A_S B_S^T, which is an integer below 2^28.
// Thread t < kEpiThreads gets row tile_row(), columns tile_col() .. + 63.  park: 128 KB of memory for this
// tile (not with LEAD).  False, for all threads, if a wait ran out; call it with all kThreads.
template <bool LEAD, typename Out>
__device__ __forceinline__ bool tile_product(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B,
                                             int64_t rows, int64_t kp, int64_t i0, int64_t j0, unsigned char* smem,
                                             double* __restrict__ park, Out (&out)[64], uint32_t stall)
{
    __shared__ Control c;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t tiles = (smem_addr(smem) + 1023) & ~1023u;
    const int blocks = (int)(kp / BK);
    const int64_t plane = rows * kp;
    if (LEAD) {
        A += S * plane;
        B += S * plane;
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&c.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < kSlots; ++k) {
            mbar_init(&c.full[k], 1);
            mbar_init(&c.empty[k], 1);
        }
        mbar_init(&c.sums_full, 1);
        mbar_init(&c.drained, 1);
        mbar_init(&c.sums_empty, kEpiThreads / 32);
        c.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = c.tmem;
    if (warp == 8) {
        if (lane == 0)
            copy_tiles<LEAD>(c, tiles, A + i0 / BM * (kp / BK) * kTileValues, B + j0 / BN * (kp / BK) * kTileValues, plane, blocks,
                             stall);
        __syncwarp();
    } else if (warp == 9) {
        if (lane == 0) issue_products<LEAD>(c, tiles, tmem, blocks);
        __syncwarp();
    } else {
        long long acc[64];
#pragma unroll
        for (int q = 0; q < 64; ++q) acc[q] = 0;
        const uint32_t mine = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 64 * (warp >> 2);
        uint32_t chunk = 0;
        bool ok = true;
        for (int p = LEAD ? kPasses - 1 : 0; p < kPasses && ok; ++p) {
            const Pass q = pass_of(p);
            const int step = q.chunk_blocks(), top = p == 0 ? S - 1 : kSmallLevels - 1;
            for (int k0 = 0; k0 < blocks; k0 += step, ++chunk) {
                ok = __all_sync(0xffffffffu, wait(c, &c.sums_full, chunk & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int l = q.lo; l <= q.hi; ++l) {
                    const int w = LEAD ? 1 : 1 << 7 * (top - l);
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        uint32_t v[16];
                        // one statement, so that no use of v moves above the wait
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
                            "tcgen05.wait::ld.sync.aligned;"
                            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                              "=r"(v[15])
                            : "r"(mine + (uint32_t)(l - q.lo) * BN + 16 * h) : "memory");
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            acc[16 * h + e] += (long long)__float2int_rn(__uint_as_float(v[e])) * w;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&c.sums_empty);
            }
            if (!LEAD && p == 0) {
#pragma unroll
                for (int q2 = 0; q2 < 64; ++q2) {
                    park[q2 * kEpiThreads + tid] = __ll2double_rn(acc[q2]);
                    acc[q2] = 0;
                }
            }
        }
        constexpr double kSmall = 1.0 / (1ull << (12 + 7 * (S - 1) - 28)) / (1ull << 28);
        constexpr double kLarge = 1.0 / (1ull << (12 + 7 * (kSmallLevels - 1)));
#pragma unroll
        for (int q = 0; q < 64; ++q) {
            if constexpr (LEAD) out[q] = (Out)acc[q];
            else out[q] = fma(__ll2double_rn(acc[q]), kLarge, park[q * kEpiThreads + tid] * kSmall);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
    return !*(volatile int*)&c.failed;
}

__device__ __forceinline__ int tile_row() { return (int)threadIdx.x & 127; }
__device__ __forceinline__ int tile_col() { return ((int)threadIdx.x >> 7) * 64; }

}  // namespace sliced
}  // namespace symeig
