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
// What is dropped (digits past 2^-63, levels past S - 1) is 2^-63 of the row's maximum times the
// column's for each term, where FP64 rounds each by 2^-53 of its own size.  That is the smaller of the two
// while one operand's rows are spread out, their maximum no more than some hundred times a typical
// entry; the caller's other operand may be anything.  The exponent kernels check it for the operand that
// is asked to be (kMaxOverRms).  Measured against longer
// arithmetic, gradients of Toeplitz eigenvectors n = 257 .. 2047: 1.4e-16 .. 2.3e-16 of their norm, FP64 MMA
// 6.0e-16 .. 1.9e-15; Gaussian orthogonal Q, n = 600: 1.6e-16 against 1.9e-15.
// A localized operand, an infinity or a NaN sets the matrix's flag word: the sliced
// kernels return at once for it and the caller's FP64 MMA kernels, launched behind them
// with the opposite test, do the work.
//
// The product kernel: 128 x 128 tiles, 8 warps of 64 x 32 with mma.sync m16n8k16 (bf16, FP32 sums), operand
// tiles of 64 of the inner dimension in a three-stage shared-memory ring by cp.async.  45 plane
// products for S = 9: 352 TFLOP/s at n = 4096, bound by ldmatrix's shared-memory reads (98 KB a
// step of 64 for 8 warps, 768 of about 1850 cycles) beside the MMAs (1024).  With 32-deep steps and
// FP64 sums per chunk the two products of n = 2047 took 8.3 ms instead of 5.5.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

namespace symeig {
namespace sliced {

constexpr int S = 9;                      // digit planes
constexpr int BM = 128, BN = 128, BK = 64, STAGES = 3, kThreads = 256;
constexpr int kTileBytes = BM * BK * 2;   // one operand tile
constexpr int kRing = STAGES * 2 * kTileBytes;
constexpr int kSmem = kRing + BM * BN * (int)sizeof(double);   // and the small levels' sums
constexpr int kSmallLevels = 5;                                // levels from this one on are small

inline int64_t pad_rows(int64_t n) { return (n + BM - 1) / BM * BM; }
inline int64_t pad_k(int64_t n) { return (n + BK - 1) / BK * BK; }
// bf16 values of one operand's planes
inline int64_t plane_values(int64_t rows, int64_t k) { return S * pad_rows(rows) * pad_k(k); }

// A magnitude's exponent e with |x| < 2^e, or kNoScale for infinity and NaN (0 gives -1075).
constexpr int kNoScale = 1 << 20;
__device__ __forceinline__ int magnitude_exponent(uint64_t abs_bits)
{
    if (abs_bits >= 0x7FF0000000000000ull) return kNoScale;
    const int ef = (int)(abs_bits >> 52);
    if (ef > 0) return ef - 1022;
    return abs_bits == 0 ? -1075 : -1010 - (__clzll((long long)abs_bits));   // subnormal: 2^-1074 * 2^(64 - clz)
}

constexpr int kFixedBits = 6 + 7 * (S - 1);

// x 2^(kFixedBits - e) rounded to an integer (|x| < 2^e, so at most 2^62)
__device__ __forceinline__ long long fixed_point(double x, int e)
{
    // in two exact steps, so that the scale factors stay normal
    const int sh = kFixedBits - e, h = sh / 2;
    return __double2ll_rn(scalbn(scalbn(x, h), sh - h));
}

// the S balanced digits of v, plane s at d[s]
__device__ __forceinline__ void digits(long long v, int (&d)[S])
{
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
// a Toeplitz matrix reach 1.4 times their rms, Gaussian ones 4 to 5, a localized one's sqrt(n)).
// Where the squares leave the FP64 range the answer is no.
constexpr double kMaxOverRms = 16.0;
__device__ __forceinline__ bool spread(double mx, double sum, int64_t n)
{
    return mx == 0.0 || (mx > 1e-140 && mx < 1e140 && mx * mx * (double)n <= kMaxOverRms * kMaxOverRms * sum);
}

// exps[i] of the columns of X (n x cols, leading dimension ld): one block per column.
static __global__ void __launch_bounds__(256)
column_exponents_kernel(const double* __restrict__ X, int64_t ld, int64_t n, int64_t stride, int* __restrict__ exps,
                        int64_t estride, bool must_spread, int* __restrict__ flag)
{
    __shared__ unsigned long long sh[8];
    __shared__ double ss[8];
    const double* x = X + blockIdx.y * stride + (int64_t)blockIdx.x * ld;
    unsigned long long m = 0;
    double sum = 0.0;
    for (int64_t k = threadIdx.x; k < n; k += blockDim.x) {
        const double v = x[k];
        m = max(m, (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull);
        sum = fma(v, v, sum);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sh[threadIdx.x >> 5] = m;
        ss[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            m = max(m, sh[w]);
            sum += ss[w];
        }
        const int e = magnitude_exponent(m);
        exps[blockIdx.y * estride + blockIdx.x] = e;
        if (e == kNoScale || (must_spread && !spread(__longlong_as_double((long long)m), sum, n))) flag[blockIdx.y] = 1;
    }
}

// exps[i] of the rows of X (n x n): 32 rows per block.
static __global__ void __launch_bounds__(256)
row_exponents_kernel(const double* __restrict__ X, int64_t ld, int64_t n, int64_t stride, int* __restrict__ exps,
                     int64_t estride, bool must_spread, int* __restrict__ flag)
{
    __shared__ unsigned long long sh[8][32];
    __shared__ double ss[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i = (int64_t)blockIdx.x * 32 + lane;
    const double* x = X + blockIdx.y * stride;
    unsigned long long m = 0;
    double sum = 0.0;
    if (i < n)
        for (int64_t k = w; k < n; k += 8) {
            const double v = x[i + k * ld];
            m = max(m, (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull);
            sum = fma(v, v, sum);
        }
    sh[w][lane] = m;
    ss[w][lane] = sum;
    __syncthreads();
    if (w == 0 && i < n) {
        for (int q = 1; q < 8; ++q) {
            m = max(m, sh[q][lane]);
            sum += ss[q][lane];
        }
        const int e = magnitude_exponent(m);
        exps[blockIdx.y * estride + i] = e;
        if (e == kNoScale || (must_spread && !spread(__longlong_as_double((long long)m), sum, n))) flag[blockIdx.y] = 1;
    }
}

// Planes of the columns of X: plane s, column i, inner index k at planes[(s * rows + i) * kp + k]
// (rows, kp padded; zeros outside).  One thread per 8 inner indices.
static __global__ void __launch_bounds__(256)
slice_columns_kernel(const double* __restrict__ X, int64_t ld, int64_t n, int64_t stride, const int* __restrict__ exps,
                     int64_t estride, int64_t rows, int64_t kp, __nv_bfloat16* __restrict__ planes, int64_t pstride,
                     const int* __restrict__ flag)
{
    if (flag[blockIdx.z]) return;
    const int64_t k0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    const int64_t i = blockIdx.y;
    if (k0 >= kp) return;
    const double* x = X + blockIdx.z * stride + i * ld;
    const int e = i < n ? exps[blockIdx.z * estride + i] : 0;
    uint32_t out[S][4];
    int d0[S], d1[S];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int64_t k = k0 + 2 * q;
        digits(i < n && k < n ? fixed_point(x[k], e) : 0, d0);
        digits(i < n && k + 1 < n ? fixed_point(x[k + 1], e) : 0, d1);
#pragma unroll
        for (int s = 0; s < S; ++s) out[s][q] = pack(d0[s], d1[s]);
    }
    __nv_bfloat16* p = planes + blockIdx.z * pstride + i * kp + k0;
#pragma unroll
    for (int s = 0; s < S; ++s)
        *reinterpret_cast<uint4*>(p + s * rows * kp) = make_uint4(out[s][0], out[s][1], out[s][2], out[s][3]);
}

// Planes of the rows of X (n x n): as slice_columns_kernel on the transpose, through a 32 x 64
// shared tile.
static __global__ void __launch_bounds__(256)
slice_rows_kernel(const double* __restrict__ X, int64_t ld, int64_t n, int64_t stride, const int* __restrict__ exps,
                  int64_t estride, int64_t rows, int64_t kp, __nv_bfloat16* __restrict__ planes, int64_t pstride,
                  const int* __restrict__ flag)
{
    if (flag[blockIdx.z]) return;
    __shared__ double tile[64][33];   // [inner][row]
    const int64_t i0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * 64;
    const double* x = X + blockIdx.z * stride;
    for (int t = threadIdx.x; t < 64 * 32; t += blockDim.x) {
        const int r = t & 31, c = t >> 5;
        tile[c][r] = i0 + r < n && k0 + c < n ? x[i0 + r + (k0 + c) * ld] : 0.0;
    }
    __syncthreads();
    const int r = threadIdx.x >> 3, c = (threadIdx.x & 7) * 8;
    const int64_t i = i0 + r;
    if (i >= rows || k0 + c >= kp) return;
    const int e = i < n ? exps[blockIdx.z * estride + i] : 0;
    uint32_t out[S][4];
    int d0[S], d1[S];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        digits(i < n ? fixed_point(tile[c + 2 * q][r], e) : 0, d0);
        digits(i < n ? fixed_point(tile[c + 2 * q + 1][r], e) : 0, d1);
#pragma unroll
        for (int s = 0; s < S; ++s) out[s][q] = pack(d0[s], d1[s]);
    }
    __nv_bfloat16* p = planes + blockIdx.z * pstride + i * kp + k0 + c;
#pragma unroll
    for (int s = 0; s < S; ++s)
        *reinterpret_cast<uint4*>(p + s * rows * kp) = make_uint4(out[s][0], out[s][1], out[s][2], out[s][3]);
}

// ---- the product ---------------------------------------------------------------------------

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Byte offset of the 16-byte piece c (0 .. 7) of row r in an operand tile: pieces rotated so that
// the eight rows of an ldmatrix phase fall on different banks.
__device__ __forceinline__ uint32_t piece(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// The schedule of plane products: levels S-1 .. 0, chunks of the inner dimension, pairs (s, l - s),
// steps of BK.
struct Schedule {
    int l, s, ks, chunk0, chunk1, ksteps;
    __device__ __forceinline__ int chunk_steps() const { return 2048 / BK / (l + 1); }
    __device__ __forceinline__ void begin(int steps)
    {
        ksteps = steps;
        l = S - 1;
        s = 0;
        chunk0 = ks = 0;
        chunk1 = min(chunk_steps(), ksteps);
    }
    __device__ __forceinline__ bool done() const { return l < 0; }
    // the next step; true when it begins a new (level, chunk)
    __device__ __forceinline__ bool next()
    {
        if (++ks < chunk1) return false;
        ks = chunk0;
        if (++s <= l) return false;
        s = 0;
        chunk0 = ks = chunk1;
        if (chunk0 >= ksteps) {
            chunk0 = ks = 0;
            --l;
            if (l < 0) return true;
        }
        chunk1 = min(chunk0 + chunk_steps(), ksteps);
        return true;
    }
};

// One 128 x 128 tile of sum_{s+t<S} 2^(-12-7(s+t)) A_s B_t^T (planes as slice_*_kernel lays them out).
// acc[x][y][h]: this thread's elements, row 64 (warp >> 2) + 16 x + (lane >> 2) + 8 (h >> 1), column
// 32 (warp & 3) + 8 y + 2 (lane & 3) + (h & 1) of the tile.
__device__ __forceinline__ void tile_product(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B,
                                             int64_t rows, int64_t kp, int64_t i0, int64_t j0, unsigned char* smem,
                                             double (&out)[4][4][4])
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = (warp >> 2) * 64, wn = (warp & 3) * 32;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    double* park = reinterpret_cast<double*>(smem + kRing) + tid;
    float part[4][4][4];
    long long acc[4][4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                acc[x][y][h] = 0;
                part[x][y][h] = 0.0f;
            }
    const int ksteps = (int)(kp / BK);
    // this thread's pieces of a tile: rows tid / 8 + 32 q
    const int lr = tid >> 3, lc = tid & 7;
    const uint32_t dst = piece(lr, lc);   // 32 rows further is 4096 bytes further
    const __nv_bfloat16* a0 = A + (i0 + lr) * kp + lc * 8;
    const __nv_bfloat16* b0 = B + (j0 + lr) * kp + lc * 8;
    auto load = [&](const Schedule& q, int stage) {
        const uint32_t sa = sbase + stage * 2 * kTileBytes + dst, sb = sa + kTileBytes;
        const int64_t ko = (int64_t)q.ks * BK;
        const __nv_bfloat16* a = a0 + q.s * rows * kp + ko;
        const __nv_bfloat16* b = b0 + (q.l - q.s) * rows * kp + ko;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            cp_async16(sa + 4096 * t, a + 32 * t * kp);
            cp_async16(sb + 4096 * t, b + 32 * t * kp);
        }
    };
    Schedule cur, pre;
    cur.begin(ksteps);
    pre.begin(ksteps);
#pragma unroll
    for (int st = 0; st < STAGES - 1; ++st) {
        if (!pre.done()) {
            load(pre, st);
            pre.next();
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0;
    while (!cur.done()) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        {
            const int ls = (stage + STAGES - 1) % STAGES;
            if (!pre.done()) {
                load(pre, ls);
                pre.next();
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const uint32_t sa = sbase + stage * 2 * kTileBytes, sb = sa + kTileBytes;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
            uint32_t bf[2][4];
#pragma unroll
            for (int y = 0; y < 2; ++y)   // columns 16 y .. 16 y + 15: matrices (n 0-7, k 0-7), (n 0-7, k 8-15), (n 8-15, ..)
                ldmatrix4(bf[y], sb + piece(wn + 16 * y + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)));
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                uint32_t af[4];
                ldmatrix4(af, sa + piece(wm + 16 * x + (lane & 15), 2 * kk + (lane >> 4)));
#pragma unroll
                for (int y = 0; y < 4; ++y) mma(part[x][y], af, bf[y >> 1][2 * (y & 1)], bf[y >> 1][2 * (y & 1) + 1]);
            }
        }
        const int l = cur.l;
        if (cur.next()) {
            // the level's chunk is complete: into the integers
            const int w = 1 << 7 * (l >= kSmallLevels ? S - 1 - l : kSmallLevels - 1 - l);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y)
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        acc[x][y][h] += (long long)__float2int_rn(part[x][y][h]) * w;
                        part[x][y][h] = 0.0f;
                    }
            if (l == kSmallLevels && cur.l < l) {
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y)
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            park[(16 * x + 4 * y + h) * kThreads] = __ll2double_rn(acc[x][y][h]);
                            acc[x][y][h] = 0;
                        }
            }
        }
        stage = (stage + 1) % STAGES;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // the ring is free for the caller
    constexpr double kSmall = 1.0 / (1ull << (12 + 7 * (S - 1) - 28)) / (1ull << 28);
    constexpr double kLarge = 1.0 / (1ull << (12 + 7 * (kSmallLevels - 1)));
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 4; ++h)
                out[x][y][h] = fma(__ll2double_rn(acc[x][y][h]), kLarge, park[(16 * x + 4 * y + h) * kThreads] * kSmall);
}

__device__ __forceinline__ int tile_row(int x, int h)
{
    return ((int)threadIdx.x >> 7) * 64 + 16 * x + (((int)threadIdx.x & 31) >> 2) + 8 * (h >> 1);
}
__device__ __forceinline__ int tile_col(int y, int h)
{
    return (((int)threadIdx.x >> 5) & 3) * 32 + 8 * y + 2 * ((int)threadIdx.x & 3) + (h & 1);
}

}  // namespace sliced
}  // namespace symeig
