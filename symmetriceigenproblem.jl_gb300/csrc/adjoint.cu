// adjoint.cu -- reverse-mode derivative of the tridiagonal eigensolve.
//
// For T = Q diag(lam) Q^T (columns of Q the eigenvectors of the symmetric tridiagonal with
// diagonal d and off-diagonal e), a loss L(lam, Q) with gradients glam = dL/dlam and
// gQ = dL/dQ has
//     Abar = Q M Q^T,   M = diag(glam) + F o (Q^T gQ),   F_ij = 1 / (lam_j - lam_i)  (i != j),
//     dL/dd_i = Abar_ii,   dL/de_i = Abar_{i,i+1} + Abar_{i+1,i}.
// (F_ii = 0, and F_ij = 0 where lam_i == lam_j: the formula assumes separated eigenvalues.)
// The reference has no derivative; this is the pullback behind the Julia rrule and the torch
// autograd Function of the host bindings.  Q is the solver's output, so no rotation history
// is stored.
//
// Two FP64 GEMMs with fused epilogues, on the bf16 tensor cores by exact slices (sliced_gemm.cuh)
// from n = kSlicedMin on, else (and where Q is localized, the slices would lose accuracy or an operand
// holds an infinity or NaN, which the device decides) on the FP64 MMA
// (dmma_tile.cuh: mma.sync m8n8k4 .f64; tcgen05 has no f64 kind):
//   1. G = Q^T gQ, epilogue M_ij = i == j ? glam_i : G_ij / (lam_j - lam_i), M stored.
//   2. P = Q M, epilogue: per row i the partial sums over the CTA's columns k of
//        P_ik Q_ik (-> dd_i),  P_ik Q_{i+1,k} and P_ik Q_{i-1,k} (-> de_i, de_{i-1}),
//      written per column tile; Abar itself is never stored.
//   3. a reduction over column tiles in a fixed order (deterministic).
// A batch of matrices of one order runs with blockIdx.z = matrix.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "symeig.h"
#include "symeig_common.cuh"
#include "dmma_tile.cuh"
#include "sliced_gemm.cuh"

namespace symeig {
namespace {

using dmma::BM;
using dmma::BN;
constexpr int kAdjThreads = dmma::kThreads;

// 1. M = diag(glam) + F o (Q^T gQ), M column-major with leading dimension n.
__global__ void __launch_bounds__(kAdjThreads)
adjoint_m_kernel(const double* __restrict__ Q, int64_t ldq, const double* __restrict__ gQ,
                 int64_t ldg, const double* __restrict__ lam, const double* __restrict__ glam,
                 int64_t n, double* __restrict__ Mout, int64_t strideQ, int64_t strideG,
                 int64_t strideM, const int* __restrict__ only_if)
{
    if (only_if && !only_if[blockIdx.z]) return;   // the sliced kernel did it
    __shared__ dmma::Smem sm;
    const int64_t z = blockIdx.z;
    Q += z * strideQ;
    gQ += z * strideG;
    Mout += z * strideM;
    lam += z * n;
    glam += z * n;
    const int64_t i0 = (int64_t)blockIdx.y * BM, j0 = (int64_t)blockIdx.x * BN;
    double acc[4][4][2];
    // A(i, k) = Q(k, i): k contiguous; B(k, j) = gQ(k, j): k contiguous
    dmma::tile_gemm(Q, ldq, 1, gQ, 1, ldg, n, n, n, i0, j0, 0, n, acc, sm);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int grp = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t i = i0 + wm + x * 8 + grp;
                const int64_t j = j0 + wn + y * 8 + tig * 2 + h;
                if (i >= n || j >= n) continue;
                double v;
                if (i == j) {
                    v = glam[i];
                } else {
                    const double gap = lam[j] - lam[i];
                    v = gap != 0.0 ? acc[x][y][h] / gap : 0.0;
                }
                Mout[i + j * n] = v;
            }
}

// 2. P = Q M and the per-row partial sums of the CTA's columns (see the file comment).
// part: [3][n_col_tiles][n]: 0 = P_ik Q_ik, 1 = P_ik Q_{i+1,k}, 2 = P_ik Q_{i-1,k}.
__global__ void __launch_bounds__(kAdjThreads)
adjoint_p_kernel(const double* __restrict__ Q, int64_t ldq, const double* __restrict__ M,
                 int64_t n, double* __restrict__ part, int64_t strideQ, int64_t strideM,
                 int64_t stridePart, const int* __restrict__ only_if)
{
    if (only_if && !only_if[blockIdx.z]) return;
    __shared__ dmma::Smem sm;
    __shared__ double red[3][2][BM];
    const int64_t z = blockIdx.z;
    Q += z * strideQ;
    M += z * strideM;
    part += z * stridePart;
    const int64_t i0 = (int64_t)blockIdx.y * BM, k0 = (int64_t)blockIdx.x * BN;
    double acc[4][4][2];
    // A(i, j) = Q(i, j): i contiguous; B(j, k) = M(j, k): j contiguous
    dmma::tile_gemm(Q, 1, ldq, M, 1, n, n, n, n, i0, k0, 0, n, acc, sm);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int grp = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const int r = wm + x * 8 + grp;
        const int64_t i = i0 + r;
        double sd = 0.0, su = 0.0, sl = 0.0;
        if (i < n) {
#pragma unroll
            for (int y = 0; y < 4; ++y)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int64_t k = k0 + wn + y * 8 + tig * 2 + h;
                    if (k >= n) continue;
                    const double p = acc[x][y][h];
                    sd = fma(p, Q[i + k * ldq], sd);
                    if (i + 1 < n) su = fma(p, Q[i + 1 + k * ldq], su);
                    if (i >= 1) sl = fma(p, Q[i - 1 + k * ldq], sl);
                }
        }
        // the 4 lanes of a group hold the same row: sum them
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            sd += __shfl_xor_sync(0xffffffffu, sd, o);
            su += __shfl_xor_sync(0xffffffffu, su, o);
            sl += __shfl_xor_sync(0xffffffffu, sl, o);
        }
        if (tig == 0) {
            red[0][warp & 1][r] = sd;
            red[1][warp & 1][r] = su;
            red[2][warp & 1][r] = sl;
        }
    }
    __syncthreads();
    const int64_t tiles = (n + BN - 1) / BN;
    for (int r = threadIdx.x; r < BM; r += blockDim.x) {
        const int64_t i = i0 + r;
        if (i >= n) continue;
#pragma unroll
        for (int t = 0; t < 3; ++t)
            part[((int64_t)t * tiles + blockIdx.x) * n + i] = red[t][0][r] + red[t][1][r];
    }
}

// 3. dd_i = sum_tiles part0[i];  de_i = sum_tiles (part1[i] + part2[i+1]).
// part holds the FP64 MMA's column tiles, or with `fallback` given and clear the sliced kernel's (counted).
__global__ void adjoint_reduce_kernel(const double* __restrict__ part, int64_t n, double* __restrict__ gd,
                                      double* __restrict__ ge, int64_t stridePart, const int* __restrict__ fallback,
                                      int* __restrict__ sliced_count)
{
    const int64_t z = blockIdx.y;
    if (fallback && blockIdx.x == 0 && threadIdx.x == 0 && !fallback[z]) atomicAdd(sliced_count, 1);
    part += z * stridePart;
    gd += z * n;
    ge += z * (n > 1 ? n - 1 : 0);
    const int64_t tiles = fallback && !fallback[blockIdx.y] ? (n + sliced::BN - 1) / sliced::BN : (n + BN - 1) / BN;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double sd = 0.0, se = 0.0;
        for (int64_t t = 0; t < tiles; ++t) {
            sd += part[(0 * tiles + t) * n + i];
            if (i + 1 < n) se += part[(1 * tiles + t) * n + i] + part[(2 * tiles + t) * n + i + 1];
        }
        gd[i] = sd;
        if (i + 1 < n) ge[i] = se;
    }
}

// ---- the same on the bf16 tensor cores (sliced_gemm.cuh) -------------------------------------

// Before 1.: whether the slices keep FP64's accuracy in every entry of Q^T gQ (sliced_gemm.cuh; a column
// of zeros is exact, and M's diagonal takes none).  `need`: the least L.
__global__ void __launch_bounds__(sliced::kThreads, 1)
sliced_m_check_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, const int* ea,
                      const int* eb, int64_t n, int64_t rows, int64_t kp, int64_t pstride, float need,
                      int* __restrict__ fallback, sliced::Report report)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int64_t z = blockIdx.z;
    wait_previous_launch();
    const bool skip = fallback[z] != 0;
    if (__syncthreads_or(skip)) return;
    const int64_t i0 = (int64_t)blockIdx.y * sliced::BM, j0 = (int64_t)blockIdx.x * sliced::BN;
    float L[64];
    bool poor = false;
    if (!sliced::tile_product<true>(A + z * pstride, B + z * pstride, rows, kp, i0, j0, smem, nullptr, L, report.stall)) {
        if (threadIdx.x == 0) report.timeout(fallback[z]);
        return;
    }
    const int64_t i = i0 + sliced::tile_row();
    if (threadIdx.x < sliced::kEpiThreads && i < n && ea[z * n + i] != sliced::kZeroScale) {
#pragma unroll
        for (int q = 0; q < 64; ++q) {
            const int64_t j = j0 + sliced::tile_col() + q;
            if (j < n && j != i && L[q] < need && eb[z * n + j] != sliced::kZeroScale) poor = true;
        }
    }
    if (__syncthreads_or(poor) && threadIdx.x == 0) fallback[z] = 1;
}

// Before 2.: whether they keep it in the gradient's entries.  dd_i = sum_k Q_ik P_ik has from P = Q M the errors
//   FP64    2^-53 sum_k |Q_ik| sum_j |Q_ij| |M_jk| >= 2^(-65 + ea_i) sum_k |Q_ik| 2^eb_k L_ik,
//   slices  sqrt(n) 2^-63 2^ea_i sum_k |Q_ik| 2^eb_k
// (as scales, and n for both as bounds), so  sum_k |Q_ik| 2^eb_k (L_ik - need) >= 0  is asked of every row, and the
// same with the weights |Q_{i+1,k}| and |Q_{i-1,k}| for de_i and de_{i-1}.  A CTA leaves its columns'
// part of the three sums in `margin`; the last one of a row of tiles adds them up.  The terms are in FP32
// about the tile's largest column, on the safe side: a weight below 2^-60 of its row's largest counts as
// 2^-60 against and as 0 for the slices, and a column below 2^-60 of the tile's largest fails.
__global__ void __launch_bounds__(sliced::kThreads, 1)
sliced_p_check_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, const int* ea,
                      const int* eb, const double* __restrict__ Q, int64_t n, int64_t rows, int64_t kp,
                      int64_t pstride, float need, double* __restrict__ margin, int64_t stride_margin,
                      int* __restrict__ done, int* __restrict__ fallback, sliced::Report report)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ float red[3][2][sliced::BM], scale[sliced::BN];
    __shared__ int top, last;
    const int64_t z = blockIdx.z;
    wait_previous_launch();
    const bool skip = fallback[z] != 0;
    if (__syncthreads_or(skip)) return;
    Q += z * n * n;
    margin += z * stride_margin;
    ea += z * n;
    eb += z * n;
    const int64_t i0 = (int64_t)blockIdx.y * sliced::BM, k0 = (int64_t)blockIdx.x * sliced::BN;
    if (threadIdx.x == 0) top = sliced::kZeroScale;
    __syncthreads();
    int e = sliced::kZeroScale;
    if (threadIdx.x < sliced::BN && k0 + threadIdx.x < n) e = eb[k0 + threadIdx.x];
    if (threadIdx.x < sliced::BN) atomicMax(&top, e);
    __syncthreads();
    bool poor = e != sliced::kZeroScale && e < top - 60;
    if (threadIdx.x < sliced::BN) scale[threadIdx.x] = e == sliced::kZeroScale || poor ? 0.0f : exp2f((float)(e - top));
    float L[64];
    if (!sliced::tile_product<true>(A + z * pstride, B + z * pstride, rows, kp, i0, k0, smem, nullptr, L, report.stall)) {
        if (threadIdx.x == 0) report.timeout(fallback[z]);
        return;
    }
    if (__syncthreads_or(poor)) {
        if (threadIdx.x == 0) fallback[z] = 1;
        return;
    }
    const int r = sliced::tile_row();
    const int64_t i = i0 + r;
    if (threadIdx.x < sliced::kEpiThreads) {
        // the neighbouring rows' weights are the neighbouring lanes'; past a warp's ends lanes 0 and 31 read them
        const int lane = threadIdx.x & 31;
        const int64_t edge = lane == 0 ? i - 1 : i + 1;
        const bool ok = i < n, edge_ok = (lane == 0 || lane == 31) && edge >= 0 && edge < n;
        const int e_row = ok ? ea[i] : 0, e_edge = edge_ok ? ea[edge] : 0;
        // L through shared memory (the operand tiles are done with) and a loop: unrolled, the code that each
        // CTA runs once cost its fetches, 44 us at n = 300
        float* Ls = reinterpret_cast<float*>(smem) + sliced::tile_col() * sliced::BM + r;
#pragma unroll
        for (int q = 0; q < 64; ++q) Ls[q * sliced::BM] = L[q];
        const double* x = Q + i + (k0 + sliced::tile_col()) * n;
        const int64_t to_edge = edge - i;
        const int cols = (int)max((int64_t)0, min((int64_t)64, n - k0 - sliced::tile_col()));
        float m0 = 0.0f, mu = 0.0f, ml = 0.0f;
#pragma unroll 8
        for (int q = 0; q < cols; ++q) {
            const float v = (Ls[q * sliced::BM] - need) * scale[sliced::tile_col() + q];
            const float w = sliced::weight(ok ? x[q * n] : 0.0, e_row), we = sliced::weight(edge_ok ? x[q * n + to_edge] : 0.0, e_edge);
            const float wu = __shfl_down_sync(0xffffffffu, w, 1), wl = __shfl_up_sync(0xffffffffu, w, 1);
            m0 += sliced::weighted(w, v);
            mu += sliced::weighted(lane == 31 ? we : wu, v);
            ml += sliced::weighted(lane == 0 ? we : wl, v);
        }
        const int half = threadIdx.x >> 7;
        red[0][half][r] = m0;
        red[1][half][r] = mu;
        red[2][half][r] = ml;
    }
    __syncthreads();
    const int64_t tiles = gridDim.x;
    if (threadIdx.x < sliced::BM && i < n)
#pragma unroll
        for (int t = 0; t < 3; ++t)
            margin[((int64_t)t * tiles + blockIdx.x) * n + i] = scalbn((double)red[t][0][r] + (double)red[t][1][r], top);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&done[z * gridDim.y + blockIdx.y], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < sliced::BM && i < n)
        for (int t = 0; t < 3; ++t) {
            double m = 0.0;
            for (int64_t b = 0; b < tiles; ++b) m += __ldcg(&margin[((int64_t)t * tiles + b) * n + i]);
            poor |= !(m >= 0.0);
        }
    if (__syncthreads_or(poor) && threadIdx.x == 0) fallback[z] = 1;
}

// 1. as adjoint_m_kernel.  A: planes of Q's columns with exponents ea; B: of gQ's columns with eb.
__global__ void __launch_bounds__(sliced::kThreads, 1)
sliced_m_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, const int* ea,
                const int* eb, const double* __restrict__ lam, const double* __restrict__ glam, int64_t n,
                int64_t rows, int64_t kp, int64_t pstride, double* __restrict__ Mout, double* __restrict__ park,
                int* __restrict__ fallback, sliced::Report report)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int64_t z = blockIdx.z;
    wait_previous_launch();
    const bool skip = fallback[z] != 0;
    if (__syncthreads_or(skip)) return;
    lam += z * n;
    glam += z * n;
    Mout += z * n * n;
    park += ((z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * sliced::BM * sliced::BN;
    const int64_t i0 = (int64_t)blockIdx.y * sliced::BM, j0 = (int64_t)blockIdx.x * sliced::BN;
    double acc[64];
    if (!sliced::tile_product<false>(A + z * pstride, B + z * pstride, rows, kp, i0, j0, smem, park, acc, report.stall)) {
        if (threadIdx.x == 0) report.timeout(fallback[z]);
        return;
    }
    const int64_t i = i0 + sliced::tile_row();
    if (threadIdx.x >= sliced::kEpiThreads || i >= n) return;
    const int e = ea[z * n + i];
    const double li = lam[i];
#pragma unroll
    for (int q = 0; q < 64; ++q) {
        const int64_t j = j0 + sliced::tile_col() + q;
        if (j >= n) continue;
        double v;
        if (i == j) {
            v = glam[i];
        } else {
            const double gap = lam[j] - li;
            v = gap != 0.0 ? scalbn(acc[q], e + eb[z * n + j]) / gap : 0.0;
        }
        Mout[i + j * n] = v;
    }
}

// 2. as adjoint_p_kernel.  A: planes of Q's rows with exponents ea; B: of M's columns with eb.
__global__ void __launch_bounds__(sliced::kThreads, 1)
sliced_p_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, const int* ea,
                const int* eb, const double* __restrict__ Q, int64_t n, int64_t rows, int64_t kp,
                int64_t pstride, double* __restrict__ part, int64_t stridePart, double* __restrict__ park,
                int* __restrict__ fallback, sliced::Report report)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ double red[3][2][sliced::BM];
    const int64_t z = blockIdx.z;
    wait_previous_launch();
    const bool skip = fallback[z] != 0;
    if (__syncthreads_or(skip)) return;
    Q += z * n * n;
    part += z * stridePart;
    park += ((z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * sliced::BM * sliced::BN;
    const int64_t i0 = (int64_t)blockIdx.y * sliced::BM, k0 = (int64_t)blockIdx.x * sliced::BN;
    double acc[64];
    if (!sliced::tile_product<false>(A + z * pstride, B + z * pstride, rows, kp, i0, k0, smem, park, acc, report.stall)) {
        if (threadIdx.x == 0) report.timeout(fallback[z]);
        return;
    }
    const int r = sliced::tile_row();
    if (threadIdx.x < sliced::kEpiThreads) {
        const int64_t i = i0 + r;
        double sd = 0.0, su = 0.0, sl = 0.0;
        if (i < n) {
            const int e = ea[z * n + i];
            // eight columns at a time: shorter sums round less
#pragma unroll
            for (int q0 = 0; q0 < 64; q0 += 8) {
                double td = 0.0, tu = 0.0, tl = 0.0;
#pragma unroll
                for (int q = q0; q < q0 + 8; ++q) {
                    const int64_t k = k0 + sliced::tile_col() + q;
                    if (k >= n) continue;
                    const double p = scalbn(acc[q], e + eb[z * n + k]);
                    td = fma(p, Q[i + k * n], td);
                    if (i + 1 < n) tu = fma(p, Q[i + 1 + k * n], tu);
                    if (i >= 1) tl = fma(p, Q[i - 1 + k * n], tl);
                }
                sd += td;
                su += tu;
                sl += tl;
            }
        }
        const int half = threadIdx.x >> 7;
        red[0][half][r] = sd;
        red[1][half][r] = su;
        red[2][half][r] = sl;
    }
    __syncthreads();
    const int64_t tiles = (n + sliced::BN - 1) / sliced::BN;
    if (threadIdx.x < sliced::BM && i0 + r < n)
#pragma unroll
        for (int t = 0; t < 3; ++t)
            part[((int64_t)t * tiles + blockIdx.x) * n + i0 + r] = red[t][0][r] + red[t][1][r];
}

// Eigenvalue-only loss (gQ = 0): dd_i = sum_k glam_k Q_ik^2, de_i = 2 sum_k glam_k Q_ik Q_{i+1,k}.
__global__ void adjoint_lambda_only_kernel(const double* __restrict__ Q, int64_t ldq,
                                           const double* __restrict__ glam, int64_t n,
                                           double* __restrict__ gd, double* __restrict__ ge,
                                           int64_t strideQ)
{
    const int64_t z = blockIdx.y;
    Q += z * strideQ;
    glam += z * n;
    gd += z * n;
    ge += z * (n > 1 ? n - 1 : 0);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double sd = 0.0, se = 0.0;
        for (int64_t k = 0; k < n; ++k) {
            const double q = Q[i + k * ldq];
            sd = fma(glam[k] * q, q, sd);
            if (i + 1 < n) se = fma(glam[k] * q, Q[i + 1 + k * ldq], se);
        }
        gd[i] = sd;
        if (i + 1 < n) ge[i] = 2.0 * se;
    }
}

}  // namespace

// From this order on the products run on the bf16 tensor cores where Q is spread out.  FP64 MMA against
// sliced, one matrix: n = 256 694 / 344 us, 300 810 / 363, 512 1304 / 427, 1000 4693 / 641, 2047 32.8 / 1.89 ms;
// 25 of n = 300 3612 / 757 us, 256 of n = 512 127.5 / 14.0 ms.  A localized Q pays for the question and the kernels that
// return at once: about 25 us, of 700 at n = 256 and 4690 at 1000, 0.3 ms of 127.5 for 256 of n = 512; below
// n = 256 it would be above 4 %.  The rule leaves the count out, so that a matrix has the same bits
// alone and in a batch.
static constexpr int64_t kSlicedMin = 256;
// Matrices sliced at once: their planes take at most this many bytes (one matrix always fits).
static constexpr int64_t kSlicedBytes = (int64_t)512 << 20;

// The planes of larger orders would take 160 GB and more.
static constexpr int64_t kSlicedMax = 65408;

bool adjoint_sliced(int64_t n) { return n >= kSlicedMin && n <= kSlicedMax; }

// (and 32767 at most: slice_columns_kernel's blockIdx.y counts two operands)
static int64_t sliced_group(int64_t count, int64_t n)
{
    const int64_t per = 2 * 2 * sliced::plane_values(n, n);
    return std::max<int64_t>(1, std::min(std::min<int64_t>(count, 32767), kSlicedBytes / per));
}

// The slices' own scratch: of a group two operands' planes and the tiles' small sums; of all matrices the
// operands' exponents, a flag and a counter a row of tiles.
size_t adjoint_planes_bytes(int64_t count, int64_t n)
{
    const int64_t g = sliced_group(count, n), r = sliced::pad_rows(n);
    return (size_t)(g * (2 * sliced::plane_values(n, n) * 2 + r * r * (int64_t)sizeof(double)) +
                    count * (2 * n + 1 + r / sliced::BM) * (int64_t)sizeof(int) + 512);
}

// Device-pointer adjoint for `count` matrices of order n stored back to back (Q, gQ with
// leading dimension n and stride n*n; lam, glam, gd with stride n; ge with stride n-1).
// scratch: adjoint_scratch_doubles(count, n) doubles.  planes: adjoint_planes_bytes(count, n) bytes, only where
// adjoint_sliced(n), or null for the FP64 MMA.
// err[0]: the handle's error word; err[1] counts the matrices that took the slices.
int adjoint_dev(cudaStream_t s, int64_t count, int64_t n, const double* lam, const double* Q,
                const double* glam, const double* gQ, double* gd, double* ge, double* scratch,
                void* planes, int* err, int32_t stall)
{
    if (count <= 0 || n <= 0) return SYMEIG_OK;
    const int64_t tiles = (n + BN - 1) / BN;
    const int64_t strideQ = n * n, strideM = n * n, stridePart = 3 * tiles * n;
    if (count > 65535) return SYMEIG_ERR_SIZE;
    if (!gQ) {
        adjoint_lambda_only_kernel<<<dim3((unsigned)((n + 127) / 128), (unsigned)count), 128, 0, s>>>(
            Q, n, glam, n, gd, ge, strideQ);
        return cudaGetLastError() == cudaSuccess ? SYMEIG_OK : SYMEIG_ERR_CUDA;
    }
    double* Mbuf = scratch;
    double* part = scratch + count * strideM;
    const dim3 grid((unsigned)tiles, (unsigned)((n + BM - 1) / BM), (unsigned)count);
    if (!planes) {
        adjoint_m_kernel<<<grid, kAdjThreads, 0, s>>>(Q, n, gQ, n, lam, glam, n, Mbuf, strideQ, strideQ, strideM, nullptr);
        adjoint_p_kernel<<<grid, kAdjThreads, 0, s>>>(Q, n, Mbuf, n, part, strideQ, strideM, stridePart, nullptr);
        adjoint_reduce_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)count), 256, 0, s>>>(part, n, gd, ge, stridePart, nullptr, nullptr);
        return cudaGetLastError() == cudaSuccess ? SYMEIG_OK : SYMEIG_ERR_CUDA;
    }
    for (const void* k : {(const void*)sliced_m_kernel, (const void*)sliced_p_kernel, (const void*)sliced_m_check_kernel,
                          (const void*)sliced_p_check_kernel})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sliced::kSmem) != cudaSuccess)
            return SYMEIG_ERR_CUDA;
    const sliced::Report report{err, stall > 0 ? (uint32_t)stall : 0xffffffffu};
    const int64_t group = sliced_group(count, n), rows = sliced::pad_rows(n), kp = sliced::pad_k(n);
    const int64_t pstride = sliced::plane_values(n, n);
    // 256-byte aligned: the planes' 16-byte pieces
    unsigned char* base = (unsigned char*)(((uintptr_t)planes + 255) & ~(uintptr_t)255);
    __nv_bfloat16* PA = (__nv_bfloat16*)base;
    __nv_bfloat16* PB = PA + group * pstride;
    double* park = (double*)(PB + group * pstride);
    int* ea = (int*)(park + group * rows * rows);   // from here on of all matrices
    int* eb = ea + count * n;
    int* flag = eb + count * n;
    int* done = flag + count;
    const int64_t ntiles = (n + sliced::BN - 1) / sliced::BN;
    const float need = (float)(sliced::kLeadFactor * std::sqrt((double)n));
    const unsigned all = (unsigned)count;
    const unsigned cblocks = (unsigned)((rows * (kp / 8) + 255) / 256);
    const unsigned eblocks = (unsigned)((n + sliced::kExpWarps - 1) / sliced::kExpWarps);
    // The FP64 MMA takes the matrices that fall back in one launch each, whatever the groups: by groups the last waves of
    // their tiles cost 3 % of 256 matrices of n = 512.  In a chain (launch_after) the launches that return at
    // once overlap.
    if (cudaMemsetAsync(flag, 0, count * (1 + ntiles) * sizeof(int), s) != cudaSuccess) return SYMEIG_ERR_CUDA;
    sliced::column_exponents_kernel<<<dim3(eblocks, all, 2), 32 * sliced::kExpWarps, 0, s>>>(sliced::Operand{Q, ea, PA, true},
                                                                            sliced::Operand{gQ, eb, PB, false}, n, flag);
    for (int64_t z = 0; z < count; z += group) {
        const unsigned g = (unsigned)std::min<int64_t>(group, count - z);
        const dim3 sgrid((unsigned)ntiles, (unsigned)ntiles, g);
        launch_after(sliced::slice_columns_kernel, dim3(cblocks, 2 * g), 256, 0, s,
                     sliced::Operand{Q + z * strideQ, ea + z * n, PA, true}, sliced::Operand{gQ + z * strideQ, eb + z * n, PB, false},
                     (int)g, n, rows, kp, pstride, flag + z);
        launch_after(sliced_m_check_kernel, sgrid, sliced::kThreads, sliced::kSmem, s, PA, PB, ea + z * n, eb + z * n, n, rows, kp,
                     pstride, need, flag + z, report);
        launch_after(sliced_m_kernel, sgrid, sliced::kThreads, sliced::kSmem, s, PA, PB, ea + z * n, eb + z * n, lam + z * n,
                     glam + z * n, n, rows, kp, pstride, Mbuf + z * strideM, park, flag + z, report);
    }
    adjoint_m_kernel<<<grid, kAdjThreads, 0, s>>>(Q, n, gQ, n, lam, glam, n, Mbuf, strideQ, strideQ, strideM, flag);
    launch_after(sliced::row_exponents_kernel, dim3((unsigned)((n + 31) / 32), all), 1024, 0, s, Q, n, ea, flag);
    const sliced::Operand om{Mbuf, eb, PB, false};
    launch_after(sliced::column_exponents_kernel, dim3(eblocks, all, 1), 32 * sliced::kExpWarps, 0, s, om, om, n, flag);
    for (int64_t z = 0; z < count; z += group) {
        const unsigned g = (unsigned)std::min<int64_t>(group, count - z);
        const dim3 sgrid((unsigned)ntiles, (unsigned)ntiles, g);
        const sliced::Operand oz{Mbuf + z * strideM, eb + z * n, PB, false};
        double* pz = part + z * stridePart;
        launch_after(sliced::slice_rows_kernel, dim3((unsigned)((kp + 63) / 64), (unsigned)((rows + 31) / 32), g), 256, 0, s,
                     Q + z * strideQ, n, ea + z * n, rows, kp, PA, pstride, flag + z);
        launch_after(sliced::slice_columns_kernel, dim3(cblocks, g), 256, 0, s, oz, oz, (int)g, n, rows, kp, pstride,
                     flag + z);
        // (pz: the margins, before the partial sums take their place)
        launch_after(sliced_p_check_kernel, sgrid, sliced::kThreads, sliced::kSmem, s, PA, PB, ea + z * n, eb + z * n,
                     Q + z * strideQ, n, rows, kp, pstride, need, pz, stridePart, done + z * ntiles, flag + z, report);
        launch_after(sliced_p_kernel, sgrid, sliced::kThreads, sliced::kSmem, s, PA, PB, ea + z * n, eb + z * n, Q + z * strideQ, n,
                     rows, kp, pstride, pz, stridePart, park, flag + z, report);
    }
    adjoint_p_kernel<<<grid, kAdjThreads, 0, s>>>(Q, n, Mbuf, n, part, strideQ, strideM, stridePart, flag);
    adjoint_reduce_kernel<<<dim3((unsigned)((n + 255) / 256), all), 256, 0, s>>>(part, n, gd, ge, stridePart, flag, err + 1);
    return cudaGetLastError() == cudaSuccess ? SYMEIG_OK : SYMEIG_ERR_CUDA;
}

int64_t adjoint_scratch_doubles(int64_t count, int64_t n)
{
    const int64_t tiles = (n + BN - 1) / BN;
    return count * (n * n + 3 * tiles * n);
}

}  // namespace symeig
