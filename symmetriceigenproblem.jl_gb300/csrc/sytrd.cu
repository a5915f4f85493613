// sytrd.cu -- dense symmetric -> tridiagonal reduction and its orthogonal factor: the step
// before qr_algorithm! when the input is a dense symmetric matrix.  The reference has none
// (its callers supply a SymTridiagonal); this follows LAPACK's dsytrd / dlatrd / dorgtr with
// UPLO = 'L'.
//
// A (n x n, column-major, both triangles stored) = Q T Q^T with T symmetric tridiagonal
// (d, e) and Q = H_0 H_1 ... H_{n-2},  H_j = I - tau_j v_j v_j^T,  v_j = (0, .., 0, 1, x_j)
// with the 1 in row j+1.  Panels of NB = 64 columns:
//   for each column j of a panel (i = j - p earlier reflectors of the panel):
//     a(j:n, j) -= V W(j, 0:i)^T + W V(j, 0:i)^T            (the panel's updates, lazily)
//     reflector of a(j+1:n, j):  beta = -sign(alpha) ||(alpha, x)||,  tau = (beta - alpha)/beta,
//       x /= alpha - beta   (dlarfg; x == 0 gives tau = 0, H = I)
//     w = tau (A22 v - W (V^T v) - V (W^T v));   w -= (tau/2) (w^T v) v
//   after the panel:  A(q:n, q:n) -= V W^T + W V^T     (q = p + pb; both triangles)
// A column is three launches, one per global reduction it needs (the reflector's norm; A22 v with
// V^T v and W^T v; w^T v): each block redoes the small reductions of the launch before it, so
// nothing but these three orders waits on the whole grid, and each sum is split over enough
// threads that no thread chains more than about 16 FP64 operations of 64 cycles.  At the sizes
// that fit L2 the reduction is bound by these latencies, not by the FP64 pipe: n = 1300 takes
// 27.0 ms (with programmatic dependent launches, which hide 6 us a column of launch latency),
// against 165 ms for six launches a column with one thread per row and a block reduction per
// earlier reflector.
// The trailing update is one FP64 tensor-core GEMM (dmma_tile.cuh) of inner dimension 2 pb.
// Every reduction sums in a fixed order, so results are deterministic.
// On exit, as in LAPACK: A's diagonal and first subdiagonal hold T, x_j lies below the
// subdiagonal of column j, tau_j in tau.
//
// orgtr forms Q by backward accumulation of the panels in compact WY form (dlarft / dlarfb):
//   Q(R, R) -= (V T) (V^T Q(R, R)),   R = rows and columns p+1 .. n-1,
// with T the pb x pb upper-triangular factor from V^T V; V^T V and V^T Q are long inner sums
// and run split over K.
//
// Range: the reflector norms are plain sums of squares, so |a_ij| must lie within 2^+-500
// (the host entry points scale A by a power of two into [2^-2, 2^2] around its largest entry).
#include <cuda_runtime.h>

#include "dmma_tile.cuh"
#include "launch_after.cuh"
#include "symeig.h"
#include "symeig_common.cuh"

namespace symeig {
namespace {

constexpr int NB = 64;    // panel width
constexpr int RB = 32;    // rows per block of the column kernels: one warp's lanes, 8 warps share the sums
constexpr int RG = 8;     // warps per such block
constexpr int SR = 128;   // rows per block of the matrix-vector product (two threads per row)

// Inner-dimension chunk of orgtr's split-K products for order n.  A 64 x 64 tile over 512 rows
// occupies one SM's FP64 pipe for 640 us; at n = 1300 that left 63 CTAs for 152 SMs (636 us a
// product, 126 us with 64).  Larger orders have tiles enough, and there the partial tiles' memory
// counts.
__host__ __device__ inline int64_t split_rows(int64_t n) { return n <= 2048 ? 64 : n <= 4096 ? 128 : n <= 8192 ? 256 : 512; }

// Columns per block of the matrix-vector product over m rows and columns: enough blocks to fill
// 152 SMs several times at small m, at most 64 partial sums per row up to m = 16384.
__host__ __device__ inline int symv_cols(int64_t m) { return m <= 2048 ? 32 : m <= 4096 ? 64 : m <= 8192 ? 128 : 256; }

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sum of a[0 .. n) by one warp, the same in every lane, in a fixed order
__device__ __forceinline__ double warp_sum_of(const double* __restrict__ a, int n)
{
    double s0 = 0.0, s1 = 0.0;
    int k = threadIdx.x & 31;
    for (; k + 32 < n; k += 64) {
        s0 += a[k];
        s1 += a[k + 32];
    }
    if (k < n) s0 += a[k];
    return warp_sum(s0 + s1);
}

// The scratch of one panel, shared by the column kernels.
struct Panel {
    double* A;
    int64_t lda, n;
    int pb;
    double *VW, *WV;     // n x 2 pb: [V W] and [W V]
    double *part;        // norm partials, one per RB rows
    double *dots;        // V^T v (NB), W^T v (NB)
    double *ypart;       // A22 v partials, one row of n per column chunk
    double *wraw;        // w before its (tau/2)(w.v) v correction
    double *wpart;       // w.v partials, one per RB rows
    double *sc;          // tau, 1/(alpha - beta), beta of the current column
};

// Finish column j-1's w (i >= 1: w += -(tau/2)(w.v) v, from wraw and wpart), then, unless
// fix_only, apply the panel's i earlier reflectors to column j:
//   a(j:n, j) -= V W(j,:)^T + W V(j,:)^T;   part[b] = sum over the block's rows >= j+2 of a^2.
// The earlier reflectors are split over the block's warps.
__global__ void __launch_bounds__(RB * RG)
column_kernel(Panel P, int64_t j, int i, int nparts, int fix_only)
{
    __shared__ double vj[NB], wj[NB], acc[RG][RB], a2s;
    wait_previous_launch();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t n = P.n;
    if (i > 0) {
        if (wp == 0) {
            const double s = warp_sum_of(P.wpart, nparts);
            if (lane == 0) a2s = -0.5 * P.sc[0] * s;
        }
        for (int t = threadIdx.x; t < i; t += blockDim.x) {
            vj[t] = P.VW[j + (int64_t)t * n];
            if (t < i - 1) wj[t] = P.VW[j + (int64_t)(P.pb + t) * n];
        }
        __syncthreads();
        if (threadIdx.x == 0) wj[i - 1] = fma(a2s, vj[i - 1], P.wraw[j]);
        __syncthreads();
    }
    const int64_t r = j + (int64_t)blockIdx.x * RB + lane;
    const bool ok = r < n;
    double u = 0.0, v = 0.0;
    if (ok) {
        if (i > 0 && wp == (i - 1) % RG) {   // the warp that holds reflector i-1 completes its w
            const double vl = P.VW[r + (int64_t)(i - 1) * n];
            const double wl = fma(a2s, vl, P.wraw[r]);
            P.VW[r + (int64_t)(P.pb + i - 1) * n] = wl;
            P.WV[r + (int64_t)(i - 1) * n] = wl;
            u = vl * wj[i - 1];
            v = wl * vj[i - 1];
        }
        if (!fix_only)
#pragma unroll 4
            for (int t = wp; t < i - 1; t += RG) {
                u = fma(P.VW[r + (int64_t)t * n], wj[t], u);
                v = fma(P.VW[r + (int64_t)(P.pb + t) * n], vj[t], v);
            }
    }
    if (fix_only) return;
    acc[wp][lane] = u + v;
    __syncthreads();
    if (wp != 0) return;
    double x2 = 0.0;
    if (ok) {
        double s = 0.0;
#pragma unroll
        for (int g = 0; g < RG; ++g) s += acc[g][lane];
        const double a = P.A[r + j * P.lda] - s;
        P.A[r + j * P.lda] = a;
        if (r >= j + 2) x2 = a * a;
    }
    x2 = warp_sum(x2);
    if (lane == 0) P.part[blockIdx.x] = x2;
}

// The reflector's scalars (dlarfg) from the norm partials: tau, 1/(alpha - beta), beta.
__device__ __forceinline__ void reflector(double alpha, double s, double& tau, double& scale, double& beta)
{
    if (s == 0.0) {
        tau = 0.0;
        beta = alpha;
        scale = 0.0;
    } else {
        const double nrm = sqrt(fma(alpha, alpha, s));
        beta = alpha >= 0.0 ? -nrm : nrm;
        tau = (beta - alpha) / beta;
        scale = 1.0 / (alpha - beta);
    }
}

// Column j's reflector and the products with its v (v(j+1) = 1, v = a scale below).  Blocks with
// blockIdx.y < chunks: ypart[chunk][r] = sum over the chunk's columns c of A(r, c) v(c), rows and
// columns j+1 .. n-1.  The other blocks, one warp per earlier reflector t: dots[t] = V_t . v and
// dots[NB + t] = W_t . v.
__global__ void __launch_bounds__(2 * SR)
products_kernel(Panel P, int64_t j, int i, int nparts, int chunks, double* __restrict__ d, double* __restrict__ e,
                double* __restrict__ tau_out)
{
    __shared__ double vs[256], half[SR], scs[3];
    wait_previous_launch();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t n = P.n, m = n - j - 1;
    const double* col = P.A + j * P.lda;
    if (wp == 0) {
        const double s = warp_sum_of(P.part, nparts);
        double tau, scale, beta;
        reflector(col[j + 1], s, tau, scale, beta);
        if (lane == 0) {
            scs[0] = tau;
            scs[1] = scale;
            scs[2] = beta;
            if (blockIdx.x == 0 && blockIdx.y == 0) {
                P.sc[0] = tau;
                P.sc[1] = scale;
                P.sc[2] = beta;
                d[j] = col[j];
                e[j] = beta;
                tau_out[j] = tau;
            }
        }
    }
    __syncthreads();
    const double scale = scs[1];
    if ((int)blockIdx.y >= chunks) {
        // dot products: the blocks' warps over t = 0 .. 2 i - 1
        const int first = ((int)(blockIdx.y - chunks) * (int)gridDim.x + (int)blockIdx.x) * (2 * SR / 32) + wp;
        for (int t = first; t < 2 * i; t += (int)(gridDim.y - chunks) * (int)gridDim.x * (2 * SR / 32)) {
            const double* x = P.VW + (int64_t)(t < i ? t : P.pb + t - i) * n;
            double s0 = lane == 0 ? x[j + 1] : 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            int64_t r = j + 2 + lane;
            for (; r + 96 < n; r += 128) {
                s0 = fma(x[r], col[r] * scale, s0);
                s1 = fma(x[r + 32], col[r + 32] * scale, s1);
                s2 = fma(x[r + 64], col[r + 64] * scale, s2);
                s3 = fma(x[r + 96], col[r + 96] * scale, s3);
            }
            for (; r < n; r += 32) s0 = fma(x[r], col[r] * scale, s0);
            const double s = warp_sum((s0 + s1) + (s2 + s3));
            if (lane == 0) P.dots[t < i ? t : NB + t - i] = s;
        }
        return;
    }
    const int gch = symv_cols(m);
    const int64_t c0 = j + 1 + (int64_t)blockIdx.y * gch;
    const int len = (int)(n - c0 < gch ? n - c0 : gch);
    for (int c = threadIdx.x; c < len; c += blockDim.x) vs[c] = c0 + c == j + 1 ? 1.0 : col[c0 + c] * scale;
    __syncthreads();
    const int rl = threadIdx.x % SR, h = threadIdx.x / SR;   // row, half of the chunk's columns
    const int64_t r = j + 1 + (int64_t)blockIdx.x * SR + rl;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (r < n) {
        const double* a = P.A + r + c0 * P.lda;
        int c = h * (gch / 2);
        const int end = min(len, c + gch / 2);
#pragma unroll 4
        for (; c + 3 < end; c += 4) {
            a0 = fma(a[c * P.lda], vs[c], a0);
            a1 = fma(a[(c + 1) * P.lda], vs[c + 1], a1);
            a2 = fma(a[(c + 2) * P.lda], vs[c + 2], a2);
            a3 = fma(a[(c + 3) * P.lda], vs[c + 3], a3);
        }
        for (; c < end; ++c) a0 = fma(a[c * P.lda], vs[c], a0);
    }
    const double y = (a0 + a1) + (a2 + a3);
    if (h == 1) half[rl] = y;
    __syncthreads();
    if (h == 0 && r < n) P.ypart[(int64_t)blockIdx.y * n + r] = y + half[rl];
}

// w = tau (A22 v - W (V^T v) - V (W^T v)) into wraw, wpart[b] = (w . v) over the block's rows; v
// into VW column i, WV column pb + i and A below the subdiagonal, beta on it.
__global__ void __launch_bounds__(RB * RG)
w_kernel(Panel P, int64_t j, int i, int chunks)
{
    __shared__ double c1[NB], c2[NB], acc[RG][RB];
    wait_previous_launch();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t n = P.n;
    for (int t = threadIdx.x; t < i; t += blockDim.x) {
        c1[t] = P.dots[t];
        c2[t] = P.dots[NB + t];
    }
    __syncthreads();
    const double tau = P.sc[0], scale = P.sc[1], beta = P.sc[2];
    const int64_t r = j + 1 + (int64_t)blockIdx.x * RB + lane;
    const bool ok = r < n;
    double y = 0.0, u = 0.0, v = 0.0;
    if (ok) {
#pragma unroll 8
        for (int b = wp; b < chunks; b += RG) y += P.ypart[(int64_t)b * n + r];
#pragma unroll 4
        for (int t = wp; t < i; t += RG) {
            u = fma(P.VW[r + (int64_t)(P.pb + t) * n], c1[t], u);
            v = fma(P.VW[r + (int64_t)t * n], c2[t], v);
        }
    }
    acc[wp][lane] = y - (u + v);
    __syncthreads();
    if (wp != 0) return;
    double wv = 0.0;
    if (ok) {
        double s = 0.0;
#pragma unroll
        for (int g = 0; g < RG; ++g) s += acc[g][lane];
        const double w = tau * s;
        double* a = P.A + r + j * P.lda;
        const double vr = r == j + 1 ? 1.0 : *a * scale;
        *a = r == j + 1 ? beta : vr;
        P.VW[r + (int64_t)i * n] = vr;
        P.WV[r + (int64_t)(P.pb + i) * n] = vr;
        P.wraw[r] = w;
        wv = w * vr;
    }
    wv = warp_sum(wv);
    if (lane == 0) P.wpart[blockIdx.x] = wv;
}

// A(q:n, q:n) -= [V W] [W V]^T  (inner dimension 2 pb).  Tiles on and below the diagonal compute;
// those below also write their transpose, so both triangles stay equal (a product for each
// triangle cost twice the tensor-pipe time: 5.1 ms of the n = 1300 reduction).
__global__ void __launch_bounds__(dmma::kThreads)
trailing_update_kernel(double* __restrict__ A, int64_t lda, int64_t n, int64_t q, int pb,
                       const double* __restrict__ VW, const double* __restrict__ WV)
{
    if (blockIdx.x > blockIdx.y) return;
    __shared__ dmma::Smem sm;
    const int64_t m = n - q;
    const int64_t i0 = (int64_t)blockIdx.y * dmma::BM, j0 = (int64_t)blockIdx.x * dmma::BN;
    double acc[4][4][2];
    dmma::tile_gemm(VW + q, 1, n, WV + q, n, 1, m, m, 2 * pb, i0, j0, 0, 2 * pb, acc, sm);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t ii = i0 + dmma::tile_row(x), jj = j0 + dmma::tile_col(y, h);
                if (ii >= m || jj >= m || ii < jj) continue;
                const double v = A[(q + ii) + (q + jj) * lda] - acc[x][y][h];
                A[(q + ii) + (q + jj) * lda] = v;
                if (ii != jj) A[(q + jj) + (q + ii) * lda] = v;
            }
}

__global__ void last_diag_kernel(const double* __restrict__ A, int64_t lda, int64_t n, double* __restrict__ d)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) d[n - 1] = A[(n - 1) + (n - 1) * lda];
}

// ---- orgtr ---------------------------------------------------------------------------------

__global__ void identity_kernel(double* __restrict__ Q, int64_t ldq, int64_t n)
{
    const int64_t total = n * n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = t % n, c = t / n;
        Q[r + c * ldq] = r == c ? 1.0 : 0.0;
    }
}

// Vp (m x pb, leading dimension m): column i is v_{p+i} on rows p+1 .. n-1
__global__ void extract_v_kernel(const double* __restrict__ A, int64_t lda, int64_t n, int64_t p,
                                 int pb, double* __restrict__ Vp)
{
    const int64_t m = n - p - 1;
    const int64_t total = m * pb;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t l = t % m, i = t / m;
        const int64_t r = p + 1 + l, jj = p + i;
        double v;
        if (r < jj + 1) v = 0.0;
        else if (r == jj + 1) v = 1.0;
        else v = A[r + jj * lda];
        Vp[l + i * m] = v;
    }
}

// split-K partial tiles of op(X)[M x K] op(Y)[K x N] for M, N <= 64 (one tile), K chunk z:
// out[z][i + 64 j]
__global__ void __launch_bounds__(dmma::kThreads)
splitk_tile_kernel(const double* __restrict__ a, int64_t a_si, int64_t a_sk,
                   const double* __restrict__ b, int64_t b_sk, int64_t b_sj, int64_t M, int64_t N,
                   int64_t K, int64_t kch, double* __restrict__ out)
{
    __shared__ dmma::Smem sm;
    const int64_t kb = (int64_t)blockIdx.z * kch;
    const int64_t i0 = (int64_t)blockIdx.y * dmma::BM, j0 = (int64_t)blockIdx.x * dmma::BN;
    double acc[4][4][2];
    dmma::tile_gemm(a, a_si, a_sk, b, b_sk, b_sj, M, N, K, i0, j0, kb, kb + kch, acc, sm);
    const int64_t tiles_m = (M + dmma::BM - 1) / dmma::BM;
    double* o = out + ((int64_t)blockIdx.z * tiles_m * ((N + dmma::BN - 1) / dmma::BN) +
                       (int64_t)blockIdx.x * tiles_m + blockIdx.y) * dmma::BM * dmma::BN;
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 2; ++h) o[dmma::tile_row(x) + dmma::BM * dmma::tile_col(y, h)] = acc[x][y][h];
}

// Y[pb x m] (leading dimension pb) = sum over K chunks of the split-K tiles of Vp^T Q
__global__ void reduce_tiles_kernel(const double* __restrict__ part, int64_t M, int64_t N,
                                    int nk, double* __restrict__ Y, int64_t ldy)
{
    const int64_t tiles_m = (M + dmma::BM - 1) / dmma::BM, tiles_n = (N + dmma::BN - 1) / dmma::BN;
    const int64_t total = M * N;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t % M, jcol = t / M;
        const int64_t ti = i / dmma::BM, tj = jcol / dmma::BN;
        const int64_t off = (tj * tiles_m + ti) * dmma::BM * dmma::BN + (i % dmma::BM) + dmma::BM * (jcol % dmma::BN);
        double s = 0.0;
        for (int z = 0; z < nk; ++z) s += part[(int64_t)z * tiles_m * tiles_n * dmma::BM * dmma::BN + off];
        Y[i + jcol * ldy] = s;
    }
}

// G_p = V_p^T V_p of every panel (blockIdx.x), K chunk blockIdx.z: out[panel][z][i + 64 k].  The
// reflectors are read in place from A (unit diagonal, zeros above).
__global__ void __launch_bounds__(dmma::kThreads)
gram_kernel(const double* __restrict__ A, int64_t lda, int64_t n, int64_t kch, int nk, double* __restrict__ out)
{
    __shared__ double V[NB][NB + 1];
    const int64_t p = (int64_t)blockIdx.x * NB;
    const int pb = (int)(n - 1 - p < NB ? n - 1 - p : NB);
    const int64_t r0 = p + 1 + (int64_t)blockIdx.z * kch;   // first row of the chunk
    if (r0 >= n) return;                                     // (its slot is not read)
    const int64_t r1 = r0 + kch < n ? r0 + kch : n;
    double* o = out + ((int64_t)blockIdx.x * nk + blockIdx.z) * NB * NB;
    // thread: 4 x 8 outputs of the 64 x 64 tile
    const int ti = (threadIdx.x % 16) * 4, tj = (threadIdx.x / 16) * 8;
    double acc[4][8] = {};
    for (int64_t rb = r0; rb < r1; rb += NB) {
        for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
            const int l = t % NB, c = t / NB;
            const int64_t r = rb + l, jj = p + c;
            double v = 0.0;
            if (r < r1 && c < pb && r >= jj + 1) v = r == jj + 1 ? 1.0 : A[r + jj * lda];
            V[c][l] = v;
        }
        __syncthreads();
        if (tj + 7 >= ti)   // only i <= k is used
            for (int l = 0; l < NB; ++l) {
                double x[4], y[8];
#pragma unroll
                for (int u = 0; u < 4; ++u) x[u] = V[ti + u][l];
#pragma unroll
                for (int u = 0; u < 8; ++u) y[u] = V[tj + u][l];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int w = 0; w < 8; ++w) acc[u][w] = fma(x[u], y[w], acc[u][w]);
            }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 8; ++w) o[(ti + u) + (int64_t)NB * (tj + w)] = acc[u][w];
}

// T (pb x pb upper triangular, leading dimension NB) of every panel (blockIdx.x) from G = V^T V
// and tau:  T(i, i) = tau_i,  T(r, i) = -tau_i sum_{c = r}^{i-1} T(r, c) G(c, i)   (dlarft,
// forward).  Eight lanes share a row's sum; column i of T replaces column i of G.
__global__ void __launch_bounds__(8 * NB)
tfactor_kernel(const double* __restrict__ part, int64_t n, int64_t kch, int nk, const double* __restrict__ tau_all,
               double* __restrict__ T_all)
{
    __shared__ double S[NB][NB + 1];
    const int64_t p = (int64_t)blockIdx.x * NB;
    const int pb = (int)(n - 1 - p < NB ? n - 1 - p : NB);
    const int chunks = (int)((n - 1 - p + kch - 1) / kch);
    const double* __restrict__ tau = tau_all + p;
    const double* __restrict__ g = part + (int64_t)blockIdx.x * nk * NB * NB;
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        double s = 0.0;
#pragma unroll 4
        for (int z = 0; z < chunks; ++z) s += g[(int64_t)z * NB * NB + t];
        S[t % NB][t / NB] = s;
    }
    __syncthreads();
    const int r = threadIdx.x >> 3, q = threadIdx.x & 7;
    for (int i = 0; i < pb; ++i) {
        double s = 0.0;
        for (int c = r + q; c < i; c += 8) s = fma(S[r][c], S[c][i], s);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        __syncthreads();
        if (q == 0) S[r][i] = r < i ? -tau[i] * s : r == i ? tau[i] : 0.0;
        __syncthreads();
    }
    double* __restrict__ T = T_all + (int64_t)blockIdx.x * NB * NB;
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) T[t] = t / NB < pb ? S[t % NB][t / NB] : 0.0;
}

// VT[m x pb] = Vp T: 32 rows and 16 columns per block, two columns per thread.
constexpr int VC = 16;
__global__ void __launch_bounds__(256)
vt_kernel(const double* __restrict__ Vp, int64_t m, int pb, const double* __restrict__ T,
          double* __restrict__ VT)
{
    __shared__ double Ts[NB][VC];
    const int i0 = blockIdx.y * VC;
    for (int t = threadIdx.x; t < NB * VC; t += blockDim.x) Ts[t % NB][t / NB] = T[t % NB + (i0 + t / NB) * NB];
    __syncthreads();
    const int64_t l = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const int i = 2 * (threadIdx.x >> 5);
    if (l >= m) return;
    double s0 = 0.0, s1 = 0.0, u0 = 0.0, u1 = 0.0;
    const int end = min(pb, i0 + i + 2);   // T is upper triangular
    int c = 0;
#pragma unroll 4
    for (; c + 1 < end; c += 2) {
        const double x = Vp[l + (int64_t)c * m], y = Vp[l + (int64_t)(c + 1) * m];
        s0 = fma(x, Ts[c][i], s0);
        s1 = fma(x, Ts[c][i + 1], s1);
        u0 = fma(y, Ts[c + 1][i], u0);
        u1 = fma(y, Ts[c + 1][i + 1], u1);
    }
    if (c < end) {
        const double x = Vp[l + (int64_t)c * m];
        s0 = fma(x, Ts[c][i], s0);
        s1 = fma(x, Ts[c][i + 1], s1);
    }
    if (i0 + i < pb) VT[l + (int64_t)(i0 + i) * m] = s0 + u0;
    if (i0 + i + 1 < pb) VT[l + (int64_t)(i0 + i + 1) * m] = s1 + u1;
}

// Q(R, R) -= VT Y   (R = p+1 .. n-1; inner dimension pb)
__global__ void __launch_bounds__(dmma::kThreads)
wy_update_kernel(double* __restrict__ Q, int64_t ldq, int64_t p1, int64_t m, int pb,
                 const double* __restrict__ VT, const double* __restrict__ Y)
{
    __shared__ dmma::Smem sm;
    const int64_t i0 = (int64_t)blockIdx.y * dmma::BM, j0 = (int64_t)blockIdx.x * dmma::BN;
    double acc[4][4][2];
    dmma::tile_gemm(VT, 1, m, Y, 1, pb, m, m, pb, i0, j0, 0, pb, acc, sm);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t ii = i0 + dmma::tile_row(x), jj = j0 + dmma::tile_col(y, h);
                if (ii < m && jj < m) Q[(p1 + ii) + (p1 + jj) * ldq] -= acc[x][y][h];
            }
}

__global__ void maxabs_kernel(const double* __restrict__ A, int64_t lda, int64_t n, double* __restrict__ out)
{
    __shared__ double sh[32];
    double m = 0.0;
    const int64_t total = n * n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x)
        m = fmax(m, fabs(A[(t % n) + (t / n) * lda]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r = fmax(r, sh[k]);
        // non-negative doubles order as their bit patterns
        atomicMax(reinterpret_cast<unsigned long long*>(out), (unsigned long long)__double_as_longlong(r));
    }
}

__global__ void scale_kernel(double* __restrict__ A, int64_t lda, int64_t n, double f)
{
    const int64_t total = n * n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x)
        A[(t % n) + (t / n) * lda] *= f;
}

__global__ void tridiag_unscale_kernel(double* __restrict__ A, int64_t lda, int64_t n, double* __restrict__ d,
                                       double* __restrict__ e, double f)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        d[t] *= f;
        A[t + t * lda] = d[t];
        if (t + 1 < n) {
            e[t] *= f;
            A[t + 1 + t * lda] = e[t];
        }
    }
}

inline unsigned blocks_for(int64_t rows, int per) { return (unsigned)((rows + per - 1) / per); }

}  // namespace

cudaError_t launch_dense_maxabs(const double* A, int64_t lda, int64_t n, double* out, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), s);
    if (e != cudaSuccess) return e;
    if (n <= 0) return cudaSuccess;
    maxabs_kernel<<<608, 256, 0, s>>>(A, lda, n, out);
    return cudaGetLastError();
}

cudaError_t launch_dense_scale(double* A, int64_t lda, int64_t n, double f, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    scale_kernel<<<1216, 256, 0, s>>>(A, lda, n, f);
    return cudaGetLastError();
}

cudaError_t launch_tridiag_unscale(double* A, int64_t lda, int64_t n, double* d, double* e, double f,
                                   cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    tridiag_unscale_kernel<<<(unsigned)((n + 255) / 256 < 1216 ? (n + 255) / 256 : 1216), 256, 0, s>>>(A, lda, n, d, e, f);
    return cudaGetLastError();
}

// Column chunks of the matrix-vector product: at most this many for order n.
static int64_t symv_max_chunks(int64_t n) { return n <= 16384 ? 64 : (n + 255) / 256; }

// Partial tiles of orgtr's split-K products: those of Vp^T Q for the first (largest) panel, or of
// all panels' Gram matrices.
static int64_t orgtr_part_doubles(int64_t n)
{
    const int64_t nk = blocks_for(n, (int)split_rows(n));
    return nk * blocks_for(n, NB) * (int64_t)NB * NB;
}

// Scratch (doubles) of sytrd_dev / orgtr_dev for order n.
int64_t dense_scratch_doubles(int64_t n)
{
    const int64_t rb = (n + RB - 1) / RB;
    const int64_t sytrd = 2 * n * 2 * NB + 2 * rb + 2 * NB + symv_max_chunks(n) * n + n + 8;
    const int64_t orgtr = 3 * n * NB + orgtr_part_doubles(n) + blocks_for(n, NB) * (int64_t)NB * NB + 8;
    return sytrd > orgtr ? sytrd : orgtr;
}

// A (n x n, lda) -> d (n), e (n-1), tau (n-1); A overwritten as by LAPACK dsytrd('L').
int sytrd_dev(cudaStream_t s, int64_t n, double* A, int64_t lda, double* d, double* e, double* tau,
              double* scratch)
{
    if (n <= 0) return SYMEIG_OK;
    const int64_t rb = (n + RB - 1) / RB;
    Panel P{};
    P.A = A;
    P.lda = lda;
    P.n = n;
    P.VW = scratch;
    P.WV = P.VW + n * 2 * NB;
    P.part = P.WV + n * 2 * NB;
    P.wpart = P.part + rb;
    P.dots = P.wpart + rb;
    P.ypart = P.dots + 2 * NB;
    P.wraw = P.ypart + symv_max_chunks(n) * n;
    P.sc = P.wraw + n;
    for (int64_t p = 0; p < n - 1; p += NB) {
        const int pb = (int)(n - 1 - p < NB ? n - 1 - p : NB);
        P.pb = pb;
        for (int i = 0; i < pb; ++i) {
            const int64_t j = p + i, m = n - j - 1;                // rows j+1 .. n-1
            const unsigned blocks = blocks_for(n - j, RB);         // rows j .. n-1
            const unsigned blocks1 = blocks_for(m, RB), sr = blocks_for(m, SR);
            const unsigned chunks = blocks_for(m, symv_cols(m));
            // blocks for the 2 i dot products beside the chunks'
            const unsigned extra = i > 0 ? blocks_for(blocks_for(2 * i, 2 * SR / 32), (int)sr) : 0;
            launch_after(column_kernel, dim3(blocks), RB * RG, 0, s, P, j, i, (int)blocks, 0);
            launch_after(products_kernel, dim3(sr, chunks + extra), 2 * SR, 0, s, P, j, i, (int)blocks, (int)chunks, d, e, tau);
            launch_after(w_kernel, dim3(blocks1), RB * RG, 0, s, P, j, i, (int)chunks);
        }
        const int64_t q = p + pb;
        launch_after(column_kernel, dim3(blocks_for(n - q, RB)), RB * RG, 0, s, P, q, pb, (int)blocks_for(n - q, RB), 1);
        const unsigned t = blocks_for(n - q, dmma::BM);
        trailing_update_kernel<<<dim3(t, t), dmma::kThreads, 0, s>>>(A, lda, n, q, pb, P.VW, P.WV);
    }
    last_diag_kernel<<<1, 32, 0, s>>>(A, lda, n, d);
    return cudaGetLastError() == cudaSuccess ? SYMEIG_OK : SYMEIG_ERR_CUDA;
}

// Q (n x n, ldq) = H_0 ... H_{n-2} from sytrd_dev's A and tau.
int orgtr_dev(cudaStream_t s, int64_t n, const double* A, int64_t lda, const double* tau, double* Q,
              int64_t ldq, double* scratch)
{
    if (n <= 0) return SYMEIG_OK;
    identity_kernel<<<1216, 256, 0, s>>>(Q, ldq, n);
    if (n == 1) return cudaGetLastError() == cudaSuccess ? SYMEIG_OK : SYMEIG_ERR_CUDA;
    double* Vp = scratch;
    double* VT = Vp + n * NB;
    double* Y = VT + n * NB;
    double* part = Y + NB * n;
    double* T = part + orgtr_part_doubles(n);
    const int64_t kch = split_rows(n);
    const unsigned panels = blocks_for(n - 1, NB), nk_max = blocks_for(n - 1, (int)kch);
    // the T factors of all panels depend on the reflectors alone
    gram_kernel<<<dim3(panels, 1, nk_max), dmma::kThreads, 0, s>>>(A, lda, n, kch, (int)nk_max, part);
    tfactor_kernel<<<panels, 8 * NB, 0, s>>>(part, n, kch, (int)nk_max, tau, T);
    for (int64_t p = (int64_t)(panels - 1) * NB; p >= 0; p -= NB) {
        const int pb = (int)(n - 1 - p < NB ? n - 1 - p : NB);
        const int64_t m = n - p - 1;
        extract_v_kernel<<<blocks_for(m * pb, 256) < 1216 ? blocks_for(m * pb, 256) : 1216, 256, 0, s>>>(A, lda, n, p, pb, Vp);
        const unsigned nk = blocks_for(m, (int)kch);
        vt_kernel<<<dim3(blocks_for(m, 32), blocks_for(pb, VC)), 256, 0, s>>>(Vp, m, pb, T + (p / NB) * NB * NB, VT);
        // Y = Vp^T Q(R, R) (pb x m): B(k, j) = Q(p+1+k, p+1+j)
        const double* QR = Q + (p + 1) + (p + 1) * ldq;
        const unsigned tn = blocks_for(m, dmma::BN);
        splitk_tile_kernel<<<dim3(tn, 1, nk), dmma::kThreads, 0, s>>>(Vp, m, 1, QR, 1, ldq, pb, m, m, kch, part);
        reduce_tiles_kernel<<<blocks_for(pb * m, 256) < 4096 ? blocks_for(pb * m, 256) : 4096, 256, 0, s>>>(part, pb, m, (int)nk, Y, pb);
        const unsigned tm = blocks_for(m, dmma::BM);
        wy_update_kernel<<<dim3(tm, tm), dmma::kThreads, 0, s>>>(Q, ldq, p + 1, m, pb, VT, Y);
    }
    return cudaGetLastError() == cudaSuccess ? SYMEIG_OK : SYMEIG_ERR_CUDA;
}

}  // namespace symeig
