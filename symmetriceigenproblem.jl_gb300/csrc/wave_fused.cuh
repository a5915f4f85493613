// wave_fused.cuh -- the wave-window Givens tile with F waves fused per iteration.
//
// The tile of wave_common.cuh applies one wave (KB rotations, one dependent chain) at a time, so
// a warp has one rotation in flight and a launch with few warps per SM sub-partition waits on
// its latency.  Here an iteration applies the F waves t = F j .. F j + F - 1 together: step q of
// it applies rotation q - f of wave f, for every f, and these F rotations touch disjoint
// columns -- wave f's pair is (F j + 2 f - q - 1, F j + 2 f - q) -- and only need steps before q:
// F independent chains instead of one, the same rotations in the same order on every element
// (same bits).  A thread's window holds the KB + F columns from F j - KB to F j + F - 1; after
// the iteration the lowest F of them are final for its layer group and go to the next group,
// which is D = (KB + F) / F iterations behind.  As before, the groups of a row are neighbouring
// lanes of one warp, group 0 reads Q, group G - 1 writes it, and the (c, s) table streams through
// a two-slot shared-memory ring by cp.async.bulk with bounded waits.
//
// Rows are spread over the SMs by the block size: every SM gets one CTA of as many warps as its
// share of the rows needs (kSms), in the fewest equal rounds when that exceeds what fits
// (max_warps), so no SM carries more rows than another by more than one warp.
//
// KB and G are chosen per pass (choose, apply_fused.cuh): the layers of a pass are padded to G * KB with KB
// even (or, FP64, 1), not to 64, and a short Q takes more lane groups (32 / G rows per warp).
//
// FP64 (SHIFT): the products run on the integer pipes (int_mul.cuh), about 1550 instructions per
// iteration of KB = 8, F = 2; the window moves down by F registers after each iteration, so the
// loop body is one iteration and stays in the instruction cache.  FP32: D iterations are unrolled
// and the window rotates by renaming.
#pragma once

#include "wave_common.cuh"

namespace symeig {
namespace fused {

using wave::bulk_load;
using wave::mbar_init;
using wave::mbar_wait_bounded;
using wave::st_pred;

constexpr int kSms = 152;   // GB300

// PD: iterations group 0 reads ahead.  NI: iterations per chunk of the table, as many as two
// chunks of 23 KB hold: two CTA barriers per chunk keep the warps together (16384 x 8192, 64
// layers: 31.2 ms with 9 KB chunks, 30.8 with 22 KB; without barriers, each warp waiting by itself
// and the last one refilling a slot, 31.3 and 31.0 ms, the warps then share no instruction
// fetches).
template <typename T, int KB_, int G_, int F_>
struct Shape {
    using P2 = typename Pair<T>::type;
    static constexpr bool SHIFT = sizeof(T) == 8;
    static constexpr int KB = KB_, G = G_, F = F_, W = KB_ + F_, D = (KB_ + F_) / F_, RPW = 32 / G_;
    static constexpr int LAYERS = KB * G;
    static constexpr int GSTRIDE = KB * F * (int)sizeof(P2) + 16;   // padded: the groups' pairs lie in other banks
    static constexpr int ITER = G * GSTRIDE;
    static constexpr int NI = SHIFT ? (23552 / ITER < 16 ? 23552 / ITER : 16) : D * (D * ITER <= 8192 ? 2 : 1);
    static constexpr int PD = SHIFT ? 1 : D;
    static constexpr int CHUNK = NI * ITER;
    // warps per CTA that fit an SM's registers: 72 per thread for FP64 (KB <= 8), FP32 up to 122
    static constexpr int MAX_WARPS = SHIFT ? 27 : (KB > 8 && F == 4) ? 16 : 20;
    static_assert(KB % F == 0 && CHUNK % 16 == 0 && GSTRIDE % 16 == 0 && 2 * CHUNK <= 48 * 1024, "layout");
    __host__ __device__ static int64_t iterations(int64_t n) { return (n - 1 + KB) / F + 1 + (int64_t)(G - 1) * D; }
    __host__ __device__ static int64_t chunks(int64_t n) { return (iterations(n) + NI - 1) / NI; }
    __host__ __device__ static int64_t table_bytes(int64_t n) { return chunks(n) * (int64_t)CHUNK; }
    // values a thread carries across a launch boundary (column segments)
    static constexpr int STATE = W + PD * F + F;
};

// Table entry (iteration j, group g, wave f, layer l of the group).  The F pairs of step q = l + f
// are adjacent; steps q >= KB fall on the slots that steps q - KB < F leave unused.
template <typename T, typename S, typename Tsrc>
__device__ __forceinline__ void table_entry(unsigned char* table, int64_t idx, const Tsrc* grid, int64_t grid_rows,
                                            const int32_t* place, int64_t c0, int64_t n_loc, int64_t L0,
                                            int64_t layers)
{
    const int f = (int)(idx % S::F), l = (int)((idx / S::F) % S::KB), g = (int)((idx / (S::F * S::KB)) % S::G);
    const int64_t j = idx / ((int64_t)S::F * S::KB * S::G);
    const int64_t i_loc = S::F * (j - (int64_t)g * S::D) + f - 1 - l;
    const int64_t lay = (int64_t)g * S::KB + l;
    Tsrc c = Tsrc(1), s = Tsrc(0);
    if (i_loc >= 0 && i_loc <= n_loc - 2 && lay < layers) {
        const int64_t i = c0 + i_loc, L = L0 + lay;
        if (place == nullptr || L < (int64_t)place[i]) {
            const Tsrc* p = grid + 2 * (i + L * grid_rows);
            c = p[0];
            s = p[1];
        }
    }
    typename S::P2 v;
    v.x = (T)c;
    v.y = (T)s;
    const int pos = ((l + f) % S::KB) * S::F + f;
    *(typename S::P2*)(table + j * S::ITER + g * S::GSTRIDE + pos * (int)sizeof(typename S::P2)) = v;
}

// The rotations of one iteration.  `base` rotates the window's slots (0 with SHIFT); callers pass
// a constant of an unrolled loop.
template <typename T, typename S>
__device__ __forceinline__ void rotations(T (&win)[S::W], const unsigned char* cs, const int base, const T nz)
{
    constexpr int KB = S::KB, F = S::F, W = S::W;
#pragma unroll
    for (int q = 0; q < KB + F - 1; ++q) {
        if constexpr (sizeof(T) == 8) {
            double2 p[F];
            double sy[F], sx[F];
            bool sp[F], any = false;
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const int l = q - f;
                if (l < 0 || l >= KB) continue;
                p[f] = *reinterpret_cast<const double2*>(cs + ((q % KB) * F + f) * 16);
                const SplitFactor s = split_factor(p[f].y);
                sp[f] = s.special;
                sy[f] = mul_rn_int(s, win[(KB + f - l + base) % W], sp[f]);
                sx[f] = mul_rn_int(s, win[(KB + f - 1 - l + base) % W], sp[f]);
                any |= sp[f];
            }
            // one vote per step: the products the integer path does not cover, on the FP64 pipe
            if (__any_sync(0xffffffffu, any)) {
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    const int l = q - f;
                    if (l < 0 || l >= KB) continue;
                    if (sp[f]) {
                        const double2 t = fma_pair_call(p[f].y, win[(KB + f - l + base) % W],
                                                        win[(KB + f - 1 - l + base) % W], nz);
                        sy[f] = t.x;
                        sx[f] = t.y;
                    }
                }
            }
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const int l = q - f;
                if (l < 0 || l >= KB) continue;
                double& x = win[(KB + f - 1 - l + base) % W];
                double& y = win[(KB + f - l + base) % W];
                x = __fma_rn(p[f].x, x, sy[f]);
                y = __fma_rn(p[f].x, y, -sx[f]);
            }
        } else {
            float2 p[F];
#pragma unroll
            for (int f = 0; f < F; f += 2) {
                const float4 v = *reinterpret_cast<const float4*>(cs + ((q % KB) * F + f) * 8);
                p[f] = make_float2(v.x, v.y);
                p[f + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const int l = q - f;
                if (l < 0 || l >= KB) continue;
                rot(win[(KB + f - 1 - l + base) % W], win[(KB + f - l + base) % W], p[f].x, p[f].y);
            }
        }
    }
}

// Rows [row0, row0 + RPW * warps) of Q through chunks [c_begin, c_end) of the pass's table; see
// wave::wave_tile for the arguments (element (row, col) is Q[row * rs + col * ldq]; `stall` is the
// test hook; SEG restores a thread's registers from `state` unless c_begin is 0 and saves them
// unless c_end is n_chunks).  False when a bounded wait gave up.
// Chunk c reads the columns below F ((c + 1) NI + PD) and finishes those below
// F ((c + 1) NI - (G - 1) D) - KB.
template <typename T, typename S, bool SEG>
__device__ __forceinline__ bool tile(T* __restrict__ Q, int64_t ldq, int64_t m, int64_t row0, int32_t n,
                                     const unsigned char* __restrict__ table, int32_t n_chunks, const T nz,
                                     unsigned char* ring, uint64_t* bar, int64_t rs, int32_t stall,
                                     int32_t c_begin_arg, int32_t c_end_arg, T* __restrict__ state, int* check)
{
    constexpr int KB = S::KB, G = S::G, F = S::F, W = S::W, RPW = S::RPW, D = S::D, PD = S::PD;
    const int tid = threadIdx.x, lane = tid & 31, g = lane / RPW, rl = lane - g * RPW;
    const int32_t c_begin = SEG ? c_begin_arg : 0, c_end = SEG ? c_end_arg : n_chunks;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
        for (int b = 0; b < 2; ++b)
            if (c_begin + b < c_end && c_begin + b < stall)
                bulk_load(ring + b * S::CHUNK, table + (int64_t)(c_begin + b) * S::CHUNK, S::CHUNK, &bar[b]);
    }
    __syncthreads();
    // checked builds test every address of Q that is read or written
#ifdef SYMEIG_DEVICE_CHECKS
    auto in_extent = [&](const T* p) { return wave::index_ok(check, wave::offset_in_extent(p - Q, ldq, rs, m, n)); };
#else
    auto in_extent = [](const T*) { return true; };
#endif
    const int64_t row = row0 + (int64_t)(tid >> 5) * RPW + rl;
    const bool row_ok = row < m;
    T* __restrict__ q0 = Q + (row_ok ? row : 0) * rs;
    const bool storer = g == G - 1 && row_ok;
    T win[W], ahead[PD][F], xout[F];
    if (!SEG || c_begin == 0) {
#pragma unroll
        for (int i = 0; i < W; ++i) win[i] = T(0);
#pragma unroll
        for (int f = 0; f < F; ++f) xout[f] = T(0);
#pragma unroll
        for (int a = 0; a < PD; ++a)
#pragma unroll
            for (int f = 0; f < F; ++f)
                ahead[a][f] = a * F + f < n && in_extent(q0 + (int64_t)(a * F + f) * ldq) ? q0[(int64_t)(a * F + f) * ldq] : T(0);
    } else {
        const T* s = state + tid;   // value-major
        const int nt = blockDim.x;
#pragma unroll
        for (int i = 0; i < W; ++i) win[i] = s[(int64_t)i * nt];
#pragma unroll
        for (int a = 0; a < PD; ++a)
#pragma unroll
            for (int f = 0; f < F; ++f) ahead[a][f] = s[(int64_t)(W + a * F + f) * nt];
#pragma unroll
        for (int f = 0; f < F; ++f) xout[f] = s[(int64_t)(W + PD * F + f) * nt];
    }
    // the first column the next iteration reads and the first it finishes (group G - 1)
    int32_t ld_col = F * (c_begin * S::NI + PD), st_col = F * (c_begin * S::NI - (G - 1) * D) - KB;
    const T* lp = q0 + (int64_t)ld_col * ldq;
    T* sp = q0 + (int64_t)st_col * ldq;
    constexpr int U = S::SHIFT ? 1 : D;   // iterations unrolled
    for (int32_t c = c_begin; c < c_end; ++c) {
        const int b = (c - c_begin) & 1;
        const bool ok = mbar_wait_bounded(&bar[b], (uint32_t)((c - c_begin) >> 1) & 1u);
        if (__syncthreads_or(!ok)) return false;
        const unsigned char* cs = ring + b * S::CHUNK + g * S::GSTRIDE;
#pragma unroll 1
        for (int it = 0; it < S::NI; it += U) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int base = S::SHIFT ? 0 : (u * F) % W;
                const int a = S::SHIFT ? 0 : u % PD;
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    const T up = __shfl_up_sync(0xffffffffu, xout[f], RPW);
                    win[(KB + f + base) % W] = g == 0 ? ahead[a][f] : up;
                    T next = T(0);
                    if (ld_col + f < n && in_extent(lp + f * ldq)) next = lp[f * ldq];
                    ahead[a][f] = next;
                }
                ld_col += F;
                lp += F * ldq;
                rotations<T, S>(win, cs + (it + u) * S::ITER, base, nz);
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    xout[f] = win[(f + base) % W];
                    const bool in = storer && (uint32_t)(st_col + f) < (uint32_t)n;
                    st_pred(sp + f * ldq, xout[f], in && in_extent(sp + f * ldq));
                }
                st_col += F;
                sp += F * ldq;
                if constexpr (S::SHIFT) {
#pragma unroll
                    for (int i = 0; i < KB; ++i) win[i] = win[i + F];
                }
            }
        }
        __syncthreads();
        if (tid == 0 && c + 2 < c_end && c + 2 < stall) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bulk_load(ring + b * S::CHUNK, table + (int64_t)(c + 2) * S::CHUNK, S::CHUNK, &bar[b]);
        }
    }
    if (SEG && c_end < n_chunks) {
        T* s = state + tid;
        const int nt = blockDim.x;
#pragma unroll
        for (int i = 0; i < W; ++i) s[(int64_t)i * nt] = win[i];
#pragma unroll
        for (int a = 0; a < PD; ++a)
#pragma unroll
            for (int f = 0; f < F; ++f) s[(int64_t)(W + a * F + f) * nt] = ahead[a][f];
#pragma unroll
        for (int f = 0; f < F; ++f) s[(int64_t)(W + PD * F + f) * nt] = xout[f];
    }
    return true;
}

}  // namespace fused
}  // namespace symeig
