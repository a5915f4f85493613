// apply_fused.cuh -- launches of the fused-wave tile (wave_fused.cuh) for one precision; included by
// apply_f64.cu and apply_f32.cu.
//
// The shape of a pass (G lane groups of KB layers, F waves fused) follows from the rows m of the
// launch and its layers.
//
// FP64.  Time per column of a pass is about rounds * ceil(W / 4) * KB * u(ceil(W / 4)) * o(KB): W the warps
// of an SM's CTA, one FP64 unit per four of them.  u, the time of a rotation of one warp on a
// sub-partition that holds w warps, falls as the warps hide each other's integer products, and
// small KB adds the per-iteration work (shuffles, Q, the window's move).  Measured, n = 4096,
// 64 layers, ms (KB x G, the model's choice marked):
//   m        8 x 8    4 x 16   2 x 32    before (one wave at a time)
//   1000       -       2.41     1.84*      5.2
//   2500       -       3.97     3.36*      6.0
//   4096      6.47     5.06     4.75*      7.8
//   6144      8.01     7.09*    7.94      10.7
//   9000      9.61*   10.1        -       16.0
//   12288    13.4*      -         -       17.0
//   16384    15.7*      -         -       17.0
// and 128 layers: m = 2500 8 x 16 8.02, 4 x 32 6.14*; m = 12288 two passes of 8 x 8 26.8, 4 x 32 25.7*.
//
// FP32.  16 layers a group, four waves fused, in CTAs of up to 16 warps; G = 4 (64 layers a pass) from
// 3072 rows, where its 8 rows per warp still fill the SMs, else G = 8 (128 layers a pass).
// n = 4096, 64 layers, TFLOP/s: m = 2048 8 x 8 13.1, 16 x 4 11.1 (before 8.6); 4096 19.9, 21.6 (15.1);
// 8192 22.8, 25.6 (21.6); 16384 27.0, 27.1 (26.3); 128 layers: 4096 25.3, 11000 28.2 (two passes before: 21).
// Its ceiling is the register file's operand bandwidth: the arithmetic alone (no table reads, no
// shuffles) runs at 36.9 TFLOP/s, 0.5 of the FMA peak.
#pragma once

#include <algorithm>

#include "symeig_common.cuh"
#include "wave_fused.cuh"

namespace symeig {
namespace fused {

struct Choice {
    int G, KB, F;
    int64_t per;    // layers per pass
};

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Warps per CTA and CTAs of an m-row launch.
struct Launch {
    unsigned blocks;
    int warps;
};
inline Launch launch_of(int64_t m, int rows_per_warp, int max_warps)
{
    const int64_t per_sm = ceil_div(ceil_div(m, kSms), rows_per_warp);
    const int64_t warps = ceil_div(per_sm, ceil_div(per_sm, max_warps));
    return {(unsigned)ceil_div(m, warps * rows_per_warp), (int)warps};
}

// The padded layers of a group for `per` layers over G groups.
template <typename T> inline int group_layers(int64_t per, int G)
{
    const int kb = (int)ceil_div(per, G);
    if (sizeof(T) == 8) return kb == 1 && G == 32 ? 1 : 2 * (int)ceil_div(kb, 2);
    return G == 4 ? 4 * (int)ceil_div(kb, 4) : 2 * (int)ceil_div(kb, 2);
}

// `one_pass`: a shape whose single pass holds all the layers (those of a pass that the choice for
// the whole apply made).
template <typename T> inline Choice choose(int64_t m, int64_t layers, bool one_pass = false)
{
    if (sizeof(T) == 4) {
        const int G = layers <= 64 && m >= 3072 ? 4 : 8;
        const int64_t passes = ceil_div(layers, 16 * G), per = ceil_div(layers, passes);
        int KB = group_layers<T>(per, G);
        int F = KB % 4 == 0 ? 4 : 2;
        // 17 to 20 warps fit an SM with two waves fused (102 registers), 16 with four
        const int64_t per_sm = ceil_div(ceil_div(m, kSms), 32 / G);
        if (G == 8 && F == 4 && KB > 8 && per_sm > 16 && per_sm <= 20) F = 2;
        return {G, KB, F, per};
    }
    static const double u[8] = {0.0, 0.60, 0.42, 0.335, 0.31, 0.30, 0.285, 0.28};
    Choice best{0, 0, 0, 0};
    double best_cost = 0.0;
    for (int G = 8; G <= 32; G *= 2) {
        const int64_t passes = ceil_div(layers, 8 * G), per = ceil_div(layers, passes);
        if (one_pass && passes > 1) continue;
        const int KB = group_layers<T>(per, G);
        const int64_t per_sm = ceil_div(ceil_div(m, kSms), 32 / G), rounds = ceil_div(per_sm, 27);
        const int64_t w = ceil_div(ceil_div(per_sm, rounds), 4);
        const double o = KB == 1 ? 2.0 : KB == 2 ? 1.18 : KB == 4 ? 1.03 : 1.0;
        const double cost = (double)(passes * rounds * w * KB) * u[std::min<int64_t>(w, 7)] * o;
        if (best.G == 0 || cost < best_cost) {
            best_cost = cost;
            best = {G, KB, KB == 1 ? 1 : 2, per};
        }
    }
    return best;
}

template <typename Tsrc, typename T, typename S>
__global__ void __launch_bounds__(256)
table_kernel(unsigned char* __restrict__ table, int64_t total, const Tsrc* __restrict__ grid, int64_t grid_rows,
             const int32_t* __restrict__ place, int64_t c0, int64_t n_loc, int64_t L0, int64_t layers)
{
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x)
        table_entry<T, S, Tsrc>(table, idx, grid, grid_rows, place, c0, n_loc, L0, layers);
}

template <typename T, typename S, bool SEG>
__global__ void __launch_bounds__(32 * S::MAX_WARPS, 1)
wave_kernel(T* __restrict__ Q, int64_t ldq, int64_t m, int32_t n_loc, const unsigned char* __restrict__ table,
            int32_t n_chunks, int* __restrict__ err, const T nz, int64_t rs, int32_t stall, int32_t c_begin,
            int32_t c_end, T* __restrict__ state)
{
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ __align__(8) uint64_t bar[2];
    const int64_t row0 = (int64_t)blockIdx.x * ((blockDim.x >> 5) * S::RPW);
    T* st = SEG ? state + (int64_t)blockIdx.x * S::STATE * blockDim.x : nullptr;
    if (!tile<T, S, SEG>(Q, ldq, m, row0, n_loc, table, n_chunks, nz, ring, bar, rs, stall, c_begin, c_end, st, err)) {
        if (threadIdx.x == 0) atomicOr(err, 1);
    }
}

template <typename Tsrc, typename T, typename S>
cudaError_t build_table(const Tsrc* grid, int64_t grid_rows, const int32_t* place, const ApplyPass& pass, void* table,
                        cudaStream_t stream)
{
    const int64_t total = S::chunks(pass.n_loc) * S::NI * S::G * S::KB * S::F;
    const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(total, 256), kSms * 16);
    table_kernel<Tsrc, T, S><<<blocks, 256, 0, stream>>>((unsigned char*)table, total, grid, grid_rows, place, pass.c0,
                                                         pass.n_loc, pass.L0, pass.layers);
    return cudaGetLastError();
}

template <typename T, typename S, bool SEG>
cudaError_t launch_wave(T* Q, int64_t ldq, int64_t m, const ApplyPass& pass, const void* table, int* err,
                        cudaStream_t stream, int32_t c_begin = 0, int32_t c_end = 0, void* state = nullptr)
{
    const Launch L = launch_of(m, S::RPW, S::MAX_WARPS);
    wave_kernel<T, S, SEG><<<L.blocks, 32 * L.warps, 2 * S::CHUNK, stream>>>(
        Q + pass.c0 * ldq, ldq, m, (int32_t)pass.n_loc, (const unsigned char*)table, (int32_t)S::chunks(pass.n_loc), err,
        (T)-0.0, pass.rs, pass.stall > 0 ? pass.stall : 0x7fffffff, c_begin, c_end, (T*)state);
    return cudaGetLastError();
}

// Calls f with the Shape of `ch`; the KB that exist are those group_layers gives.
template <typename T, typename Fn> auto with_shape(const Choice& ch, Fn&& f)
{
    if constexpr (sizeof(T) == 8) {
#define SYMEIG_KB(G)                                                                                   \
        switch (ch.KB) {                                                                               \
            case 2: return f(Shape<T, 2, G, 2>{});                                                     \
            case 4: return f(Shape<T, 4, G, 2>{});                                                     \
            case 6: return f(Shape<T, 6, G, 2>{});                                                     \
            default: return f(Shape<T, 8, G, 2>{});                                                    \
        }
        if (ch.G == 8) SYMEIG_KB(8)
        if (ch.G == 16) SYMEIG_KB(16)
        if (ch.KB == 1) return f(Shape<T, 1, 32, 1>{});
        SYMEIG_KB(32)
#undef SYMEIG_KB
    } else {
        if (ch.G == 4) switch (ch.KB) {
            case 4: return f(Shape<T, 4, 4, 4>{});
            case 8: return f(Shape<T, 8, 4, 4>{});
            case 12: return f(Shape<T, 12, 4, 4>{});
            default: return f(Shape<T, 16, 4, 4>{});
        }
        if (ch.F == 4) switch (ch.KB) {
            case 4: return f(Shape<T, 4, 8, 4>{});
            case 8: return f(Shape<T, 8, 8, 4>{});
            case 12: return f(Shape<T, 12, 8, 4>{});
            default: return f(Shape<T, 16, 8, 4>{});
        }
        switch (ch.KB) {
            case 2: return f(Shape<T, 2, 8, 2>{});
            case 6: return f(Shape<T, 6, 8, 2>{});
            case 10: return f(Shape<T, 10, 8, 2>{});
            case 12: return f(Shape<T, 12, 8, 2>{});
            case 14: return f(Shape<T, 14, 8, 2>{});
            default: return f(Shape<T, 16, 8, 2>{});
        }
    }
}

// The column-segment launches exist for fewer shapes; a pass of at most 64 layers fits one of them.
template <typename T> inline Choice choose_segmented(int64_t m, int64_t layers)
{
    Choice ch = choose<T>(m, layers, true);
    if (sizeof(T) == 8) {
        if (ch.KB < 2) ch = {16, 2, 2, layers};
        const int cap = 64 / ch.G;   // 8, 4, 2
        ch.KB = cap;
        ch.F = 2;
    } else {
        ch.KB = ch.G == 4 ? 16 : 8;
        ch.F = 4;
    }
    ch.per = layers;
    return ch;
}
template <typename T, typename Fn> auto with_segmented(const Choice& ch, Fn&& f)
{
    if constexpr (sizeof(T) == 8) {
        if (ch.G == 8) return f(Shape<T, 8, 8, 2>{});
        if (ch.G == 16) return f(Shape<T, 4, 16, 2>{});
        return f(Shape<T, 2, 32, 2>{});
    } else {
        if (ch.G == 4) return f(Shape<T, 16, 4, 4>{});
        return f(Shape<T, 8, 8, 4>{});
    }
}

}  // namespace fused

template <typename T> int64_t fused_layers_per_pass(int64_t m, int64_t layers) { return fused::choose<T>(m, layers).per; }

// Bytes of the largest table of passes of `layers` layers, whatever the rows.
template <typename T> size_t fused_table_bytes(int64_t n_loc, int64_t layers)
{
    size_t b = 0;
    // every row count takes one of these group counts; KB rises with the layers of a pass
    for (int G = sizeof(T) == 8 ? 8 : 4; G <= (sizeof(T) == 8 ? 32 : 8); G *= 2) {
        const int64_t per = std::min<int64_t>(layers, (sizeof(T) == 8 ? 8 : 16) * G);
        for (int F = 1; F <= 4; F *= 2) {
            if (sizeof(T) == 8 ? F == 4 : F == 1) continue;
            fused::Choice ch{G, fused::group_layers<T>(per, G), F, per};
            if (sizeof(T) == 8) ch.F = ch.KB == 1 ? 1 : 2;
            else if (G == 4) ch.F = 4;
            else if (F == 4) ch.KB = 4 * (int)fused::ceil_div(ch.KB, 4);
            b = std::max(b, fused::with_shape<T>(ch, [&](auto s) { return (size_t)decltype(s)::table_bytes(n_loc); }));
        }
    }
    if (layers <= 64)   // the column segments' shapes hold 64 layers whatever the pass has
        for (int G = 4; G <= 32; G *= 2)
            b = std::max(b, fused::with_segmented<T>({G, 0, 0, 0}, [&](auto s) { return (size_t)decltype(s)::table_bytes(n_loc); }));
    return (b + 255) & ~(size_t)255;
}

template <typename Tsrc, typename T>
cudaError_t fused_pass(T* Q, int64_t ldq, int64_t m, const Tsrc* grid, int64_t grid_rows, const int32_t* place,
                       const ApplyPass& pass, void* table, int* err, cudaStream_t stream, cudaEvent_t ev_begin,
                       cudaEvent_t ev_end, int what)
{
    if (pass.n_loc < 2 || pass.layers <= 0) return cudaSuccess;
    if (m <= 0) return cudaSuccess;   // the table's shape follows from the rows
    return fused::with_shape<T>(fused::choose<T>(m, pass.layers, true), [&](auto s) {
        using S = decltype(s);
        if (S::LAYERS < pass.layers) return cudaErrorInvalidValue;
        cudaError_t e = cudaSuccess;
        if (what & kPassTable) e = fused::build_table<Tsrc, T, S>(grid, grid_rows, place, pass, table, stream);
        if (e != cudaSuccess || !(what & kPassWave)) return e;
        if (ev_begin) cudaEventRecord(ev_begin, stream);
        e = fused::launch_wave<T, S, false>(Q, ldq, m, pass, table, err, stream);
        if (ev_end) cudaEventRecord(ev_end, stream);
        return e;
    });
}

// The host-pointer apply of one pass of k <= 64 layers, streamed by column segments.  The
// caller's column-major Q (host memory, leading dimension lda) goes to the device buffer dQ
// (leading dimension m) in column chunks on io.s_in; the pass runs as io.nseg launches over
// consecutive chunk ranges of its table on `stream`, each waiting for the columns its chunks
// read and carrying its registers to the next launch in io.state; the columns a launch finishes
// (all of them after the last) go back on io.s_out as soon as it ends.  So the copies in both
// directions overlap the kernels, and every launch runs the whole m-row grid.  Only stream
// events order the three streams.
template <typename T>
cudaError_t fused_host_segmented(T* dQ, int64_t m, const T* d_cs, const ApplyPass& pass, void* table, int* err,
                                 cudaStream_t stream, const HostStream& io)
{
    const int64_t n = pass.n_loc;
    return fused::with_segmented<T>(fused::choose_segmented<T>(m, pass.layers), [&](auto s) {
        using S = decltype(s);
        cudaError_t e = fused::build_table<T, T, S>(d_cs, n - 1, nullptr, pass, table, stream);
        if (e != cudaSuccess) return e;
        const int64_t n_chunks = S::chunks(n);
        const int nseg = (int)std::max<int64_t>(1, std::min<int64_t>(io.nseg, n_chunks));
        const size_t esz = sizeof(T);
        T* host = (T*)io.host;
        int64_t in_lo = 0, out_lo = 0;
        // copies in and kernels first, then the copies out: with pageable host memory a copy out
        // blocks the calling thread until it is done, and must not hold back the next copy in
        for (int j = 0; j < nseg; ++j) {
            const int64_t cb = (int64_t)j * n_chunks / nseg, ce = (int64_t)(j + 1) * n_chunks / nseg;
            const int64_t in_hi = std::min<int64_t>(n, S::F * (ce * S::NI + S::PD));
            if (in_hi > in_lo) {
                e = cudaMemcpy2DAsync(dQ + in_lo * m, m * esz, host + in_lo * io.lda, io.lda * esz, m * esz,
                                      in_hi - in_lo, cudaMemcpyHostToDevice, io.s_in);
                if (e != cudaSuccess) return e;
                in_lo = in_hi;
            }
            if ((e = cudaEventRecord(io.ev_in[j], io.s_in)) != cudaSuccess) return e;
            if ((e = cudaStreamWaitEvent(stream, io.ev_in[j], 0)) != cudaSuccess) return e;
            e = fused::launch_wave<T, S, true>(dQ, m, m, pass, table, err, stream, (int32_t)cb, (int32_t)ce, io.state);
            if (e != cudaSuccess) return e;
            if ((e = cudaEventRecord(io.ev_seg[j], stream)) != cudaSuccess) return e;
        }
        for (int j = 0; j < nseg; ++j) {
            const int64_t ce = (int64_t)(j + 1) * n_chunks / nseg;
            const int64_t out_hi = j == nseg - 1 ? n
                : std::max<int64_t>(0, std::min<int64_t>(n, S::F * (ce * S::NI - (int64_t)(S::G - 1) * S::D) - S::KB));
            if ((e = cudaStreamWaitEvent(io.s_out, io.ev_seg[j], 0)) != cudaSuccess) return e;
            if (out_hi > out_lo) {
                e = cudaMemcpy2DAsync(host + out_lo * io.lda, io.lda * esz, dQ + out_lo * m, m * esz, m * esz,
                                      out_hi - out_lo, cudaMemcpyDeviceToHost, io.s_out);
                if (e != cudaSuccess) return e;
                out_lo = out_hi;
            }
        }
        return cudaSuccess;
    });
}

// Device memory of the registers the segments of an m-row launch carry, whichever shape it takes.
template <typename T> size_t fused_state_bytes(int64_t m)
{
    size_t b = 0;
    for (int G = 4; G <= 32; G *= 2)
        b = std::max(b, fused::with_segmented<T>({G, 0, 0, 0}, [&](auto s) {
            using S = decltype(s);
            const fused::Launch L = fused::launch_of(m, S::RPW, S::MAX_WARPS);
            return (size_t)L.blocks * 32 * L.warps * S::STATE * sizeof(T);
        }));
    return b;
}

}  // namespace symeig
