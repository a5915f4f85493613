// chase.cu -- the FP64 bulge-chase kernel: one flush of qr_algorithm! on the device.
//
// Restates, on one warp, the inner loop of qr_algorithm! (src/bulge_chasing.jl:166-279):
// the deflation scan (:205-222, is_offdiagonal_small :7-8), the layer capacity rule
// (:226-230), the Wilkinson shift (:239-265) and single_shift! (:11-144) with
// get_rotation / LinearAlgebra.givensAlgorithm (src/simple_givens.jl:20-23).  The sweep is a
// strict dependency chain and runs on one warp (sweep_warp); the O(n) scans (deflation, thickest
// column) use all 32 lanes with ballots.  Rotations go to a Julia-layout (c,s) grid: at
// grid[i, ++thickness[i]] as the reference records them, or (the default) at the sweep's
// exact-order layer described at chase_kernel.
//
// Every floating-point operation is an explicit _rn intrinsic.  Inside single_shift! the
// reference runs under @fastmath; this kernel and the CPU oracle fuse the first product of
// each `u*a + v*b` (see symeig_common.cuh).  Outside it (givensAlgorithm, the shift, the
// deflation test) the arithmetic is plain IEEE without contraction, as Julia compiles it.
// Division and square root are the correctly rounded __ddiv_rn / __dsqrt_rn, so the kernel
// reproduces the oracle's rotation stream bit for bit.
//
// The kernel never traps and never waits on another kernel: a flush ends by itself and
// reports CHASE_FLUSH, CHASE_CONVERGED or CHASE_MAXITER in ChaseState.
#include "symeig_common.cuh"
#include "givens.cuh"
#include "givens_int.cuh"

namespace symeig {

namespace {

using namespace gv;

// is_offdiagonal_small(H, j, tol), 1-based j (src/bulge_chasing.jl:7-8).
__device__ __forceinline__ bool is_small(const double* dv, const double* ev, int64_t j, double tol)
{
    return fabs(ev[j - 1]) <= __dmul_rn(tol, __dadd_rn(fabs(dv[j - 1]), fabs(dv[j])));
}

// False only where is_small is false, from the exponent fields: |e| >= 2^(xe-1023), while
// tol (|d_j| + |d_j+1|) < 2^(xt-1023+1) 2^(max(xd)-1023+2), unless the sum is infinite (xd >= 2046, where
// every xe below xt + 1026 passes the second test and those from there on the first, with xe = 0) or tol is
// (kNoTol).  An FP64 instruction costs 64 cycles, so the scan runs the exact test only where this cannot
// decide.
constexpr int32_t kNoTol = 4096;   // above every xe
__device__ __forceinline__ int32_t tol_exponent(double tol)
{
    const int32_t xt = (__double2hiint(tol) >> 20) & 0x7FF;
    return xt == 0x7FF ? kNoTol : xt;
}
__device__ __forceinline__ bool maybe_small(double e, double d0, double d1, int32_t xt)
{
    const int32_t xe = (__double2hiint(e) >> 20) & 0x7FF;
    const int32_t xd = max((__double2hiint(d0) >> 20) & 0x7FF, (__double2hiint(d1) >> 20) & 0x7FF);
    return (uint32_t)(xe - 1) >= (uint32_t)(xt + 1025) || xe < xt + xd - 1020;
}

// Wilkinson shift from the trailing 2x2 block [a c; c b] (src/bulge_chasing.jl:239-265), by a
// warp: the three divisions by the scale in three lanes at once (650 cycles each).
__device__ __forceinline__ double wilkinson_shift(double a, double b, double c)
{
    const int lane = threadIdx.x & 31;
    const double scale = __dadd_rn(__dadd_rn(fabs(a), __dmul_rn(2.0, fabs(c))), fabs(b));
    const double q = __ddiv_rn(lane == 0 ? a : lane == 1 ? c : b, scale);
    const double H11 = __shfl_sync(0xffffffffu, q, 0), H12 = __shfl_sync(0xffffffffu, q, 1),
                 H22 = __shfl_sync(0xffffffffu, q, 2);
    const double t = __dmul_rn(__dadd_rn(H11, H22), 0.5);   // (H11 + H22) / 2
    const double p = __dmul_rn(__dsub_rn(H11, t), __dsub_rn(H22, t));
    const double sq = __dsqrt_rn(fabs(__dsub_rn(p, __dmul_rn(H12, H12))));
    const double l1 = __dadd_rn(t, sq), l2 = __dsub_rn(t, sq);
    const double lam = fabs(__dsub_rn(H22, l1)) < fabs(__dsub_rn(H22, l2)) ? l1 : l2;
    return __dmul_rn(lam, scale);
}

__device__ __forceinline__ double fsum(double u, double a, double v, double b, double nz)
{
    // u*a + v*b with the first product fused
    return __fma_rn(u, a, mulz(v, b, nz));
}

// u*a - v*b with the first product fused
__device__ __forceinline__ double fdif(double u, double a, double v, double b, double nz)
{
    return __fma_rn(u, a, neg(mulz(v, b, nz)));
}

// Record (c,s) of rotation i (1-based).  thick[i] is the reference's layer_thickness (it
// drives the capacity rule); place[i] is the grid layer used, equal to thick[i] in reference
// mode (layer <= 0) or the sweep's common layer in exact-order mode.
__device__ __forceinline__ void record(double* grid, int32_t* thick, int32_t* place, int64_t rows,
                                       int64_t i, int32_t layer, double c, double s)
{
    const int32_t t = thick[i - 1] + 1;
    thick[i - 1] = t;
    if (layer <= 0) layer = t;
    place[i - 1] = layer;
    double* p = grid + 2 * ((i - 1) + (int64_t)(layer - 1) * rows);
    p[0] = c;
    p[1] = s;
}

// single_shift!(H, from, to, mu, givens, layer_thickness) (src/bulge_chasing.jl:11-144).
// dv/ev are 0-based arrays; from/to 1-based.  Values the sweep itself produced travel in
// registers; only untouched entries are loaded.
__device__ void single_shift(double* __restrict__ dv, double* __restrict__ ev, int64_t from,
                             int64_t to, double mu, double* __restrict__ grid,
                             int32_t* __restrict__ thick, int32_t* __restrict__ place,
                             int64_t rows, int32_t layer, double nz)
{
    const double H11 = dv[from - 1], H21 = ev[from - 1], H22 = dv[from];
    double c, s, nrm;
    givens_fast(__dsub_rn(H11, mu), H21, c, s, nrm, nz);
    const double H11p = fsum(c, H11, s, H21, nz);
    const double H21p = fdif(c, H21, s, H11, nz);
    const double H12p = fsum(c, H21, s, H22, nz);
    const double H22p = fdif(c, H22, s, H21, nz);
    const double H11pp = fsum(H11p, c, H12p, s, nz);
    const double H12pp = fdif(H12p, c, H11p, s, nz);
    const double H22pp = fdif(H22p, c, H21p, s, nz);
    dv[from - 1] = H11pp;
    dv[from] = H22pp;
    ev[from - 1] = H12pp;
    double bulge = 0.0;
    double e_next = 0.0;  // ev[i] (1-based) entering step i
    if (from + 2 <= to) {
        const double H23 = ev[from];
        bulge = mulz(s, H23, nz);
        e_next = mulz(c, H23, nz);
        ev[from] = e_next;
    }
    record(grid, thick, place, rows, from, layer, c, s);

    double p1 = H12pp;      // ev[i-1] (1-based) entering step i
    double B11 = H22pp;     // dv[i]   (1-based) entering step i
    // untouched entries for the first loop step
    double B22_n = (from + 1 <= to - 1) ? dv[from + 1] : 0.0;
    double B23_n = (from + 3 <= to) ? ev[from + 1] : 0.0;
    for (int64_t i = from + 1; i <= to - 1; ++i) {
        const double B22 = B22_n, B23 = B23_n;
        // prefetch for step i+1: dv[i+2], ev[i+2] (1-based)
        if (i + 1 <= to - 1) B22_n = dv[i + 1];
        if (i + 3 <= to) B23_n = ev[i + 1];
        givens_fast(p1, bulge, c, s, nrm, nz);
        ev[i - 2] = nrm;
        const double B21 = e_next;
        const double B11p = fsum(c, B11, s, B21, nz);
        const double B21p = fdif(c, B21, s, B11, nz);
        const double B12p = fsum(c, B21, s, B22, nz);
        const double B22p = fdif(c, B22, s, B21, nz);
        const double B11pp = fsum(B11p, c, B12p, s, nz);
        const double B12pp = fdif(B12p, c, B11p, s, nz);
        const double B22pp = fdif(B22p, c, B21p, s, nz);
        dv[i - 1] = B11pp;
        dv[i] = B22pp;
        ev[i - 1] = B12pp;
        if (i + 2 <= to) {
            bulge = mulz(s, B23, nz);
            e_next = mulz(c, B23, nz);
            ev[i] = e_next;
        }
        record(grid, thick, place, rows, i, layer, c, s);
        p1 = B12pp;
        B11 = B22pp;
    }
}

// ---- the sweep on one warp ---------------------------------------------------------------
//
// single_shift! is one dependency chain per step: (f, g) -> r = sqrt(f^2 + g^2) -> c = f/r,
// s = g/r -> the 2x2 update -> next (f, g).  On GB300 a dependent FP64 instruction costs 64
// cycles and a warp has one in flight at a time, whatever its active lanes; an FP64 result that
// an integer instruction or a shuffle reads costs 40 more.  So a step is built of few FP64
// instructions, each doing several products in different lanes:
//   the rotation on the integer pipes in every lane (givens_int.cuh),
//   level 1  p1 = m1 a1:        s B21 | s B22 | -s B11 | -s B21 | s B23 (next bulge) | -0
//   level 2  v2 = c a2 + p1:    B11'  | B12'  | B21'   | B22'   | (bulge)            | c B23
//   level 3  p3 = v2 m3:     -B11' s  | B12' s| -B21' s|        | bulge^2            |
//   level 4  v4 = oth c + p3:  B12''  | B11'' | B22''                  (oth = v2 of lane ^ 1)
//   lane (of 8)                  0    |   1   |   2    |   3    |   4                |   5
// then x = B12''^2 + bulge^2 for the next rotation: six FP64 levels.  B22'' (lane 2) and c B23
// (lane 5) are the next step's B11 and B21.  The lanes' operands are picked by bit masks: the
// same selections written as ternaries compiled to divergent branches and cost 330 cycles.
// The step's results go to memory during the next step: lane 1 stores dv, lane 2 ev, lanes 4
// and 5 the pair (c, s), one masked store.  Measured 890 to 1040 cycles per step, against 1802 for the
// two-warp Newton form this replaces and 1130 for a split over four warps with named barriers
// (the warps' FP64 instructions queue for the SM's one unit).
//
// Step i (1-based, from .. to-1) is the reference's first rotation for i = from and its loop
// body otherwise; both have the same 2x2 update.  Of the entries the reference writes and
// later overwrites within the sweep only the final ones are stored: dv[from-1 .. to-1]
// (0-based), ev[from-1 .. to-3] = the norms r of steps from+1 .. to-1 and ev[to-2] = the last
// B12''.  The grid slot of rotation i is column `layer` (ONE_LAYER: exact order) or
// thick[i-1] + 1 (the reference's placement; thick is updated by the caller after the sweep).
// Every rotation is givensAlgorithm's, correctly rounded, so the bits are the reference's.
__device__ __forceinline__ double lane_sel(uint32_t mask, double a, double b)
{
    const uint32_t lo = ((uint32_t)__double2loint(a) & mask) | ((uint32_t)__double2loint(b) & ~mask);
    const uint32_t hi = ((uint32_t)__double2hiint(a) & mask) | ((uint32_t)__double2hiint(b) & ~mask);
    return __hiloint2double((int)hi, (int)lo);
}

// x with the sign bit cleared where `keep` lacks it and flipped where `flip` has it
__device__ __forceinline__ double lane_sign(double x, uint32_t keep, uint32_t flip)
{
    return __hiloint2double((int)(((uint32_t)__double2hiint(x) & keep) ^ flip), __double2loint(x));
}

// Store forced to a predicated instruction (no branch).
__device__ __forceinline__ void st_if(double* p, double v, bool pred)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f64 [%0], %1;\n\t}"
                 ::"l"(p), "d"(v), "r"((unsigned)pred) : "memory");
}

__device__ __forceinline__ double lane_get(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// The lanes' roles (lane & 7) as masks and sign bits.
struct SweepLanes {
    uint32_t m0, m1, m2, m3, m4, m5;  // all ones in the lane of that role
    uint32_t keep1, flip1, flip3;     // signs of s in levels 1 and 3
};

__device__ __forceinline__ SweepLanes sweep_lanes()
{
    const int role = threadIdx.x & 7;
    const uint32_t sg = 0x80000000u;
    SweepLanes L;
    L.m0 = role == 0 ? ~0u : 0u;
    L.m1 = role == 1 ? ~0u : 0u;
    L.m2 = role == 2 ? ~0u : 0u;
    L.m3 = role == 3 ? ~0u : 0u;
    L.m4 = role == 4 ? ~0u : 0u;
    L.m5 = role == 5 ? ~0u : 0u;
    L.keep1 = role == 5 ? ~sg : ~0u;   // |s| times -0 is -0, so lane 5's level 2 is c B23 exactly
    L.flip1 = (role == 2 || role == 3) ? sg : 0u;
    L.flip3 = (role == 0 || role == 2) ? sg : 0u;
    return L;
}

// What a sweep carries from step to step: the next rotation's (f, g) and x = f^2 + g^2, the
// lanes' v2 and v4, and the last rotation.
struct SweepRegs {
    double f, g, x, v2, v4, c, s, r;
};

// H11, H21: dv[from], ev[from] (1-based) of the sweep's block.
__device__ __forceinline__ SweepRegs sweep_begin(double H11, double H21, double mu, double nz)
{
    SweepRegs S;
    S.f = __dsub_rn(H11, mu);
    S.g = H21;
    S.x = __dadd_rn(mulz(S.f, S.f, nz), mulz(H21, H21, nz));
    S.v4 = H11;   // lane 2's v4 is B11, lane 5's v2 is B21
    S.v2 = H21;
    S.c = S.s = S.r = 0.0;
    return S;
}

// This lane's result of the last step: lane 1 B11'', lane 2 r, lane 4 c, lane 5 s.
__device__ __forceinline__ double sweep_result(const SweepLanes& L, const SweepRegs& S)
{
    return lane_sel(L.m1, S.v4, lane_sel(L.m2, S.r, lane_sel(L.m4, S.c, S.s)));
}

// One step with the entries B22 = dv[i+1], B23 = ev[i+1] (1-based i).  `emit` puts the last
// step's result away, `fetch` starts the loads of the next step's entries.
// The order of the statements matters: the compiler keeps the shuffles and memory operations
// about where they stand, and these wait in one queue with the FP64 instructions.  96 orders were
// timed in place, all with the same results (n = 750 default solve 180 to 215 ms, eigenvalues of
// n = 1500 by multishift 52 to 58 ms, 256 small ones in a batch 60 to 74 ms); this one is best
// or near it in all three.
template <typename Emit, typename Fetch>
__device__ __forceinline__ void sweep_step(const SweepLanes& L, SweepRegs& S, double B22, double B23, double nz,
                                           Emit emit, Fetch fetch)
{
    // the lanes' operands that the entries alone give; the others are B11 or B21
    const double e1 = lane_sel(L.m1, B22, lane_sel(L.m5, -0.0, B23)), e2 = lane_sel(L.m3, B22, lane_sel(L.m5, B23, 0.0));
    const double B11 = lane_get(S.v4, 2), B21 = lane_get(S.v2, 5);
    double c, s, r;
    IntRot K;
    givens_int(S.f, S.g, S.x, c, s, r, K);
    fetch();
    emit(sweep_result(L, S));
    const double a1 = lane_sel(L.m1 | L.m4 | L.m5, e1, lane_sel(L.m2, B11, B21));
    const double a2 = lane_sel(L.m3 | L.m4 | L.m5, e2, lane_sel(L.m0, B11, B21));
    double p1 = __fma_rn(lane_sign(s, L.keep1, L.flip1), a1, nz);
    double v2 = __fma_rn(c, a2, p1);
    double p3 = __fma_rn(v2, lane_sel(L.m4, p1, lane_sign(s, ~0u, L.flip3)), nz);
    double v4 = __fma_rn(__shfl_xor_sync(0xffffffffu, v2, 1), c, p3);
    if (__any_sync(0xffffffffu, !K.in_range || K.undecided != 0u)) {
        const Rot3 o = givens_fix(S.f, S.g, K, nz);
        c = o.c; s = o.s; r = o.r;
        p1 = __fma_rn(lane_sign(s, L.keep1, L.flip1), a1, nz);
        v2 = __fma_rn(c, a2, p1);
        p3 = __fma_rn(v2, lane_sel(L.m4, p1, lane_sign(s, ~0u, L.flip3)), nz);
        v4 = __fma_rn(__shfl_xor_sync(0xffffffffu, v2, 1), c, p3);
    }
    const double f = lane_get(v4, 0), g = lane_get(p1, 4), gg = lane_get(p3, 4);
    S.x = __dadd_rn(mulz(f, f, nz), gg);
    S.v2 = v2; S.v4 = v4;
    S.f = f; S.g = g;
    S.c = c; S.s = s; S.r = r;
}

template <bool ONE_LAYER>
__device__ void sweep_warp(double* __restrict__ dv, double* __restrict__ ev, int64_t from, int64_t to,
                           double mu, double* __restrict__ grid, const int32_t* __restrict__ thick,
                           int64_t rows, int32_t layer, double nz)
{
    const int lane = threadIdx.x & 31, role = lane & 7;
    const SweepLanes L = sweep_lanes();
    const int steps = (int)(to - from);
    SweepRegs S = sweep_begin(dv[from - 1], ev[from - 1], mu, nz);
    double B22n = dv[from], B23n = 2 <= steps ? ev[from] : 0.0;
    // where this lane's result of the step before the current one goes
    double* out = role == 1 ? dv + from - 2 : role == 2 ? ev + from - 3
                                            : grid + 2 * ((from - 2) + (int64_t)(layer - 1) * rows) + (role == 5);
    const int out_step = role >= 4 ? 2 : 1;
    const bool stores = lane == 1 || lane == 2 || lane == 4 || lane == 5;
    const double *ld = dv + from + 1, *le = ev + from + 1;   // entries of step k + 1
    int32_t t_out = 0, t_cur = 0, t_next = 0;   // thick of the stored, the current and the next rotation
    if (!ONE_LAYER) t_cur = thick[from - 1];
    auto put = [&](double v, bool first, bool second) {
        double* p = out;
        if (!ONE_LAYER && role >= 4) p += (int64_t)(t_out + 1 - layer) * 2 * rows;
        st_if(p, v, stores && !first && !(role == 2 && second));   // the first rotation has no r entry
        out += out_step;
    };
#pragma unroll 1
    for (int k = 0; k < steps; ++k) {
        sweep_step(L, S, B22n, B23n, nz, [&](double v) { put(v, k == 0, k == 1); },
                   [&] {
                       B22n = k + 2 <= steps ? *ld : 0.0;
                       B23n = k + 3 <= steps ? *le : 0.0;
                       ++ld;
                       ++le;
                       if (!ONE_LAYER) t_next = k + 2 <= steps ? thick[from + k] : 0;
                   });
        t_out = t_cur;
        t_cur = t_next;
    }
    put(sweep_result(L, S), false, steps == 1);
    st_if(dv + to - 1, S.v4, lane == 2);
    st_if(ev + to - 2, S.f, lane == 0);
    __syncwarp();
}

constexpr int kScanUnroll = 8;  // chunks of 32 entries per round of the deflation scan

__device__ __forceinline__ int32_t warp_max(int32_t v)
{
    return __reduce_max_sync(0xffffffffu, v);
}

// The start of the unreduced block that ends at `to`: the largest j+1 with is_small(j), j in
// [start, to-1], or start.  kScanUnroll chunks of 32 per round: their loads are issued
// together, so a long block costs one memory latency per 32 * kScanUnroll entries.
__device__ __forceinline__ int64_t block_start(const double* dv, const double* ev, int64_t start, int64_t to,
                                               double tol)
{
    const int lane = threadIdx.x & 31;
    const int32_t xt = tol_exponent(tol);
    for (int64_t base = to - 1; base >= start; base -= 32 * kScanUnroll) {
        bool may[kScanUnroll];
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            const int64_t j = base - 32 * u - lane;
            may[u] = j >= start && maybe_small(ev[j - 1], dv[j - 1], dv[j], xt);
        }
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            if (!__any_sync(0xffffffffu, may[u])) continue;
            const int64_t j = base - 32 * u - lane;
            const unsigned mask = __ballot_sync(0xffffffffu, may[u] && is_small(dv, ev, j, tol));
            if (mask) return base - 32 * u - (__ffs(mask) - 1) + 1;
        }
    }
    return start;
}

// max(0, a[lo .. hi]) by a warp
__device__ __forceinline__ int32_t warp_range_max(const int32_t* a, int64_t lo, int64_t hi)
{
    int32_t v = 0;
#pragma unroll 8
    for (int64_t q = lo + (threadIdx.x & 31); q <= hi; q += 32) v = max(v, a[q]);
    return warp_max(v);
}

// What a sweep over [from, to] meets: the thickest column, the exact-order layer (see chase_kernel)
// and the least filled slot among its rotations' columns.
struct SweepRoom {
    int32_t thickest, layer, least;
};
__device__ __forceinline__ SweepRoom sweep_room(const int32_t* thick, const int32_t* place, int64_t from, int64_t to,
                                                int64_t n)
{
    int32_t t = 0, hi = 0, lo = INT32_MAX;
    const int32_t after = to <= n - 1 ? place[to - 1] : 0, before = from >= 2 ? place[from - 2] - 1 : 0;
#pragma unroll 4
    for (int64_t q = from - 1 + (threadIdx.x & 31); q <= to - 1; q += 32) {
        t = max(t, thick[q]);
        if (q < to - 1) {
            const int32_t p = place[q];
            hi = max(hi, p);
            lo = min(lo, p);
        }
    }
    SweepRoom r;
    r.thickest = warp_max(t);
    r.layer = 1 + max(warp_max(hi), max(after, before));
    r.least = __reduce_min_sync(0xffffffffu, lo);
    return r;
}
// The identity in the slots the jump to `layer` skips.
__device__ __forceinline__ void fill_skipped(double* grid, const int32_t* place, int64_t from, int64_t to,
                                             int32_t layer, int64_t rows)
{
    for (int64_t q = from - 1 + (threadIdx.x & 31); q <= to - 2; q += 32)
        for (int32_t g = place[q] + 1; g < layer; ++g) {
            double* p = grid + 2 * (q + (int64_t)(g - 1) * rows);
            p[0] = 1.0;
            p[1] = 0.0;
        }
}

// ---- multishift batches (chase_mode 3) -----------------------------------------------------
//
// Shifts of a batch of nb <= kMaxBulges bulges over the block [from, to] (1-based): nb
// eigenvalues of the block's trailing w x w principal submatrix, w = min(kShiftWindow * nb,
// to - from + 1), ascending -- those ranked about the bottom diagonal entry (with r the number
// of the window's eigenvalues below dv[to], the ranks k0 .. k0 + nb - 1,
// k0 = min(max(r - nb / 2, 0), w - nb)).  A window twice the batch approximates the
// eigenvalues that belong to the bottom rows better than the square of the batch's own size
// (measured in the oracle's restatement: 0.95-1.02x the reference's sweeps for case A at
// n = 4096-8192, against 1.43-1.53x).
// The window is scaled by an exact power of two to max |entry| in [0.5, 1).  The rank r and
// a bracket of each eigenvalue come from bisection on FP32 Sturm counts; the shift itself is
// then refined in FP64 by a safeguarded Newton iteration on the characteristic polynomial
// p(x) = det(T_w - x I): one pass of the three-term recurrence gives p, p' and, from the
// signs of the leading minors p_i, the FP64 Sturm count at x, which moves an FP64 bracket
// [A, B] of the eigenvalue; a Newton step that is not finite or leaves [A, B] is replaced by
// the bracket's midpoint.  The recurrence is rescaled by exact powers of two whenever the
// exponent of p_i leaves [-600, 600]: over 128 rows of a window whose diagonal lies close to
// the shift, the unscaled p_i underflows (about 1e-362 in case A), which made every Newton
// step non-finite and left the shifts at FP32 accuracy.  Warp 0 of the controller sets up the
// window (batch_shifts_setup) and each bulge's CTA solves for its own shift (bulge_shift).
constexpr int kShiftWindow = 2;
constexpr int kWinMax = kShiftWindow * kMaxBulges;

// Number of the scaled window's eigenvalues below x, from the FP32 pivots of
// T - x I = L D L^T (a negative pivot per eigenvalue below x).
__device__ __forceinline__ int window_count32(const float* sd, const float* se2, int w, float x)
{
    constexpr float kPiv = 1e-30f;
    float q = sd[0] - x;
    int cnt = q < 0.0f;
    for (int i = 1; i < w; ++i) {
        if (fabsf(q) < kPiv) q = -kPiv;
        q = (sd[i] - x) - se2[i - 1] / q;
        cnt += q < 0.0f;
    }
    return cnt;
}

// p(x), p'(x) and the number of eigenvalues below x of the scaled window, in FP64, step by step:
// dd the diagonal, nbb[i] = -e_{i-1}^2.  The windows that meet an exact zero of a leading minor.
__device__ __noinline__ void char_poly(const double* dd, const double* nbb, int w, double x, double& p, double& dp,
                                       int& below)
{
    double p0 = 1.0, p1 = dd[0] - x, q0 = 0.0, q1 = -1.0;
    int cnt = p1 < 0.0;
    for (int i = 1; i < w; ++i) {
        const double aa = dd[i] - x, nb = nbb[i];
        const double p2 = __fma_rn(aa, p1, __dmul_rn(nb, p0));
        const double q2 = __fma_rn(aa, q1, __fma_rn(nb, q0, -p1));
        // a sign change of the leading minors is an eigenvalue below x; an exact zero takes
        // the sign opposite to its predecessor's (the pivot convention of the FP32 counts)
        cnt += (p2 == 0.0) ? 1 : ((p2 < 0.0) != (p1 < 0.0));
        p0 = p1;
        p1 = (p2 == 0.0) ? -copysign(1e-300, p1) : p2;
        q0 = q1;
        q1 = q2;
        // keep p1 within 2^+-600 by exact power-of-two scaling of the whole recurrence state
        const int e = (int)((__double_as_longlong(p1) >> 52) & 0x7FF) - 1023;
        if ((e > 600 && e < 1024) || e < -600) {
            const double sc = __longlong_as_double((long long)(1023 - e) << 52);   // 2^-e, exact
            p0 *= sc;
            p1 *= sc;
            q0 *= sc;
            q1 *= sc;
        }
    }
    p = p1;
    dp = q1;
    below = cnt;
}

// Warp 0 of the controller: the scaled window into bs, its Gershgorin interval, and the rank of the
// first shift.  sd, se2, sea: kWinMax-entry shared arrays.
__device__ void batch_shifts_setup(const double* __restrict__ dv, const double* __restrict__ ev, int64_t from,
                                   int64_t to, int nb, BulgeScratch* __restrict__ bs, float* sd, float* se2, float* sea)
{
    const int lane = threadIdx.x & 31;
    constexpr int H = kWinMax / 32;
    const int w = (int)min((int64_t)kShiftWindow * nb, to - from + 1);
    const int64_t r0 = to - w;  // 0-based first row of the window
    // lane holds entries q = lane + 32 h of the window
    double dq[H], eq[H];
    double mx = 0.0;
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int q = lane + 32 * h;
        dq[h] = q < w ? dv[r0 + q] : 0.0;
        eq[h] = q < w - 1 ? ev[r0 + q] : 0.0;
        mx = fmax(mx, fmax(fabs(dq[h]), fabs(eq[h])));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (!(mx > 0.0) || !isfinite(mx)) {
        // a zero block is already diagonal; a non-finite one is left to the sweep
        for (int j = lane; j < nb; j += 32) bs->shifts[j] = dv[to - nb + j];
        if (lane == 0) bs->win_trivial = 1;
        __syncwarp();
        return;
    }
    int ex;
    frexp(mx, &ex);
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int q = lane + 32 * h;
        const double dsc = ldexp(dq[h], -ex), esc = ldexp(eq[h], -ex);
        const float ef = (float)esc;
        sd[q] = (float)dsc;
        se2[q] = ef * ef;
        sea[q] = fabsf(ef);
        if (q < w) {
            bs->win_d[q] = dsc;
            bs->win_e[q] = esc;
        }
    }
    __syncwarp();
    // Gershgorin interval of the window
    float lo = 3.0f, hi = -3.0f;
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int q = lane + 32 * h;
        if (q < w) {
            const float rad = (q >= 1 ? sea[q - 1] : 0.0f) + (q < w - 1 ? sea[q] : 0.0f);
            lo = fminf(lo, sd[q] - rad);
            hi = fmaxf(hi, sd[q] + rad);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    int k0 = 0;
    if (w > nb) k0 = min(max(window_count32(sd, se2, w, sd[w - 1]) - nb / 2, 0), w - nb);
    if (lane == 0) {
        bs->win_w = w;
        bs->win_k0 = k0;
        bs->win_ex = ex;
        bs->win_trivial = 0;
        bs->win_lo = lo - 1e-6f;
        bs->win_hi = hi + 1e-6f;
    }
    __syncwarp();
}

// A bulge's copy of the window.
struct ShiftSmem {
    float sd[kWinMax], se2[kWinMax];
    double dd[kWinMax], nbb[kWinMax + 1];      // diagonal; nbb[i] = -e_{i-1}^2, nbb[0] = 0
    double aa[kWinMax + 1], p[kWinMax + 1];    // dd - x; the leading minors at x
};

// p(x), p'(x) and the count by one warp: even lanes carry the minors, odd lanes their derivatives one
// step behind, so a step is two FP64 instructions for both (p_i = aa p_{i-1} + RN(nbb p_{i-2}),
// q_i = aa q_{i-1} + RN(nbb q_{i-2} - p_{i-1}), char_poly's operations).  The rescaling is
// checked every eight steps against 2^+-300 (a step shrinks a minor by less than 2^-105 and grows it
// by less than 4) and changes no bit of p / p'.
__device__ __forceinline__ void char_poly_warp(ShiftSmem& sm, int w, double x, double& p, double& dp, int& below)
{
    const int lane = threadIdx.x & 31;
    const bool odd = lane & 1;
    for (int i = lane; i < w; i += 32) sm.aa[i] = __dsub_rn(sm.dd[i], x);
    if (lane == 0) sm.aa[w] = 0.0;
    __syncwarp();
    const double* aa = sm.aa - odd;
    const double* bb = sm.nbb - odd;
    const uint32_t m = odd ? ~0u : 0u;
    double z0 = odd ? 0.0 : 1.0, z1 = odd ? 0.0 : sm.aa[0];
    if (lane == 0) sm.p[0] = z1;
#pragma unroll 1
    for (int s = 1; s <= w; ++s) {
        const double up = __shfl_sync(0xffffffffu, z0, lane & 30);
        const double add = lane_sel(m, lane_sign(up, ~0u, 0x80000000u), -0.0);
        const double z2 = __fma_rn(aa[s], z1, __fma_rn(bb[s], z0, add));
        z0 = z1;
        z1 = z2;
        if (lane == 0) sm.p[s] = z2;
        if ((s & 7) == 0) {
            const int hi = __shfl_sync(0xffffffffu, __double2hiint(z1), 0);
            const int e = ((hi >> 20) & 0x7FF) - 1023;
            if ((e > 300 && e < 1024) || (e < -300 && e > -1023)) {
                const double sc = __longlong_as_double((long long)(1023 - e) << 52);   // 2^-e, exact
                z0 *= sc;
                z1 *= sc;
            }
        }
    }
    __syncwarp();
    p = lane_get(z0, 0);
    dp = lane_get(z1, 1);
    int cnt = 0;
    bool zero = false;
    for (int i = lane; i < w; i += 32) {
        const double pi = sm.p[i];
        zero |= pi == 0.0;
        cnt += (pi < 0.0) != (i > 0 && sm.p[i - 1] < 0.0);
    }
    if (__any_sync(0xffffffffu, zero)) {
        char_poly(sm.dd, sm.nbb, w, x, p, dp, below);
        return;
    }
    below = __reduce_add_sync(0xffffffffu, cnt);
}

// Shift j of the batch, by one warp of bulge j's CTA, every CTA at once: FP32 bisection to a bracket,
// five levels a round (lane n of 1 .. 31 counts at the midpoint a bisection would reach at node n
// of its tree, so the path is the bisection's), then the safeguarded FP64 Newton iteration.  One
// thread per shift in the controller, 40 levels and both recurrences in sequence, took about
// 285 us for 64 shifts of a 128-row window (n = 2000 multishift solve 125 ms, 113 ms this way).
__device__ double bulge_shift(const BulgeScratch* bs, int j, ShiftSmem& sm)
{
    const int lane = threadIdx.x & 31;
    if (bs->win_trivial) return bs->shifts[j];
    const int w = bs->win_w, k = bs->win_k0 + j;
    for (int q = lane; q < w; q += 32) {
        const double d = bs->win_d[q], e = bs->win_e[q];
        const float ef = (float)e;
        sm.sd[q] = (float)d;
        sm.se2[q] = ef * ef;
        sm.dd[q] = d;
        sm.nbb[q + 1] = -(e * e);
    }
    if (lane == 0) sm.nbb[0] = 0.0;
    __syncwarp();
    float a = bs->win_lo, b = bs->win_hi;
    const int depth = 31 - __clz(lane | 1);
    for (int it = 0; it < 40; it += 5) {
        float na = a, nb = b, mid = 0.0f;
        bool valid = lane > 0;
        for (int l = 0; l <= depth; ++l) {
            mid = 0.5f * (na + nb);
            valid = valid && mid > na && mid < nb;
            if (l < depth) {
                if ((lane >> (depth - 1 - l)) & 1) na = mid;
                else nb = mid;
            }
        }
        const unsigned above = __ballot_sync(0xffffffffu, window_count32(sm.sd, sm.se2, w, mid) > k);
        const unsigned ok = __ballot_sync(0xffffffffu, valid);
        bool done = false;
        for (int l = 0, node = 1; l < 5; ++l) {
            if (!((ok >> node) & 1u)) {
                done = true;
                break;
            }
            mid = 0.5f * (a + b);
            if ((above >> node) & 1u) {
                b = mid;
                node = 2 * node;
            } else {
                a = mid;
                node = 2 * node + 1;
            }
        }
        if (done) break;
    }
    // FP64 refinement inside a bracket kept by FP64 Sturm counts
    double A = (double)a - 4e-7, B = (double)b + 4e-7;
    double x = 0.5 * ((double)a + (double)b);
    for (int it = 0; it < 5; ++it) {
        double p, dp;
        int below;
        char_poly_warp(sm, w, x, p, dp, below);
        if (below > k) B = x;
        else A = x;
        const double step = p / dp;
        // converged: a step below the last bits ends the iteration first (such a step can
        // land on the bracket's edge, which the safeguard below would turn into a jump)
        if (fabs(step) <= 4e-16 * fabs(x) + 1e-300) break;
        double xn = x - step;
        if (!(xn > A && xn < B)) xn = 0.5 * (A + B);
        x = xn;
    }
    return ldexp(x, bs->win_ex);
}

// The bulges of a batch.  Bulge j (CTA j) runs the one-warp sweep with shift shifts[j] over the
// batch's block, a few steps behind bulge j-1, reading only what bulge j-1 has stored: step k of
// a sweep stores dv[k-1] and ev[k-2] (0-based; its last step also dv[k] and ev[k-1]), so the
// entries of step i (dv[i], ev[i]) need bulge j-1 through step min(i+2, to-1).
// Three warps.  The sweep's warp (0) touches only shared memory: warp 1 fetches the entries of
// the next steps as far as bulge j-1's progress allows, warp 2 stores the results and releases
// the bulge's own progress (st.release.gpu, whose fence would hold the sweep for about 700
// cycles).  They work in chunks of `every` steps, two buffers each way, handed over by named
// barriers, each used by one producer (bar.arrive) and one consumer (bar.sync) that strictly
// alternate: full[b] before a buffer is read, empty[b] before it is written again.
// Warp 1 reads the progress word with ld.acquire.gpu only when the value it holds is too small,
// and dv/ev through L2 (ld.global.cg), never from a stale L1 line.  Bulge j waits only for bulge
// j-1 and the CTAs are co-resident (one cooperative launch), so the waits form one chain that
// starts at bulge 0, which waits for none.  Every wait on another bulge is bounded (about 2 s of
// SM clock): one that gives up sets the device error word, and the warp carries on without
// waiting, so the barriers still complete; the call then reports the error.
// `hold` (the test hook of symeig_set_test_stall, bulge 0 only) withholds every release, so
// the next bulge's wait runs out.
// With the two-warp Newton sweep that waited, loaded and stored by itself a step cost 1.15 us:
// the whole n = 2000 multishift solve took 175 ms and takes 137 ms, n = 3001 with FP32 Q and a
// random diagonal 514 and 348 ms.

__device__ __forceinline__ long long ld_acquire_gpu(const long long* p)
{
    long long v;
    asm volatile("ld.acquire.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_gpu(long long* p, long long v)
{
    asm volatile("st.release.gpu.global.s64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Every lane polls with its own acquire load, and the warp moves on together: when all lanes
// saw the value needed (it keeps their minimum, which every lane has synchronised with, the
// progress word only growing) or when any lane's wait ran out.
struct PipeWait {
    const long long* pred;  // progress word of the bulge ahead; null for bulge 0
    int* err;
    long long known;        // the smallest value the warp's lanes last read (warp-uniform)
    __device__ __forceinline__ void until(long long need)
    {
        if (pred == nullptr || known >= need) return;
        const long long t0 = clock64();
        for (;;) {
            long long v = ld_acquire_gpu(pred);
            if (__all_sync(0xffffffffu, v >= need)) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
                known = v;
                return;
            }
            const bool give_up = *(volatile int*)err != 0 || clock64() - t0 > 4000000000LL;
            if (__any_sync(0xffffffffu, give_up)) {
                if ((threadIdx.x & 31) == 0) atomicExch(err, 1);
                known = 0x7fffffffffffffffLL;  // stop waiting for the rest of the sweep
                return;
            }
        }
    }
};

constexpr int kMaxRelease = 64;   // largest chunk (symeig_set_multishift's release_every)
enum : int { kBarInFull = 1, kBarInEmpty = 3, kBarOutFull = 5, kBarOutEmpty = 7 };   // two each

__device__ __forceinline__ void nb_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void nb_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

struct BulgeRing {
    double2 in[2][kMaxRelease];       // (dv[i], ev[i]) of the chunk's steps
    double out[2][kMaxRelease][4];    // (B11'', r, c, s)
    double first[2];                  // dv[from-1], ev[from-1]
    double last[2];                   // the last step's B22'', B12''
};

__device__ __forceinline__ void bulge_sweep(BulgeRing& R, int steps, int every, double mu, double nz)
{
    const int lane = threadIdx.x & 31, role = lane & 7;
    const SweepLanes L = sweep_lanes();
    const bool stores = lane == 1 || lane == 2 || lane == 4 || lane == 5;
    const int item = role == 1 ? 0 : role == 2 ? 1 : role == 4 ? 2 : 3;
    const uint32_t out0 = (uint32_t)__cvta_generic_to_shared(&R.out[0][0][item]);
    nb_sync(kBarInFull);
    SweepRegs S = sweep_begin(R.first[0], R.first[1], mu, nz);
    uint32_t at = out0;   // where the last step's result goes
    int b = 0;
    for (int k0 = 0; k0 < steps; k0 += every, b ^= 1) {
        if (k0 > 0) nb_sync(kBarInFull + b);
        if (k0 >= 2 * every) nb_sync(kBarOutEmpty + b);
        const int len = min(every, steps - k0);
        const double2* in = R.in[b];
#pragma unroll 1
        for (int q = 0; q < len; ++q) {
            const double2 B = in[q];
            sweep_step(L, S, B.x, B.y, nz, [&](double v) {
                asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.shared.f64 [%0], %1;\n\t}"
                             ::"r"(at), "d"(v), "r"((unsigned)(stores && k0 + q > 0)) : "memory");
            }, [] {});
            if (q == 0 && k0 > 0) {
                __syncwarp();
                nb_arrive(kBarOutFull + (b ^ 1));
            }
            at = out0 + (uint32_t)((b * kMaxRelease + q) * 4 * sizeof(double));
        }
        if (k0 + 2 * every < steps) nb_arrive(kBarInEmpty + b);   // only a buffer that is filled again
    }
    if (stores) {
        const double v = sweep_result(L, S);
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
    }
    if (lane == 2) R.last[0] = S.v4;
    if (lane == 0) R.last[1] = S.f;
    __syncwarp();
    nb_arrive(kBarOutFull + (b ^ 1));
}

__device__ __forceinline__ void bulge_fetch(BulgeRing& R, const double* __restrict__ dv, const double* __restrict__ ev,
                                            int64_t from, int64_t to, int steps, int every, PipeWait pw)
{
    const int lane = threadIdx.x & 31;
    int b = 0;
    for (int k0 = 0; k0 < steps; k0 += every, b ^= 1) {
        const int len = min(every, steps - k0);
        if (k0 >= 2 * every) nb_sync(kBarInEmpty + b);
        // the chunk's last step is i = from + k0 + len - 1
        pw.until(min(from + k0 + len + 1, to - 1));
        if (k0 == 0 && lane == 0) {
            R.first[0] = __ldcg(dv + from - 1);
            R.first[1] = __ldcg(ev + from - 1);
        }
        for (int q = lane; q < len; q += 32) {
            const int64_t i = from + k0 + q;
            R.in[b][q] = make_double2(__ldcg(dv + i), i + 2 <= to ? __ldcg(ev + i) : 0.0);
        }
        __syncwarp();
        nb_arrive(kBarInFull + b);
    }
}

__device__ __forceinline__ void bulge_store(BulgeRing& R, double* __restrict__ dv, double* __restrict__ ev, int64_t from,
                                            int64_t to, double* __restrict__ grid, const int32_t* __restrict__ thick,
                                            int64_t rows, int32_t layer, int32_t jofs, int steps, int every,
                                            long long* __restrict__ my_prog, bool hold)
{
    const int lane = threadIdx.x & 31;
    int b = 0;
    for (int k0 = 0; k0 < steps; k0 += every, b ^= 1) {
        const int len = min(every, steps - k0);
        nb_sync(kBarOutFull + b);
        for (int t = lane; t < 4 * len; t += 32) {
            const int q = t >> 2, item = t & 3;
            const int64_t i = from + k0 + q;   // 1-based step
            const double v = R.out[b][q][item];
            if (item == 0) {
                dv[i - 1] = v;
            } else if (item == 1) {
                if (k0 + q > 0) ev[i - 2] = v;
            } else {
                const int32_t Lr = layer > 0 ? layer : thick[i - 1] + 1 + jofs;
                grid[2 * ((i - 1) + (int64_t)(Lr - 1) * rows) + (item - 2)] = v;
            }
        }
        if (k0 + every >= steps && lane == 0) {
            dv[to - 1] = R.last[0];
            ev[to - 2] = R.last[1];
        }
        __syncwarp();
        if (k0 + 2 * every < steps) nb_arrive(kBarOutEmpty + b);
        if (!hold && lane == 0) st_release_gpu(my_prog, from + k0 + len - 1);
    }
}

// One CTA of three warps per bulge; dynamic shared memory (kBatchSmem) keeps one CTA per SM, so
// no two bulges share an SM's FP64 unit.
constexpr int kBatchSmem = 120 * 1024;

__global__ void __launch_bounds__(96, 1)
bulge_batch_kernel(const ChaseState* __restrict__ st, double* dv, double* ev, double* __restrict__ grid,
                   const int32_t* __restrict__ thick, BulgeScratch* __restrict__ bs,
                   int* __restrict__ err)
{
    __shared__ BulgeRing ring;
    __shared__ ShiftSmem shift;
    const int j = blockIdx.x;
    if (st->status != CHASE_BATCH) return;  // a launch queued ahead after the batches ended
    const int32_t nb = st->b_bulges;
    if (j >= nb) return;
    const int64_t n = st->n, from = st->b_from, to = st->b_to;
    const int64_t rows = n > 1 ? n - 1 : 1;
    const int32_t L0 = st->b_layer0;
    const int steps = (int)(to - from), every = st->ms_prog_mask + 1;
    const int warp = threadIdx.x >> 5;
    if (warp == 0) {
        bulge_sweep(ring, steps, every, bulge_shift(bs, j, shift), st->neg_zero);
    } else if (warp == 1) {
        bulge_fetch(ring, dv, ev, from, to, steps, every, PipeWait{j > 0 ? &bs->prog[j - 1] : nullptr, err, -1});
    } else {
        bulge_store(ring, dv, ev, from, to, grid, thick, rows, L0 > 0 ? L0 + j : 0, j, steps, every, &bs->prog[j],
                    st->test_stall != 0 && j == 0);
    }
}

// One flush: the reference's inner loop from `to = last_block_ends_at` until the matrix is
// split into converged parts, every block has reached max_layers, or iter > maxiter.
// Warp 0 runs the control flow, the O(n) scans with ballots and the sweeps (sweep_warp); warp 1
// shares the O(n) updates.  In chase modes 1 and 2 every sweep runs in the
// reference form on one thread (mode 2: after the warp's sweep, undone from the copy `bak`, 2n
// doubles, of the entries it may change).
//
// Exact-order placement (st->exact_order != 0).  The reference applies a flush's grid in
// layer-major order, which equals the order the chase made the rotations only while every
// sweep meets equal layer counts on its indices; when a split block re-merges it does not,
// and the reference's Q loses accuracy.  In exact-order mode every rotation of a sweep over
// [from, to] goes to the single layer
//     L = 1 + max(place[from..to-1], place[to], place[from-1] - 1)
// and skipped slots are set to (1,0), so the layer-major order of the grid is the chase's
// order.  The chase itself (and so every eigenvalue) is the reference's.  A sweep whose layer
// would exceed the grid's capacity ends the flush early (st->early_flushes counts these).
struct Decision {
    int64_t from, to;
    double mu;
    int32_t layer;
    int32_t action;  // 0 stop, 1 sweep, 2 no sweep this iteration, 3 multishift batch
    int32_t bulges;  // action 3: sweeps of the batch
};

__global__ void __launch_bounds__(64, 1)
chase_kernel(ChaseState* __restrict__ st, double* __restrict__ dv, double* __restrict__ ev,
             double* __restrict__ grid, int32_t* __restrict__ thick, int32_t* __restrict__ place,
             double* __restrict__ bak, BulgeScratch* __restrict__ bs, int32_t resume_only)
{
    __shared__ Decision dec;
    __shared__ float ms_d[kWinMax], ms_e2[kWinMax], ms_ea[kWinMax];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int64_t n = st->n;
    const int64_t start = st->start;
    const double tol = st->tol;
    const double nz = st->neg_zero;
    const int32_t max_layers = st->max_layers;
    const int32_t grid_layers = st->grid_layers;
    const bool exact = st->exact_order != 0;
    const int64_t maxiter = st->maxiter;
    const int32_t mode = st->chase_mode;
    const int32_t ms_bulges = min(max(st->ms_bulges, 2), kMaxBulges);
    const int32_t ms_min = min(max(st->ms_min_bulges, 2), ms_bulges);
    const int64_t ms_rows = max(st->ms_rows, 4);
    int64_t iter = st->iter;
    int64_t lbe = st->last_block_ends_at;
    const int64_t rows = n > 1 ? n - 1 : 1;
    int64_t redone = 0;

    // chase_mode 3 returns to the host for each multishift batch; the launch after the batch
    // resumes the flush where it stopped, first recording the batch in thick/place: every
    // index of its block got one layer per bulge (bulge j at layer thick + 1 + j, or at the
    // exact-order layer b_layer0 + j).
    const bool resume = st->resume != 0;
    if (resume_only && !resume) return;  // a launch queued ahead after the batches ended
    if (!resume) {
        for (int64_t q = threadIdx.x; q < n; q += 64) {
            thick[q] = 0;
            place[q] = 0;
        }
    } else {
        const int32_t nbk = st->b_bulges, L0 = st->b_layer0;
        for (int64_t q = st->b_from - 1 + threadIdx.x; q < st->b_to - 1; q += 64) {
            const int32_t t = thick[q] + nbk;
            thick[q] = t;
            place[q] = L0 > 0 ? L0 + nbk - 1 : t;
        }
    }
    __syncthreads();

    bool did = resume && st->r_did != 0;
    int64_t rotations = resume ? st->r_rotations : 0, min_from = resume ? st->r_min_from : n + 1;
    int64_t max_to = resume ? st->r_max_to : 0, early = resume ? st->r_early : 0;
    int32_t status = CHASE_RUNNING;
    int64_t to = resume ? st->r_to : lbe;
    Decision last{};

    for (;;) {
        if (warp == 0) {
            Decision d{0, 0, 0.0, 0, 2, 1};
            if (iter > maxiter) {
                status = CHASE_MAXITER;
                d.action = 0;
            } else if (to <= start) {
                d.action = 0;
            } else {
                const int64_t from = block_start(dv, ev, start, to, tol);
                if (from == to) {
                    if (lane == 0) ev[from - 2] = 0.0;
                    if (to == lbe) lbe -= 1;
                    to -= 1;
                } else {
                    const SweepRoom room = sweep_room(thick, place, from, to, n);
                    const int32_t mx = room.thickest;
                    if (mx == max_layers) {
                        to = from - 1;
                    } else {
                        int32_t layer = 0;
                        bool go = true;
                        if (exact) {
                            layer = room.layer;
                            if (layer > grid_layers) {
                                early = 1;
                                go = false;
                                d.action = 0;
                            } else if (room.least < layer - 1) {
                                fill_skipped(grid, place, from, to, layer, rows);
                            }
                        }
                        if (go) {
                            // mode 3: as many bulges as the block's length, its layer room
                            // (the capacity rule of that many single sweeps) and maxiter allow
                            int64_t nbl = 1;
                            if (mode == 3) {
                                int64_t cap = (int64_t)max_layers - mx;
                                if (exact) cap = min(cap, (int64_t)grid_layers - layer + 1);
                                nbl = min(min((int64_t)ms_bulges, (to - from + 1) / ms_rows), cap);
                                nbl = min(nbl, maxiter - iter + 1);
                                // a batch too small to repay its launches and shift solve
                                // runs as one sweep with the reference's shift
                                if (nbl < ms_min) nbl = 1;
                            }
                            if (nbl >= 2) {
                                batch_shifts_setup(dv, ev, from, to, (int)nbl, bs, ms_d, ms_e2, ms_ea);
                                d.bulges = (int32_t)nbl;
                                d.action = 3;
                            } else {
                                d.mu = wilkinson_shift(dv[to - 2], dv[to - 1], ev[to - 2]);
                                d.action = 1;
                            }
                            d.from = from;
                            d.to = to;
                            d.layer = layer;
                            did = true;
                            iter += nbl >= 2 ? nbl : 1;
                            rotations += (nbl >= 2 ? nbl : 1) * (to - from);
                            min_from = min(min_from, from);
                            max_to = max(max_to, to);
                        }
                    }
                }
                if (d.action == 2 && to <= start) d.action = 0;
            }
            if (lane == 0) dec = d;
        }
        __syncthreads();
        const Decision d = dec;
        last = d;
        if (d.action == 3) {
            // the batch runs in its own launch
            break;
        }
        if (d.action == 1) {
            // entries the sweep may change: dv[from-1 .. to-1], ev[from-1 .. to-2] (0-based)
            const int64_t q0 = d.from - 1, q1 = d.to - 1;
            const bool redo = mode == 1 || mode == 2;
            if (mode == 2) {
                for (int64_t q = q0 + threadIdx.x; q <= q1; q += 64) {
                    bak[q] = dv[q];
                    if (q < q1) bak[n + q] = ev[q];
                }
                __syncthreads();
            }
            if (mode != 1) {
                if (warp == 0) {
                    if (d.layer > 0) sweep_warp<true>(dv, ev, d.from, d.to, d.mu, grid, thick, rows, d.layer, nz);
                    else sweep_warp<false>(dv, ev, d.from, d.to, d.mu, grid, thick, rows, d.layer, nz);
                }
                __syncthreads();
                if (mode == 2) {
                    for (int64_t q = q0 + threadIdx.x; q <= q1; q += 64) {
                        dv[q] = bak[q];
                        if (q < q1) ev[q] = bak[n + q];
                    }
                    ++redone;
                }
            }
            if (redo) {
                // the reference form on one thread; it updates thick/place itself
                __syncthreads();
                if (threadIdx.x == 0)
                    single_shift(dv, ev, d.from, d.to, d.mu, grid, thick, place, rows, d.layer, nz);
            } else {
                for (int64_t q = q0 + threadIdx.x; q < q1; q += 64) {
                    const int32_t t = thick[q] + 1;
                    thick[q] = t;
                    place[q] = d.layer > 0 ? d.layer : t;
                }
            }
        }
        __syncthreads();
        if (d.action == 0) break;  // both warps leave on the same decision
    }

    if (last.action == 3) {
        // hand the batch to the host: its block, its layers, and the loop state to resume
        for (int q = threadIdx.x; q < last.bulges; q += 64) bs->prog[q] = -1;
        if (threadIdx.x == 0) {
            st->status = CHASE_BATCH;
            st->resume = 1;
            st->b_bulges = last.bulges;
            st->b_from = last.from;
            st->b_to = last.to;
            st->b_layer0 = last.layer;
            st->r_did = did ? 1 : 0;
            st->r_to = to;
            st->r_rotations = rotations;
            st->r_min_from = min_from;
            st->r_max_to = max_to;
            st->r_early = early;
            st->iter = iter;
            st->last_block_ends_at = lbe;
            st->redone_sweeps += redone;
            st->batches += 1;
        }
        return;
    }
    if (warp == 0) {
        int32_t kmax = 0;
        for (int64_t q = lane; q < n; q += 32) kmax = max(kmax, place[q]);
        kmax = warp_max(kmax);
        if (lane == 0) {
            if (status == CHASE_RUNNING) status = did ? CHASE_FLUSH : CHASE_CONVERGED;
            st->status = status;
            st->iter = iter;
            st->last_block_ends_at = lbe;
            st->rotations = rotations;
            st->min_from = min_from;
            st->max_to = max_to;
            st->max_thickness = kmax;
            st->total_rotations += rotations;
            st->early_flushes += early;
            st->redone_sweeps += redone;
            st->resume = 0;
        }
    }
}

// ---- batched chase: one warp per matrix ---------------------------------------------------
//
// Each warp runs its own matrix's flush with the one-warp sweep: its six FP64 instructions per
// step (64 cycles each) leave the FP64 unit of the SM room for the warps beside it, the scans
// use all lanes, and no matrix waits for another's sweep length.  One lane per matrix, which
// this replaces, shared every FP64 instruction among 32 chases but ran the warp's longest
// sweeps and serial scans for all of them (256 matrices of n = 32 .. 320 with FP64 Q, the whole
// call: 354 ms, 79 ms with one warp per matrix).

// One flush of one matrix by one warp (the same steps, in the same order, as chase_kernel).
__device__ void chase_flush_warp(ChaseState* __restrict__ st, double* __restrict__ dv,
                                 double* __restrict__ ev, double* __restrict__ grid,
                                 int32_t* __restrict__ thick, int32_t* __restrict__ place)
{
    const int lane = threadIdx.x & 31;
    const int64_t n = st->n;
    const int64_t start = st->start;
    const double tol = st->tol;
    const double nz = st->neg_zero;
    const int32_t max_layers = st->max_layers;
    const int32_t grid_layers = st->grid_layers;
    const bool exact = st->exact_order != 0;
    const int64_t maxiter = st->maxiter;
    int64_t iter = st->iter;
    int64_t lbe = st->last_block_ends_at;
    const int64_t rows = n > 1 ? n - 1 : 1;

    for (int64_t q = lane; q < n; q += 32) {
        thick[q] = 0;
        place[q] = 0;
    }
    __syncwarp();
    bool did = false;
    int64_t rotations = 0, min_from = n + 1, max_to = 0, early = 0;
    int32_t status = CHASE_RUNNING;
    int64_t to = lbe;
    for (;;) {
        if (iter > maxiter) { status = CHASE_MAXITER; break; }
        if (to <= start) break;
        const int64_t from = block_start(dv, ev, start, to, tol);
        if (from == to) {
            if (lane == 0) ev[from - 2] = 0.0;
            __syncwarp();
            if (to == lbe) lbe -= 1;
            to -= 1;
        } else {
            const SweepRoom room = sweep_room(thick, place, from, to, n);
            if (room.thickest == max_layers) {
                to = from - 1;
            } else {
                int32_t layer = 0;
                if (exact) {
                    layer = room.layer;
                    if (layer > grid_layers) { early = 1; break; }
                    if (room.least < layer - 1) fill_skipped(grid, place, from, to, layer, rows);
                }
                const double mu = wilkinson_shift(dv[to - 2], dv[to - 1], ev[to - 2]);
                if (layer > 0) sweep_warp<true>(dv, ev, from, to, mu, grid, thick, rows, layer, nz);
                else sweep_warp<false>(dv, ev, from, to, mu, grid, thick, rows, layer, nz);
                for (int64_t q = from - 1 + lane; q < to - 1; q += 32) {
                    const int32_t t = thick[q] + 1;
                    thick[q] = t;
                    place[q] = layer > 0 ? layer : t;
                }
                __syncwarp();
                did = true;
                iter += 1;
                rotations += to - from;
                min_from = min(min_from, from);
                max_to = max(max_to, to);
            }
        }
        if (to <= start) break;
    }
    const int32_t kmax = warp_range_max(place, 0, n - 1);
    if (lane == 0) {
        if (status == CHASE_RUNNING) status = did ? CHASE_FLUSH : CHASE_CONVERGED;
        st->status = status;
        st->iter = iter;
        st->last_block_ends_at = lbe;
        st->rotations = rotations;
        st->min_from = min_from;
        st->max_to = max_to;
        st->max_thickness = kmax;
        st->total_rotations += rotations;
        st->early_flushes += early;
    }
}

constexpr int kBatchWarps = 4;   // most matrices per CTA, one on each SM sub-partition

__global__ void __launch_bounds__(32 * kBatchWarps)
chase_batched_kernel(const BatchMat* __restrict__ mats, const int32_t* __restrict__ order,
                     int32_t count, ChaseState* __restrict__ states, double* __restrict__ d,
                     double* __restrict__ e, double* __restrict__ grids,
                     int32_t* __restrict__ thick, int32_t* __restrict__ place)
{
    const int32_t k = (int32_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    if (k >= count) return;
    const int32_t i = order[k];
    ChaseState* st = states + i;
    const int32_t s0 = st->status;
    if (s0 == CHASE_CONVERGED || s0 == CHASE_MAXITER) return;
    const BatchMat mt = mats[i];
    chase_flush_warp(st, d + mt.doff, e + mt.eoff, grids + mt.goff, thick + mt.doff, place + mt.doff);
}

// get_rotation(f, g) (src/simple_givens.jl:20-23) elementwise: form 0 as the chase computes it
// (givens_int.cuh), form 1 the reference form (givens).
__global__ void get_rotation_kernel(int64_t count, const double* __restrict__ f,
                                    const double* __restrict__ g, double* __restrict__ c,
                                    double* __restrict__ s, double* __restrict__ r, int32_t form,
                                    double nz)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double fi = f[i], gi = g[i];
        double ci, si, ri;
        if (form == 1) givens(fi, gi, ci, si, ri);
        else {
            const Rot3 o = givens_any(fi, gi, nz);
            ci = o.c; si = o.s; ri = o.r;
        }
        c[i] = ci;
        s[i] = si;
        r[i] = ri;
    }
}

}  // namespace

cudaError_t launch_get_rotation(int64_t count, const double* f, const double* g, double* c,
                                double* s, double* r, int32_t form, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int64_t blocks = (count + 255) / 256 < 1216 ? (count + 255) / 256 : 1216;
    get_rotation_kernel<<<(unsigned)blocks, 256, 0, stream>>>(count, f, g, c, s, r, form, -0.0);
    return cudaGetLastError();
}

cudaError_t launch_chase(ChaseState* state, double* d, double* e, double* grid, int32_t* thick,
                         int32_t* place, double* bak, BulgeScratch* bs, int32_t resume_only,
                         cudaStream_t stream)
{
    chase_kernel<<<1, 64, 0, stream>>>(state, d, e, grid, thick, place, bak, bs, resume_only);
    return cudaGetLastError();
}

cudaError_t launch_bulge_batch(const ChaseState* state, double* d, double* e, double* grid,
                               const int32_t* thick, BulgeScratch* bs, int* err, int32_t bulges,
                               cudaStream_t stream)
{
    if (bulges < 2 || bulges > kMaxBulges) return cudaErrorInvalidValue;
    cudaError_t ce = cudaFuncSetAttribute(bulge_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kBatchSmem);
    if (ce != cudaSuccess) return ce;
    void* args[] = {(void*)&state, (void*)&d, (void*)&e, (void*)&grid, (void*)&thick, (void*)&bs, (void*)&err};
    return cudaLaunchCooperativeKernel((const void*)bulge_batch_kernel, dim3((unsigned)bulges), dim3(96), args,
                                       (size_t)kBatchSmem, stream);
}

cudaError_t launch_chase_batched(const BatchMat* mats, const int32_t* order, int32_t count,
                                 ChaseState* states, double* d, double* e, double* grids,
                                 int32_t* thick, int32_t* place, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    // One matrix per SM while there are enough SMs (chases on one SM queue for its FP64 unit: 16 of
    // n = 50 .. 250 31.3 against 32.1 ms).  From there four, so that the round's apply beside
    // it has SMs of its own (256 of n = 200 .. 256, FP64 Q: 68.5 ms, 77.2 with two per CTA).
    const int32_t warps = count <= 152 ? 1 : kBatchWarps;
    chase_batched_kernel<<<(unsigned)((count + warps - 1) / warps), 32 * warps, 0, stream>>>(mats, order, count, states, d,
                                                                                            e, grids, thick, place);
    return cudaGetLastError();
}

}  // namespace symeig
