// givens.cuh -- LinearAlgebra.givensAlgorithm (LAPACK 3.2 DLARTG port, called by get_rotation,
// src/simple_givens.jl:20-23) on the device, in forms that give identical bits:
//
//   givens()        the reference form, branch by branch, with __dsqrt_rn / __ddiv_rn;
//   givens_fast()   the same with its branch tests on the integer pipe;
//   givens_int()    (givens_int.cuh) the plain branch (the one a bulge chase takes) in fixed
//                   point on the integer pipes.
//
// On GB300 an FP64 instruction holds its warp for ~64 cycles and FP64 compares count as FP64
// instructions, so the branch tests are done on bit patterns.
#pragma once
#include <cstdint>

namespace symeig {
namespace gv {

// ---- bit-pattern tests on the integer pipe ----------------------------------------------
__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ uint64_t abs_bits(double x) { return bits(x) & 0x7FFFFFFFFFFFFFFFull; }
__device__ __forceinline__ bool nan_bits(uint64_t a) { return a > 0x7FF0000000000000ull; }
__device__ __forceinline__ double neg(double x) { return from_bits(bits(x) ^ 0x8000000000000000ull); }
__device__ __forceinline__ double neg_if(double x, bool p)
{
    return from_bits(bits(x) ^ (p ? 0x8000000000000000ull : 0ull));
}
// x < 0.0
__device__ __forceinline__ bool is_negative(double x)
{
    const uint64_t b = bits(x), a = b & 0x7FFFFFFFFFFFFFFFull;
    return (b >> 63) != 0 && a != 0 && !nan_bits(a);
}
// a*b as an FMA with a -0.0 addend supplied at run time: bit-identical to the product, and an
// FP64 FMA issues faster than an FP64 multiply on GB300.
__device__ __forceinline__ double mulz(double a, double b, double nz) { return __fma_rn(a, b, nz); }

__device__ __forceinline__ double jl_max(double a, double b) { return (a > b || a != a) ? a : b; }

// Which branch of givensAlgorithm (f, g) takes: 0 g == 0, 1 f == 0, 2 scaled down,
// 3 scaled up, 4 plain (also when f or g is NaN: the NaN scale fails both range tests).
__device__ __forceinline__ int givens_case(double f, double g)
{
    const uint64_t af = abs_bits(f), ag = abs_bits(g);
    if (ag == 0) return 0;
    if (af == 0) return 1;
    if (nan_bits(af) || nan_bits(ag)) return 4;
    const uint64_t m = af > ag ? af : ag;
    if (m >= 0x5E40000000000000ull) return 2;  // max(|f|,|g|) >= 2^485
    if (m <= 0x21A0000000000000ull) return 3;  // max(|f|,|g|) <= 2^-485
    return 4;
}

// The sign convention of givensAlgorithm: flip (c, s, r) when |f| > |g| and c < 0.
__device__ __forceinline__ bool givens_flip(double f, double g, double c)
{
    const uint64_t af = abs_bits(f), ag = abs_bits(g);
    return af > ag && !nan_bits(af) && !nan_bits(ag) && is_negative(c);
}

// LinearAlgebra.givensAlgorithm, branch by branch.
__device__ __forceinline__ void givens(double f, double g, double& cs, double& sn, double& r)
{
    const double safmn2 = 0x1p-485;
    const double safmx2 = 0x1p+485;
    if (g == 0.0) {
        cs = 1.0; sn = 0.0; r = f;
    } else if (f == 0.0) {
        cs = 0.0; sn = 1.0; r = g;
    } else {
        double f1 = f, g1 = g;
        double scale = jl_max(fabs(f1), fabs(g1));
        if (scale >= safmx2) {
            int count = 0;
            do {
                ++count;
                f1 = __dmul_rn(f1, safmn2); g1 = __dmul_rn(g1, safmn2);
                scale = jl_max(fabs(f1), fabs(g1));
            } while (scale >= safmx2 && count < 20);
            r = __dsqrt_rn(__dadd_rn(__dmul_rn(f1, f1), __dmul_rn(g1, g1)));
            cs = __ddiv_rn(f1, r); sn = __ddiv_rn(g1, r);
            for (int i = 0; i < count; ++i) r = __dmul_rn(r, safmx2);
        } else if (scale <= safmn2) {
            int count = 0;
            do {
                ++count;
                f1 = __dmul_rn(f1, safmx2); g1 = __dmul_rn(g1, safmx2);
                scale = jl_max(fabs(f1), fabs(g1));
            } while (scale <= safmn2 && count < 64);  // 64 steps cover every subnormal
            r = __dsqrt_rn(__dadd_rn(__dmul_rn(f1, f1), __dmul_rn(g1, g1)));
            cs = __ddiv_rn(f1, r); sn = __ddiv_rn(g1, r);
            for (int i = 0; i < count; ++i) r = __dmul_rn(r, safmn2);
        } else {
            r = __dsqrt_rn(__dadd_rn(__dmul_rn(f1, f1), __dmul_rn(g1, g1)));
            cs = __ddiv_rn(f1, r); sn = __ddiv_rn(g1, r);
        }
        if (fabs(f) > fabs(g) && cs < 0.0) { cs = -cs; sn = -sn; r = -r; }
    }
}

// givensAlgorithm with its branch tests on the integer pipe and its products issued as FMAs.
__device__ __forceinline__ void givens_fast(double f, double g, double& cs, double& sn, double& r,
                                            double nz)
{
    if (givens_case(f, g) != 4) {
        givens(f, g, cs, sn, r);
        return;
    }
    r = __dsqrt_rn(__dadd_rn(mulz(f, f, nz), mulz(g, g, nz)));
    cs = __ddiv_rn(f, r);
    sn = __ddiv_rn(g, r);
    if (givens_flip(f, g, cs)) { cs = neg(cs); sn = neg(sn); r = neg(r); }
}

// the hardware's 1/sqrt(x), relative error about 2^-20 (measured), its low word zero
__device__ __forceinline__ double rsqrt_seed(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

}  // namespace gv
}  // namespace symeig
