// givens_int.cuh -- givensAlgorithm's plain branch (src/simple_givens.jl:20-23) with the square
// root and the two quotients on the integer pipes.
//
// On GB300 a dependent FP64 instruction costs 64 cycles, a 32-bit integer one 4 to 5 and a
// 32 x 32 -> 64-bit multiply-add about 5.  Newton steps in FP64 are a chain of ten instructions
// after x = f^2 + g^2 (719 cycles measured); here one table seed (18
// cycles) and fixed-point arithmetic on 64-bit integers give r = RN(sqrt x), c = RN(f/r) and
// s = RN(g/r) in 307 cycles, each from an interval that holds the exact value.  Where an
// interval straddles a rounding boundary (3.8 % of the rotations of a chase) givens_exact
// decides by the exact remainder, so the results are always the correctly rounded ones.
//
// Method.  x = 2^(2k) X, X in [1, 4) with 54 bits; y = 1/sqrt(X) in (1/2, 1], R = sqrt(X) = X y.
//   y0  the hardware's seed (rsqrt.approx.ftz.f64, 21 bits), e = 1 - X y0^2, |e| < 2^-18 (tested: a
//       seed further off takes the reference form),
//   y   = y0 (1 + e/2 + 3/8 e^2 + 5/16 e^3), the binomial series of (1 - e)^(-1/2); the next
//         term is below 2^-73.
// All products are exact integers or truncated towards a known side.  In units of 2^-64,
//   0 <= 1/sqrt(X) - y < 3:  e is truncated at 2^-67 (1/16 of a unit), e^2 enters with E = e
//   truncated at 2^-49 and is itself truncated at 2^-66, the two terms at 2^-68 (together below
//   0.6), the sum at 2^-64 (1), and one unit is subtracted so that the side is known (and X = 1
//   does not wrap).
// In units of 2^-62, 0 <= sqrt(X) - R < 3 X/4 + 2 <= 5 (R the product X y less at most 2 for
//   its truncations); kWinR = 6.
// c: with D = r - R (|D| <= 2^9 units of 2^-62) and C0 = F y, F = |f|'s significand,
//   F/r = C0 - C0 y D up to second order (2^-104).  In units of 2^-63 C0 is short by less than
//   F 3/2 + 2 <= 5, and C0 y D exceeds its value by less than 2 C0 y (3 X/4 + 2) = F (1.5 + 4/X)
//   <= 11 (D is too large by R's shortfall), plus 2 for truncations: below 18; kWinC = 20.
// A host model of these steps against 113-bit arithmetic (6e6 random and structured pairs)
// measured [0.99, 2.27] for y, [0.29, 3.92] for R and [1.2, 14.1] for c and s.
#pragma once
#include "givens.cuh"

namespace symeig {
namespace gv {

constexpr uint32_t kWinR = 6, kWinC = 20;

__device__ __forceinline__ uint32_t lo32(uint64_t v) { return (uint32_t)v; }
__device__ __forceinline__ uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }
__device__ __forceinline__ uint64_t mulw(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
// the 53-bit significand of a normal number's bits
__device__ __forceinline__ uint64_t significand(uint64_t b)
{
    return (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
}

// floor(a b / 2^64) or one less (the lowest partial product is left out)
__device__ __forceinline__ uint64_t mulhi64(uint64_t a, uint64_t b)
{
    const uint64_t p1 = mulw(lo32(a), hi32(b));
    const uint64_t p2 = mulw(hi32(a), lo32(b)) + lo32(p1);
    return mulw(hi32(a), hi32(b)) + hi32(p1) + hi32(p2);
}

// The fixed-point form's range, from the high words: max(|f|, |g|) in [2^-450, 2^450) and
// min >= 2^-400 max by the exponent fields (so f, g are nonzero and finite, givensAlgorithm takes
// its plain branch, x and r are normal and |c|, |s| >= 2^-401).
__device__ __forceinline__ bool in_range_hi(uint32_t fh, uint32_t gh)
{
    const uint32_t ef = (fh >> 20) & 0x7FFu, eg = (gh >> 20) & 0x7FFu;
    const uint32_t mx = max(ef, eg), mn = min(ef, eg);
    return mx - 573u <= 899u && mn + 400u >= mx;
}

// What givens_int leaves for givens_exact.
struct IntRot {
    uint64_t X, y, R, Cf, Cg;
    uint32_t kr;         // biased exponent of r
    uint32_t undecided;  // nonzero: an interval straddles a rounding boundary
    bool in_range;
};

// The sign convention: flip (c, s, r) when |f| > |g| and f < 0 (then c = f/r < 0).
__device__ __forceinline__ uint32_t flip_sign(uint64_t fb, uint64_t gb)
{
    const uint64_t af = fb & 0x7FFFFFFFFFFFFFFFull, ag = gb & 0x7FFFFFFFFFFFFFFFull;
    return af > ag ? hi32(fb) & 0x80000000u : 0u;
}

// q = RN(a / r) from C0 = |a|'s significand times y, D and kr.  EXACT decides a straddling
// interval by the sign of a - (midpoint) r, an integer far below 2^63 (Mr: r's significand);
// else `undecided` collects it.
template <bool EXACT>
__device__ __forceinline__ double quot_int(uint64_t ab, uint64_t Mr, uint32_t yh, int32_t D, uint32_t kr,
                                           uint32_t flip, uint64_t C0, uint32_t& undecided)
{
    const uint32_t T = __umulhi(hi32(C0), yh);                       // C0 y, units 2^-31
    const int64_t corr = ((int64_t)T * (int64_t)D) >> 30;            // C0 y D, units 2^-63
    const uint64_t C = C0 - (uint64_t)corr - 1;
    const uint32_t big = hi32(C) >> 31;                              // quotient >= 1: round at bit 11
    const uint32_t half = 512u << big;
    const uint64_t Cr = C + half;
    const uint32_t straddle = ((lo32(Cr) & (2 * half - 1)) + kWinC) & (2 * half);
    uint64_t M = Cr >> (10u + big);
    if (EXACT) {
        const int64_t d = (int64_t)((significand(ab) << (54u - big)) - (2 * M + 1) * Mr);
        if (straddle && d > 0) M += 1;
    } else {
        undecided |= straddle;
    }
    const uint32_t ef = ((uint32_t)(ab >> 52) & 0x7FFu) - kr + 1021u + big;
    const uint32_t sign = (hi32(ab) & 0x80000000u) ^ flip;
    return __hiloint2double((int)(((ef << 20) + hi32(M)) | sign), (int)lo32(M));
}

// (c, s, r) of givensAlgorithm(f, g), x = RN(RN(f f) + RN(g g)), sign convention applied.  The
// results hold where K.in_range and K.undecided == 0; givens_fix gives them elsewhere.
__device__ __forceinline__ void givens_int(double f, double g, double x, double& c, double& s, double& r, IntRot& K)
{
    const uint64_t fb = bits(f), gb = bits(g), xb = bits(x);
    const uint32_t xh = hi32(xb);
    const uint32_t ex = xh >> 20;
    const uint32_t p = ~ex & 1u;                                     // odd exponent: X in [2, 4)
    const uint32_t kr = (ex + 1023u) >> 1;
    const uint64_t X = (((uint64_t)((xh & 0xFFFFFu) | 0x100000u) << 32) | lo32(xb)) << p;
    const uint32_t Xl = lo32(X), Xh = hi32(X);
    // y0 2^21, linear in the seed's bits so that y0 = 1 (and a seed just below 1/2) are covered
    const uint32_t y0 = (uint32_t)__double2hiint(rsqrt_seed(x)) + ((kr - 2044u) << 20);
    const uint64_t A = mulw(y0, y0);
    const uint64_t t0 = mulw(Xl, lo32(A));
    const uint64_t t1 = mulw(Xl, hi32(A)) + hi32(t0);
    const uint64_t t2 = mulw(Xh, lo32(A)) + t1;
    const uint32_t t2l = lo32(t2), t2h = hi32(t2) + Xh * hi32(A);
    // X y0^2 = (1 - e) 2^94 in units of 2^-94; e modulo 2^64 in units of 2^-67
    const uint32_t eql = ~__funnelshift_l(lo32(t0), t2l, 5);
    const int32_t eqh = (int32_t)~__funnelshift_l(t2l, t2h, 5);
    K.in_range = ((uint32_t)(eqh + 0x20000) & 0xFFFC0000u) == 0u &&  // |e| < 2^-18
                 in_range_hi(hi32(fb), hi32(gb));
    const int32_t E = (int32_t)__funnelshift_r(eql, (uint32_t)eqh, 18);
    const int32_t e2 = __mulhi(E, E);
    const int32_t e3 = __mulhi(e2, E);
    // units 2^-68; 0 <= e2 <= 2^30, so 3 e2 needs the unsigned word
    const int32_t qs = (int32_t)((3u * (uint32_t)e2) >> 1) + (((e3 >> 4) * 5) >> 15);
    const int64_t w = (int64_t)mulw(eql, y0) + (int64_t)qs * (int64_t)(int32_t)y0;
    const int64_t v = (int64_t)eqh * (int64_t)(int32_t)y0 + (int64_t)((uint64_t)(y0 << 4) << 32);
    const uint64_t y = ((uint64_t)v << 7) + (uint64_t)(w >> 25) - 1;
    K.X = X;
    K.y = y;
    K.kr = kr;
    K.R = mulhi64(X << 10, y);
    K.Cg = mulhi64(significand(gb) << 11, y);
    K.Cf = mulhi64(significand(fb) << 11, y);
    const uint64_t Rr = K.R + 512;
    const uint32_t low = lo32(Rr) & 1023u;
    K.undecided = (low + kWinR) & 1024u;
    const int32_t D = 512 - (int32_t)low;
    const uint32_t flip = flip_sign(fb, gb);
    const uint64_t M = Rr >> 10;
    s = quot_int<false>(gb, M, hi32(y), D, kr, flip, K.Cg, K.undecided);
    c = quot_int<false>(fb, M, hi32(y), D, kr, flip, K.Cf, K.undecided);
    r = __hiloint2double((int)((((kr - 1u) << 20) + hi32(M)) | flip), (int)lo32(M));
}

struct Rot3 {
    double c, s, r;
};

// The undecided rotations: the same intervals, each straddling one resolved by the exact
// remainder (modulo 2^64, where its sign is known to survive).
static __device__ __noinline__ Rot3 givens_exact(double f, double g, uint64_t X, uint64_t y, uint64_t R,
                                                 uint64_t Cf, uint64_t Cg, uint32_t kr)
{
    const uint64_t fb = bits(f), gb = bits(g);
    const uint64_t Rr = R + 512;
    const uint32_t low = lo32(Rr) & 1023u;
    uint64_t M = Rr >> 10;
    int32_t D = 512 - (int32_t)low;
    if ((low + kWinR) & 1024u) {
        // sqrt(X) against the midpoint M + 1/2 (units 2^-52): X 2^54 - (2 M + 1)^2
        const int64_t d = (int64_t)((X << 54) - (2 * M + 1) * (2 * M + 1));
        if (d > 0) {
            M += 1;
            D += 1024;
        }
    }
    const uint32_t flip = flip_sign(fb, gb);
    uint32_t unused = 0;
    Rot3 o;
    o.r = __hiloint2double((int)((((kr - 1u) << 20) + hi32(M)) | flip), (int)lo32(M));
    o.c = quot_int<true>(fb, M, hi32(y), D, kr, flip, Cf, unused);
    o.s = quot_int<true>(gb, M, hi32(y), D, kr, flip, Cg, unused);
    return o;
}

// The rotations out of the fixed-point form's range: the reference form.
static __device__ __noinline__ Rot3 givens_outside(double f, double g, double nz)
{
    Rot3 o;
    givens_fast(f, g, o.c, o.s, o.r, nz);
    return o;
}

__device__ __forceinline__ Rot3 givens_fix(double f, double g, const IntRot& K, double nz)
{
    return K.in_range ? givens_exact(f, g, K.X, K.y, K.R, K.Cf, K.Cg, K.kr) : givens_outside(f, g, nz);
}

// givensAlgorithm(f, g) as the chase computes it.
__device__ __forceinline__ Rot3 givens_any(double f, double g, double nz)
{
    Rot3 o;
    IntRot K;
    givens_int(f, g, __dadd_rn(mulz(f, f, nz), mulz(g, g, nz)), o.c, o.s, o.r, K);
    if (!K.in_range || K.undecided) o = givens_fix(f, g, K, nz);
    return o;
}

}  // namespace gv
}  // namespace symeig
