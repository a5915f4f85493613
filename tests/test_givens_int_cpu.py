"""The fixed-point rotation (givens_int.cuh) compiled for the host (no GPU), with seeds of every error that its
range test lets through: whatever 1/sqrt seed the hardware gives, the results are givensAlgorithm's, correctly
rounded, or the range test turns the pair away."""
from __future__ import annotations

import shutil
import subprocess
import sys

import pytest

PROGRAM = r'''
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
using std::fabs; using std::max; using std::min;
static inline long long __double_as_longlong(double x) { long long b; std::memcpy(&b, &x, 8); return b; }
static inline double __longlong_as_double(long long b) { double x; std::memcpy(&x, &b, 8); return x; }
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static inline double __hiloint2double(int h, int l) { return __longlong_as_double((long long)(((uint64_t)(uint32_t)h << 32) | (uint32_t)l)); }
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __dsqrt_rn(double a) { return std::sqrt(a); }
static inline double __ddiv_rn(double a, double b) { return a / b; }
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline int32_t __mulhi(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32); }
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)((((uint64_t)hi << 32) | lo) >> s); }
#define rsqrt_seed hardware_seed
#include "givens.cuh"
#undef rsqrt_seed
static double seed_error;   // relative, before the low word is cut off as the hardware leaves it
namespace symeig { namespace gv {
inline double rsqrt_seed(double x)
{
    return from_bits(bits((double)((1.0L + seed_error) / sqrtl((long double)x))) & 0xFFFFFFFF00000000ull);
}
} }
#include "givens_int.cuh"
using namespace symeig::gv;
int main()
{
    std::mt19937_64 gen(5);
    std::uniform_real_distribution<double> u(0.0, 1.0), w(-1.0, 1.0);
    long wrong = 0, pairs = 0;
    // the error e of X y0^2 is about twice the seed's; the range test asks |e| < 2^-18
    for (double top : {0x1p-24, 0x1p-21, 0x1p-20, 0.8 * 0x1p-19, 0.99 * 0x1p-19, 1.5 * 0x1p-19}) {
        long in = 0;
        for (int k = 0; k < 400000; ++k, ++pairs) {
            seed_error = k & 1 ? top * w(gen) : (k & 2 ? top : -top) * (1.0 - 0.01 * u(gen));
            double f = std::ldexp(1.0 + u(gen), (int)(gen() % 41) - 20), g = std::ldexp(1.0 + u(gen), (int)(gen() % 41) - 20);
            if (k % 5 == 0) g = f * (1.0 + 0x1p-52 * (double)((int)(gen() % 13) - 6));   // c, s near sqrt(1/2)
            if (k % 7 == 0) { f = 3.0 * std::ldexp(1.0, k % 9); g = f / 3.0 * 4.0; }     // exact quotients
            if (gen() & 1) f = -f;
            if (gen() & 1) g = -g;
            IntRot K;
            double c, s, r, rc, rs, rr;
            givens_int(f, g, f * f + g * g, c, s, r, K);
            in += K.in_range;
            const Rot3 o = givens_any(f, g, -0.0);
            givens(f, g, rc, rs, rr);
            wrong += bits(o.c) != bits(rc) || bits(o.s) != bits(rs) || bits(o.r) != bits(rr);
        }
        if (in == 0) ++wrong;   // the fixed-point form itself has to run at every error
    }
    std::printf("%ld of %ld\n", wrong, pairs);
    return wrong != 0;
}
'''


def test_every_seed_of_the_range_test(pkg, tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    b = sys.modules[pkg.__name__ + ".build"]
    src, exe = tmp_path / "seed.cpp", tmp_path / "seed"
    src.write_text(PROGRAM)
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(b.CSRC), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
