"""The host rules of the fused-wave apply (no GPU): for every row count and layer count each pass's
shape exists and holds the pass's layers, and the table and segment-state scratch, which are sized
without knowing the shape, hold what any launch needs."""
from __future__ import annotations

import subprocess
import sys

PROGRAM = r'''
#include "apply_fused.cuh"
#include <cstdio>
using namespace symeig;
using namespace symeig::fused;
static long bad = 0;
template <typename T> void check(int64_t m, int64_t layers, int64_t n)
{
    const Choice c = choose<T>(m, layers);
    const size_t have = fused_table_bytes<T>(n, layers);
    if (c.per < 1) ++bad;
    for (int64_t left = layers; left > 0; left -= c.per) {
        const int64_t l = left < c.per ? left : c.per;
        const Choice q = choose<T>(m, l, true);
        with_shape<T>(q, [&](auto s) {
            using S = decltype(s);
            const Launch L = launch_of(m, S::RPW, S::MAX_WARPS);
            if (S::G != q.G || S::KB != q.KB || S::F != q.F || S::LAYERS < l) ++bad;
            if ((size_t)S::table_bytes(n) > have) ++bad;
            if (L.warps < 1 || L.warps > S::MAX_WARPS || (int64_t)L.blocks * L.warps * S::RPW < m) ++bad;
            // every column is read and finished by the last iteration
            if (S::F * (S::iterations(n) - 1 - (int64_t)(S::G - 1) * S::D) - S::KB + S::F - 1 < n - 1) ++bad;
            return 0;
        });
    }
    if (layers <= 64)
        with_segmented<T>(choose_segmented<T>(m, layers), [&](auto s) {
            using S = decltype(s);
            const Launch L = launch_of(m, S::RPW, S::MAX_WARPS);
            if (S::LAYERS < layers || (size_t)S::table_bytes(n) > have) ++bad;
            if ((size_t)L.blocks * 32 * L.warps * S::STATE * sizeof(T) > fused_state_bytes<T>(m)) ++bad;
            return 0;
        });
}
int main()
{
    for (int64_t m = 1; m < 60000; m += 1 + m / 9)
        for (int64_t k = 1; k <= 700; k += k < 300 ? 1 : 37)
            for (int64_t n : {2, 3, 77, 1000}) {
                check<double>(m, k, n);
                check<float>(m, k, n);
            }
    std::printf("%ld\n", bad);
    return bad != 0;
}
'''


def test_shapes_and_scratch(pkg, tmp_path):
    b = sys.modules[pkg.__name__ + ".build"]
    src, exe = tmp_path / "rules.cu", tmp_path / "rules"
    src.write_text(PROGRAM)
    r = subprocess.run([b.nvcc(), *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-O1", "-I", str(b.CSRC),
                        "-I", str(b.ROOT / "include"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (r.returncode, r.stdout.strip()) == (0, "0")
