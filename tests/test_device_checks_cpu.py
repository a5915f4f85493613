"""The address test of the checked build (wave::offset_in_extent), on the host: it holds for every element of a
pass's extent in both layouts and fails for the addresses that a wrong row, column, stride or lane would give."""
from __future__ import annotations

import subprocess
import sys

PROGRAM = r'''
#include "wave_common.cuh"
#include <cstdio>
using symeig::wave::offset_in_extent;
int main()
{
    long bad = 0;
    for (int64_t m : {1, 7, 33}) for (int64_t n : {2, 20, 65}) for (int64_t pad : {1, 3, 40}) {
        // column-major with leading dimension m + pad, and the transposed view of the row rotations
        const int64_t layout[2][2] = {{m + pad, 1}, {1, n + pad}};
        for (const auto& l : layout) {
            const int64_t ldq = l[0], rs = l[1];
            auto at = [&](int64_t row, int64_t col) { return offset_in_extent(row * rs + col * ldq, ldq, rs, m, n); };
            for (int64_t r = 0; r < m; ++r)
                for (int64_t c = 0; c < n; ++c) bad += !at(r, c);
            for (int64_t c = 0; c < n; ++c) bad += at(m, c);                    // the row past the last
            for (int64_t r = 0; r < m; ++r) bad += at(r, n);                    // the column past the last
            bad += at(-1, 0) + at(0, -1) + at(m, n);
            bad += offset_in_extent(n * (m + pad) * (n + pad), ldq, rs, m, n);  // another stride altogether
        }
    }
    std::printf("%ld\n", bad);
    return bad != 0;
}
'''


def test_address_test(pkg, tmp_path):
    b = sys.modules[pkg.__name__ + ".build"]
    src, exe = tmp_path / "extent.cu", tmp_path / "extent"
    src.write_text(PROGRAM)
    r = subprocess.run([b.nvcc(), *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(b.CSRC),
                        "-I", str(b.ROOT / "include"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (r.returncode, r.stdout.strip()) == (0, "0")
