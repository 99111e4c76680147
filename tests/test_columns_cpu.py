"""The adjoint's column kernels (csrc/fr_columns.h) give every voxel to exactly one thread, in all three
arrangements of a block's columns, on the CPU: extents around the arrangements' limits, row pitches
with and without padding, column depths that divide the extent and that do not."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastreg_gb300" / "csrc"

CHECK = r"""
#include "fr_columns.h"
#include <cstdio>
#include <vector>
int main() {
    const int xs[] = {2, 3, 4, 5, 11, 16, 31, 32, 33, 64, 65, 128, 257}, ys[] = {2, 4, 7, 8, 9, 32, 33, 64, 130};
    const int zs[] = {2, 3, 8, 17, 40};
    int seen_kind = 0;
    for (int X : xs)
        for (int Y : ys)
            for (int Z : zs)
                for (int pitch : {X, (X + 3) / 4 * 4})
                    for (int depth : {1, 2, 6, 16}) {
                        frg::Columns C(pitch, X, Y);
                        C.depth = depth;
                        seen_kind |= 1 << C.shape;
                        auto place = [&](int b, int t, int& x, int& y, int& z0, int& z1) {
                            if (C.shape == frg::kTileColumns) C.place<frg::kTileColumns>(b, t, Z, x, y, z0, z1);
                            else if (C.shape == frg::kFlatColumns) C.place<frg::kFlatColumns>(b, t, Z, x, y, z0, z1);
                            else C.place<frg::kLayeredColumns>(b, t, Z, x, y, z0, z1);
                        };
                        std::vector<char> seen((size_t)X * Y * Z, 0);
                        for (int b = 0; b < C.blocks(Z); ++b)
                            for (int t = 0; t < 256; ++t) {
                                int x, y, z0, z1;
                                place(b, t, x, y, z0, z1);
                                if (x < 0 || y < 0 || z0 < 0 || z1 > Z) return std::printf("outside\n"), 1;
                                int x0, y0, a0, a1;  // a warp's lanes share their slices
                                place(b, t & ~31, x0, y0, a0, a1);
                                if (a0 != z0 || a1 != z1) return std::printf("a warp of two layers\n"), 1;
                                if (x >= X || y >= Y) continue;
                                for (int z = z0; z < z1; ++z)
                                    if (seen[x + (size_t)X * (y + (size_t)Y * z)]++) return std::printf("twice\n"), 1;
                            }
                        for (char c : seen)
                            if (!c) return std::printf("%d %d %d: a voxel without a thread\n", X, Y, Z), 1;
                    }
    return seen_kind == 7 ? 0 : (std::printf("arrangements %d\n", seen_kind), 1);
}
"""


def test_every_voxel_has_one_thread(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "columns.cpp").write_text(CHECK)
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", str(CSRC), str(tmp_path / "columns.cpp"), "-o",
                    str(tmp_path / "columns")], check=True)
    r = subprocess.run([str(tmp_path / "columns")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
