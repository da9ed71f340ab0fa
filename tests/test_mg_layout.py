"""The layout of a multigrid level in shared memory and the length of the buffer that keeps a copy
of it, compiled for the host from the header that the kernels use: every flat index of an odd row
pitch falls inside the length, each on an element of its own, with the colours apart, for odd and
even sides (an odd nx with an even ny has one element of padding beyond (nx + 4)(ny + 3) nodes)."""
import subprocess

from jd_lepic_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "mg_layout.h"
int main() {
    for (int nx = 1; nx <= 70; nx++)
        for (int ny = 1; ny <= 70; ny++) {
            const int RP = mg_pitch(nx + 3), RH = ny + 3, PS = mg_plane(RP, RH);
            const long long len = mg_level_len(nx, ny);
            if (RP < nx + 3 || !(RP & 1) || len < 2ll * PS || len < (long long)RP * RH) { printf("%d %d\n", nx, ny); return 1; }
            std::vector<char> used((size_t)len, 0);
            for (int j = 0; j < RH; j++)
                for (int i = 0; i < RP; i++) {
                    const int q = i + j * RP, t = (q & 1) * PS + (q >> 1);
                    if (t >= len || used[t]++ || (q & 1) != ((i + j) & 1)) { printf("%d %d %d %d\n", nx, ny, i, j); return 1; }
                }
        }
    // the case that a length of (nx + 3)(ny + 3) + ny + 3 is one short of
    return mg_level_len(3, 2) == 36 && mg_level_len(33, 20) == 852 ? 0 : 2;
}
"""


def test_level_length(tmp_path):
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
