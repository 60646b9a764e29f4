"""G2P's test whether a particle's stencils lie in the shared-memory tile (g2p_box.h), compiled for the host with overflow
checks: the integers that far and infinite positions saturate to are outside every tile, without an overflow."""
import os
import subprocess

from slosh_b200 import build

SOURCE = """
#include <climits>
#include <cstdio>
#include "g2p_box.h"
static bool tile_axis(int b0, int b1, int o, int n, int (&at)[2]) {
    at[0] = slosh::tile_place(b0, o);
    at[1] = slosh::tile_place(b1, o);
    return slosh::tile_holds(at[0], at[1], n);
}
int main() {
    const int far[] = {INT_MIN, -2147483520, -1073741824, 1073741824, 2147483520, INT_MAX}, near[] = {-1073741823, -5, 4000, 1073741823};
    const int origins[] = {0, 1, 7, 2040}, sizes[] = {3, 8, 40};
    int bad = 0;
    for (int o : origins)
        for (int n : sizes) {
            int at[2];
            for (int b : far) bad += tile_axis(b, b, o, n, at);
            for (int b : near) bad += tile_axis(b, b - 1, o, n, at) || tile_axis(b, b, o, n, at);
            for (int b0 = o - 3; b0 < o + n + 3; ++b0)
                for (int b1 = b0 - 1; b1 <= b0; ++b1) {
                    const bool want = b1 - o >= 0 && b0 + 1 - o <= n - 1;
                    const bool in = tile_axis(b0, b1, o, n, at);
                    bad += in != want || (in && (at[0] != b0 - o || at[1] != b1 - o));
                }
        }
    std::printf("%d\\n", bad);
    return bad != 0;
}
"""


def test_tile_axis(tmp_path):
    (tmp_path / "box.cpp").write_text(SOURCE)
    exe = str(tmp_path / "box")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all", "-I",
                    os.path.join(build.HERE, "csrc"), str(tmp_path / "box.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.strip() == "0"
