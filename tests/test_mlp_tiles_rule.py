"""The rule that cuts the output of a network's GEMM into tiles (bec_b200/csrc/mlp_tiles.h), compiled for the host: for every
padded width and every tile width of a launch, whole tiles, and as many CTAs as it takes to cover the matrix."""
import os
import subprocess

from bec_b200.build import CSRC

PROGRAM = r"""
#include "mlp_tiles.h"
#include <cstdio>
int main()
{
    int bad = 0;
    for (int n = 64; n <= 4096; n += 64)
        for (int m = 64; m <= 16384; m += 64)
            for (int tn = 16; tn <= kWidestTile; tn *= 2) {
                const int w = tile_cols(n, tn);
                if (w < 16 || w > tn || n % w || (long long)tile_ctas(m, n, tn) * kTileRows * w != (long long)m * n)
                    if (bad++ < 5) std::printf("%d x %d, tiles of %d: %d wide, %d CTAs\n", m, n, tn, w, tile_ctas(m, n, tn));
            }
    return bad != 0;
}
"""


def test_every_tile_has_its_cta(tmp_path):
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, cwd=os.path.dirname(exe))
    assert r.returncode == 0, r.stdout
