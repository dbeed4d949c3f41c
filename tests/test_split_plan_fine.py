"""The ensemble's finer cut of small blocks (ForceConfig::fine_ni) stays
inside the partials a cluster has, n * batch_max_split(nj_pad, min_tiles)
records, and covers the j-set (no GPU: the planner runs on the host)."""
import os
import shutil
import subprocess

import pytest

from starlab_b200 import build

SOURCE = r"""
#include <cstdio>
#include "kernels.h"
using namespace g6;
int main() {
    for (int kmode : {kKernF64, kKernMixedP})
        for (int mt : {1, 2, 4, 8})
            for (int h : {1, 2, 4, 8})
                for (int n = 1; n <= 40000; n += n < 1200 ? 1 : 97) {
                    const int T = tile_of(kmode), nj_pad = (n + T - 1) / T * T;
                    for (int ni : {1, 2, 3, 8, 16, 17, 32, 33, 64, 127, 128, 129, 256, 512}) {
                        if (ni > n) break;
                        ForceConfig c{32, 1, 8, h, 592};
                        c.min_tiles = mt;
                        c.fine_ni = kEnsFineNi;
                        ForceParams p{};
                        p.ni = ni;
                        p.nj = n;
                        p.nj_pad = nj_pad;
                        int nt = 0;
                        batch_plan(kmode, c, p, nt);
                        const bool covers = (long long)p.nsplit * p.jper >= nj_pad && (p.nsplit - 1) * p.jper < nj_pad;
                        const bool fits = (long long)p.nsplit * ni <= (long long)n * batch_max_split(kmode, nj_pad, mt);
                        if (!covers || !fits || p.jper % T) {
                            std::printf("kmode %d mt %d h %d n %d ni %d: nsplit %d jper %d\n", kmode, mt, h, n, ni,
                                        p.nsplit, p.jper);
                            return 1;
                        }
                    }
                }
    std::printf("ok\n");
}
"""


def test_small_blocks_stay_inside_their_partials(tmp_path):
    nvcc = build.NVCC if os.path.exists(build.NVCC) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "fine.cu", str(tmp_path / "fine")
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets",
                    "-I" + os.path.join(build.PKG, "csrc"), "-o", exe, str(src)], check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
