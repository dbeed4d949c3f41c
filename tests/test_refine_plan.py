"""The refinement's FP64 pass as it is planned on the device stays inside the
buffers of its call (no GPU: the planner runs on the host, see
tests/refine_plan_check.cu)."""
import os
import shutil
import subprocess

import pytest

from starlab_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_refinement_plans_stay_inside_their_buffers(tmp_path):
    nvcc = build.NVCC if os.path.exists(build.NVCC) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "refine_plan_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets",
                    "-I" + os.path.join(build.PKG, "csrc"), "-o", exe, os.path.join(HERE, "refine_plan_check.cu")],
                   check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("ok "), out.stdout + out.stderr
    checked, waves = map(int, out.stdout.split()[1:])
    assert checked > 10000 and waves > 1000
