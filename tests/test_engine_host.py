"""The engine's host code where no GPU is needed: engine.cu on a fake CUDA
runtime with fake kernels (tests/engine_host.h), one small program per
behaviour, each of which prints "ok" or what went wrong."""
import os
import shutil
import subprocess

import pytest

from starlab_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("program", ["failed_call", "no_memory", "upload_during_call", "status_words", "open", "retry"])
def test_engine_host(program, tmp_path):
    nvcc = build.NVCC if os.path.exists(build.NVCC) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / program)
    r = subprocess.run([nvcc, "-x", "cu", "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets",
                        "-I" + os.path.join(build.PKG, "csrc"), "-I" + HERE, "-o", exe,
                        os.path.join(HERE, "engine_host_%s.cpp" % program)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
