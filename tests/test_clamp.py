"""The projections of the FP64 steps compare doubles by their bits (sih-26_gb300/csrc/common.cuh
clamp_box); tests/host/clamp_check.cu holds them to floating-point comparisons on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_projections_by_bits(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    from sankhya_gb300 import _paths, build

    exe = str(tmp_path / "clamp_check")
    subprocess.run([nvcc] + build.ARCH + ["-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                                          _paths.CSRC_DIR,
                                          os.path.join(ROOT, "tests", "host", "clamp_check.cu"),
                                          "-lcudart", "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
