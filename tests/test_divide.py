"""The row proximal step's quotient (sih-26_gb300/csrc/common.cuh divide): tests/host/divide_check.cu holds
it to IEEE division on the CPU, past the largest number too."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    from sankhya_gb300 import _paths, build

    exe = str(tmp_path / "divide_check")
    subprocess.run([nvcc] + build.ARCH + ["-O2", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler",
                                          "-ffp-contract=off", "-I", _paths.CSRC_DIR,
                                          os.path.join(ROOT, "tests", "host", "divide_check.cu"),
                                          "-lcudart", "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
