"""The meetings of a cooperative grid's blocks (csrc/common.cuh, GridMeet). What the host says for each
error word on the CPU; on the GPU tests/host/meet_check.cu lets a meeting run out (a block that never
comes) and meets again."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build(tmp_path, name, source):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    from sankhya_gb300 import _paths, build

    exe = str(tmp_path / name)
    subprocess.run([nvcc] + build.ARCH + ["-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                                          _paths.CSRC_DIR, source, "-lcudart", "-o", exe], check=True)
    return exe


def test_messages(tmp_path):
    source = tmp_path / "messages.cu"
    source.write_text('#include <cstdio>\n#include "common.cuh"\n'
                      'int main() { std::printf("%s\\n%s\\n", sgb::fault_message(sgb::kCopyFault), '
                      'sgb::fault_message(sgb::kMeetFault)); }\n')
    out = subprocess.run([_build(tmp_path, "messages", str(source))], capture_output=True, text=True)
    copy, meet = out.stdout.splitlines()
    assert "copy" in copy and "meet" in meet


@pytest.mark.gpu
def test_a_meeting_runs_out(tmp_path):
    exe = _build(tmp_path, "meet_check", os.path.join(ROOT, "tests", "host", "meet_check.cu"))
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    print(run.stdout)
    assert run.returncode == 0 and run.stdout.rstrip().endswith("OK"), run.stdout
