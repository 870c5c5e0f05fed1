"""The storage that the batch engine reserves for basis matrices (csrc/batch.cuh, basis_places):
tests/host/basis_places_check.cu holds the bound to the slices' rules on the CPU; on the GPU a batch of
wide LPs with a dense row takes memory by its bases, not by the row."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from sankhya_gb300 import capi
from sankhya_gb300.model import LP

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bound_on_the_slices(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    from sankhya_gb300 import _paths, build

    exe = str(tmp_path / "basis_places_check")
    subprocess.run([nvcc] + build.ARCH + ["-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                                          _paths.INCLUDE_DIR, "-I", _paths.CSRC_DIR,
                                          os.path.join(ROOT, "tests", "host", "basis_places_check.cu"),
                                          "-lcudart", "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.startswith("OK"), run.stdout


@pytest.mark.gpu
def test_wide_lps_with_a_dense_row():
    torch = pytest.importorskip("torch")
    m, n, count = 100, 50000, 8
    rng = np.random.default_rng(0)
    lps = []
    for _ in range(count):
        rows = [np.sort(np.unique(np.append(rng.integers(1, m, 3), 0))) for _ in range(n)]
        starts = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
        rows = np.concatenate(rows)
        x = rng.uniform(0.0, 2.0, n)
        v = rng.normal(size=len(rows))
        ax = np.bincount(rows, v * np.repeat(x, np.diff(starts)), m)
        lps.append(LP(m, n, starts.astype(np.int32), rows.astype(np.int32), v, rng.normal(size=n),
                      np.zeros(n), np.full(n, 2.0), ax, ax))
    with capi.BatchEngine(0) as eng:
        eng.set_schedule(1, 256)
        eng.load(lps)
        eng.solve(tolerance=1e-4, stop_rule="relative", iteration_limit=400)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        eng.adjoint([np.ones(n)] * count, [np.ones(m)] * count, np.ones(count))
        used = before - torch.cuda.mem_get_info()[0]
    # Vectors: 4 doubles, 2 ints and a byte a column and 25 words a row; a workspace of 128 x 128 an LP.
    assert used <= count * (45 * n + 200 * m + 24 * 12800 + 4 * 128 * 128) + (64 << 20), used
