"""The FP64 passes' sliced layouts (csrc/slices.cuh).

* On the CPU, `tests/host/slices_check.cu` checks plan_slices on every row count around a slice
  and a group, and on row lengths around the long-row limit (64) and a piece (2,048).
* On the GPU, the preconditioner, the products and a short FP64 solve over the same lengths
  against the oracle: the scaling bit for bit; products within (2 + n_i) u sum |a_ij| |x_j| of the
  oracle's, u = 2^-53 and n_i the row's entries (each side rounds once or twice per entry); the
  solve's point after 40 accepted steps within 1e-9 (its rounding differences, measured at 1e-13
  on LPs of these sizes, grow with the iterations).
"""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

from sankhya_gb300 import capi
from sankhya_gb300.model import LP

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sliced_layouts(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    from sankhya_gb300 import _paths, build

    build.build_engine()
    objdir = os.path.join(os.path.dirname(_paths.ENGINE_LIB), "obj")
    objs = [os.path.join(objdir, s.replace(".cu", ".o")) for s in build.CUDA_SOURCES]
    exe = str(tmp_path / "slices_check")
    cmd = ([nvcc] + build.ARCH + ["-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                                  _paths.INCLUDE_DIR, "-I", _paths.CSRC_DIR,
                                  os.path.join(ROOT, "tests", "host", "slices_check.cu")] + objs +
           ["-lcudart", "-o", exe])
    proc = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert proc.returncode == 0, proc.stdout
    run = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                         timeout=300)
    assert run.returncode == 0 and run.stdout.startswith("OK"), run.stdout


def lp_with_rows(lengths, n, seed):
    """An LP whose row i has lengths[i] entries (at distinct random columns), with feasible
    equality and range rows around a point of the box."""
    rng = np.random.default_rng(seed)
    m = len(lengths)
    rows = [np.sort(rng.choice(n, size=k, replace=False)) for k in lengths]
    r = np.repeat(np.arange(m), [len(c) for c in rows])
    c = np.concatenate(rows) if m else np.zeros(0, int)
    order = np.lexsort((r, c))
    r, c = r[order], c[order]
    v = rng.normal(size=len(r))
    starts = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(c, minlength=n), out=starts[1:])
    x = rng.uniform(0, 10, n)
    ax = np.bincount(r, v * x[c], m)
    slack = np.where(rng.random(m) < 0.5, 0.0, 1.0)
    return LP(m, n, starts, r.astype(np.int32), v, rng.normal(size=n), np.zeros(n),
              np.full(n, 10.0), ax - slack, ax + slack)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,longest", [(1, 1, 1), (31, 40, 12), (129, 257, 30), (130, 70, 66),
                                         (40, 2060, 2050), (300, 6200, 6150)])
def test_slices_match_the_oracle(oracle, m, n, longest):
    rng = np.random.default_rng(m + n)
    lengths = rng.integers(0, min(n, 21), size=m)
    for k, want in enumerate((longest, 0, 64, 65, 2048, 2049)):
        if k < m and want <= min(n, longest):
            lengths[(k * 37) % m] = want
    lp = lp_with_rows(lengths, n, seed=m)
    a = LP(lp.rows, lp.cols, lp.col_starts, lp.row_index, np.abs(lp.values), lp.col_cost,
           lp.col_lower, lp.col_upper, lp.row_lower, lp.row_upper)
    u = 2.0 ** -53
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        x, y = rng.normal(size=n), rng.normal(size=m)
        for op, v, f, entries in ((0, x, "multiply", lengths),
                                  (1, y, "transpose_multiply", np.diff(lp.col_starts))):
            bound = (2 + entries) * u * getattr(oracle, f)(a, np.abs(v))
            assert np.all(np.abs(eng.spmv(op, v) - getattr(oracle, f)(lp, v)) <= bound)
        dr, dc, values, norm = eng.scaling()
        ref = oracle.build_scaling(lp)
        assert np.array_equal(dr, ref["row"]) and np.array_equal(dc, ref["col"])
        assert np.array_equal(values, ref["values"])
        got = eng.solve(tolerance=1e-13, iteration_limit=40)
        px, _, py = eng.solution()
    ref = oracle.solve(lp, tolerance=1e-13, iteration_limit=40)
    if ref.status_name != "iteration_limit" or got.status_name != "iteration_limit":
        # The smallest LPs are solved before the limit: the points are then both optimal.
        assert got.status_name == ref.status_name
        assert abs(got.objective - ref.objective) <= 1e-6 * max(1.0, abs(ref.objective))
        return
    scale = max(1.0, np.abs(ref.col_value).max())
    assert np.abs(px - ref.col_value).max() <= 1e-9 * scale
    assert np.abs(py - ref.row_dual).max() <= 1e-9 * max(1.0, np.abs(ref.row_dual).max())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(20, 30), (100, 200), (200, 400), (450, 900), (1300, 2600),
                                 (3500, 3900)])
def test_resident_steps_match_the_oracle(oracle, m, n):
    """LPs on clusters of 1, 2, 4, 8 and 16 blocks and one past them: iteration limits are exact
    inside and at the end of an evaluation period, and the point after 40 accepted steps is the
    oracle's within 1e-9."""
    lp = lp_with_rows(np.random.default_rng(n).integers(0, 21, size=m), n, seed=n)
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        for limit in (1, 41, 85):
            assert eng.solve(tolerance=1e-13, iteration_limit=limit).iterations == limit
        points = []
        for _ in range(2):
            eng.solve(tolerance=1e-13, iteration_limit=40)
            points.append(eng.solution())
        x, _, y = points[0]
        assert all(np.array_equal(a, b) for a, b in zip(*points))
    ref = oracle.solve(lp, tolerance=1e-13, iteration_limit=40)
    assert np.abs(x - ref.col_value).max() <= 1e-9 * max(1.0, np.abs(ref.col_value).max())
    assert np.abs(y - ref.row_dual).max() <= 1e-9 * max(1.0, np.abs(ref.row_dual).max())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(1, 1), (33, 31), (64, 256), (700, 700), (1500, 1400)])
def test_resident_setup_gives_the_bits_of_the_launches(monkeypatch, m, n):
    """Scaled in one cluster kernel or over launches (a window capacity turns the cluster off):
    maxima, ascending sums and products are the same operations, so the scaled LP has the same bits;
    the norm differs by the order of sums of 1,500 non-negative terms (1,500 * 2^-52 at most)."""
    lp = lp_with_rows(np.random.default_rng(n).integers(1, min(n, 20) + 1, size=m), n, seed=n)
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        got = eng.scaling(3)
    monkeypatch.setenv("SANKHYA_GB300_WINDOW_CAP", "0")
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        want = eng.scaling(3)
    for g, w in zip(got[:-1], want[:-1]):
        np.testing.assert_array_equal(g, w)
    assert abs(got[-1] - want[-1]) <= 4e-13 * want[-1]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,per_column,band", [(0, 33, 0, 2), (1, 1, 1, 0), (31, 33, 3, 1),
                                                 (128, 129, 5, 0), (40, 300, 20, 30)])
def test_qp_slices_match_the_oracle(oracle, m, n, per_column, band):
    """The QP passes on sliced items (lanes left to the engine) around a slice and a group, with
    no rows, and with columns on both sides of the long-item limit: the oracle's status and
    iteration count, and its point within 1e-9 of its scale, as every QP parity test."""
    from sankhya_gb300.model import random_qp

    qp = random_qp(17 + n, m, n, per_column=per_column, hessian_band=band)
    ref = oracle.solve_qp(qp, tolerance=1e-8, iteration_limit=1500)
    with capi.QpEngine(0) as eng:
        eng.load(qp)
        got = eng.solve(tolerance=1e-8, iteration_limit=1500)
        x, d, y = eng.solution()
    assert (got.status_name, got.iterations) == (ref.status_name, ref.iterations)
    for a, b in ((x, ref.col_value), (d, ref.col_dual), (y, ref.row_dual)):
        assert np.all(np.abs(a - b) <= 1e-9 * max(1.0, np.abs(b).max() if len(b) else 0.0))


@pytest.mark.gpu
@pytest.mark.parametrize("lengths,n,limit", [([40] * 900, 1500, 60), ([], 1025, 60), ([1100, 600, 65, 64] + [3] * 700, 1100, 177),
                                             ([7] * 6000, 9000, 101), ([2] * 1300, 40, 50)])
def test_qp_steps_in_one_launch_match_the_oracle(oracle, lengths, n, limit):
    """QPs past 1,024 items, whose check periods run in one cooperative launch: no rows, rows in
    chunks, rows of more than 32 entries, limits that end inside a period, more rows than columns;
    the oracle's iteration count, its point within 1e-9 of its scale, as every QP parity test, and
    the same bits twice."""
    from sankhya_gb300.model import QP, banded_hessian

    lp = lp_with_rows(lengths, n, seed=n)
    qp = QP(lp, *banded_hessian(n, 2, seed=n))
    ref = oracle.solve_qp(qp, tolerance=1e-12, iteration_limit=limit)
    with capi.QpEngine(0) as eng:
        eng.load(qp)
        got = eng.solve(tolerance=1e-12, iteration_limit=limit)
        x, d, y = eng.solution()
        eng.solve(tolerance=1e-12, iteration_limit=limit)
        assert all(np.array_equal(a, b) for a, b in zip(eng.solution(), (x, d, y)))
    assert (got.status_name, got.iterations) == (ref.status_name, ref.iterations)
    for a, b in ((x, ref.col_value), (d, ref.col_dual), (y, ref.row_dual)):
        assert np.all(np.abs(a - b) <= 1e-9 * max(1.0, np.abs(b).max() if len(b) else 0.0))


@pytest.mark.gpu
@pytest.mark.parametrize("lengths,n", [([2100, 4100, 65, 64] + [3] * 500, 4300), ([6] * 5000, 8000),
                                       ([2] * 9000, 60)])
def test_pdhg_steps_in_one_launch_match_the_oracle(oracle, lengths, n):
    """LPs past the resident kernel, whose steps run in one cooperative launch: rows of several
    pieces, more blocks for one side than for the other; iteration limits are exact inside and at
    the end of an evaluation period, and the point after 40 accepted steps is the oracle's within
    1e-9."""
    lp = lp_with_rows(lengths, n, seed=n)
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        for limit in (1, 41, 85):
            assert eng.solve(tolerance=1e-13, iteration_limit=limit).iterations == limit
        points = []
        for _ in range(2):
            eng.solve(tolerance=1e-13, iteration_limit=40)
            points.append(eng.solution())
        x, _, y = points[0]
        assert all(np.array_equal(a, b) for a, b in zip(*points))
    ref = oracle.solve(lp, tolerance=1e-13, iteration_limit=40)
    assert np.abs(x - ref.col_value).max() <= 1e-9 * max(1.0, np.abs(ref.col_value).max())
    assert np.abs(y - ref.row_dual).max() <= 1e-9 * max(1.0, np.abs(ref.row_dual).max())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(1, 2), (33, 70), (900, 1500), (5000, 9000)])
def test_mixed_steps_in_one_launch(monkeypatch, m, n):
    """The mixed method's steps in one cooperative launch (windows that hold the whole vectors) and over
    launches (a window capacity of half the longer vector): limits are exact inside and at the end
    of a period, and objectives at a relative KKT of 1e-6 agree to 1e-4, a hundred times the KKT."""
    lp = lp_with_rows(np.random.default_rng(n).integers(1, min(n, 12) + 1, size=m), n, seed=n)
    runs = []
    for cap in (None, str(max(4, max(m, n) // 2))):
        if cap is not None:
            monkeypatch.setenv("SANKHYA_GB300_WINDOW_CAP", cap)
        with capi.PdhgEngine(0) as eng:
            eng.load(lp)
            for limit in (1, 41, 85):
                r = eng.solve(tolerance=1e-13, precision="mixed", iteration_limit=limit)
                assert r.iterations == limit or r.converged
            runs.append(eng.solve(tolerance=1e-6, precision="mixed", iteration_limit=200000))
    assert {r.status_name for r in runs} <= {"optimal", "feasible"}
    assert abs(runs[0].objective - runs[1].objective) <= 1e-4 * max(1.0, abs(runs[1].objective))
