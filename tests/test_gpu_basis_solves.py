"""The basis solves of the adjoint and the polish (k_batch_adjoint, k_batch_polish) in each form of
their storage, from the known vertex: bases around a slice (32 lines), one held wholly in shared
memory (700), one with its vectors there (2,500) and one with its two gathered vectors (5,300).
Gradients agree with dense solves of the planted basis to the adjoint's bar, 1e-5 relative to
max(1, |gradient|); the polished point stays on the vertex to 1e-9.
"""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [3, 31, 32, 33, 700, 2500, 5300])
def test_basis_solves_from_the_vertex(m):
    lps = [lpgen.planted_nondegenerate(m, 2 * m, min(5, m), seed=70 + s)
           for s in range(2 if m < 2000 else 1)]
    rng = np.random.default_rng(m)
    gxs = [rng.standard_normal(lp.cols) for lp in lps]
    gys = [rng.standard_normal(lp.rows) for lp in lps]
    with capi.BatchEngine(0) as eng:
        eng.set_schedule(1, 256)
        eng.load(lps)
        eng.solve(tolerance=0.05, stop_rule="relative", iteration_limit=50000)
        for k, lp in enumerate(lps):
            cols = np.repeat(np.arange(lp.cols), np.diff(lp.col_starts))
            reduced = lp.col_cost - np.bincount(cols, lp.values * lp.lam[lp.row_index], lp.cols)
            eng.set_point(k, lp.x0, reduced, lp.lam)
        items, info = eng.polish()
        grads = eng.adjoint(gxs, gys, np.ones(len(lps)))
        points = [eng.solution(k) for k in range(len(lps))]
    for lp, gx, gy, g, p, i in zip(lps, gxs, gys, grads, points, info):
        assert i["status"] == 0 and g["status"] == 0, (i, g["status"], g["residual"])
        assert np.abs(p[0] - lp.x0).max() <= 1e-9 * max(1.0, np.abs(lp.x0).max())
        cols = np.repeat(np.arange(lp.cols), np.diff(lp.col_starts))
        basic = (lp.x0 > lp.col_lower) & (lp.x0 < lp.col_upper)
        a = np.zeros((lp.rows, lp.cols))
        a[lp.row_index, cols] = lp.values
        pb = np.linalg.solve(a[:, basic].T, gx[basic])
        q = np.linalg.solve(a[:, basic], gy)
        dc = lp.x0.copy()
        dc[basic] += q
        db = pb + lp.lam
        d = gx - a.T @ pb + (lp.col_cost - a.T @ lp.lam)
        for got, want in ((g["dc"], dc), (g["drl"] + g["dru"], db),
                          (g["dl"], np.where(~basic & (lp.x0 <= lp.col_lower), d, 0.0)),
                          (g["du"], np.where(~basic & (lp.x0 >= lp.col_upper), d, 0.0))):
            assert np.all(np.abs(got - want) <= 1e-5 * np.maximum(1.0, np.abs(want)))


@pytest.mark.parametrize("m", [64, 480, 513, 1000, 1024])
def test_factored_solves_from_far(m):
    """The dense FP32 factors and their FP64 refinement (dense_lu.cuh), past one panel, one and two
    column runs, and at the largest basis a block factors, from a point that is not the vertex: both
    systems' residuals reach the conjugate gradients' 1e-13, in a few steps."""
    lps = [lpgen.planted_nondegenerate(m, 2 * m, 4, seed=170 + s) for s in range(3)]
    rng = np.random.default_rng(m)
    with capi.BatchEngine(0) as eng:
        eng.set_schedule(1, 256)
        eng.load(lps)
        eng.solve(tolerance=0.05, stop_rule="relative", iteration_limit=50000)
        for k, lp in enumerate(lps):
            cols = np.repeat(np.arange(lp.cols), np.diff(lp.col_starts))
            reduced = lp.col_cost - np.bincount(cols, lp.values * lp.lam[lp.row_index], lp.cols)
            basic = (lp.x0 > lp.col_lower) & (lp.x0 < lp.col_upper)
            x = lp.x0 + np.where(basic, 1e-7 * rng.standard_normal(lp.cols), 0.0)
            eng.set_point(k, x, reduced, lp.lam * (1.0 + 1e-7))
        _, info = eng.polish()
        grads = eng.adjoint([rng.standard_normal(lp.cols) for lp in lps],
                            [rng.standard_normal(lp.rows) for lp in lps], np.ones(3))
        points = [eng.solution(k) for k in range(3)]
    for lp, i, g, p in zip(lps, info, grads, points):
        assert i["status"] == 0 and g["status"] == 0
        assert max(*i["residual"], *g["residual"]) <= 1e-13
        assert 0 < max(*i["iterations"], *g["iterations"]) <= 10
        assert np.abs(p[0] - lp.x0).max() <= 1e-9 * max(1.0, np.abs(lp.x0).max())
