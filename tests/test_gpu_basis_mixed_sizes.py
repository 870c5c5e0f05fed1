"""An LP's basis solves do not depend on the rest of its batch: bases that are factored densely and bases
too large for it, together and alone, give the same gradients and the same polished points bit for bit,
and the small ones are factored in either batch (a few refinement steps, not hundreds of iterations)."""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen

pytestmark = pytest.mark.gpu


def run(lps, gxs, gys):
    with capi.BatchEngine(0) as eng:
        eng.set_schedule(1, 256)
        eng.load(lps)
        eng.solve(tolerance=0.05, stop_rule="relative", iteration_limit=50000)
        for k, lp in enumerate(lps):
            cols = np.repeat(np.arange(lp.cols), np.diff(lp.col_starts))
            reduced = lp.col_cost - np.bincount(cols, lp.values * lp.lam[lp.row_index], lp.cols)
            eng.set_point(k, lp.x0 * (1.0 + 1e-9), reduced, lp.lam)
        _, info = eng.polish()
        grads = eng.adjoint(gxs, gys, np.ones(len(lps)))
        return [(g, eng.solution(k), i) for k, (g, i) in enumerate(zip(grads, info))]


def test_alone_and_together():
    sizes = [40, 300, 1024, 1025, 1100]
    lps = [lpgen.planted_nondegenerate(m, 2 * m, 4, seed=900 + m) for m in sizes]
    rng = np.random.default_rng(0)
    gxs = [rng.standard_normal(lp.cols) for lp in lps]
    gys = [rng.standard_normal(lp.rows) for lp in lps]
    together = run(lps, gxs, gys)
    for k, m in enumerate(sizes):
        (g, point, info), = run([lps[k]], [gxs[k]], [gys[k]])
        other, other_point, _ = together[k]
        assert g["status"] == other["status"] == 0
        for key in ("dc", "drl", "dru", "dl", "du"):
            assert np.array_equal(g[key], other[key]), (m, key)
        for a, b in zip(point, other_point):
            assert np.array_equal(a, b), m
        assert g["iterations"] == other["iterations"]
        assert (max(g["iterations"]) <= 10) == (m <= 1024), (m, g["iterations"])
