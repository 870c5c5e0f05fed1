"""Basis matrices that are singular, with right-hand sides in their range (an equality row that repeats
another one, times a factor that is exact or rounds): the dense FP32 factors cannot tell the null space
from rounding and are refused, and the conjugate gradients give the solution of least length, as dense
pseudo-inverses do.

The tolerance: the solves stop at a residual of 1e-13 of the right-hand side's length, and the planted
bases' largest singular value is below 1e4 times their least that is not zero, so 1e-8 of the solution's
length leaves a factor of ten. That holds where a pass of the iterations ends by its residual: always
for the systems with the transpose, for the others where the row is repeated exactly (else the second
pass runs to its limit on rounding and wanders in the null space, by up to 5e-3 of the length).
"""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen
from sankhya_gb300.model import LP


def repeated_row(m, n, factor, seed):
    """A planted nondegenerate LP with one more equality row, `factor` times row 0, and one more basic
    column; (lp, x, reduced costs, multipliers, dense matrix, basic columns)."""
    lp = lpgen.planted_nondegenerate(m, n, min(5, m), seed=seed).contiguous()
    cols = np.repeat(np.arange(n), np.diff(lp.col_starts))
    a = np.zeros((m + 1, n))
    a[lp.row_index, cols] = lp.values
    a[m] = factor * a[0]
    free = (lp.x0 > lp.col_lower) & (lp.x0 < lp.col_upper)
    new = np.flatnonzero(~free)[0]
    lo, up = lp.col_lower.copy(), lp.col_upper.copy()
    lo[new], up[new] = lp.x0[new] - 1.0, lp.x0[new] + 1.0
    lam = np.append(lp.lam, 0.05)
    lam[0] -= 0.05 * factor
    cost = lp.col_cost.copy()
    reduced = cost - a.T @ lam
    cost[new] -= reduced[new]
    reduced[new] = 0.0
    c, r = np.nonzero(a.T)
    starts = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=n))])
    out = LP(m + 1, n, starts.astype(np.int32), r.astype(np.int32), a.T[c, r].copy(), cost, lo, up,
             np.append(lp.row_lower, factor * lp.row_lower[0]),
             np.append(lp.row_upper, factor * lp.row_upper[0])).contiguous()
    free[new] = True
    return out, lp.x0, reduced, lam, a, free


@pytest.mark.gpu
@pytest.mark.parametrize("factor", [1.0, 3.0, -0.7])
@pytest.mark.parametrize("m", [40, 60, 300])
def test_gradients_of_least_length(m, factor):
    lp, x, reduced, lam, a, basic = repeated_row(m, 2 * m, factor, seed=7 + m)
    rng = np.random.default_rng(m)
    gy = rng.normal(size=m + 1)
    gy[m] = factor * gy[0]
    gx = a.T @ rng.normal(size=m + 1)
    with capi.BatchEngine(0) as eng:
        eng.set_schedule(1, 256)
        eng.load([lp])
        eng.solve(tolerance=0.05, stop_rule="relative", iteration_limit=2000)
        eng.set_point(0, x, reduced, lam)
        g = eng.adjoint([gx], [gy], np.zeros(1))[0]
    basis = a[:, basic]
    assert basis.shape == (m + 1, m + 1)
    singular = np.linalg.svd(basis, compute_uv=False)
    assert singular[-1] <= 1e-14 * singular[0] and singular[0] <= 1e4 * singular[-2]
    inverse = np.linalg.pinv(basis, rcond=1e-10)
    q, p = inverse @ gy, inverse.T @ gx[basic]
    assert g["status"] == 0
    assert np.linalg.norm(g["dc"][basic] - q) <= (1e-8 if factor == 1.0 else 0.05) * np.linalg.norm(q)
    assert np.linalg.norm(g["drl"] + g["dru"] - p) <= 1e-8 * np.linalg.norm(p)
