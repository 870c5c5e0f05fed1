"""Basis solves whose dense FP32 factors refine quickly, slowly or not at all (values over six orders of
magnitude, rows and columns scaled by as much: condition numbers of 1e1 to 1e14), with the conjugate
gradients taking over for both systems or for the second one only. What the engine reports as solved is
solved: the residual against longdouble products is within the engine's 1e-11 of the right-hand side's
length, and what the residual's own rounding adds where it is formed in FP64, 2 (k + 2) u |B| |q| for
lines of k entries. Well-conditioned bases are all solved.
"""
import numpy as np
import pytest

from sankhya_gb300 import capi
from sankhya_gb300.model import LP

pytestmark = pytest.mark.gpu


def planted(n, seed, kind):
    """(lp, x, reduced costs, multipliers, basis): n equality rows, n basic columns, n at their bound."""
    rng = np.random.default_rng(seed)
    basis = np.zeros((n, n))
    for j in range(n):
        i = rng.choice(n, 5, replace=False)
        v = rng.normal(size=5)
        basis[i, j] = np.sign(v) * 10 ** rng.uniform(-3, 3, 5) if kind == "log" else v
    basis[np.arange(n), rng.permutation(n)] += 1.0
    if kind == "scaled":
        basis = 10 ** rng.uniform(-3, 3, n)[:, None] * basis * 10 ** rng.uniform(-3, 3, n)[None, :]
    other = np.zeros((n, n))
    for j in range(n):
        other[rng.choice(n, 3, replace=False), j] = rng.normal(size=3)
    a = np.hstack([basis, other])
    x = np.concatenate([np.full(n, 0.5), np.zeros(n)])
    lam = rng.normal(size=n)
    reduced = np.concatenate([np.zeros(n), rng.uniform(1.0, 2.0, n)])
    b = a @ x
    c, r = np.nonzero(a.T)
    starts = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=2 * n))])
    lp = LP(n, 2 * n, starts.astype(np.int32), r.astype(np.int32), a.T[c, r].copy(),
            a.T @ lam + reduced, np.zeros(2 * n), np.ones(2 * n), b, b).contiguous()
    return lp, x, reduced, lam, basis, rng


@pytest.mark.parametrize("kind,n", [("normal", 50), ("normal", 300), ("log", 50), ("log", 300),
                                    ("scaled", 50)])
def test_reported_as_solved_is_solved(kind, n):
    for seed in range(6):
        lp, x, reduced, lam, basis, rng = planted(n, seed, kind)
        gx, gy = rng.normal(size=2 * n), rng.normal(size=n)
        with capi.BatchEngine(0) as eng:
            eng.set_schedule(1, 256)
            eng.load([lp])
            eng.solve(tolerance=0.5, stop_rule="relative", iteration_limit=200)
            eng.set_point(0, x, reduced, lam)
            g = eng.adjoint([gx], [gy], np.zeros(1))[0]
        assert g["status"] == 0 or kind != "normal", (seed, g["residual"])
        if g["status"] != 0:
            continue
        for s, u, h in ((basis, g["dc"][:n], gy), (basis.T, g["drl"] + g["dru"], gx[:n])):
            wide = s.astype(np.longdouble) @ u.astype(np.longdouble) - h
            entries = (s != 0).sum(axis=1)
            rounding = np.linalg.norm(2 * (entries + 2) * 2.0 ** -53 * (np.abs(s) @ np.abs(u)))
            assert np.linalg.norm(wide.astype(float)) <= 1e-11 * np.linalg.norm(h) + rounding, seed
