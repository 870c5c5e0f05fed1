"""The mixed method's step kernels in each form of their chunk layouts (chunks.cuh): packed entries where
the windows hold all of them, entries as the layout has them elsewhere, split layouts of either kind, and
long rows in pieces; with chunks of a few entries, of half their places, one more, and full. The point of
a solve to a relative 1e-6 meets it by the oracle's own evaluation."""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen

pytestmark = pytest.mark.gpu

LPS = {f"{k} a column": (lambda k=k: lpgen.planted_blocks(6, 150, 300, k, seed=k)) for k in (1, 3, 4, 8, 9)}
LPS["long rows"] = lambda: lpgen.planted_uniform(40, 4000, 5, seed=5)  # rows of about 500 entries


@pytest.mark.parametrize("cap", [None, "0", "64", "256"])
@pytest.mark.parametrize("shape", list(LPS))
def test_forms_meet_the_tolerance(monkeypatch, oracle, shape, cap):
    if cap is None:
        monkeypatch.delenv("SANKHYA_GB300_WINDOW_CAP", raising=False)
    else:
        monkeypatch.setenv("SANKHYA_GB300_WINDOW_CAP", cap)
    lp = LPS[shape]()
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        r = eng.solve(tolerance=1e-6, precision="mixed", stop_rule="relative", iteration_limit=400000)
        x, _, y = eng.solution()
    assert r.converged, r.message
    res, _, _ = oracle.evaluate(lp, x, -lp.sense * y)
    assert max(res["primal"], res["dual"], res["gap"]) <= 1e-6 * (1 + 1e-9), res
    # Without windows nothing is staged; with small ones the columns' vector is, in part.
    assert (max(r.staged_fraction) == 0.0) == (cap == "0"), r.staged_fraction
    assert np.isfinite(x).all() and np.isfinite(y).all()
