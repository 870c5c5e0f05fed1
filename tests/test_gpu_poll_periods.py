"""Where a solve's steps are cut into launches does not show in its points: the same bits whatever
steps_per_poll, for LPs that run resident, in one launch a period, and in the mixed method."""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen

LPS = {
    "resident": lambda: lpgen.planted_uniform(60, 120, 5, seed=3),
    "resident general": lambda: lpgen.planted_general(300, 600, 4, seed=3, free=False),
    "steps uniform": lambda: lpgen.planted_uniform(5000, 10001, 5, seed=3),
    "steps zipf": lambda: lpgen.planted_zipf(5000, 10001, 200000, seed=3),
}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", sorted(LPS))
def test_points_do_not_depend_on_the_poll_period(shape, precision):
    with capi.PdhgEngine(0) as eng:
        eng.load(LPS[shape]())
        want = None
        for steps in (0, 1, 7, 47, 48, 49, 130):
            r = eng.solve(tolerance=1e-12, iteration_limit=200, precision=precision,
                          steps_per_poll=steps)
            got = (*eng.solution(), r.iterations, r.attempts)
            want = want or got
            for a, b in zip(got, want):
                assert np.array_equal(a, b), steps
