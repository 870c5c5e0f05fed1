"""A batch engine that is loaded again keeps no buffer that is too small and no point of the batch
before: after a small batch in the mixed method with its adjoint, a larger one gives exactly what a
fresh engine gives, read in order, backwards and one by one."""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen

pytestmark = pytest.mark.gpu


def solve(eng, lps, order):
    eng.set_schedule(1, 256)
    eng.load(lps)
    items, _ = eng.solve(tolerance=1e-4, stop_rule="relative", iteration_limit=20000,
                         precision="mixed")
    points = {k: eng.solution(k) for k in order}
    rng = np.random.default_rng(1)
    grads = eng.adjoint([rng.standard_normal(lp.cols) for lp in lps],
                        [rng.standard_normal(lp.rows) for lp in lps], np.ones(len(lps)))
    return items, points, grads


@pytest.mark.parametrize("order", ["forward", "backward", "one"])
def test_reload_with_a_larger_batch(order):
    small = [lpgen.planted_nondegenerate(12, 24, 4, seed=1)]
    large = [lpgen.planted_nondegenerate(40 + 7 * k, 80 + 15 * k, 5, seed=k) for k in range(9)]
    ks = {"forward": range(9), "backward": range(8, -1, -1), "one": [4]}[order]
    with capi.BatchEngine(0) as eng:
        solve(eng, small, [0])
        got = solve(eng, large, ks)
    with capi.BatchEngine(0) as eng:
        want = solve(eng, large, range(9))
    for a, b in zip(got[0], want[0]):
        assert (a.status, a.iterations, a.objective) == (b.status, b.iterations, b.objective)
    for k in ks:
        for u, v in zip(got[1][k], want[1][k]):
            assert np.array_equal(u, v)
    for a, b in zip(got[2], want[2]):
        assert a["status"] == b["status"]
        for key in ("dc", "drl", "dru", "dl", "du"):
            assert np.array_equal(a[key], b[key])
