"""The memory estimate (sankhya_gb300_estimate_memory) against the device memory that goes when an LP is
loaded and solved, FP64 and then mixed: never less, on even and on skewed patterns, and not more than
four times as much."""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen
from sankhya_gb300.model import LP


def one_long_row_in(group, m):
    """Every `group`-th row has 64 entries, the others one."""
    rng = np.random.default_rng(1)
    n = 2 * m
    lengths = np.ones(m, np.int64)
    lengths[::group] = 64
    rows = np.repeat(np.arange(m), lengths)
    cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) if k > 1 else
                           rng.integers(0, n, 1) for k in lengths])
    order = np.lexsort((rows, cols))
    starts = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    return LP(m, n, starts.astype(np.int32), rows[order].astype(np.int32),
              rng.normal(size=len(rows)), rng.normal(size=n), np.zeros(n), np.full(n, 2.0),
              np.full(m, -1.0), np.full(m, 1.0))


SHAPES = {
    "uniform": lambda: lpgen.planted_uniform(400000, 800000, 3, seed=1),
    "zipf": lambda: lpgen.planted_zipf(100000, 200001, 4000000, seed=1),
    "blocks": lambda: lpgen.planted_blocks(32, 15625, 31250, 9, seed=1),
    "general": lambda: lpgen.planted_general(100000, 200001, 4, seed=1, free=False),
    "one long row in 128": lambda: one_long_row_in(128, 200000),
    "one long row in 7": lambda: one_long_row_in(7, 100000),
    "small": lambda: lpgen.planted_uniform(3000, 6001, 5, seed=1),
}


@pytest.mark.gpu
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_estimate_bounds_what_goes(shape):
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    with capi.PdhgEngine(0) as eng:  # the kernels and their stacks are loaded
        eng.load(lpgen.planted_uniform(9000, 18001, 5, seed=3))
        for precision in ("fp64", "mixed"):
            eng.solve(iteration_limit=40, precision=precision)
    lp = SHAPES[shape]().contiguous()
    before = free()
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        for precision in ("fp64", "mixed"):
            eng.solve(iteration_limit=80, precision=precision)
            used = before - free()
            estimate = capi.estimate_memory(lp.rows, lp.cols, lp.nnz, precision)
            print(shape, precision, used / 1e6, estimate / 1e6)
            assert used <= estimate, (used, estimate)
            assert estimate <= 4 * used + (64 << 20), (used, estimate)
