"""A QP layout that cannot be built (no device memory left for it) leaves no trace: the engine reports the
memory error, and its next solves, with the lanes it had before and with those that failed, give what a
fresh engine gives."""
import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen
from sankhya_gb300.model import QP, banded_hessian

pytestmark = pytest.mark.gpu


def test_solves_after_a_layout_without_memory():
    torch = pytest.importorskip("torch")
    lp = lpgen.planted_uniform(400000, 800000, 8, seed=2)
    qp = QP(lp, *banded_hessian(lp.cols, 2, 2)).contiguous()
    options = [dict(column_lanes=4, row_lanes=4), dict()]

    def point(eng, o):
        eng.solve(tolerance=1e-9, iteration_limit=100, **o)
        return eng.solution()

    want = []
    for o in options:
        with capi.QpEngine(0) as eng:
            eng.load(qp)
            want.append(point(eng, o))
    with capi.QpEngine(0) as eng:
        eng.load(qp)
        first = point(eng, options[0])
        torch.cuda.synchronize()
        # The sliced copies take 200 MB; leave 64.
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
        with pytest.raises(capi.EngineError) as failure:
            point(eng, options[1])
        del hold
        torch.cuda.empty_cache()
        assert "cudaErrorMemoryAllocation" in str(failure.value)
        again, other = point(eng, options[0]), point(eng, options[1])
    for got, ref in ((first, want[0]), (again, want[0]), (other, want[1])):
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
