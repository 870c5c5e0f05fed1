"""Solves beside a kernel that holds part of the SMs for seconds (a batch in another thread): the ones that
run their periods in cooperative launches, which need every SM, run in launches of single passes then. They
finish while the batch still runs, with the bits they have alone; and with the SMs free again the periods
are single launches again (fewer kernels)."""
import threading
import time

import numpy as np
import pytest

from sankhya_gb300 import capi, lpgen
from sankhya_gb300.model import QP, banded_hessian

pytestmark = pytest.mark.gpu

LIMIT = dict(tolerance=1e-13, iteration_limit=400)


def jobs():
    lp = lpgen.planted_uniform(60000, 120001, 5, seed=3)
    zipf = lpgen.planted_zipf(5000, 10001, 200000, seed=3)
    small = lpgen.planted_uniform(9000, 18001, 5, seed=4)
    qp = QP(lpgen.planted_uniform(20000, 40003, 5, seed=5), *banded_hessian(40003, 2, 5))
    for load, options in ((lp, {}), (zipf, {}), (small, dict(precision="mixed")), (qp, None)):
        eng = capi.QpEngine(0) if options is None else capi.PdhgEngine(0)
        eng.load(load)
        yield eng, LIMIT if options is None else dict(LIMIT, **options)


def run(eng, options):
    r = eng.solve(**options)
    return (*eng.solution(), r.iterations), r.kernel_launches


def test_solves_beside_a_batch():
    work = list(jobs())
    alone = [run(*job) for job in work]
    batch = capi.BatchEngine(0)
    batch.set_schedule(1, 512)
    batch.load([lpgen.planted_uniform(2500, 5001, 6, seed=9 + k) for k in range(90)])
    t = time.perf_counter()
    batch.solve(tolerance=1e-13, iteration_limit=1000)
    limit = int(1000 * 6.0 / (time.perf_counter() - t))
    thread = threading.Thread(target=lambda: batch.solve(tolerance=1e-14, iteration_limit=limit))
    thread.start()
    try:
        time.sleep(0.7)
        beside = [run(*job) for job in work for _ in range(2)]
        still = thread.is_alive()
    finally:
        thread.join()
    after = [run(*job) for job in work]
    assert still, "the solves waited for the batch"
    for k, (want, launches) in enumerate(alone):
        for got, _ in (beside[2 * k], beside[2 * k + 1], after[k]):
            for a, b in zip(got, want):
                assert np.array_equal(a, b), k
        assert beside[2 * k][1] > launches and after[k][1] == launches, k
    for eng, _ in work:
        eng.close()
    batch.close()
