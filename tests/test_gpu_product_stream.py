"""Device products of a caller who names no stream (PdhgEngine.spmv_device without a stream, or with
handle 0): they run on the legacy default stream, so what the caller wrote there before is in the
product and what the caller reads there after is the result, with no synchronisation between; and
products of two engines, which share the fixed scratch, come one after the other.

The references are the host product's (the same kernel on the same layout): equal bit for bit.
"""
import ctypes

import numpy as np
import pytest

from sankhya_gb300 import capi
from sankhya_gb300.model import LP

CALLS = 40


def lp_of_lengths(lengths, n, seed):
    """Rows of the given lengths over n columns; the last column holds an entry of every row."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for i, k in enumerate(lengths):
        c = np.append(rng.choice(n - 1, size=k - 1, replace=False), n - 1)
        rows.append(np.full(k, i))
        cols.append(c)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((rows, cols))
    starts = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    m = len(lengths)
    return LP(m, n, starts.astype(np.int32), rows[order].astype(np.int32),
              rng.normal(size=len(rows)), rng.normal(size=n), np.zeros(n), np.full(n, 10.0),
              np.full(m, -1.0), np.full(m, 1.0)).contiguous()


def skewed(seed, m=5000, n=9000):
    """Rows of 1, 64, 65, 2,047, 2,048, 2,049 and 6,500 entries, the others of up to 20; the last
    column has an entry of every row."""
    lengths = np.random.default_rng(seed).integers(1, 21, size=m)
    lengths[[0, 1, 2, 3, 4, 5, 6]] = [1, 64, 65, 2047, 2048, 2049, 6500]
    lengths[-1] = 6500
    return lp_of_lengths(lengths, n, seed)


def _cudart():
    for name in ("libcudart.so.13", "libcudart.so", "libcudart.so.12"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            continue
    pytest.skip("no shared CUDA runtime to make a blocking stream with")


@pytest.mark.gpu
@pytest.mark.parametrize("engines", [1, 2])
def test_products_without_a_stream_follow_the_default_stream(engines):
    torch = pytest.importorskip("torch")
    lps = [skewed(seed) for seed in range(3, 3 + engines)]
    rng = np.random.default_rng(8)
    xs = rng.standard_normal((CALLS, lps[0].cols))
    ys = rng.standard_normal((CALLS, lps[0].rows))
    engs = [capi.PdhgEngine(0) for _ in lps]
    try:
        for eng, lp in zip(engs, lps):
            eng.load(lp)
        want = [([eng.spmv(0, x) for x in xs], [eng.spmv(1, y) for y in ys]) for eng in engs]
        xd, yd = torch.from_numpy(xs).cuda(), torch.from_numpy(ys).cuda()
        bufs = [tuple(torch.zeros(k, dtype=torch.float64, device="cuda")
                      for k in (lp.cols, lp.rows, lp.rows, lp.cols)) for lp in lps]
        got = [([], []) for _ in engs]
        torch.cuda.synchronize()
        for call in range(CALLS):
            # Work ahead of the inputs: the products must wait for it.
            torch.cuda._sleep(200_000)
            for eng, (x, y, ax, aty), g in zip(engs, bufs, got):
                x.copy_(xd[call])
                y.copy_(yd[call])
                handle = torch.cuda.current_stream().cuda_stream
                eng.spmv_device(0, x.data_ptr(), ax.data_ptr(), stream=handle or None)
                eng.spmv_device(1, y.data_ptr(), aty.data_ptr(), stream=handle)
            for (x, y, ax, aty), g in zip(bufs, got):
                g[0].append(ax.clone())
                g[1].append(aty.clone())
        for (wax, waty), (gax, gaty) in zip(want, got):
            for call in range(CALLS):
                assert np.array_equal(gax[call].cpu().numpy(), wax[call]), call
                assert np.array_equal(gaty[call].cpu().numpy(), waty[call]), call
    finally:
        for eng in engs:
            eng.close()


@pytest.mark.gpu
def test_a_scaling_after_a_product_without_a_stream():
    """The next preconditioning rewrites the scaled values that the product reads: it waits."""
    torch = pytest.importorskip("torch")
    lp = skewed(11)
    v = np.random.default_rng(1).standard_normal(lp.cols)
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        eng.scaling(0)
        want = eng.spmv(0, v, scaled=True)
        x = torch.from_numpy(v).cuda()
        out = torch.zeros(lp.rows, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(5):
            out.zero_()
            torch.cuda._sleep(200_000)
            eng.spmv_device(0, x.data_ptr(), out.data_ptr(), scaled=True)
            eng.scaling(0)
            assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
def test_without_a_stream_while_a_blocking_stream_is_captured():
    """The legacy stream may not be used then: the engine's stream carries the product, and the
    capture goes on."""
    torch = pytest.importorskip("torch")
    rt = _cudart()
    lp = skewed(12)
    v = np.random.default_rng(2).standard_normal(lp.cols)
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        want = eng.spmv(0, v)
        x = torch.from_numpy(v).cuda()
        out = torch.zeros(lp.rows, dtype=torch.float64, device="cuda")
        eng.spmv_device(0, x.data_ptr(), out.data_ptr())  # the scratch's set-up
        torch.cuda.synchronize()
        out.zero_()
        torch.cuda.synchronize()
        stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
        assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0  # a blocking stream
        try:
            assert rt.cudaStreamBeginCapture(stream, 2) == 0  # relaxed
            eng.spmv_device(0, x.data_ptr(), out.data_ptr())
            assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
            rt.cudaGraphDestroy(graph)
        finally:
            rt.cudaStreamDestroy(stream)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_products_beside_solves(precision):
    torch = pytest.importorskip("torch")
    lp = skewed(13)
    rng = np.random.default_rng(3)
    x, y = rng.standard_normal(lp.cols), rng.standard_normal(lp.rows)
    with capi.PdhgEngine(0) as eng:
        eng.load(lp)
        want = eng.spmv(0, x), eng.spmv(1, y)
        eng.solve(tolerance=1e-12, iteration_limit=120, precision=precision)
        points = eng.solution()
        side = torch.cuda.Stream()
        xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        outs = [(torch.zeros(lp.rows, dtype=torch.float64, device="cuda"),
                 torch.zeros(lp.cols, dtype=torch.float64, device="cuda")) for _ in range(200)]
        torch.cuda.synchronize()
        for solve in range(4):
            for ax, aty in outs[50 * solve:50 * solve + 50]:
                eng.spmv_device(0, xd.data_ptr(), ax.data_ptr(), stream=side.cuda_stream)
                eng.spmv_device(1, yd.data_ptr(), aty.data_ptr(), stream=side.cuda_stream)
            eng.solve(tolerance=1e-12, iteration_limit=120, precision=precision)
            for got, ref in zip(eng.solution(), points):
                assert np.array_equal(got, ref), solve
        side.synchronize()
        for ax, aty in outs:
            assert np.array_equal(ax.cpu().numpy(), want[0])
            assert np.array_equal(aty.cpu().numpy(), want[1])
