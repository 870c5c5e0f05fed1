"""The staged share that a solve reports is that of the kernels it ran in: all for a resident FP64 solve,
none for one whose periods are one cooperative launch (its layouts have a window for the column pass, since
4,000 rows fit one), and the windows' for the passes by themselves."""
import pytest

from sankhya_gb300 import capi, lpgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,cap,want", [(60, 120, None, (1.0, 1.0)),
                                                (4000, 9001, None, (0.0, 0.0)),
                                                (4000, 9001, "4096", (1.0, None))])
def test_staged_share(monkeypatch, rows, cols, cap, want):
    if cap is None:
        monkeypatch.delenv("SANKHYA_GB300_WINDOW_CAP", raising=False)
    else:
        monkeypatch.setenv("SANKHYA_GB300_WINDOW_CAP", cap)
    with capi.PdhgEngine(0) as eng:
        eng.load(lpgen.planted_uniform(rows, cols, 5, seed=1))
        r = eng.solve(tolerance=1e-9, iteration_limit=80)
    for got, ref in zip(r.staged_fraction, want):
        assert ref is None or got == ref, r.staged_fraction
