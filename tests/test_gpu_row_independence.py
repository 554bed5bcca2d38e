"""A cell has the same bits whatever is searched beside it: alone, with some of
the codes, with all of them, and with the Doppler grid in chunks — what lets
the gathered shares of a search equal one search of all codes
(sharding.py)."""
import numpy as np
import pytest

from conftest import unpack_codes

pytestmark = pytest.mark.gpu

CASES = [
    # block, K, folded length, two-sided, statistic
    (500, 3, 0, False, 0),      # two passes
    (1736, 40, 0, False, 0),
    (2046, 20, 0, False, 1),
    (4000, 10, 0, False, 0),    # compile-time passes
    (4000, 7, 0, True, 0),
    (4092, 7, 0, True, 0),
    (5000, 4, 0, False, 0),
    (5005, 5, 0, False, 0),     # four passes
    (8184, 3, 2046, False, 0),
    (5720, 1, 0, False, 0),
    (10230, 3, 0, False, 0),
    (20460, 2, 0, False, 0),
]


@pytest.mark.parametrize("n,k,fold,two_sided,stat", CASES)
def test_cell_bits_alone_and_in_company(ctx, golden_codes, monkeypatch, n, k, fold, two_sided, stat):
    from ugsdr_gb300 import _lib as L
    chips = unpack_codes(golden_codes, "gps_l1ca")
    mode = L.SPECTRUM_TWO_SIDED if two_sided else L.SPECTRUM_ONE_SIDED
    raw = np.random.default_rng(n).integers(-60, 61, (n * k, 2)).astype(np.int8)
    codes = [ctx.code_put(chips[p], n, n // fold if fold else 1, mode) for p in range(32)]

    def cells(handles, span):
        job = ctx.make_job(raw, L.SAMPLES_CI8, n * 1e3, n, k, handles, span, 500.0, fold_samples=fold, statistic=stat,
                           spectrum_mode=mode)
        return ctx.acquire(job, cells=True)[1]

    try:
        every = cells(codes, 5000.0)
        for c in (0, 9, 31):
            assert cells(codes[c:c + 1], 0.0)[0, 0].tobytes() == every[c, 10].tobytes()
        for c0, c1, half in ((0, 1, 10), (4, 6, 2), (8, 16, 5), (16, 32, 10)):
            some = cells(codes[c0:c1], half * 500.0)
            assert some.tobytes() == every[c0:c1, 10 - half:11 + half].tobytes(), (c0, c1, half)
        monkeypatch.setenv("UGSDR_SPECTRA_BUDGET_MB", "1")
        assert cells(codes, 5000.0).tobytes() == every.tobytes()
    finally:
        for h in codes:
            ctx.code_release(h)
