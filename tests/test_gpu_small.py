"""Single-CTA kernels (acq_small.cuh) against the oracle: two to four passes,
odd and even first radices, both register classes, the K blocks of a row on one
CTA or split over a cluster (few rows) with a remainder, one- and two-sided
spectra, both statistics and every sample type."""
import numpy as np
import pytest

from conftest import unpack_codes
from test_gpu_acquire import check_vs_oracle, run_engine, to_complex

pytestmark = pytest.mark.gpu

CASES = [
    # n, K, Doppler bins each side, sample type, two-sided, statistic
    (62, 3, 1, "ci8", False, 0),       # 31 x 2
    (1023, 1, 2, "cf32", False, 0),    # 31 x 11 x 3, a block of one
    (1736, 5, 1, "ci16", False, 1),    # 31 x 8 x 7
    (2046, 20, 2, "ci8", False, 0),    # split over a cluster: 8 CTAs, 3 blocks each with a remainder
    (2048, 9, 100, "ri8", True, 0),    # no split: 201 rows of 9 blocks
    (3375, 7, 1, "ci16", False, 0),    # 27 x 25 x 5
    (4000, 4, 1, "ci8", True, 1),
    (4092, 10, 60, "cf32", False, 0),
    (5005, 2, 1, "ci8", False, 0),     # 13 x 11 x 7 x 5: four passes
    (5600, 3, 1, "ci16", True, 0),
]


@pytest.mark.parametrize("n,k,half,sample_type,two_sided,stat", CASES)
def test_small_blocks_vs_oracle(ctx, oracle, golden_codes, n, k, half, sample_type, two_sided, stat):
    from ugsdr_gb300 import _lib as L, signals
    chips = unpack_codes(golden_codes, "gps_l1ca")[6]
    fs = n * 1e3
    em = signals.Emitter(chips, 1.023e6, 300.5, 100.0, 60.0, data_rate=0.0)
    raw = signals.synthesize([em], fs, n * k, 20.0, sample_type, seed=n)
    mode = L.SPECTRUM_TWO_SIDED if two_sided else L.SPECTRUM_ONE_SIDED
    span, step = 100.0 * half, 100.0
    res, cells = run_engine(ctx, raw, fs, n, k, [chips], 1, span, step, spectrum_mode=mode, statistic=stat)
    x, code = to_complex(raw), oracle.upsample(chips, n)
    if half <= 2:
        check_vs_oracle(res[0], *(oracle.acquire(x, n, k, code, fs, span, step, stat=stat, spectrum_mode=mode, double=d)
                                  for d in (False, True)))
    else:  # the bins around the peak's, searched alone
        lo = [c for c in cells[0][half - 1:half + 4]]
        few, few_cells = run_engine(ctx, raw, fs, n, k, [chips], 1, 0.0, step, spectrum_mode=mode, statistic=stat)
        want = oracle.acquire(x, n, k, code, fs, 0.0, step, stat=stat, spectrum_mode=mode, double=True)
        for got in (lo[1], few_cells[0][0]):
            assert int(got["index"]) == int(want["index"])
            for f in ("level", "mean", "std"):
                assert abs(float(got[f]) - want[f]) <= 1e-4 * abs(want[f])
