"""Pair kernels of the four-step inverse (acq_pairs.cuh) against the natural
CTA-tile kernels (warp_cols 0) on splits that cover every prime radix, odd and
even halves, both register classes and tile widths, row remainders, one- and
two-sided spectra and both statistics; and, against the oracle, the block
sizes one CTA could hold that run the four-step kernels."""
import numpy as np
import pytest

from conftest import unpack_codes
from test_gpu_acquire import check_vs_oracle, run_engine, to_complex

pytestmark = pytest.mark.gpu

# both paths: float transforms of at most 2^19 points, each within 5e-7 of 64
# bits, and sums of three blocks
RTOL = 2e-6
SIZES = [13800, 14872, 16000, 16384, 20460, 25840, 27405, 33250, 38192, 40920, 65536, 81840, 133000, 152768, 163840, 204600,
         332500, 381920, 500000]


@pytest.mark.parametrize("n", SIZES)
def test_pair_kernels_vs_natural_layout(ctx, golden_codes, n):
    from ugsdr_gb300 import _lib as L, signals
    chips = unpack_codes(golden_codes, "galileo_e1b")
    two_sided, stat, k = n % 3 == 0, int(n % 5 == 0), 1 + n % 3
    mode = L.SPECTRUM_TWO_SIDED if two_sided else L.SPECTRUM_ONE_SIDED
    fs = float(n * 250)  # one 4 ms period
    step = 125.0
    rate = len(chips[0]) / 0.004
    em = signals.Emitter(chips[1], rate, 1234.25, step, 58.0, data_rate=0.0)
    raw = signals.synthesize([em], fs, n * k, 20.0, "ci16", seed=n)
    codes = [ctx.code_put(chips[p], n, 1, mode) for p in range(3)]
    job = ctx.make_job(raw, L.SAMPLES_CI16, fs, n, k, codes, step, step, statistic=stat, spectrum_mode=mode)
    try:
        assert ctx.tile_shape(n)["warp_cols"] == 1
        got, gc = ctx.acquire(job, cells=True)
        ctx.set_tile_shape(n, dict(n1=ctx.tile_shape(n)["n1"], warp_cols=0))
        want, wc = ctx.acquire(job, cells=True)
    finally:
        ctx.set_tile_shape(n, None)
        for h in codes:
            ctx.code_release(h)
    for f in ("level", "mean", "std"):
        np.testing.assert_allclose(gc[f], wc[f], rtol=RTOL * (1 + stat))
    assert (got[1].index, got[1].doppler_bin) == (want[1].index, want[1].doppler_bin)
    assert got[1].doppler_bin == 2 and abs(got[1].index - 1234.25 / rate * fs) < 0.7 * fs / rate


@pytest.mark.parametrize("n,two_sided", [(5720, False), (6944, True), (8184, False), (9548, False), (10230, True), (11440, False)])
def test_small_four_step_blocks_vs_oracle(ctx, oracle, golden_codes, n, two_sided):
    from ugsdr_gb300 import _lib as L, signals
    chips = unpack_codes(golden_codes, "gps_l1ca")
    fs, k = n * 1e3, 2
    em = signals.Emitter(chips[4], 1.023e6, 300.5, 500.0, 52.0, data_rate=0.0)
    raw = signals.synthesize([em], fs, n * k, 20.0, "ci8", seed=n)
    mode = L.SPECTRUM_TWO_SIDED if two_sided else L.SPECTRUM_ONE_SIDED
    res, _ = run_engine(ctx, raw, fs, n, k, [chips[4]], 1, 1000, 500, spectrum_mode=mode)
    x, code = to_complex(raw), oracle.upsample(chips[4], n)
    check_vs_oracle(res[0], *(oracle.acquire(x, n, k, code, fs, 1000, 500, double=d, spectrum_mode=mode) for d in (False, True)))
