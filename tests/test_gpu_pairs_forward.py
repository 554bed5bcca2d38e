"""Forward pair kernels against the forward kernels they replaced
(UGSDR_NO_WARP_FWD_ROWS): every sample type, the front-end mix, radices up to
32, ragged column and row tiles, several items per CTA, one- and two-sided
spectra.  The same inverse kernels read both, so what differs is the forward
stage; the bar is that of test_gpu_pairs.py."""
import numpy as np
import pytest

from conftest import unpack_codes

pytestmark = pytest.mark.gpu

RTOL = 2e-6
CASES = [
    # n, K, Doppler bins each side, sample type, front end, two-sided
    (10230, 3, 2, "ci8", 0.0, False),
    (13800, 2, 1, "ci16", 2e5, True),
    (26970, 1, 2, "cf32", 0.0, False),      # 29 x 31 x 30
    (30752, 5, 3, "ri8", -1e5, False),      # 31 x 31 x 32
    (40920, 2, 2, "ci8", 0.0, True),
    (50000, 4, 20, "ci16", 5e5, False),     # four items per CTA
    (152768, 1, 1, "cf32", 0.0, False),
    (204600, 3, 1, "ri8", 1e6, False),
    (332500, 1, 1, "ci16", 0.0, True),
    (984064, 1, 0, "ci8", 0.0, False),      # radices 31 and 32 on both sides
]


@pytest.mark.parametrize("n,k,half,sample_type,fe,two_sided", CASES)
def test_forward_pair_kernels_vs_former_ones(ctx, golden_codes, monkeypatch, n, k, half, sample_type, fe, two_sided):
    from ugsdr_gb300 import _lib as L
    chips = unpack_codes(golden_codes, "gps_l1ca")
    rng = np.random.default_rng(n)
    shape = n * k if sample_type == "ri8" else (n * k, 2)
    if sample_type == "cf32":
        raw = rng.normal(0, 20, shape).astype(np.float32)
    else:
        raw = rng.integers(-60, 61, shape).astype(np.int16 if sample_type == "ci16" else np.int8)
    st = {"ci8": L.SAMPLES_CI8, "ci16": L.SAMPLES_CI16, "cf32": L.SAMPLES_CF32, "ri8": L.SAMPLES_RI8}[sample_type]
    mode = L.SPECTRUM_TWO_SIDED if two_sided else L.SPECTRUM_ONE_SIDED
    codes = [ctx.code_put(chips[p], n, 1, mode) for p in range(2)]
    job = ctx.make_job(raw, st, n * 1e3, n, k, codes, 500.0 * half, 500.0, frontend_frequency=fe, spectrum_mode=mode)
    try:
        monkeypatch.delenv("UGSDR_NO_WARP_FWD_ROWS", raising=False)
        got = ctx.acquire(job, cells=True)[1]
        monkeypatch.setenv("UGSDR_NO_WARP_FWD_ROWS", "1")
        want = ctx.acquire(job, cells=True)[1]
    finally:
        for h in codes:
            ctx.code_release(h)
    assert got.tobytes() != want.tobytes()  # two sets of kernels ran
    for f in ("level", "mean", "std"):
        np.testing.assert_allclose(got[f], want[f], rtol=RTOL)
