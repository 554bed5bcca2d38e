"""Folded searches on transforms of the folded length (acq_folded.cuh) against
the general folded path (N-point transforms, UGSDR_NO_FOLD_FIRST): every form
the rule accepts gives the same peak and Doppler bin of planted signals and the
same statistics, and what it does not accept (a replica that does not repeat,
folded after the magnitude) gives the general path's very bits."""
import numpy as np
import pytest

from conftest import unpack_codes

pytestmark = pytest.mark.gpu

# float sums of at most 20 terms and transforms of up to 2^19 points, each
# within 3e-7 of 64 bits on its own path
RTOL = 2e-6

CASES = [
    # fs, ms, K, folds per ms-count, sample type, statistic, two-sided, front-end frequency
    (2.046e6, 2, 1, "ci8", 0, False, 0.0),     # one CTA either way, smallest block
    (4e6, 3, 2, "ci16", 1, True, 0.0),         # three folds: sqrt(1 / F) is not a power of two
    (4e6, 4, 2, "ci8", 0, False, 1.25e5),      # four-step -> the 4,000-point compile-time plan, translated
    (9.548e6, 4, 1, "cf32", 1, False, 0.0),    # odd radices
    (20.46e6, 5, 1, "ci16", 0, True, -3e6),    # four-step -> four-step (20,460)
    (50e6, 2, 2, "ci8", 0, False, 0.0),        # -> the warp-owned 50,000-point kernels
]


def search(ctx, monkeypatch, general, job, cells=True):
    if general:
        monkeypatch.setenv("UGSDR_NO_FOLD_FIRST", "1")
    else:
        monkeypatch.delenv("UGSDR_NO_FOLD_FIRST", raising=False)
    return ctx.acquire(job, cells=cells)


@pytest.mark.parametrize("coherent", [True, False])
@pytest.mark.parametrize("fs,ms,k,sample_type,stat,two_sided,fe", CASES)
def test_folded_length_vs_general(ctx, golden_codes, monkeypatch, fs, ms, k, sample_type, stat, two_sided, fe, coherent):
    from ugsdr_gb300 import _lib as L, signals
    ca = unpack_codes(golden_codes, "gps_l1ca")
    st = {"ci8": L.SAMPLES_CI8, "ci16": L.SAMPLES_CI16, "cf32": L.SAMPLES_CF32}[sample_type]
    mode = L.SPECTRUM_TWO_SIDED if two_sided else L.SPECTRUM_ONE_SIDED
    m, n = int(fs / 1000), int(fs / 1000) * ms
    step = 500.0 / ms
    ems = [signals.Emitter(ca[0], 1.023e6, 100.0, 3 * step - fe, 55.0, 0.0), signals.Emitter(ca[2], 1.023e6, 700.3, -2 * step - fe, 52.0, 0.0)]
    raw = signals.synthesize(ems, fs, n * k, 20.0, sample_type, seed=7)
    codes = [ctx.code_put(ca[p], n, ms, mode) for p in range(3)]
    job = ctx.make_job(raw, st, fs, n, k, codes, 4 * step, step, fold_samples=m, fold_coherent=coherent, statistic=stat,
                       spectrum_mode=mode, frontend_frequency=fe)
    want, wc = search(ctx, monkeypatch, True, job)
    got, gc = search(ctx, monkeypatch, False, job)
    for h in codes:
        ctx.code_release(h)
    for f in ("level", "mean", "std"):
        np.testing.assert_allclose(gc[f], wc[f], rtol=RTOL * (2 if stat else 1))
    for i in (0, 2):  # the planted signals
        assert (got[i].index, got[i].doppler_bin) == (want[i].index, want[i].doppler_bin)
    assert [g.doppler_bin for g in (got[0], got[2])] == [7, 2]


@pytest.mark.parametrize("mask,repeats", [(0b0110, 4), (0b0001, 4), (0, 2)])
def test_magnitude_fold_of_a_replica_that_does_not_repeat(ctx, golden_codes, monkeypatch, mask, repeats):
    """Signs per period, or a period of two folds: the general path, bit for
    bit where it has no atomics (one CTA); complex folds still fold first.
    Signs that cancel over the folds leave nothing but rounding of either
    path (a few 1e-7 of the unfolded correlation)."""
    from ugsdr_gb300 import _lib as L, signals
    ca = unpack_codes(golden_codes, "gps_l1ca")
    raw = signals.synthesize([signals.Emitter(ca[0], 1.023e6, 50.0, 250.0, 55.0, 0.0)], 2.046e6, 8184, 20.0, "ci8", seed=3)
    chips = np.tile(ca[0], 4 // repeats) * (1.0 if repeats == 4 else np.repeat([1.0, -1.0], 1023).astype(np.float32))
    h = ctx.code_put(chips, 8184, repeats, sign_mask=mask, sign_segment=2046)
    for coherent in (True, False):
        job = ctx.make_job(raw, L.SAMPLES_CI8, 2.046e6, 8184, 1, [h], 500, 125, fold_samples=2046, fold_coherent=coherent)
        _, wc = search(ctx, monkeypatch, True, job)
        _, gc = search(ctx, monkeypatch, False, job)
        if coherent:
            assert gc.tobytes() == wc.tobytes()
        elif mask == 0b0001:
            np.testing.assert_allclose(gc["level"], wc["level"], rtol=RTOL)
        else:
            whole = ctx.acquire(ctx.make_job(raw, L.SAMPLES_CI8, 2.046e6, 8184, 1, [h], 500, 125), cells=True)[1]
            assert max(gc["level"].max(), wc["level"].max()) < RTOL * whole["level"].max()
    ctx.code_release(h)
