"""Which folded searches run on transforms of the folded length, told from the
general path's (UGSDR_NO_FOLD_FIRST) by the kernels launched: not those of a
few samples, nor of hundreds of folds, whose mixing is a serial chain."""
import numpy as np
import pytest

from conftest import unpack_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,first", [(4000, 2, False), (4000, 100, False), (4000, 125, False), (4096, 128, True), (40000, 50, False),
                                       (40000, 200, True), (65536, 128, True), (131072, 128, False), (140000, 280, True),
                                       (166400, 320, False), (38192, 9548, True), (614400, 1024, True), (2046000, 2046, True)])
def test_folds_first_where_the_mix_is_short(ctx, golden_codes, monkeypatch, n, m, first):
    from ugsdr_gb300 import _lib as L
    chips = unpack_codes(golden_codes, "gps_l1ca")
    raw = np.random.default_rng(n).integers(-60, 61, (n, 2)).astype(np.int8)
    h = ctx.code_put(chips[0], n, n // m)

    def launches(general):
        if general:
            monkeypatch.setenv("UGSDR_NO_FOLD_FIRST", "1")
        else:
            monkeypatch.delenv("UGSDR_NO_FOLD_FIRST", raising=False)
        job = ctx.make_job(raw, L.SAMPLES_CI8, n * 1e3, n, 1, [h], 500.0, 500.0, fold_samples=m, fold_coherent=False)
        before = ctx.launch_count()
        res = ctx.acquire(job)
        return ctx.launch_count() - before, res[0]

    try:
        (general, want), (got_launches, got) = launches(True), launches(False)
    finally:
        ctx.code_release(h)
    assert (got_launches != general) == first
    assert got.level == pytest.approx(want.level, rel=1e-5) and got.std == pytest.approx(want.std, rel=1e-4)
