"""Samples of any magnitude that float holds the correlation of: a search of
complex-float samples times 10^e gives 10^e (statistic |.|) or 10^2e (|.|^2)
times the cells of the samples themselves, on every kernel of the four-step
path.  The bar: the scaled samples' own rounding, 2^-24, in level, mean and
deviation alike; 2e-6 leaves both runs' transforms their 5e-7."""
import numpy as np
import pytest

from conftest import unpack_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stat,exponents", [(0, (9, 12, 13, -12, -18)), (1, (6, 12, -12))])
@pytest.mark.parametrize("n,fold", [(10230, 0), (20460, 0), (40920, 0), (50000, 0), (40920, 20460), (100000, 50000), (500000, 0)])
def test_cells_scale_with_the_samples(ctx, golden_codes, n, fold, stat, exponents):
    from ugsdr_gb300 import _lib as L
    chips = unpack_codes(golden_codes, "gps_l1ca")
    x = np.random.default_rng(n).normal(0, 1, (n * 3, 2)).astype(np.float32)
    h = ctx.code_put(chips[0], n, n // fold if fold else 1)

    def cells(samples):
        job = ctx.make_job(samples, L.SAMPLES_CF32, n * 1e3, n, 3, [h], 500.0, 500.0, fold_samples=fold, fold_coherent=False,
                           statistic=stat)
        return ctx.acquire(job, cells=True)[1]

    try:
        want = cells(x)
        for e in exponents:
            got = cells((x * 10.0 ** e).astype(np.float32))
            for f in ("level", "mean", "std"):
                np.testing.assert_allclose(got[f].astype(np.float64) / 10.0 ** (e * (1 + stat)), want[f], rtol=2e-6 * (1 + stat))
    finally:
        ctx.code_release(h)
