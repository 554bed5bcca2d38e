"""Standard deviation of searches of many blocks against 64 bits, on every
column kernel: pair (one CTA could hold the block, or not), warp-owned,
natural layout, and the folded search on its folded length.

The bar: an accumulator's K float additions round to about 2^-24 sqrt(K) / 3 of
the mean, the mean is sqrt(3.7 K) sigmas, and errors independent over N cells
move the deviation by 1 / sqrt(N) of that: at most 2e-7 here.  Transforms and
twiddles add a few 1e-7.  Squares summed about zero in float lose 2^-24 of
(mean / sigma)^2 = 3.7 K instead, several 1e-6."""
import numpy as np
import pytest

from conftest import unpack_codes

pytestmark = pytest.mark.gpu

RTOL = 1.5e-6
CASES = [
    # block, K, folded length, tile shape
    (10230, 500, 0, None),
    (8184, 500, 0, None),
    (20460, 400, 0, None),
    (16000, 400, 0, dict(warp_cols=0)),
    (50000, 250, 0, None),
    (40920, 200, 20460, None),
]


@pytest.mark.parametrize("n,k,fold,shape", CASES)
def test_deviation_of_many_blocks(ctx, golden_codes, n, k, fold, shape):
    from ugsdr_gb300 import _lib as L
    chips = unpack_codes(golden_codes, "gps_l1ca")
    raw = np.random.default_rng(n).integers(-60, 61, (n * k, 2)).astype(np.int8)
    repeats = n // fold if fold else 1
    if shape:
        ctx.set_tile_shape(n, shape)
    codes = [ctx.code_put(chips[p], n, repeats) for p in range(4)]
    try:
        job = ctx.make_job(raw, L.SAMPLES_CI8, n * 1e3, n, k, codes, 0.0, 500.0, fold_samples=fold, fold_coherent=False)
        _, cells = ctx.acquire(job, cells=True)
    finally:
        for h in codes:
            ctx.code_release(h)
        if shape:
            ctx.set_tile_shape(n, None)
    x = np.fft.fft((raw[:, 0] + 1j * raw[:, 1].astype(np.float64)).reshape(k, n))
    for p in range(4):
        code = np.tile(chips[p], repeats)[np.arange(n, dtype=np.int64) * (1023 * repeats) // n].astype(np.float64)
        spec = np.conj(np.fft.fft(code))
        spec[n // 2 + 1:] = 0
        acc = np.zeros(fold or n)
        for b in range(k):
            y = 2 * np.fft.ifft(x[b] * spec)
            acc += np.abs(y.reshape(-1, fold).sum(0) if fold else y)
        assert abs(cells["mean"][p, 0] / acc.mean() - 1) < 5e-7
        assert abs(cells["std"][p, 0] / acc.std(ddof=1) - 1) < RTOL
