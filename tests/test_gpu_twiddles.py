"""Inter-step twiddles of the pair kernels against 64 bits: forward transforms
(ugsdr_dft) of splits with radices up to 32 on both sides.

The bar: a recurrence of seven products carries its step's rounding (rms 3.4e-8)
seven times at most, rms 1.4e-7 over a butterfly; the passes of a million-point
transform 1.2e-7, the twiddles' own arguments 0.8e-7: 2e-7 in all, 3e-7 with a
margin.  A recurrence of 31 products adds 6e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31 * 32 * 31 * 32, 31 * 31 * 31 * 31, 32 * 29 * 31 * 29, 1000000, 332500, 204600, 65536, 40920])
def test_four_step_dft_vs_64_bits(ctx, n):
    rng = np.random.default_rng(n)
    x = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(np.complex64)
    want = np.fft.fft(x.astype(np.complex128))
    assert np.linalg.norm(ctx.dft(x) - want) <= 3e-7 * np.linalg.norm(want)
