"""The detector on samples that are not numbers: a column of NaN has its
candidates from the lowest bin on, each the first that the one before it did
not null (+-3 bins), as the maximum of the magnitudes' bit patterns gives
them."""
import numpy as np
import pytest

from ugsdr_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 1120, 40000])
def test_nan_columns_from_the_lowest_bin(ctx, n):
    det = ctx.jamming_detect(np.full(n, np.nan + 1j * np.nan, np.complex64), 4e6)
    got = [(d["type"], d["frequency_bin"]) for d in det]
    assert got == [(t, 4 * r) for r in range(8) for t in (L.INTERFERENCE_NARROWBAND, L.INTERFERENCE_WIDEBAND)]
    assert all(np.isnan(d["jammer_to_noise"]) for d in det)
