"""Interference stage at the edges of its tiles against the oracle: one column,
a batch of 32 columns and its neighbours, columns and samples that end inside
a run of output slots, one run per octet and several waves of them.  Bars as
in test_gpu_jamming.py."""
import numpy as np
import pytest

from test_gpu_jamming import same_detections

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jammed", [True, False])
@pytest.mark.parametrize("n", [128, 129, 159, 160, 1119, 1120, 1121, 1152, 3205, 8192 + 127, 262144 + 33, 1500001])
def test_ragged_lengths_vs_oracle(ctx, oracle, n, jammed):
    rng = np.random.default_rng(n)
    x = (rng.normal(0, 0.5, n) + 1j * rng.normal(0, 0.5, n)).astype(np.complex64)
    if jammed:
        x += (10 * np.exp(2j * np.pi * 20 / 128 * np.arange(n))).astype(np.complex64)
    ref_det, ref = oracle.jamming(x, 4e6)
    y = x.copy()
    same_detections(ctx.jamming_suppress(y, 4e6), ref_det)
    assert np.abs(y - ref).max() <= 1e-4 * np.abs(x).max()
