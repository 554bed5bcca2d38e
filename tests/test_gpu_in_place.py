"""Single-CTA inverse kernels with the passes in place, at the edges of their
plans: first radices odd and even, the padding of a group of rows at its
smallest and largest, butterflies short of and beyond a round of threads, the
compile-time 4,000-point kernel, and clusters of every size with and without a
remainder of the K blocks.  Checks and bars as in test_gpu_small.py."""
import pytest

import test_gpu_small as small

pytestmark = pytest.mark.gpu

CASES = [
    # n, K, Doppler bins each side, sample type, two-sided, statistic
    (4000, 1, 2, "ci8", False, 0),
    (4000, 2, 1, "cf32", False, 1),
    (4000, 7, 1, "ci16", False, 0),    # clusters of seven
    (4000, 17, 2, "ri8", True, 0),     # of six: three blocks each, the last two
    (4000, 10, 100, "ci8", False, 0),  # 201 rows
    (4096, 8, 1, "ci8", False, 0),     # 16 x 16 x 16: even first radix, clusters of eight
    (4096, 3, 1, "ci16", True, 1),
    (2500, 19, 1, "ci8", False, 0),
    (3600, 5, 1, "cf32", True, 0),
    (4913, 3, 1, "ci8", False, 0),     # 17 x 17 x 17
    (5456, 4, 2, "ci16", False, 0),    # 31 x 16 x 11
    (5488, 6, 1, "ri8", False, 1),     # 28 x 14 x 14
]


@pytest.mark.parametrize("n,k,half,sample_type,two_sided,stat", CASES)
def test_in_place_blocks_vs_oracle(ctx, oracle, golden_codes, n, k, half, sample_type, two_sided, stat):
    small.test_small_blocks_vs_oracle(ctx, oracle, golden_codes, n, k, half, sample_type, two_sided, stat)
