"""Tile shapes say what runs: on a split of the pair kernels the widths asked
for are those of its tiles, widths the pair kernels do not have take it to the
natural layout (the same bits as asking for that), and the tuner measures no
set of kernels twice under different names."""
import numpy as np
import pytest

from conftest import unpack_codes
from ugsdr_gb300 import _lib as L

pytestmark = pytest.mark.gpu

KEY = ("n1", "cols", "rows", "warp_cols", "warp_rows")


@pytest.mark.parametrize("n", [16000, 20460, 40920])
def test_widths_on_a_pair_split(ctx, golden_codes, n):
    chips = unpack_codes(golden_codes, "gps_l1ca")
    raw = np.random.default_rng(n).integers(-60, 61, (n * 2, 2)).astype(np.int8)
    codes = [ctx.code_put(chips[p], n) for p in range(3)]
    job = ctx.make_job(raw, L.SAMPLES_CI8, n * 1e3, n, 2, codes, 1000.0, 500.0)

    def with_shape(**shape):
        ctx.set_tile_shape(n, shape)
        return ctx.tile_shape(n), ctx.acquire(job, cells=True)[1]

    try:
        rule = ctx.tile_shape(n)
        assert rule["cols"] in (4, 8) and rule["rows"] in (4, 8) and (rule["warp_cols"], rule["warp_rows"]) == (1, 0)
        want = ctx.acquire(job, cells=True)[1]
        for cols, rows in ((4, 4), (8, 4), (4, 8), (8, 8), (0, 8), (4, 0)):
            got, cells = with_shape(cols=cols, rows=rows)
            assert (got["cols"], got["rows"], got["warp_cols"], got["warp_rows"]) == (cols or got["cols"], rows or got["rows"], 1, 0)
            for f in ("level", "mean", "std"):
                np.testing.assert_allclose(cells[f], want[f], rtol=2e-6)
        for cols, rows in ((2, 2), (1, 4), (4, 2), (2, 0)):
            got, cells = with_shape(cols=cols, rows=rows)
            assert got["warp_cols"] == 0 and got["cols"] == cols and got["rows"] == (rows or got["rows"])
            asked, same = with_shape(cols=cols, rows=rows, warp_cols=0)
            assert asked == got and same.tobytes() == cells.tobytes()
        got, cells = with_shape(cols=2, rows=2, warp_cols=1)
        assert {k: got[k] for k in KEY} == {k: rule[k] for k in KEY} and cells.tobytes() == want.tobytes()
        ctx.set_tile_shape(n, None)
        tried = ctx.autotune([job])
        mine = [t for t in tried if t["block_samples"] == n]
        assert len({tuple(t[k] for k in KEY) for t in mine}) == len(mine) >= 2
        assert all(t["warp_rows"] == 0 and (not t["warp_cols"] or (t["cols"] in (4, 8) and t["rows"] in (4, 8))) for t in mine)
    finally:
        ctx.set_tile_shape(n, None)
        for h in codes:
            ctx.code_release(h)
    assert ctx.tile_shape(n) == rule
