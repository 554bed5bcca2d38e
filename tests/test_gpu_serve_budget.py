"""Served searches under a small memory budget: a search whose full scratch
exceeds the budget runs with fewer rows (or Doppler bins) per launch, with the
same bits as without a budget, and one that cannot is still refused."""
import numpy as np
import pytest

from conftest import unpack_codes
from ugsdr_gb300 import _lib as L
from ugsdr_gb300.api import Server

pytestmark = pytest.mark.gpu

FIELDS = ("index", "doppler_bin", "level", "mean", "std", "snr")


@pytest.mark.parametrize("n,k,fold,budget_mb", [(10230, 20, 0, 128), (10230, 20, 0, 16), (8184, 20, 0, 100), (40920, 8, 0, 200),
                                                (20460, 4, 10230, 24)])
def test_small_budgets_run_in_smaller_batches(ctx, golden_codes, n, k, fold, budget_mb):
    chips = unpack_codes(golden_codes, "gps_l1ca")
    raw = np.random.default_rng(n).integers(-60, 61, (n * k, 2)).astype(np.int8)
    codes = [ctx.code_put(chips[p], n, n // fold if fold else 1) for p in range(32)]
    try:
        job = ctx.make_job(raw, L.SAMPLES_CI8, n * 1e3, n, k, codes, 10000.0, 500.0, fold_samples=fold, fold_coherent=False)
        want = ctx.acquire(job)
        srv = Server(ctx, max_inflight=1, memory_budget=budget_mb << 20)
        ticket = srv.submit(job)
        srv.drain()
        got = srv.poll(ticket)
        assert srv.stats()["device_bytes"] <= budget_mb << 20
        srv.close()
        tiny = Server(ctx, max_inflight=1, memory_budget=1 << 18)  # not even the samples
        ticket = tiny.submit(job)
        tiny.drain()
        with pytest.raises(L.UgsdrError) as e:
            tiny.poll(ticket)
        assert e.value.status == L.E_NOMEM
        tiny.close()
    finally:
        for h in codes:
            ctx.code_release(h)
    for a, b in zip(got, want):
        assert [getattr(a, f) for f in FIELDS] == [getattr(b, f) for f in FIELDS]
