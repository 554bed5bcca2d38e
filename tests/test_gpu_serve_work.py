"""The server's estimate of a search's work (its trace): that of the transforms
the search runs, so that a folded search counts as one of the folded length
beside its mixing, and a few of them leave the measured rate, by which the
server tells long searches from short ones, where it is."""
import re

import numpy as np
import pytest

from conftest import unpack_codes
from ugsdr_gb300 import _lib as L
from ugsdr_gb300.api import Server

pytestmark = pytest.mark.gpu


def submitted_work(ctx, job, capfd):
    capfd.readouterr()
    srv = Server(ctx, max_inflight=1)
    ticket = srv.submit(job)
    srv.drain()
    srv.poll(ticket)
    srv.close()
    return float(re.search(r"submit ticket \d+ work (\S+)", capfd.readouterr().err).group(1))


@pytest.mark.parametrize("m,folds,k,coherent", [(2046, 4, 3, True), (9548, 4, 1, False), (50000, 20, 2, True)])
def test_folded_work_is_that_of_the_folded_length(ctx, golden_codes, monkeypatch, capfd, m, folds, k, coherent):
    monkeypatch.setenv("UGSDR_SERVER_TRACE", "1")
    chips = unpack_codes(golden_codes, "gps_l1ca")
    raw = np.zeros((m * folds * k, 2), np.int8)
    codes = [ctx.code_put(chips[p], m * folds, folds) for p in range(8)]
    short = [ctx.code_put(chips[p], m) for p in range(8)]
    try:
        folded = submitted_work(ctx, ctx.make_job(raw, L.SAMPLES_CI8, m * 1e3, m * folds, k, codes, 1000.0, 250.0, fold_samples=m,
                                                  fold_coherent=coherent), capfd)
        plain = submitted_work(ctx, ctx.make_job(raw[:m * k], L.SAMPLES_CI8, m * 1e3, m, k, short, 1000.0, 250.0), capfd)
        general = submitted_work(ctx, ctx.make_job(raw, L.SAMPLES_CI8, m * 1e3, m * folds, k, codes, 1000.0, 250.0), capfd)
    finally:
        for h in codes + short:
            ctx.code_release(h)
    cells = 8 * 9 * k
    assert plain == pytest.approx(cells * m, rel=0.01) and general == pytest.approx(cells * m * folds, rel=0.01)
    assert plain < folded < 2 * plain and folded < 0.5 * general
