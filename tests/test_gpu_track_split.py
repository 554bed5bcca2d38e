"""A bank's state between calls: one run of many epochs and the same epochs in
several runs give the same bits, in both NCO modes (the carrier phase is the
64-bit fraction of a cycle or the reference's radians)."""
import numpy as np
import pytest

from conftest import unpack_codes
from ugsdr_gb300 import _lib as L
from ugsdr_gb300 import signals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fs", [4e6, 20e6])
@pytest.mark.parametrize("nco_mode", [0, 1])
def test_epochs_in_several_runs(ctx, golden_codes, nco_mode, fs):
    from ugsdr_gb300.api import TrackBank
    ca = unpack_codes(golden_codes, "gps_l1ca")
    ms, spm = 24, int(fs // 1000)
    raw, truth = signals.gps_l1_config(seed=5, codes={p: ca[p] for p in range(6)}, fs=fs, ms=ms, visible=3, cn0=(45, 50),
                                       max_doppler=3000)
    chans = [dict(code=t["prn"], fs=fs, code_frequency=1.023e6, code_phase=float(round(t["code_phase_samples"])),
                  carrier_frequency=t["doppler"] + 3.0, carrier_phase=0.7) for t in truth]

    def run(pieces):
        bank = TrackBank(ctx, chans, [ca[p] for p in range(6)], nco_mode=nco_mode)
        out, at = [], 0
        for n in pieces:
            out.append(bank.run(raw[at * spm:(at + n) * spm], L.SAMPLES_CI8, n))
            at += n
        bank.close()
        return np.concatenate(out).tobytes()

    whole = run([ms])
    assert run([ms // 2, ms // 2]) == whole
    assert run([1, 5, 18]) == whole
