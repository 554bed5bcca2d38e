"""Performance cases: what a user of the library has it do, through the Python
layer over the C ABI (ugsdr_gb300.api).

Five kinds of call, each over the range it has in use:

  search        Context.acquire: one PRN x Doppler x code-phase search, from a
                1 ms block at 1.7 MHz to a 20 ms block at 50 MHz (1,736 to
                1,000,000 points), host or device capture, int8 / int16 /
                float I/Q, one- or two-sided spectra, folded or not, with the
                front end (IF translate, resampling) or without
  batch         Context.acquire_batch: every system of one wideband capture
  track         TrackBank.run / run_device: a correlator bank over one stretch
                of capture, from a receiver's dozen channels to 256
  interference  Context.jamming_suppress: detection and suppression, in place
                on a device capture
  observables   observables and preamble_search over a bank's outputs

Every input is synthesised from the seed: signals of the named systems with
uniform delay, Doppler and C/N0 in additive white Gaussian noise.  The context
and its code spectra are made once per process, as a receiver keeps them.

Single-precision results (level, mean, sigma: ugsdr_acq_cell's floats, which
AcqResult widens to double) are returned as float32; values computed in double
stay float64.
"""
import functools
import math

import numpy as np
import torch

from ugsdr_gb300 import _lib as L
from ugsdr_gb300 import api, signals

DEV = "cuda:0"
SIGMA = 20.0          # noise per I / Q component, LSB
TRACK_CFG = dict(early_late=0.15, very_early_late=0.5, pll_bw=15.0, dll_bw=1.0, fll_bw=0.0)
TYPES = {"ci8": L.SAMPLES_CI8, "ci16": L.SAMPLES_CI16, "cf32": L.SAMPLES_CF32, "ri8": L.SAMPLES_RI8}
# signal id, codes the system has, chip rate (E1B: half-chips), code period in ms
SYSTEMS = {"gps": (L.GPS_L1CA, 32, 1.023e6, 1), "l5i": (L.GPS_L5I, 32, 10.23e6, 1),
           "e1b": (L.GALILEO_E1B, 36, 2.046e6, 4), "glo": (L.GLONASS_L1OF, 1, 0.511e6, 1)}
# the request mix's rates, and the other rates of the captures the tests search
RATES = (1.736e6, 2.046e6, 4e6, 4.092e6, 9.548e6, 10.23e6, 16.384e6, 20.46e6, 33.25e6, 38.192e6, 50e6)
BATCH_CENTER = 1590e6


# ---------------------------------------------------------------- the cases
def _search(name, system, fs, t_ms, k, n_codes, span, step, sample_type="ci8", device=False, cells=False, fold=0,
            two_sided=False, abs2=False, fs_in=0.0, if_hz=0.0, nh10=False):
    case = dict(kind="search", system=system, fs=fs, t_ms=t_ms, k=k, n_codes=n_codes, span=span, step=step,
                sample_type=sample_type, device=device, cells=cells, fold=fold, two_sided=two_sided, abs2=abs2,
                fs_in=fs_in, if_hz=if_hz, nh10=nh10)
    return dict(case, name=name) if name else case


def listed():
    return [
        # a hot re-acquisition request: 8 PRNs, 4 ms of host int8 capture; latency
        # and launches count.  Its per-cell records are read as well
        _search("short_gps_4mhz", "gps", 4e6, 1, 4, 8, 5000.0, 500.0, cells=True),
        # a receiver's cold start at its narrowest front end, odd block size
        _search("cold_gps_2mhz", "gps", 2.046e6, 1, 20, 32, 5000.0, 500.0, sample_type="ci16"),
        # the plain GPS L1 C/A search: 32 PRNs x 21 bins x 4,000 x 10 blocks
        _search("plain_gps_4mhz", "gps", 4e6, 1, 10, 32, 5000.0, 500.0),
        # the drop-in engine's GPS search (four periods coherently, folded to 1 ms
        # after the magnitude) at the rate it picks for a 38.192 MHz capture
        _search("engine_gps_9mhz", "gps", 9.548e6, 4, 1, 32, 5000.0, 125.0, device=True, fold=1),
        # a mid-size request of the served mix: Galileo E1B, 4 ms at 10.23 MHz
        _search("e1b_10mhz", "e1b", 10.23e6, 4, 10, 36, 5000.0, 125.0, sample_type="ci16", device=True),
        # weak-signal L5I: real int8 at 40 MHz, IF 10 MHz, resampled to 20.46 MHz on
        # the device, 10 ms coherent with the NH10 code wiped off, x 20 blocks
        _search("weak_l5i_20mhz", "l5i", 20.46e6, 10, 20, 16, 1000.0, 25.0, sample_type="ri8", device=True,
                fs_in=40e6, if_hz=10e6, nh10=True),
        # the longest coherent block: 20 ms at 50 MHz (1,000,000 points), folded to
        # one code period before the magnitude
        _search("long_gps_50mhz", "gps", 50e6, 20, 2, 12, 1000.0, 25.0, sample_type="ci16", device=True, fold=2),
        # one 40 ms, 50 MHz int16 capture searched for every system at once: GPS L1
        # C/A, 14 GLONASS letters, Galileo E1B
        dict(name="multi_50mhz", kind="batch", fs=50e6, ms=40, gps=32, letters=14, e1b=36, step=250.0),
        # the tracking bank at capacity: 256 channels at 20 MHz, 200 ms
        dict(name="track_256ch_20mhz", kind="track", fs=20e6, channels=256, epochs=200, sample_type="ci16", device=True),
        # a receiver's bank in real time: 12 channels, 100 ms of host int8 samples
        dict(name="track_12ch_4mhz", kind="track", fs=4e6, channels=12, epochs=100, sample_type="ci8", device=False),
        # the antijamming stage over 400 ms at 50 MHz, a CW jammer on an STFT bin
        dict(name="interference_50mhz", kind="interference", fs=50e6, n=20000000, jammer="cw"),
        # a minute of 256 channels' outputs turned into measurements
        dict(name="observables_256ch", kind="observables", channels=256, epochs=60000),
    ]


def draw(rng):
    kind = rng.choices(("search", "batch", "track", "interference", "observables"), (10, 1, 3, 1.5, 1.5))[0]
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    if kind == "search":
        system = rng.choice(("gps", "gps", "l5i", "e1b"))
        _, have, chip_rate, period = SYSTEMS[system]
        fs = rng.choice([r for r in RATES if r > chip_rate])
        # one code period, or several folded to one (a replica that repeats
        # correlates alike at every period), or the ten of an NH10 code
        t_ms, fold, nh10 = period, 0, False
        if system == "l5i" and rng.random() < 0.4:
            t_ms, nh10 = 10, True
        elif rng.random() < 0.45:
            t_ms, fold = period * rng.randint(2, 20 // period), rng.choice((1, 2))
        n = round(fs * t_ms / 1000)
        k = rng.randint(1, min(40, max(1, int(4e7 / n))))
        n_codes = rng.randint(1, have)
        # transform points, over the range of the listed searches
        points = log(5e5, 6e9)
        while n_codes > 1 and n_codes * k * n * 3 > points:
            n_codes = (n_codes + 1) // 2
        while k > 1 and n_codes * k * n * 3 > points:
            k = (k + 1) // 2
        step = 1000.0 / (2 * t_ms)
        half = max(1, min(int(points / (n_codes * k * n)) // 2, int(5000.0 / step)))
        return _search("", system, fs, t_ms, k, n_codes, half * step, step,
                       sample_type=rng.choice(("ci8", "ci8", "ci16", "ci16", "cf32")), device=rng.random() < 0.6,
                       cells=n_codes * (2 * half + 1) <= 100, fold=fold, two_sided=rng.random() < 0.15,
                       abs2=rng.random() < 0.15, nh10=nh10)
    if kind == "batch":
        return dict(kind="batch", fs=rng.choice((20.46e6, 38.192e6, 50e6)), ms=4 * rng.randint(1, 10), gps=rng.randint(4, 32),
                    letters=rng.randint(1, 14), e1b=rng.randint(2, 24), step=rng.choice((250.0, 500.0)))
    if kind == "track":
        fs = rng.choice((4e6, 9.548e6, 10e6, 16.384e6, 20e6, 33.25e6, 50e6))
        channels = int(log(4, 256.99))
        return dict(kind="track", fs=fs, channels=channels, epochs=rng.choice((20, 40, 100, 200)),
                    sample_type=rng.choice(("ci8", "ci16", "cf32")), device=rng.random() < 0.5)
    if kind == "interference":
        fs = rng.choice((4e6, 20.46e6, 50e6))
        return dict(kind="interference", fs=fs, n=round(fs * int(log(4, 400.99)) / 1000),
                    jammer=rng.choice(("cw", "cw", "none", "gated")))
    return dict(kind="observables", channels=int(log(8, 256.99)), epochs=int(log(2000, 60000)))


# ------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _ctx():
    stream = torch.cuda.Stream()
    ctx = api.Context(0)
    ctx.set_stream(stream.cuda_stream)
    return ctx, stream


@functools.lru_cache(maxsize=None)
def _chips(system, sv):
    return api.prn_code(SYSTEMS[system][0], sv)


@functools.lru_cache(maxsize=None)
def _code(system, sv, n, repeats, mode, mask=0, segment=0):
    return _ctx()[0].code_put(_chips(system, sv), n, repeats, spectrum_mode=mode, sign_mask=mask, sign_segment=segment)


def _synthesise(emitters, fs, n, sample_type, seed):
    """The capture on the device: emitters are dicts of chips, rate, delay
    (chips), f (Hz), cn0 (dB-Hz), data_rate (0: pilot), weight and nh10."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    t = torch.arange(n, dtype=torch.float64, device=DEV) / fs
    real = sample_type == "ri8"
    iq = torch.randn((n, 2), generator=gen, device=DEV) * SIGMA
    for e in emitters:
        chips = torch.as_tensor(e["chips"], device=DEV)
        pos = t * e["rate"] - e["delay"]
        s = chips[torch.remainder(torch.floor(pos), chips.numel()).long()]
        if e["data_rate"]:
            bits = rng.choice([-1.0, 1.0], size=int(n / fs * e["data_rate"]) + 2).astype(np.float32)
            s = s * torch.as_tensor(bits, device=DEV)[torch.floor(t * e["data_rate"]).long()]
        if e.get("nh10"):
            sec = torch.as_tensor(1.0 - 2.0 * signals.NH10, dtype=torch.float32, device=DEV)
            s = s * sec[torch.remainder(torch.floor(pos / chips.numel()), 10).long()]
        cyc = e["f"] * t + e["phase"]
        ang = (2 * math.pi * (cyc - torch.floor(cyc))).float()
        amp = SIGMA * math.sqrt(2.0 * 10 ** (e["cn0"] / 10.0) / fs) * e.get("weight", 1.0)
        iq[:, 0] += amp * (math.sqrt(2.0) if real else 1.0) * s * torch.cos(ang)
        iq[:, 1] += amp * s * torch.sin(ang)
    if sample_type == "cf32":
        return iq.contiguous()
    lim = 32767 if sample_type == "ci16" else 127
    q = torch.clamp(torch.round(iq[:, 0] if real else iq), -lim - 1, lim)
    return q.to(torch.int16 if sample_type == "ci16" else torch.int8).contiguous()


def _emitters(system, rng, count, have, carrier, cn0, data_rate, glo_letter=None):
    _, _, rate, period = SYSTEMS[system]
    out = []
    for p in rng.choice(have, min(count, have), replace=False):
        chips = _chips(system, int(p))
        out.append(dict(chips=chips, rate=rate, delay=rng.uniform(0, len(chips)), f=carrier + rng.uniform(-900, 900),
                        cn0=rng.uniform(*cn0), data_rate=data_rate, phase=rng.uniform(0, 1), sv=int(p), system=system))
    return out


def _bins(span, step):
    """The Doppler grid of ProcessBpsk's loop, accumulation included."""
    grid, d = [], -span
    while d <= span:
        grid.append(d)
        d += step
    return grid


def _search_shape(case):
    n = round(case["fs"] * case["t_ms"] / 1000)
    spm = round(case["fs"] / 1000)
    fold = spm * SYSTEMS[case["system"]][3] if case["fold"] else 0
    fs_in = case["fs_in"] or case["fs"]
    n_in = math.ceil(n * case["k"] * fs_in / case["fs"])
    return n, fold, fs_in, n_in


def _search_capture(case, seed):
    n, fold, fs_in, n_in = _search_shape(case)
    rng = np.random.default_rng(seed)
    lo = (30.0, 38.0) if case["nh10"] else (38.0, 48.0)
    ems = _emitters(case["system"], rng, max(1, case["n_codes"] // 4), case["n_codes"], case["if_hz"], lo,
                    0.0 if case["nh10"] else 50.0)
    for e in ems:
        if case["nh10"]:
            e["nh10"], e["delay"] = True, rng.uniform(0, 10 * len(e["chips"]))
    return _synthesise(ems, fs_in, n_in, case["sample_type"], seed)


def _prepare_search(case, seed):
    ctx, _ = _ctx()
    n, fold, fs_in, n_in = _search_shape(case)
    mode = L.SPECTRUM_TWO_SIDED if case["two_sided"] else L.SPECTRUM_ONE_SIDED
    repeats = case["t_ms"] // SYSTEMS[case["system"]][3]
    mask, segment = (signals.nh10_mask(), n // 10) if case["nh10"] else (0, 0)
    codes = [_code(case["system"], sv, n, repeats, mode, mask, segment) for sv in range(case["n_codes"])]
    x = _search_capture(case, seed)
    if not case["device"]:
        x = x.cpu().numpy()
    return dict(case=case, samples=x, codes=codes, n=n, n_in=n_in, fold=fold, mode=mode)


def _job(ctx, s, case):
    x = s["samples"]
    return ctx.make_job(x.data_ptr() if case["device"] else x, TYPES[case["sample_type"]], case["fs"], s["n"], case["k"],
                        s["codes"], case["span"], case["step"], n_samples=s["n_in"], on_device=case["device"],
                        intermediate_frequency=case["if_hz"], frontend_frequency=-case["if_hz"], fold_samples=s["fold"],
                        fold_coherent=case["fold"] == 1, statistic=L.STAT_ABS2 if case["abs2"] else L.STAT_ABS,
                        spectrum_mode=s["mode"], input_sampling_rate=case["fs_in"])


def _results(res):
    single = ("level", "sigma", "mean", "std", "snr")
    out = {f: np.array([getattr(r, f) for r in res], np.float32) for f in single}
    out.update({f: np.array([getattr(r, f) for r in res]) for f in ("index", "doppler_bin", "doppler", "code_offset")})
    return out


def _run_search(s):
    ctx, _ = _ctx()
    case = s["case"]
    if not case["cells"]:
        return _results(ctx.acquire(_job(ctx, s, case)))
    res, cells = ctx.acquire(_job(ctx, s, case), cells=True)
    return dict(results=_results(res), cells={f: cells[f] for f in cells.dtype.names})


# -------------------------------------------------------------------- batch
def _batch_jobs(case):
    """(system, svs, block samples, K, step, IF) of each job of the capture."""
    fs = case["fs"]
    if_l1 = 1575.42e6 - BATCH_CENTER
    one = round(fs / 1000)
    jobs = [("gps", range(case["gps"]), one, case["ms"], case["step"], if_l1)]
    jobs += [("glo", range(1), one, case["ms"], case["step"], (1602e6 + (i - 7) * 0.5625e6 - BATCH_CENTER) % fs)
             for i in range(case["letters"])]
    jobs.append(("e1b", range(case["e1b"]), 4 * one, case["ms"] // 4, case["step"] / 4, if_l1))
    return jobs


def _batch_capture(case, seed):
    rng = np.random.default_rng(seed)
    ems = []
    for system, svs, _, _, _, f_if in _batch_jobs(case):
        visible = 8 if len(svs) > 1 else int(rng.integers(0, 2))
        ems += _emitters(system, rng, visible, len(svs), f_if, (38.0, 48.0), 250.0 if system == "e1b" else 50.0)
    return _synthesise(ems, case["fs"], round(case["fs"] * case["ms"] / 1000), "ci16", seed)


def _prepare_batch(case, seed):
    codes = [[_code(system, sv, n, 1, L.SPECTRUM_ONE_SIDED) for sv in svs] for system, svs, n, _, _, _ in _batch_jobs(case)]
    return dict(case=case, samples=_batch_capture(case, seed), codes=codes)


def _run_batch(s):
    ctx, _ = _ctx()
    x = s["samples"]
    jobs = [ctx.make_job(x.data_ptr(), L.SAMPLES_CI16, s["case"]["fs"], n, k, codes, 5000.0, step, n_samples=x.shape[0],
                         on_device=True, intermediate_frequency=f_if, frontend_frequency=-f_if)
            for codes, (_, _, n, k, step, f_if) in zip(s["codes"], _batch_jobs(s["case"]))]
    return _results([r for res in ctx.acquire_batch(jobs) for r in res])


# -------------------------------------------------------------------- track
def _prepare_track(case, seed):
    """Channels on signals that repeat seamlessly with the capture (whole code
    periods, carrier cycles and data bits), so that a bank may run over the
    same capture again and stay in lock as over a longer one."""
    ctx, _ = _ctx()
    rng = np.random.default_rng(seed)
    fs, seconds = case["fs"], case["epochs"] / 1000
    n = round(fs * seconds)
    gps, e1b = 32, 36
    table = [_chips("gps", p) for p in range(gps)] + [_chips("e1b", p) for p in range(e1b)]
    ems, chans = [], []
    for i in range(case["channels"]):
        ci = int(rng.integers(0, gps + e1b))
        rate = 1.023e6 if ci < gps else 2.046e6
        delay = rng.uniform(0, len(table[ci]))
        f = round(rng.uniform(-5000, 5000) * seconds) / seconds
        ems.append(dict(chips=table[ci], rate=rate, delay=delay, f=f, cn0=rng.uniform(42, 50), phase=rng.uniform(0, 1),
                        data_rate=50.0 if ci < gps else 250.0))
        chans.append(dict(code=ci, fs=fs, code_frequency=rate, code_phase=float(round(delay / rate * fs)),
                          carrier_frequency=f + rng.uniform(-5, 5), boc=int(ci >= gps)))
    x = _synthesise(ems, fs, n, case["sample_type"], seed)
    bank = api.TrackBank(ctx, chans, table, **TRACK_CFG)
    out = None
    if case["device"]:
        out = torch.zeros((case["epochs"], case["channels"], api.TRACK_DTYPE.itemsize), dtype=torch.uint8, device=DEV)
    return dict(case=case, samples=x if case["device"] else x.cpu().numpy(), bank=bank, out=out)


def _run_track(s):
    case, bank = s["case"], s["bank"]
    if case["device"]:
        bank.run_device(s["samples"].data_ptr(), TYPES[case["sample_type"]], case["epochs"], s["out"].data_ptr())
        return dict(taps=s["out"].view(torch.float32)[:, :, :10], loops=s["out"].view(torch.float64)[:, :, 5:])
    rows = bank.run(s["samples"], TYPES[case["sample_type"]], case["epochs"])
    return {f: rows[f] for f in rows.dtype.names}


# ------------------------------------------------------------- interference
def _interference_capture(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    n = case["n"]
    x = torch.randn((n, 2), generator=gen, device=DEV) * 0.5
    if case["jammer"] != "none":
        bin_ = int(np.random.default_rng(seed).integers(5, 120))
        ph = torch.arange(n, device=DEV) * bin_ % 128 * (2 * math.pi / 128)
        amp = torch.full((n,), 10.0, device=DEV)
        if case["jammer"] == "gated":  # on in one slot of twenty
            amp = amp * (torch.arange(n, device=DEV) * 20 // n == 7)
        x[:, 0] += amp * torch.cos(ph)
        x[:, 1] += amp * torch.sin(ph)
    return x


def _prepare_interference(case, seed):
    x = _interference_capture(case, seed)
    return dict(case=case, capture=x, work=torch.empty_like(x))


def _run_interference(s):
    ctx, stream = _ctx()
    with torch.cuda.stream(stream):  # the stage works in place: the next capture arrives in the buffer
        s["work"].copy_(s["capture"])
    found = ctx.jamming_suppress(s["work"].data_ptr(), s["case"]["fs"], s["case"]["n"])
    return dict(samples=s["work"], detections=found)


# -------------------------------------------------------------- observables
def _prepare_observables(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    n_ep, n_ch = case["epochs"], case["channels"]
    f64 = dict(generator=gen, device=DEV, dtype=torch.float64)
    rec = torch.zeros((n_ep, n_ch, 22), dtype=torch.float32, device=DEV)
    rec[:, :, :10] = torch.randn((n_ep, n_ch, 10), generator=gen, device=DEV) * 40
    bits = torch.randint(0, 2, (n_ep // 20 + 1, n_ch), generator=gen, device=DEV).float() * 2 - 1
    rec[:, :, 4] += 300 * bits.repeat_interleave(20, dim=0)[:n_ep]
    d = rec.view(torch.float64)  # the taps are 0..4
    f = 2000.0 + torch.randn((n_ep, n_ch), **f64)
    err = torch.randn((n_ep, n_ch), **f64) * 0.02
    d[:, :, 5], d[:, :, 9] = f, err
    # the bank's wrapped carrier phase: the loop's running phase
    cyc = torch.cumsum(torch.cat([torch.full((1, n_ch), 2.0, dtype=torch.float64, device=DEV), f[:-1] * 1e-3]) + err * 0.25, 0)
    d[:, :, 6] = (cyc - torch.floor(cyc)) * (2 * math.pi)
    d[:, :, 7] = 5000.0 + torch.rand((1, n_ch), **f64) * 1000 + torch.randn((n_ep, n_ch), **f64) * 0.01
    d[:, :, 8] = 1.023e6
    chans = [dict(fs=20e6, intermediate_frequency=0.0, carrier_frequency=2000.0, carrier_phase=0.0, preamble_position=100,
                  range_correction_ms=68.0) for _ in range(n_ch)]
    return dict(case=case, rec=rec, chans=chans, messages=[L.NAV_GPS_LNAV] * n_ch,
                out=torch.empty((n_ep, n_ch, 4), dtype=torch.float64, device=DEV))


def _run_observables(s):
    ctx, _ = _ctx()
    shape = (s["case"]["epochs"], s["case"]["channels"])
    api.observables(ctx, s["rec"].data_ptr(), s["chans"], shape=shape, out_ptr=s["out"].data_ptr())
    # random navigation symbols give one candidate in twelve epochs
    counts, idx = api.preamble_search(ctx, s["rec"].data_ptr(), s["messages"], cap=shape[0] // 8 + 512, shape=shape,
                                      as_arrays=True)
    for row, count in zip(idx, counts):
        row[count:] = -1
    return dict(observables=s["out"], counts=counts, candidates=idx)


# ---------------------------------------------------------------- interface
def prepare(case, seed):
    return dict(search=_prepare_search, batch=_prepare_batch, track=_prepare_track, interference=_prepare_interference,
                observables=_prepare_observables)[case["kind"]](case, seed)


def run(state):
    return dict(search=_run_search, batch=_run_batch, track=_run_track, interference=_run_interference,
                observables=_run_observables)[state["case"]["kind"]](state)


def _search_work(n_codes, bins, n, k, sample_bytes, fold=0):
    """Forward transforms once per (Doppler, block), inverse ones per code too
    (5 N log2 N each), the mix, the product and the accumulated magnitude.  A
    folded search needs its mixed block and its code folded only once, and
    transforms of the folded length (the replica of a folded search repeats)."""
    m = fold or n
    fft = 5 * m * math.log2(m)
    flops = bins * k * (fft + (8 if fold else 6) * n) + n_codes * bins * k * (fft + 10 * m)
    return dict(bytes=sample_bytes + n_codes * 8 * m + n_codes * bins * 16, flops=flops)


def work(case):
    if case["kind"] == "search":
        n, fold, _, n_in = _search_shape(case)
        per = {"ci8": 2, "ci16": 4, "cf32": 8, "ri8": 1}[case["sample_type"]]
        return _search_work(case["n_codes"], len(_bins(case["span"], case["step"])), n, case["k"], per * n_in, fold)
    if case["kind"] == "batch":
        parts = [_search_work(len(svs), len(_bins(5000.0, step)), n, k, 0) for _, svs, n, k, step, _ in _batch_jobs(case)]
        return dict(bytes=sum(p["bytes"] for p in parts) + 4 * case["fs"] * case["ms"] / 1000, flops=sum(p["flops"] for p in parts))
    if case["kind"] == "track":
        # per channel-sample: the mix (6) and five complex taps (4 each)
        n = case["fs"] * case["epochs"] / 1000
        per = {"ci8": 2, "ci16": 4, "cf32": 8}[case["sample_type"]]
        return dict(bytes=per * n + 88 * case["epochs"] * case["channels"], flops=26 * n * case["channels"])
    if case["kind"] == "interference":
        # the detector's 128-point transform per 32 samples; with a wideband
        # jammer one more forward and an inverse, and the samples written
        flops = case["n"] / 32 * (5 * 128 * 7 * (3 if case["jammer"] == "cw" else 1) + 10 * 128)
        return dict(bytes=case["n"] * (16 if case["jammer"] == "cw" else 8), flops=flops)
    cells = case["channels"] * case["epochs"]
    return dict(bytes=cells * (88 + 32), flops=cells * 30)


# ------------------------------------------------------- the 64-bit results
def _lut():
    return torch.as_tensor(np.sin(np.arange(80) * (5 * math.pi / 80 / 2)).astype(np.float32).astype(np.float64), device=DEV)


def _mix64(x, fs, f, lut):
    """TableMixer: 32-bit NCO, its top 6 bits indexing the sine table."""
    f = fs + f if f < 0 else f
    adder = int(4294967296.0 * f / fs) & 0xFFFFFFFF
    i = torch.arange(x.numel(), device=DEV, dtype=torch.int64)
    idx = ((i * adder) & 0xFFFFFFFF) >> 26
    return x * torch.complex(lut[idx + 16], lut[idx])


def _complex64bit(raw, sample_type):
    if sample_type == "ri8":
        return raw.double().to(torch.complex128)
    return torch.view_as_complex(raw.double().contiguous())


def _resample64(x, fs_in, fs):
    """Zero-order hold to the common rate, then the boxcar mean."""
    g = math.gcd(round(fs_in), round(fs))
    up, m = round(fs) // g, round(fs_in) // g
    total = up * x.numel()
    run = torch.cat([torch.zeros(1, dtype=x.dtype, device=DEV), torch.cumsum(x, 0)])

    def upto(p):
        p = torch.clamp(p, max=total)
        j = torch.div(p, up, rounding_mode="floor")
        part = (p - j * up).double() / up
        return run[j] + part * torch.where(j < x.numel(), x[torch.clamp(j, max=x.numel() - 1)], torch.zeros((), dtype=x.dtype, device=DEV))

    k = torch.arange(-(-total // m), device=DEV)
    return (upto((k + 1) * m) - upto(k * m)) * up / m


def _replica(system, sv, n, repeats, mask, segment):
    chips = np.tile(_chips(system, sv), repeats).astype(np.float64)
    code = chips[(np.arange(n, dtype=np.int64) * len(chips) // n) % len(chips)]
    for b in range(32):
        if segment and (mask >> b) & 1:
            code[b * segment:(b + 1) * segment] *= -1
    return torch.as_tensor(code, device=DEV)


def _search64(x, fs, n, k, codes, span, step, fold, fold_abs, abs2, two_sided, f_if, mixed_if):
    """Every cell's level, index, mean and sigma, and each code's kept bin."""
    lut = _lut()
    if mixed_if:
        x = _mix64(x, fs, -f_if, lut)
    spec = torch.conj(torch.fft.fft(codes.to(torch.complex128)))
    if not two_sided:
        spec[:, n // 2 + 1:] = 0
    scale = 1.0 if two_sided else 2.0
    grid = _bins(span, step)
    n_codes = codes.shape[0]
    cells = {f: torch.zeros((n_codes, len(grid)), dtype=torch.int64 if f == "index" else torch.float64, device=DEV)
             for f in ("level", "index", "mean", "std")}
    group = max(1, int(4e8 // (16 * n)))
    for d, f in enumerate(grid):
        blocks = torch.fft.fft(_mix64(x[:n * k], fs, -f, lut).reshape(k, n))
        acc = torch.zeros((n_codes, fold or n), dtype=torch.float64, device=DEV)
        for c0 in range(0, n_codes, group):
            part = spec[c0:c0 + group]
            for b in range(k):
                y = torch.fft.ifft(blocks[b] * part) * scale
                if fold and not fold_abs:
                    y = y.reshape(part.shape[0], n // fold, fold).sum(1)
                y = y.abs() ** 2 if abs2 else y.abs()
                if fold and fold_abs:
                    y = y.reshape(part.shape[0], n // fold, fold).sum(1)
                acc[c0:c0 + group] += y
        top = acc.max(1)
        cells["level"][:, d], cells["index"][:, d] = top.values, top.indices
        cells["mean"][:, d], cells["std"][:, d] = acc.mean(1), acc.std(1)
    best = cells["level"].argmax(1, keepdim=True)
    kept = {f: v.gather(1, best)[:, 0].cpu().numpy() for f, v in cells.items()}
    best = best[:, 0].cpu().numpy()
    res = dict(level=kept["level"], sigma=kept["std"] + kept["mean"], mean=kept["mean"], std=kept["std"],
               snr=kept["level"] / (kept["std"] + kept["mean"]), index=kept["index"], doppler_bin=best,
               doppler=np.array(grid)[best] + f_if, code_offset=kept["index"].astype(np.float64))
    return res, {f: v.cpu().numpy() for f, v in cells.items()}


def _exact_search(case, seed):
    n, fold, fs_in, n_in = _search_shape(case)
    if case["n_codes"] * len(_bins(case["span"], case["step"])) * n * case["k"] > 2e10:
        return None
    x = _complex64bit(_search_capture(case, seed), case["sample_type"])
    if case["fs_in"]:
        x = _resample64(_mix64(x, fs_in, -case["if_hz"], _lut()) if case["if_hz"] else x, fs_in, case["fs"])
    mask, segment = (signals.nh10_mask(), n // 10) if case["nh10"] else (0, 0)
    codes = torch.stack([_replica(case["system"], sv, n, case["t_ms"] // SYSTEMS[case["system"]][3], mask, segment)
                         for sv in range(case["n_codes"])])
    res, cells = _search64(x, case["fs"], n, case["k"], codes, case["span"], case["step"], fold, case["fold"] == 1,
                           case["abs2"], case["two_sided"], case["if_hz"], case["if_hz"] != 0.0 and not case["fs_in"])
    return dict(results=res, cells=cells) if case["cells"] else res


def _exact_batch(case, seed):
    raw = _complex64bit(_batch_capture(case, seed), "ci16")
    parts = []
    for system, svs, n, k, step, f_if in _batch_jobs(case):
        codes = torch.stack([_replica(system, sv, n, 1, 0, 0) for sv in svs])
        parts.append(_search64(raw, case["fs"], n, k, codes, 5000.0, step, 0, False, False, False, f_if, True)[0])
    return {f: np.concatenate([p[f] for p in parts]) for f in parts[0]}


def _exact_interference(case, seed):
    x = torch.view_as_complex(_interference_capture(case, seed).double().contiguous())
    if case["jammer"] == "gated":
        return None  # what it is taken for hangs on the occupation vote
    if case["jammer"] == "cw":
        n = x.numel()
        cols = (n - 96) // 32
        win = 0.5 * (1 - torch.cos(torch.arange(128, device=DEV, dtype=torch.float64) * (2 * math.pi / 128)))
        s = torch.fft.fft(x.unfold(0, 128, 32)[:cols] * win.float().double())
        s[s.abs() >= 20] = 0
        y = torch.fft.ifft(s) * 2
        x = torch.zeros((cols + 3, 32), dtype=torch.complex128, device=DEV)
        for j in range(4):
            x[j:j + cols] += y[:, 32 * j:32 * j + 32]
        x = torch.cat([x.reshape(-1), torch.zeros(n, dtype=torch.complex128, device=DEV)])[:n]
    return dict(samples=torch.view_as_real(x), detections=None)


def _exact_observables(case, seed):
    s = _prepare_observables(case, seed)
    d, rec, ch = s["rec"].view(torch.float64), s["rec"], s["chans"][0]
    f, err = d[:, :, 5], d[:, :, 9]
    first = torch.full((1, case["channels"]), ch["carrier_frequency"], dtype=torch.float64, device=DEV)
    total = torch.cumsum(torch.cat([first, f[:-1]]) * 1e-3 + err * 0.25, 0)
    wrapped = d[:, :, 6] / (2 * math.pi)
    to_ms = 1000 / ch["fs"]
    offset = torch.trunc(d[ch["preamble_position"], :, 7] * to_ms)
    out = torch.empty((case["epochs"], case["channels"], 4), dtype=torch.float64, device=DEV)
    out[:, :, 0] = d[:, :, 7] * to_ms - offset + ch["range_correction_ms"]
    out[:, :, 1] = -(torch.round(total - wrapped) + wrapped)
    out[:, :, 2] = f
    out[:, :, 3] = 27 + 20 * torch.log10(rec[:, :, 4].double().abs() / rec[:, :, 5].double().std(0))
    return dict(observables=out, counts=None, candidates=None)


def exact(case, seed):
    """None for the tracking bank: its loops feed each rounding back, so no
    64-bit run of them is what a 32-bit correlator has to give."""
    return dict(search=_exact_search, batch=_exact_batch, track=lambda c, s: None, interference=_exact_interference,
                observables=_exact_observables)[case["kind"]](case, seed)
