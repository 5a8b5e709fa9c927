"""Timed cases of the beam-processing path, through the Python binding.

A case names one kind of call and its sizes:

* ``channelise``  PPF.channelise: voltages -> integrated Stokes filterbank
* ``modules``     PPF.run, stokes, integrate: the module chain of a pipeline
                  that keeps the complex spectra
* ``clip``        RFI.run on a filterbank whose history is full
* ``trials``      dedisperse: one buffer of channel rows over a trial grid
* ``module``      DedispersionModule.add: host blobs in, host spectra out
* ``search``      analyse: events of a dedispersed window
* ``beam``        Beam.process and events: one beam's whole chain, a chunk
* ``batch``       Batch.run and events: uneven beams, one chunk each

LOFAR subbands are 195.3125 kHz wide and sampled at 5.12 us.  Voltages are
seeded Gaussian noise (sigma 16 per component) with narrowband sinusoids in 3 %
of the channels, broadband bursts and dispersed pulses.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pelican-lofar_gb300"))
import pv  # noqa: E402

SUB_BW = 0.1953125  # MHz
RAW_TSAMP = 5.12e-6  # s
K_DM = 4148.741601
HISTORY = 10000  # RFI_Clipper History@maximum of the pipelines
MAX_EVENTS = 8192  # rows of a returned event table
DEV = "cuda"


def listed():
    return [
        # One station beam of 32 subbands, 65536 samples each: the smallest chunk that is streamed.
        dict(name="channelise 32x16", kind="channelise", nsub=32, nchan=16, nblocks=4096, window=4, nstokes=1,
             int16=True),
        # The full LOFAR band, 16384 integrated spectra.
        dict(name="channelise 244x16", kind="channelise", nsub=244, nchan=16, nblocks=65536, window=4, nstokes=1,
             int16=True),
        # Fine channels for high dispersion measures; a chunk that no tile divides.
        dict(name="channelise 61x64", kind="channelise", nsub=61, nchan=64, nblocks=16391, window=4, nstokes=1,
             int16=True),
        # A polarimetry pipeline: the complex spectra are kept, four Stokes parameters are integrated.
        dict(name="modules 62x32", kind="modules", nsub=62, nchan=32, nblocks=2050, window=16, nstokes=4),
        # The clipper by itself on the full band, flags asked for.
        dict(name="clip 3904x4096", kind="clip", nsub=244, nchan=16, nt=4096, npol=1, flags=True),
        # A small DM grid on one buffer, ragged in every size.
        dict(name="trials 300x496x5003", kind="trials", f_lo=110.0, bw=31 * SUB_BW, nchan=496, tsamp=327.68e-6,
             tdms=300, dm_max=60.0, nout=5003),
        # The reference module's buffering, host blobs in and host spectra out.
        dict(name="module 512x512", kind="module", nsub=32, nchan=16, buffer=16384, tdms=512, dm_max=100.0),
        # The search of one full window.
        dict(name="search 2048x16384", kind="search", tdms=2048, nsamp=16384, pow2=6, threshold=6.0),
        # One beam's chain on a small chunk: 512 channels, 512 trials.
        dict(name="beam 32x16", kind="beam", nsub=32, nchan=16, f_lo=140.0, chunk=1024, tdms=512, dm_max=100.0),
        # One beam's chain on the full band: 3904 channels, 2048 trials, 16384 spectra.
        dict(name="beam 244x16", kind="beam", nsub=244, nchan=16, f_lo=110.0, chunk=16384, tdms=2048, dm_max=500.0),
        # Eight uneven beams of the serving mix, pipelined, FP32 rings.
        dict(name="batch 8 f32", kind="batch", mix=8, nbeams=8, chunk=4096, store="f32", pipelined=True, udp=False,
             tdms_max=4096),
        # Packet-fed beams with 8-bit rings, every window in the step of its last chunk.
        dict(name="batch 4 u8", kind="batch", mix=4, nbeams=4, chunk=2048, store="u8", pipelined=False, udp=True,
             tdms_max=2048),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channelise", "channelise", "modules", "clip", "trials", "module", "search", "beam", "beam",
                       "batch"])
    if kind == "channelise":
        nchan = rng.choice([16, 16, 32, 64, 64, 128])
        nsub = _log(rng, 8, 244)
        return dict(kind=kind, nsub=nsub, nchan=nchan, nblocks=_log(rng, 1000, max(1001, 2.5e8 / (nsub * nchan))),
                    window=rng.choice([1, 4, 4, 8, 16]), nstokes=rng.choice([1, 1, 1, 4]),
                    int16=rng.choice([True, True, False]))
    if kind == "modules":
        return dict(kind=kind, nsub=_log(rng, 4, 122), nchan=rng.choice([16, 20, 32, 64, 256]),
                    nblocks=_log(rng, 64, 4096), window=rng.choice([1, 4, 16]), nstokes=rng.choice([1, 4]))
    if kind == "clip":
        nchan = rng.choice([16, 16, 64])
        return dict(kind=kind, nsub=8 * _log(rng, 4, 30), nchan=nchan, nt=_log(rng, 256, 8192),
                    npol=rng.choice([1, 1, 4]), flags=rng.choice([True, False]))
    if kind == "trials":
        return dict(kind=kind, f_lo=rng.choice([110.0, 140.0, 1215.0]), bw=round(rng.uniform(4.0, 40.0), 3),
                    nchan=_log(rng, 64, 4096), tsamp=rng.choice([327.68e-6, 1310.72e-6]), tdms=_log(rng, 16, 1024),
                    dm_max=round(rng.uniform(20.0, 200.0), 2), nout=_log(rng, 256, 16384))
    if kind == "module":
        return dict(kind=kind, nsub=_log(rng, 8, 61), nchan=16, buffer=rng.choice([16384, 32768]),
                    tdms=_log(rng, 32, 1024), dm_max=round(rng.uniform(20.0, 100.0), 2))
    if kind == "search":
        return dict(kind=kind, tdms=_log(rng, 16, 4096), nsamp=_log(rng, 512, 16384), pow2=rng.choice([4, 6, 6, 8]),
                    threshold=rng.choice([5.0, 6.0]))
    if kind == "beam":
        return dict(kind=kind, nsub=8 * _log(rng, 1, 15), nchan=rng.choice([16, 16, 32, 64]),
                    f_lo=rng.choice([110.0, 140.0]), chunk=64 * _log(rng, 8, 128), tdms=_log(rng, 32, 1024),
                    dm_max=round(rng.uniform(20.0, 200.0), 2))
    return dict(kind=kind, mix=rng.randrange(1 << 20), nbeams=rng.randrange(2, 7), chunk=rng.choice([1024, 2048, 4096]),
                store=rng.choice(["f32", "f16", "u8"]), pipelined=rng.choice([True, False]),
                udp=rng.choice([True, False]), tdms_max=rng.choice([1024, 2048]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _voltages(nsub, nchan, n, f_lo, seed, complex64=False):
    """[sub][2][n] voltages: int16 [sub][2][2n] (re, im) or complex64."""
    g, rng = _gen(seed), np.random.default_rng(seed)
    out = torch.empty((nsub, 2, 2 * n), dtype=torch.float32 if complex64 else torch.int16, device=DEV)
    nbins = nsub * nchan
    rfi = rng.choice(nbins, size=max(1, int(0.03 * nbins)), replace=False)
    bursts = rng.integers(0, max(1, n - 16), size=max(1, n // 40000))
    f_top = f_lo + nsub * SUB_BW
    pulses = [(rng.uniform(10.0, 90.0), rng.uniform(0.1, 0.9)) for _ in range(3)]
    width = min(n // 8, 400)  # 2 ms
    t = np.arange(nchan)
    for s in range(nsub):
        v = torch.randn((2, n, 2), generator=g, device=DEV) * 16.0
        f = f_lo + (s + 0.5) * SUB_BW
        for dm, pos in pulses:
            t0 = int((pos * n + K_DM * dm * (1.0 / f ** 2 - 1.0 / f_top ** 2) / RAW_TSAMP) % max(1, n - width))
            v[:, t0:t0 + width] *= 1.25
        for b in bursts:
            v[:, b:b + 16] *= 3.0
        m = n // nchan * nchan
        for ch in rfi[rfi // nchan == s] % nchan:
            ph = 2 * np.pi * ((ch - nchan // 2) / nchan * t + rng.uniform())
            tone = torch.tensor(20 * 16.0 * np.stack([np.cos(ph), np.sin(ph)], -1), dtype=torch.float32, device=DEV)
            v[:, :m].view(2, -1, nchan, 2).add_(tone)
        v = v.round_().clamp_(-32768, 32767)
        out[s] = v.reshape(2, 2 * n)
    return torch.view_as_complex(out.view(nsub, 2, n, 2)) if complex64 else out


def _packets(v, per):
    """The LOFAR packet streams (16-byte header, [subband][16 samples][pol] int16 pairs) of int16 voltages."""
    nsub, _, n2 = v.shape
    npk = n2 // 32
    body = v.view(nsub // per, per, 2, npk, 16, 2).permute(0, 3, 1, 4, 2, 5).contiguous()
    body = body.view(torch.uint8).view(nsub // per, npk, per * 128)
    head = torch.zeros((nsub // per, npk, 4), dtype=torch.int32, device=DEV)
    head[:, :, 2] = 1300000000
    head[:, :, 3] = 16 * torch.arange(npk, device=DEV, dtype=torch.int32)
    return torch.cat([head.view(torch.uint8).view(nsub // per, npk, 16), body], dim=2).reshape(-1)


def _filterbank(nt, nsub, npol, nchan, seed):
    """Integrated powers [t][sub][pol][chan] (sums of 4 x 2 x 2 squared Gaussians, mean 8192) with narrowband
    channels and bursts."""
    g, rng = _gen(seed), np.random.default_rng(seed)
    nbins = nsub * nchan
    x = torch.randn((nt, nsub, npol, nchan), generator=g, device=DEV) * 2048.0 + 8192.0
    x[:, :, 0] = x[:, :, 0].abs() + 64.0
    bad = torch.from_numpy(rng.choice(nbins, size=max(1, int(0.03 * nbins)), replace=False)).to(DEV)
    x[:, bad // nchan, 0, bad % nchan] *= 30.0
    for b in rng.integers(0, nt, size=max(1, nt // 10000)):
        x[int(b), :, 0] *= 4.0
    return x


def _bp(nbins, start, width, median, rms):
    return "\n".join(["# flat bandpass", str(nbins), repr(start), repr(start + width * nbins), repr(width), repr(rms),
                      repr(median)]) + "\n"


def _coeffs(ntaps, nchan):
    """A Kaiser-windowed sinc prototype [tap][chan], as a user's own filter."""
    n = ntaps * nchan
    t = (np.arange(n) - (n - 1) / 2.0) / nchan
    return (np.sinc(t) * np.kaiser(n, 9.0)).reshape(ntaps, nchan).astype(np.float32)


def _band(nsub, nchan, f_lo):
    foff = SUB_BW / nchan
    return f_lo - (nchan // 2) * foff, foff


def _delays(fch1, foff, nchan):
    top = fch1 + foff * (nchan - 1) if foff >= 0 else fch1
    f = top - abs(foff) * np.arange(nchan)
    return (K_DM * (1.0 / f ** 2 - 1.0 / top ** 2)).astype(np.float32)


def _shifts(k, tdms, start, step):
    """[trial][channel] sample delays, in the FP32 products the reference kernel forms."""
    v = (np.arange(tdms).astype(np.float64) * np.float64(np.float32(step)) + np.float64(np.float32(start))).astype(
        np.float32)
    return np.trunc(v[:, None] * k[None, :]).astype(np.int64)


def _beam_config(nsub, nchan, f_lo, chunk, tdms, dm_max, udp):
    fch1, foff = _band(nsub, nchan, f_lo)
    per = next(p for p in (61, 31, nsub) if nsub % p == 0)
    kw = dict(udp_packet_bytes=16 + per * 128, udp_subbands=per) if udp else {}
    return pv.beam_config(nsub=nsub, nchan_sub=nchan, window="kaiser", int_time=4, fch1=fch1, foff=foff,
                          tsamp=RAW_TSAMP * nchan * 4, tdms=tdms, dm_step=dm_max / (tdms - 1), chunk=chunk,
                          threshold=6.0, bin_pow2=6, cr=5.0, sr=4.0, history=HISTORY, zero_dming=1, prefilled=1,
                          bp_text=_bp(nsub * nchan, fch1, foff, 1000.0, 50.0), **kw), per


def _mix(c):
    """(nsub, nchan, dm_max, tdms) of the beams of a batch."""
    rng = np.random.default_rng(c["mix"])
    trials = [t for t in (256, 512, 1024, 2048, 4096) if t <= c["tdms_max"]][-3:]
    return [(int(rng.choice([31, 61, 122, 244])), int(rng.choice([16, 64])), float(rng.choice([250.0, 1000.0])),
             int(rng.choice(trials))) for _ in range(c["nbeams"])]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind in ("channelise", "modules"):
        x = _voltages(c["nsub"], c["nchan"], c["nblocks"] * c["nchan"], 110.0, seed,
                      complex64=kind == "modules" or not c["int16"])
        return dict(case=c, x=x, ppf=pv.PPF(c["nchan"], 8, coeffs=_coeffs(8, c["nchan"])))
    if kind == "clip":
        rfi = _clipper(c)
        first = _filterbank(HISTORY + 240, c["nsub"], c["npol"], c["nchan"], seed + 1)
        rfi.run(first)  # the history of a stream that has run for some seconds
        x = _filterbank(c["nt"], c["nsub"], c["npol"], c["nchan"], seed)
        return dict(case=c, rfi=rfi, x=x, work=torch.empty_like(x))
    if kind == "trials":
        k, start, step, width = _grid(c)
        x = torch.randn((c["nchan"], width), generator=_gen(seed), device=DEV)
        x[:, width // 2] += 1.0
        return dict(case=c, x=x, k=torch.from_numpy(k).to(DEV), start=start, step=step)
    if kind == "module":
        first, blob = _blobs(c, seed)
        mod = _module(c)
        mod.add(first, _tsamp(c))
        return dict(case=c, mod=mod, blob=blob)
    if kind == "search":
        x = torch.randn((c["tdms"], c["nsamp"]), generator=_gen(seed), device=DEV) * 62.0
        rng = np.random.default_rng(seed)
        for _ in range(10):
            d, t, w = int(rng.integers(c["tdms"])), int(rng.integers(c["nsamp"])), int(rng.integers(1, 16))
            x[max(0, d - 3):d + 4, t:t + w] += 62.0 * rng.uniform(3.0, 12.0)
        return dict(case=c, x=x)
    if kind == "beam":
        cfg, _ = _beam_config(c["nsub"], c["nchan"], c["f_lo"], c["chunk"], c["tdms"], c["dm_max"], False)
        x = _voltages(c["nsub"], c["nchan"], c["chunk"] * 4 * c["nchan"], c["f_lo"], seed)
        beam = pv.Beam(cfg)
        for _ in range(math.ceil(HISTORY / c["chunk"])):
            beam.process(x)
        return dict(case=c, beam=beam, x=x)
    cfgs, xs = [], []
    for i, (nsub, nchan, dm_max, tdms) in enumerate(_mix(c)):
        cfg, per = _beam_config(nsub, nchan, 110.0, c["chunk"], tdms, dm_max, c["udp"])
        v = _voltages(nsub, nchan, c["chunk"] * 4 * nchan, 110.0, seed + 100 * i)
        cfgs.append(cfg)
        xs.append(_packets(v, per) if c["udp"] else v)
    batch = pv.Batch(cfgs, tune=True, graph=True, pipelined=c["pipelined"], store=c["store"])
    for i, x in enumerate(xs):
        batch.set_input(i, x, both=True)
    for _ in range(math.ceil(HISTORY / c["chunk"])):
        batch.run()
    return dict(case=c, batch=batch)


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "channelise":
        return state["ppf"].channelise(state["x"], c["nstokes"], c["window"], 1)
    if kind == "modules":
        spectra = state["ppf"].run(state["x"])
        power = pv.stokes(spectra, c["nstokes"])
        return spectra, pv.integrate(power, c["window"])
    if kind == "clip":
        state["work"].copy_(state["x"])  # the clipper works in place: a chunk arrives fresh each time
        flags = state["rfi"].run(state["work"], flags=c["flags"])
        return (state["work"], flags) if c["flags"] else state["work"]
    if kind == "trials":
        return pv.dedisperse(state["x"], c["nout"], c["tdms"], state["k"], state["start"], state["step"])
    if kind == "module":
        return [w for w, _ in state["mod"].add(state["blob"], _tsamp(c))]
    if kind == "search":
        return _events(*pv.analyse(state["x"], c["threshold"], 62.0, c["pow2"], cap=1 << 20))
    if kind == "beam":
        beam = state["beam"]
        beam.process(state["x"])
        ev, n, first = beam.events()
        window = pv.device_array(beam.buffers()[2], (c["tdms"], c["chunk"]))
        return [window, _events(ev, n)]
    batch = state["batch"]
    batch.run()
    out = []
    for i, cfg in enumerate(batch.cfgs):
        ev, n, first = batch.events(i)
        out.append([pv.device_array(batch.buffers(i)[1], (cfg.tdms, cfg.chunk)), _events(ev, n)])
    return out


def _events(ev, n):
    """The event list as a table of a fixed number of rows (zeros after the last event) and the event count."""
    where, what = np.zeros((MAX_EVENTS, 2), np.int32), np.zeros((MAX_EVENTS, 2), np.float32)
    m = min(len(ev), MAX_EVENTS)
    where[:m, 0], where[:m, 1] = ev["dm"][:m], ev["t"][:m]
    what[:m, 0], what[:m, 1] = ev["bin_factor"][:m], ev["value"][:m]
    return dict(where=where, what=what, total=int(n))


def _clipper(c):
    nbins = c["nsub"] * c["nchan"]
    return pv.RFI(_bp(nbins, 110.0, SUB_BW / c["nchan"], 8000.0, 2000.0), cr=5.0, sr=4.0, history=HISTORY,
                  zero_dming=True)


def _grid(c):
    foff = -c["bw"] / c["nchan"]
    k = _delays(c["f_lo"] + c["bw"], foff, c["nchan"])
    start, step = 0.0, float(np.float32(c["dm_max"] / max(1, c["tdms"] - 1)) / np.float32(c["tsamp"]))
    return k, start, step, c["nout"] + int(_shifts(k, c["tdms"], start, step).max()) + 1


def _tsamp(c):
    return RAW_TSAMP * c["nchan"] * 4


def _module(c):
    fch1, foff = _band(c["nsub"], c["nchan"], 140.0)
    return pv.DedispersionModule(c["buffer"], c["tdms"], 0.0, c["dm_max"] / (c["tdms"] - 1), fch1, foff)


def _module_sizes(c):
    """(maxshift, outputs per buffer) by the module's own rule."""
    fch1, foff = _band(c["nsub"], c["nchan"], 140.0)
    k = _delays(fch1, foff, c["nsub"] * c["nchan"])
    step = np.float32(c["dm_max"] / (c["tdms"] - 1))
    ms = int(float(np.float32(step * np.float32(c["tdms"] - 1)) * k[-1]) / _tsamp(c))
    return ms, c["buffer"] - ms - (c["buffer"] - ms) % 224


def _blobs(c, seed):
    """The blob that leaves the module one blob short of a full buffer, and the blob that fills it."""
    _, nout = _module_sizes(c)
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((c["buffer"], c["nsub"], 1, c["nchan"]), dtype=np.float32)
    return x[:c["buffer"] - nout], np.ascontiguousarray(x[c["buffer"] - nout:])


def work(case):
    """Bytes that have to be read and written and operations that have to be done, by one pass."""
    c = case
    kind = c["kind"]

    def chan(nsub, nchan, nblocks, nstokes, window, elem):
        n = nsub * 2 * nblocks * nchan
        return dict(bytes=n * elem + 4 * nstokes * nsub * nchan * (nblocks // window),
                    flops=n * (32 + 5 * math.log2(max(nchan, 2)) + 4 * nstokes))

    def add(*ws):
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))

    def chain(nsub, nchan, chunk, tdms):
        nbins = nsub * nchan
        return add(chan(nsub, nchan, chunk * 4, 1, 4, 4),
                   dict(bytes=4 * tdms * chunk, flops=tdms * nbins * chunk + 10 * nbins * chunk))

    if kind == "channelise":
        return chan(c["nsub"], c["nchan"], c["nblocks"], c["nstokes"], c["window"], 4 if c["int16"] else 8)
    if kind == "modules":
        w = chan(c["nsub"], c["nchan"], c["nblocks"], c["nstokes"], c["window"], 8)
        w["bytes"] += 8 * c["nsub"] * 2 * c["nblocks"] * c["nchan"]
        return w
    if kind == "clip":
        n = c["nt"] * c["nsub"] * c["nchan"]
        return dict(bytes=n * (8 * c["npol"] + (1 if c["flags"] else 0)), flops=10 * n)
    if kind == "trials":
        return dict(bytes=4 * c["nchan"] * _grid(c)[3] + 4 * c["tdms"] * c["nout"],
                    flops=c["tdms"] * c["nchan"] * c["nout"])
    if kind == "module":
        _, nout = _module_sizes(c)
        nbins = c["nsub"] * c["nchan"]
        return dict(bytes=4 * nout * (nbins + c["tdms"]), flops=c["tdms"] * nbins * nout)
    if kind == "search":
        return dict(bytes=4 * c["tdms"] * c["nsamp"], flops=2 * c["tdms"] * c["nsamp"])
    if kind == "beam":
        return chain(c["nsub"], c["nchan"], c["chunk"], c["tdms"])
    return add(*[chain(nsub, nchan, c["chunk"], tdms) for nsub, nchan, _, tdms in _mix(c)])


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------

def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind in ("channelise", "modules"):
        return _exact_channelise(c, seed)
    if kind == "clip":
        return _exact_clip(c, seed)
    if kind == "trials":
        k, start, step, width = _grid(c)
        x = prepare(c, seed)["x"].double()
        return _exact_trials(x, _shifts(k, c["tdms"], start, step), c["nout"])
    if kind == "module":
        first, blob = _blobs(c, seed)
        nbins = c["nsub"] * c["nchan"]
        x = np.concatenate([first, blob]).reshape(c["buffer"], nbins)[:, ::-1]  # ascending band: highest first
        fch1, foff = _band(c["nsub"], c["nchan"], 140.0)
        ts = np.float32(_tsamp(c))
        sh = _shifts(_delays(fch1, foff, nbins), c["tdms"], 0.0, np.float32(c["dm_max"] / (c["tdms"] - 1)) / ts)
        return [_exact_trials(torch.from_numpy(np.ascontiguousarray(x.T)).to(DEV).double(), sh, _module_sizes(c)[1])]
    return None  # events are decisions on FP32 sums; a whole chain takes too long in 64 bits


def _exact_channelise(c, seed):
    cplx = c["kind"] == "modules" or not c["int16"]
    n, nchan, nb = c["nblocks"] * c["nchan"], c["nchan"], c["nblocks"]
    x = _voltages(c["nsub"], nchan, n, 110.0, seed, complex64=cplx)
    co = torch.from_numpy(_coeffs(8, nchan)).to(DEV).double()
    w = min(c["window"], nb)
    nu = nb // w
    nst = c["nstokes"]
    spectra = torch.empty((nb, c["nsub"], 2, nchan), dtype=torch.complex128, device=DEV) if c["kind"] == "modules" \
        else None
    out = torch.empty((nu, c["nsub"], nst, nchan), dtype=torch.float64, device=DEV)
    for s in range(c["nsub"]):
        v = x[s] if cplx else torch.view_as_complex(x[s].view(2, n, 2).float())
        v = v.to(torch.complex128).view(2, nb, nchan)
        v = torch.cat([torch.zeros((2, 7, nchan), dtype=v.dtype, device=DEV), v], 1)
        y = sum(v[:, t:t + nb] * co[t] for t in range(8))
        f = torch.fft.fft(y, dim=-1)
        if spectra is not None:
            spectra[:, s] = f.transpose(0, 1)
        px, py = f[0].abs().square(), f[1].abs().square()
        xy = f[0] * f[1].conj()
        for k, p in enumerate([px + py, px - py, 2 * xy.real, 2 * xy.imag][:nst]):
            out[:, s, k] = p[:nu * w].view(nu, w, nchan).sum(1)
    return (spectra, out) if spectra is not None else out


def _exact_trials(x, shifts, nout):
    """sum over channels c of x[c][t + shift(d, c)]."""
    out = torch.zeros((shifts.shape[0], nout), dtype=torch.float64, device=DEV)
    t = torch.arange(nout, device=DEV)
    sh = torch.from_numpy(np.ascontiguousarray(shifts.T)).to(DEV)
    for ch in range(x.shape[0]):
        out += x[ch][sh[ch][:, None] + t[None, :]]
    return out


def _exact_clip(c, seed):
    """RFI_Clipper with a flat bandpass, zero-DMing and the RMS taken from the mean, in 64 bits."""
    nbins = c["nsub"] * c["nchan"]
    first = _filterbank(HISTORY + 240, c["nsub"], c["npol"], c["nchan"], seed + 1)[:, :, 0].reshape(-1, nbins)
    full = _filterbank(c["nt"], c["nsub"], c["npol"], c["nchan"], seed)
    x = torch.cat([first, full[:, :, 0].reshape(-1, nbins)]).double().cpu().numpy()
    out = full.double().cpu().numpy()
    flags = np.zeros((c["nt"], nbins), np.uint8)
    del first, full
    H, cr, sr, cpb = HISTORY, 5.0, 4.0, nbins // 8
    bp, bp_rms = 8000.0, 2000.0
    means, rmss = [], []
    mean_run = rms_run = mean_acc = rms_acc = 0.0
    mor = 0.0
    num = bad_spectra = 0
    last_good = np.zeros(nbins)
    zeros = nbins
    for t in range(x.shape[0]):
        v = x[t]
        dm = 0.0
        if len(rmss) < H:
            b = v[:8 * cpb].reshape(8, cpb)
            m = b.mean(1)
            rmss.append(np.sqrt(np.maximum((b * b).mean(1) - m * m, 0)).min())
            rms_acc += rmss[-1]
            rms_run = rms_acc / len(rmss)
            if len(rmss) == H:
                mor = mean_run / rms_run
            low = np.append(b[:7].min(1), v[7 * cpb:].min())
            dm = np.sort(np.minimum(low, 1e6) - min(bp, 1e6))[4] + 4.0 / math.sqrt(8.0) * rms_run
        else:
            rms_run += (rmss[-1] - rmss[0]) / H
            rmss.append(abs(mean_run / mor))
            rmss.pop(0)
        clip = (v - dm) - bp > cr * rms_run
        good = ~clip
        v = np.where(clip, last_good, v)
        s = x[t][good].mean() if good.any() else math.nan
        if len(means) < H:
            means.append(s)
            mean_acc += s
            mean_run = mean_acc / len(means)
        else:
            mean_run += (means[-1] - means[0]) / H
            means.append(s)
            means.pop(0)
        g = np.append(good[:7 * cpb].reshape(7, cpb).sum(1), good[7 * cpb:].sum())
        bands = int((g < 0.8 * cpb).sum() + 4 * (g == 0).sum() + (4 if good.sum() < 0.8 * nbins else 0))
        reject = False
        if len(means) < 1000:
            reject = True
        elif s - mean_run > sr * bp_rms / math.sqrt(nbins) or bands >= 4:
            reject = True
            bad_spectra += 1
            means[-1], rmss[-1] = means[-2], rmss[-2]
        elif zeros:
            fill = (last_good == 0.0) & (v != 0.0)
            last_good[fill] = v[fill]
            zeros -= int(fill.sum())
        w = (np.full(nbins, -0.2) if reject else v) - (bp + dm)
        m = w.mean()
        r = math.sqrt(max((w * w).mean() - m * m, 0.0)) or 1.0
        if not reject:
            w = (w - m) / r
            w[w > cr] = 0.0
        bp, bp_rms = mean_run, rms_run
        u = t - (x.shape[0] - c["nt"])
        if u >= 0:
            o = out[u].transpose(1, 0, 2).reshape(c["npol"], nbins)
            o[0] = w
            o[1:] = -0.2 if reject else np.where(clip, v, o[1:])
            out[u] = o.reshape(c["npol"], c["nsub"], c["nchan"]).transpose(1, 0, 2)
            flags[u] = clip + (2 if reject else 0)
    return (out, flags) if c["flags"] else out
