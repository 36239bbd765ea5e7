"""The work that users of this framework have it do, as timed cases.

A case is one pass through the public Python interface (sfxc_gpu.correlator):
a correlator node's job -- parameters, each stream's input-node protocol
bytes, the integration, its output bytes -- a timeslice of several subbands on
one node each, a batch of uneven jobs in one graph, or a station's front end
(recording -> channels -> protocol).  Inputs are host buffers (pinned, as a
receiving process keeps them), outputs come back to the host, and both
transfers belong to the pass.  The samples are the seeded signal model of
synth.model_codes_torch: a common analytic sky signal seen through each
station's delay model, independent noise, 2-bit (or sign) quantisation.

exact() computes the same visibilities in 64 bits with torch and numpy alone,
from the same protocol bytes and delay tables.
"""
import math
import os
import struct
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sfxc-1_gb300"))

from sfxc_gpu import correlator, lib, scenario, synth, timebase  # noqa: E402

RECT, COS, HAMMING, HANN = 1, 2, 3, 4
MHZ = 1_000_000
# seconds of one recording before the first integration (the delays reach +-15 ms)
LEAD_US = 16000
BLOCK_BYTES = 2000


def listed():
    return [
        # The smallest call: two stations, one polarisation, 16 MHz, 512
        # channels, one short integration -- fringe checks during an
        # observation, where the call's latency counts.
        job("plain_small", stations=2, pols=1, rate=32 * MHZ, nchan=512, us=15625, mode="fp32"),
        # An odd small array: five stations, 1-bit, an integration that is no
        # round number, the Hamming window, a station with invalid frames, and
        # the spectra reduced to fewer output channels with the user's lag window.
        job("odd_onebit", stations=5, pols=2, rate=32 * MHZ, bits=1, nchan=1024, outch=256, us=137311, window=HAMMING,
            mode="fp32", invalid=1),
        # A continuum array of eight stations (the plain 4096-channel
        # configuration): four subbands side by side, one node each, as the
        # subbands of a timeslice are correlated.
        job("plain_fp32", stations=8, pols=2, rate=64 * MHZ, nchan=4096, us=500000, mode="fp32", subbands=4),
        # The same kind of array, 16 stations, in single precision throughout.
        job("precision_fp32", stations=16, pols=2, rate=64 * MHZ, nchan=4096, us=1000000, mode="fp32"),
        # The precision configuration: 16 stations, 32 MHz dual polarisation,
        # four subbands side by side, on the tensor cores.
        job("precision_tc", stations=16, pols=2, rate=64 * MHZ, nchan=4096, us=500000, mode="tc", subbands=4),
        # Twenty stations of three formats (32 MHz and 64 MHz 2-bit, 16 MHz
        # 1-bit) correlated over their common band: forty streams of uneven rates.
        job("mixed_wide", stations=20, pols=2, rate=64 * MHZ, nchan=4096, us=500000, mode="tc", mixed=1),
        # Spectral lines: the finest channels (32768-sample windows), one polarisation pair per station.
        job("fine_channels", stations=12, pols=2, rate=64 * MHZ, nchan=16384, us=500000, mode="tc"),
        # The coarsest channels, short dumps: transients, quick look.
        job("coarse_channels", stations=8, pols=2, rate=32 * MHZ, nchan=256, us=250000, window=COS, mode="tc"),
        # Pulsar binning: 256 phase bins and the off-pulse bin.
        job("pulsar_bins", stations=10, pols=2, rate=32 * MHZ, nchan=2048, us=1000000, mode="tc", bins=256),
        # Wide-field imaging: extra phase centres of one pointing.
        job("phase_centres", stations=8, pols=2, rate=32 * MHZ, nchan=2048, us=1000000, mode="fp32", centres=16),
        # A timeslice of uneven jobs in one graph: 40, 24 and 16 streams,
        # 4096, 16384 and 256 channels, one, four and eight integrations.
        {"name": "uneven_batch", "kind": "batch", "us": 250000},
        # One station's front end: a 16-channel VDIF recording read, its
        # channels extracted and each turned into protocol bytes.
        {"name": "front_end", "kind": "frontend", "rate": 32 * MHZ, "ms": 1000},
    ]


def job(name, *, stations, pols, rate, nchan, us, mode, bits=2, outch=0, window=HANN, subbands=1, mixed=0, bins=0,
        centres=1, invalid=0):
    d = dict(kind="job", stations=stations, pols=pols, rate=rate, bits=bits, nchan=nchan, outch=outch or nchan, us=us,
             window=window, mode=mode, subbands=subbands, mixed=mixed, bins=bins, centres=centres, invalid=invalid)
    return dict(name=name, **d) if name else d


def draw(rng):
    """Another case of the same kinds: sizes spread over the ranges the listed ones stand for."""
    kind = rng.random()
    if kind < 0.1:
        return {"kind": "frontend", "rate": rng.choice([16, 32, 64]) * MHZ,
                "ms": int(round(math.exp(rng.uniform(math.log(100), math.log(1000)))))}
    if kind < 0.2:
        return {"kind": "batch", "us": 8 * rng.randint(10000, 30000)}
    rate = rng.choice([8, 16, 32, 64]) * MHZ
    nchan = 1 << rng.randint(8, 14)
    pols = rng.choice([1, 2, 2])
    mode = rng.choice(["fp32", "tc"])
    stations = int(round(math.exp(rng.uniform(math.log(2), math.log(20)))))
    c = dict(stations=stations, pols=pols, rate=rate, nchan=nchan, mode=mode, bits=rng.choice([1, 2, 2, 2]),
             window=rng.choice([RECT, COS, HAMMING, HANN, HANN]))
    extra = rng.random()
    if extra < 0.15:
        c.update(bins=rng.choice([9, 32, 100, 256]), nchan=min(nchan, 2048), bits=2)
    elif extra < 0.3:
        c.update(centres=rng.randint(2, 16), nchan=min(nchan, 4096), mode="fp32")
    elif extra < 0.45:
        c.update(mixed=1, nchan=min(max(nchan, 512), 8192), rate=max(rate, 16 * MHZ), bits=2)
    elif extra < 0.55:
        c.update(outch=max(32, nchan // rng.choice([2, 4, 16])))
    elif extra < 0.75:
        c.update(subbands=rng.randint(2, 4))
    lo = max(15625, 6 * c["nchan"] * MHZ // c["rate"])
    per_second = stations * pols * c["rate"] * c.get("subbands", 1) * (1.3 if c.get("mixed") else 1.0)
    hi = max(lo + 1, min(1000000, int(1.0e9 / per_second * 1e6)))
    us = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return job(None, us=us, invalid=int(rng.random() < 0.15 and not c.get("mixed")), **c)


# ----------------------------------------------------------------- inputs
def _pinned():
    keep = []

    def alloc(n):
        buf = torch.empty(n, dtype=torch.uint8, pin_memory=torch.cuda.is_available())
        keep.append(buf)
        return buf.numpy()

    return alloc, keep


# sign bits of four 2-bit codes (the high bit of each)
_SIGNS = np.array([sum(((b >> (2 * k + 1)) & 1) << k for k in range(4)) for b in range(256)], dtype=np.uint8)


def _codes_of(sc, seed):
    """codes(k, nbytes) for scenario.build_job_bulk: the signal model, one sky signal per recording mode."""
    keys = sc.streams()
    device = "cuda:0" if torch.cuda.is_available() else "cpu"
    modes = {}
    for si, st in enumerate(sc.stations):
        m = sc.station_modes.get(st.number, (sc.sample_rate, sc.bits, 0))
        modes.setdefault(m, []).append(si)
    data = {}
    for q, ((rate, bits, off), members) in enumerate(sorted(modes.items())):
        k = next(i for i, (si, _) in enumerate(keys) if si == members[0])
        n = scenario.bulk_stream_bytes(sc, k) * 8 // bits
        tones = [(0.234 * sc.bandwidth, math.sqrt(2000.0 / sc.nchan))]
        gen = synth.model_codes_torch([sc.stations[si] for si in members], sc.pols, rate,
                                      float(sc.channel_freq + off), n, float(sc.sec0), sc.rho, seed * 10 + q,
                                      tones=tones, device=device)
        for (i, pol), packed in gen:
            if bits == 1:
                s = _SIGNS[packed]
                packed = s[0::2] | (s[1::2] << 4)
            data[(members[i], pol)] = packed
    return lambda k, nbytes: data[keys[k]]


def _stations(n, seed, max_delay):
    rng = np.random.Generator(np.random.PCG64(seed + 99))
    return scenario.cubic_stations(n, seed=seed, max_delay=max_delay, max_rate=3e-6,
                                   gains=list(rng.uniform(0.5, 2.0, size=n)))


def _scenario(c, seed, sb):
    st = _stations(c["stations"], 4242 + seed, 15e-3)
    rate, bw = c["rate"], c["rate"] // 2
    modes = {}
    if c["mixed"]:  # three recording modes: the job's, twice its band, and a 1-bit half of it
        for i, s in enumerate(st):
            if i % 10 in (6, 7, 8):
                modes[s.number] = (2 * rate, 2, -bw if sb % 2 else 0)
            elif i % 10 == 9:
                modes[s.number] = (rate // 2, 1, bw // 2 if sb % 2 else 0)
    extra = []
    if c["centres"] > 1:
        rng = np.random.Generator(np.random.PCG64(seed + 7))
        extra = [("PC%d" % k, list(rng.uniform(-3e-7, 3e-7, size=c["stations"]))) for k in range(1, c["centres"])]
    return scenario.Scenario(
        stations=st, pols=("R", "L")[:c["pols"]], sample_rate=rate, bandwidth=bw, bits=c["bits"],
        channel_freq=4_800_000_000 + sb * bw, nchan=c["nchan"], number_channels=c["outch"], window=c["window"],
        integration_us=c["us"], n_integrations=1, sub_integration_us=125000, lead_us=LEAD_US,
        seed=seed * 16 + sb, block_bytes=BLOCK_BYTES, frequency_nr=sb, rho=0.01, station_modes=modes,
        extra_centers=extra)


def _lag_window(n):
    """The user's lag window of a spectral reduction: 2n lags, triangular."""
    q = np.arange(2 * n)
    return (1.0 - np.minimum(q, 2 * n - q) / (1.5 * n)).astype(np.float32)


def _job(c, seed, sb, alloc):
    sc = _scenario(c, seed, sb)
    codes = _codes_of(sc, seed * 16 + sb)
    j = scenario.build_job_bulk(sc, alloc=alloc, codes=codes)
    if c["outch"] < c["nchan"]:
        j["lag_window"] = _lag_window(c["outch"])
    if c["bins"]:
        j.update(scenario.pulsar_params(sc, nbins=c["bins"], gate=(0.0, 1.0), obs_freq=4800.0))
    if c["invalid"]:  # the first station's invalid frames, one run in each of some blocks
        rec0, start, tint, slice_samples = scenario.job_timing(sc)
        dels = j["del_bytes"][0]
        sl = [(start, start + tint, slice_samples,
               correlator.delay_list(dels, start, start + tint, sc.sample_rate, sc.bits))]
        spb = sc.block_bytes * 8 // sc.bits * timebase.ticks_per_sample(sc.sample_rate)
        for k in range(c["pols"]):
            raw = codes(k, 0)
            nb = len(raw) // sc.block_bytes
            blocks = [(rec0 + b * spb, raw[b * sc.block_bytes:(b + 1) * sc.block_bytes],
                       [(100, 700)] if b % 7 == 3 else []) for b in range(nb)]
            p = correlator.write_protocol(blocks, sl, sc.sample_rate, sc.bits, sc.integration_us)
            buf = alloc(len(p[0]))
            buf[:] = np.frombuffer(p[0], dtype=np.uint8)
            j["protocols"][k] = [buf]
    return j


def _batch_jobs(c, seed, alloc):
    scs = scenario.c4_jobs(scale=c["us"] / 2e6, seed=11 + seed, subbands=(0,), fine_subbands=(0,),
                           narrow_subbands=(0,))
    return [scenario.build_job_bulk(sc, alloc=alloc, codes=_codes_of(sc, seed * 16 + i)) for i, sc in enumerate(scs)]


_TRACKS16 = [[2 * c + 1, 2 * c] for c in range(16)]


def _frontend(c, seed):
    sr = c["rate"]
    sc = scenario.Scenario(stations=scenario.cubic_stations(1, seed=5, max_delay=4e-3, max_rate=1e-6),
                           sample_rate=sr, bandwidth=sr // 2, nchan=512, integration_us=(c["ms"] - 40) * 1000 // 2,
                           n_integrations=2, lead_us=16000)
    rng = np.random.Generator(np.random.PCG64(11 + seed))
    per_frame = 8000 * 8 // 32  # 8000-byte payloads, 16 channels x 2 bits
    frames = c["ms"] * sr // 1000 // per_frame
    words = np.frombuffer(rng.bytes(frames * 8000), dtype=np.uint32)
    rec = synth.vdif_frames_array(words, payload_bytes=8000, sample_rate=sr, nchan=16, bits=2, start_mjd=sc.mjd,
                                  start_sec_of_day=sc.sec0)
    alloc, keep = _pinned()
    buf = alloc(rec.size)
    buf[:] = rec
    dels = scenario.del_tables(sc)[0]
    _, start, tint, slice_samples = scenario.job_timing(sc)
    slices = [(start + k * tint, start + (k + 1) * tint, slice_samples,
               correlator.delay_list(dels, start + k * tint, start + (k + 1) * tint, sr, 2))
              for k in range(sc.n_integrations)]
    params = dict(ref_ticks=timebase.ticks_from_mjd_sec(sc.mjd, 0.0), track_bit_rate=sr, frame_size=8000, n_tracks=32,
                  bits=2, channel_tracks=_TRACKS16)
    return buf, keep, params, slices, sc.integration_us


def prepare(case, seed):
    if case["kind"] == "frontend":
        buf, keep, params, slices, us = _frontend(case, seed)
        return dict(kind="frontend", node=correlator.CorrelatorNode(0, lib.X_FP32), rec=buf, keep=keep, params=params,
                    slices=slices, us=us, rate=case["rate"])
    alloc, keep = _pinned()
    if case["kind"] == "batch":
        jobs = _batch_jobs(case, seed, alloc)
        nodes = [correlator.CorrelatorNode(0, lib.X_TC_HILO) for _ in jobs]
        return dict(kind="batch", jobs=jobs, nodes=nodes, batch=correlator.Batch(nodes), keep=keep)
    mode = lib.X_TC_HILO if case["mode"] == "tc" else lib.X_FP32
    jobs = [_job(case, seed, sb, alloc) for sb in range(case["subbands"])]
    nodes = [correlator.CorrelatorNode(0, mode) for _ in jobs]
    pool = ThreadPoolExecutor(max_workers=len(jobs)) if len(jobs) > 1 else None
    torch.cuda.empty_cache()
    return dict(kind="job", jobs=jobs, nodes=nodes, pool=pool, keep=keep)


# ------------------------------------------------------------------- run
def _split(j, cor, tsys, n_integrations=1):
    """The output bytes of one job as arrays: headers (bytes), visibilities
    [output][baseline][channel], tsys records (bytes); views, nothing copied."""
    a = np.frombuffer(cor, dtype=np.uint8)
    nst = len(j["streams"])
    nbl = struct.unpack_from("<i", a, 8)[0]
    nuvw = struct.unpack_from("<i", a, 12)[0]
    rec = 8 + 8 * (j["number_channels"] + 1)
    head = 20 + 32 * nuvw + 24 * nst
    parts = a.reshape(-1, head + nbl * rec)
    body = parts[:, head:].reshape(parts.shape[0], nbl, rec)
    return {"head": parts[:, :head], "baselines": body[:, :, :8], "vis": body[:, :, 8:].view(np.complex64),
            "tsys": np.frombuffer(tsys, dtype=np.uint8)}


def run(state):
    if state["kind"] == "frontend":
        r = correlator.DeviceRecording(state["node"], state["rec"], "vdif", **state["params"])
        r.extract(4, 2, _TRACKS16)
        out = [r.protocol(ch, state["slices"], state["rate"], 2, state["us"]) for ch in range(16)]
        r.close()
        return [np.frombuffer(b, dtype=np.uint8) for ch in out for b in ch]
    if state["kind"] == "batch":
        outs = state["batch"].correlate(state["jobs"])
        return [_split(j, c, t) for j, (c, t) in zip(state["jobs"], outs)]
    jobs, nodes = state["jobs"], state["nodes"]
    if state["pool"] is None:
        outs = [nodes[0].correlate(jobs[0])]
    else:
        outs = list(state["pool"].map(lambda nj: nj[0].correlate(nj[1]), zip(nodes, jobs)))
    return [_split(j, c, t) for j, (c, t) in zip(jobs, outs)]


# ------------------------------------------------------------------ work
def _job_work(rates, bits, bws, us, nchan, outch, nout, nbl, job_rate):
    samples = [r * us / 1e6 for r in rates]
    rows = us / 1e6 * job_rate / nchan
    flops = 0.0
    for s, r in zip(samples, rates):
        # 256-point forward and inverse transforms with the ramp and the
        # rotation, then a windowed real transform every half window
        flops += s * (7.5 * 8 + 8 + 5.0 * math.log2(2 * nchan * r / job_rate))
    flops += 8.0 * nbl * nchan * rows
    inb = sum(s * b / 8 for s, b in zip(samples, bits))
    return inb + 8.0 * nout * nbl * (outch + 1), flops


def _n_baselines(stations, pols):
    n = stations * pols
    return n + n * (n - 1) // 2 - (stations if pols == 2 else 0)


def work(case):
    if case["kind"] == "frontend":
        n = case["ms"] / 1e3 * case["rate"] * 4
        return {"bytes": 2 * n, "flops": 0}
    if case["kind"] == "batch":
        us, b, f = case["us"], 0.0, 0.0
        for rates, bits, nchan, st, count, rate in (
                ([64e6] * 24 + [128e6] * 12 + [32e6] * 4, [2] * 36 + [1] * 4, 4096, 20, 1, 64e6),
                ([64e6] * 24, [2] * 24, 16384, 12, 4, 64e6),
                ([128e6] * 12 + [32e6] * 4, [2] * 12 + [1] * 4, 256, 8, 8, 32e6)):
            x, y = _job_work(rates, bits, None, us, nchan, nchan, count, _n_baselines(st, 2), rate)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    rates, bits = [], []
    for i in range(case["stations"]):
        r, q = case["rate"], case["bits"]
        if case["mixed"]:
            r, q = (2 * r, 2) if i % 10 in (6, 7, 8) else (r // 2, 1) if i % 10 == 9 else (r, q)
        rates += [r] * case["pols"]
        bits += [q] * case["pols"]
    nout = case["bins"] + 1 if case["bins"] else case["centres"]
    b, f = _job_work(rates, bits, None, case["us"], case["nchan"], case["outch"], nout,
                     _n_baselines(case["stations"], case["pols"]), case["rate"])
    return {"bytes": b * case["subbands"], "flops": f * case["subbands"]}


# ----------------------------------------------------------------- exact
TICKS = 512_000_000.0


class _Akima:
    """Akima's (1970) interpolation of a delay table's rows, the end slopes
    extrapolated linearly, over the rows from 2 s before the whole second of
    the integration's start to 2 s after its end."""

    def __init__(self, del_bytes, scan, start, duration):
        p = 4 + struct.unpack_from("<i", del_bytes, 0)[0]
        scans = []
        while p + 81 + 4 + 56 <= len(del_bytes):
            mjd = struct.unpack_from("<i", del_bytes, p + 81)[0]
            p += 85
            rows = []
            while p + 56 <= len(del_bytes):
                row = struct.unpack_from("<7d", del_bytes, p)
                p += 56
                if row[0] == 0 and row[4] == 0:
                    break
                rows.append(row)
            scans.append((mjd, np.array(rows)))
        mjd, rows = scans[scan]
        sec0 = rows[0, 0]
        self.begin = (mjd - 51544) * 86400 * 512_000_000 + round(sec0 * TICKS)
        t0 = math.floor((start - self.begin) / TICKS)
        t1 = math.ceil((start + duration - self.begin) / TICKS)
        lo, hi = max(0, t0 - 2), min(len(rows) - 1, t1 + 2)
        x, y = rows[lo:hi + 1, 0] - sec0, rows[lo:hi + 1, 4]
        n = len(x)
        m = np.zeros(n + 3)
        m[2:n + 1] = np.diff(y) / np.diff(x)
        m[1] = 2 * m[2] - m[3]
        m[0] = 3 * m[2] - 2 * m[3]
        m[n + 1] = 2 * m[n] - m[n - 1]
        m[n + 2] = 3 * m[n] - 2 * m[n - 1]
        w1, w2 = np.abs(m[3:] - m[2:-1]), np.abs(m[1:-2] - m[:-3])
        tot = w1 + w2
        s = np.where(tot > 0, (w1 * m[1:-2] + w2 * m[2:-1]) / np.where(tot > 0, tot, 1.0), m[2:-1])
        h = np.diff(x)
        self.x, self.y, self.b = x, y[:-1], s[:-1]
        self.c = (3 * m[2:n + 1] - 2 * s[:-1] - s[1:]) / h
        self.d = (s[:-1] + s[1:] - 2 * m[2:n + 1]) / (h * h)

    def _at(self, ticks):
        v = (np.asarray(ticks, dtype=np.int64) - self.begin).astype(np.float64) / TICKS
        i = np.clip(np.searchsorted(self.x, v, side="right") - 1, 0, len(self.y) - 1)
        return i, v - self.x[i]

    def delay(self, ticks):
        i, dx = self._at(ticks)
        return self.y[i] + dx * (self.b[i] + dx * (self.c[i] + self.d[i] * dx))

    def rate(self, ticks):
        i, dx = self._at(ticks)
        return self.b[i] + dx * (2 * self.c[i] + 3 * self.d[i] * dx)


def _samples(proto, bits, total, device):
    """The correlator's sample stream of one integration from its protocol
    bytes: data, zeros for invalid samples, one sample inserted (zero) or
    dropped at each change of the integer delay.  Returns (samples, flagged)."""
    buf = np.ascontiguousarray(proto)
    raw = buf.tobytes()
    spb, p, skip, cur, flagged = 8 // bits, 0, 0, None, 0
    starts, sizes, segs, off = [], [], [], 0

    def seg(src, n):
        if n > 0:
            if segs and src >= 0 and segs[-1][0] >= 0 and segs[-1][0] + segs[-1][1] == src:
                segs[-1][1] += n
            else:
                segs.append([src, n])

    have = 0
    while have < total:
        h = raw[p]
        if h == 0:
            n = raw[p + 1] | (raw[p + 2] << 8)
            starts.append(p + 3)
            sizes.append(n)
            seg(off + skip, n * spb - skip)
            have += n * spb - skip
            off += n * spb
            skip = 0
            p += 3 + n
        elif h == 1:
            n = raw[p + 1] | (raw[p + 2] << 8)
            flagged += n
            k = min(skip, n)
            skip -= k
            seg(-1, n - k)
            have += n - k
            p += 3
        elif h == 2:
            rem = struct.unpack_from("b", raw, p + 1)[0]
            if cur is None:
                skip = rem
            elif rem - cur == -1 or rem - cur > 1:
                seg(-1, 1)
                have += 1
            else:
                skip = 1
            cur = rem
            p += 2
        else:
            raise ValueError("protocol ended early")
    payload = np.concatenate([buf[s:s + n] for s, n in zip(starts, sizes)])
    b = torch.from_numpy(payload).to(device).to(torch.int64)
    table = torch.tensor([-7.0, -2.0, 2.0, 7.0] if bits == 2 else [-5.0, 5.0], dtype=torch.float64, device=device)
    x = table[torch.stack([(b >> (bits * k)) & ((1 << bits) - 1) for k in range(spb)], dim=1).reshape(-1)]
    zero = torch.zeros(max([n for s, n in segs if s < 0], default=0), dtype=torch.float64, device=device)
    out = torch.cat([x[s:s + n] if s >= 0 else zero[:n] for s, n in segs])
    return out[:total], flagged


def _windows(kind, n):
    i = np.arange(n, dtype=np.float64)
    w = {RECT: ((i >= n // 4) & (i < 3 * n // 4)).astype(np.float64), COS: np.sin(np.pi * i / (n - 1)),
         HAMMING: 0.54 - 0.46 * np.cos(2 * np.pi * i / (n - 1)), HANN: 0.5 * (1 - np.cos(2 * np.pi * i / (n - 1)))}
    return w[kind]


def _spectra(j, k, it, device):
    """Delay-corrected, fringe-stopped, windowed spectra [row][0..M] of stream
    k in 64 bits, and its flagged samples."""
    _, _, sr, cf, bw, _, _, bits, _, _, tab = j["streams"][k]
    M, rate = j["fft_size_correlation"], j["sample_rate"]
    tint = round(j["integration_time_us"] * 512)
    start = j["start_ticks"] + it * tint
    nr = tint // round(M / (rate / 1e6) * 512)
    nb = M // 256 * nr * sr // rate
    x, flagged = _samples(j["protocols"][k][it], bits, nb * 256, device)
    sp = _Akima(j["del_bytes"][tab], 0, start, tint)
    tps = round(TICKS / sr)
    t0 = start + np.arange(nb, dtype=np.int64) * 256 * tps
    d0, dc, d1 = sp.delay(t0), sp.delay(t0 + 128 * tps), sp.delay(t0 + 256 * tps)
    over = round(sr / (2 * bw))
    integer = np.floor(dc * sr + 0.5).astype(np.int64)
    frac = dc * sr - integer
    step = -2 * np.pi / sr * frac  # radians per Hz
    ramp0 = (integer & (4 * over - 1)) * (np.pi / (2 * over)) - step * (0.5 * bw)
    ramp1 = step * (sr / 256.0)
    fc = cf + 0.5 * bw  # upper sideband
    p0, p1 = fc * d0, fc * d1
    f0 = np.floor(p0)
    phi0, phi1 = -2 * np.pi * (p0 - f0), -2 * np.pi * (p1 - f0)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)  # noqa: E731
    y = torch.empty(nb, 256, dtype=torch.float64, device=device)
    q = torch.arange(129, dtype=torch.float64, device=device)
    n = torch.arange(256, dtype=torch.float64, device=device)
    X = torch.fft.rfft(x.view(nb, 256), dim=1)
    X[:, 0] *= 0.5
    X[:, 128] *= 0.5
    ang = T(np.mod(ramp0, 2 * np.pi))[:, None] + T(ramp1)[:, None] * q
    X = X * torch.polar(torch.ones_like(ang), -ang)
    z = torch.fft.ifft(torch.nn.functional.pad(X, (0, 127)), dim=1) * 256
    ang = T(phi0)[:, None] + T((phi1 - phi0) / 256)[:, None] * n
    y = z.real * torch.cos(ang) + z.imag * torch.sin(ang)
    rot = 2 * M * sr // rate
    hop = rot // 2
    win = T(_windows(j["window"], rot))
    rows = y.reshape(-1)[:nr * hop].unfold(0, rot, hop)  # nr - 1 windows, half overlapping
    S = torch.fft.rfft(rows * win, dim=1)
    delta = j["channel_freq"] - cf
    shift = int(abs(delta) * 2 * M // rate) * (1 if delta > 0 else -1)
    out = torch.zeros(S.shape[0], M + 1, dtype=torch.complex128, device=device)
    a, b = max(0, -shift), min(M, hop - shift)
    out[:, a:b + 1] = S[:, a + shift:b + 1 + shift]
    return out, flagged


def _pairs(j):
    st = [s[0] for s in j["streams"]]
    n = len(st)
    return [(i, i) for i in range(n)] + [(a, b) for a in range(n) for b in range(a + 1, n) if st[a] != st[b]]


def _bins(j, it, nrows, device):
    """Pulsar bin of every (row, channel): the 64-bit phase model of the polyco, in its defined order of operations."""
    nbins, g0, g1 = j["pulsar"]
    nbins += 1
    tmid, dm, ref_phase, ref_freq, obs = j["polyco"][0][:5]
    coef = j["polyco"][0][5:]
    M, day = j["fft_size_correlation"], 86400000000.0
    start = j["start_ticks"] + it * round(j["integration_time_us"] * 512)
    per_day = 86400 * 512_000_000
    mjd = 51544 + start // per_day + (start % per_day) / TICKS / 86400
    dur = M * 1e6 / j["sample_rate"]
    dt = ((mjd + dur / day) - tmid) * 1440
    ph = 0.0
    for cc in reversed(coef[1:]):
        ph = (ph + cc) * dt
    ph += (ref_phase - math.floor(ref_phase)) + dt * 60 * ref_freq + coef[0]
    rate = coef[1] + 60 * ref_freq
    freq = 0.0
    for i in range(len(coef) - 1, 1, -1):
        freq = (freq + i * coef[i]) * dt
    freq = (freq + coef[1]) / 60 + ref_freq
    k = np.arange(M + 1, dtype=np.float64)
    f = j["channel_freq"] * 1e-6 + k * (j["sample_rate"] * 1e-6 / (2 * M))
    off = (4148.808 * dm) * ((1 / (f * f) - 1 / (obs * obs)) * freq)
    r = np.arange(nrows, dtype=np.float64)
    phase = ph + ((rate * dur) * r) * 1440.0 / day
    p = torch.from_numpy(phase).to(device)[:, None] - torch.from_numpy(off).to(device)[None, :]
    p = p - torch.floor(p)
    width = g1 - g0
    b = ((p - g0) * float(nbins - 1) / width).to(torch.int64) + 1
    return torch.where((p >= g0) & (p < g1), b, torch.zeros_like(b)), nbins


def _subints(j, nrows):
    """Row ranges between the sub-integration dumps: the delay correction hands over 8192 samples at a time."""
    M, rate = j["fft_size_correlation"], j["sample_rate"]
    nsub = round(j["sub_integration_time_us"] * 512) // round(M / (rate / 1e6) * 512)
    step = max(8192 // 256, M // 256)
    out, tb, cur, first, nxt, c0, total = [], 0, 0, 0, 1, 0, (nrows + 1) * (M // 256)
    while c0 < total:
        nb = min(step, total - c0)
        nc = (nb * 256 + tb) // M - 1
        tb += nb * 256 - nc * M
        c0 += step
        if nc <= 0:
            continue
        cur += nc
        if cur == nrows or (nsub > 0 and cur >= nxt * nsub):
            out.append((first, cur))
            first = cur
            if cur != nrows:
                nxt += 1
    if first != nrows:
        out.append((first, nrows))
    return out


def _centre_weights(M, window):
    n = 2 * M - 1
    i = np.arange(2 * M, dtype=np.float64)
    f = {RECT: ((i >= n // 4) & (i < 3 * n // 4)).astype(np.float64), COS: np.sin(np.pi * i / n),
         HAMMING: 0.54 - 0.46 * np.cos(2 * np.pi * i / n), HANN: 0.5 * (1 - np.cos(2 * np.pi * i / n))}[window]
    F = np.fft.rfft(f, 4 * M)
    r = np.fft.irfft(np.abs(F) ** 2)[:M]
    return r / r[0]


def _gram(S, pairs):
    """sum over rows of S_a conj(S_b) per pair: S [stream][row][channel] -> [pair][channel]."""
    P = S.permute(2, 0, 1).contiguous()  # [channel][stream][row]
    G = torch.bmm(P, P.conj().transpose(1, 2))
    a = torch.tensor([p[0] for p in pairs], device=S.device)
    b = torch.tensor([p[1] for p in pairs], device=S.device)
    return G[:, a, b].transpose(0, 1)


def _normalised(acc, j, pairs, flagged, total):
    n, M = len(j["streams"]), j["fft_size_correlation"]
    norm = torch.clamp(acc[:n].real.sum(dim=1) / M, min=1.0)
    out = acc.clone()
    out[:n] = (acc[:n].real / norm[:, None]).to(torch.complex128)
    for p in range(n, len(pairs)):
        a, b = pairs[p]
        f = 1.0 - (flagged[a] + flagged[b]) / total  # at most one of the two has flagged samples
        out[p] = acc[p] / torch.sqrt(f * norm[a] * norm[b])
    return out


def _exact_job(j, it, device):
    spec = [_spectra(j, k, it, device) for k in range(len(j["streams"]))]
    S = torch.stack([s for s, _ in spec])
    flagged = [f for _, f in spec]
    spec = None
    pairs, nrows, M = _pairs(j), S.shape[1], j["fft_size_correlation"]
    total = nrows * M
    if "pulsar" in j:
        bins, nb = _bins(j, it, nrows, device)
        idx = (bins * (M + 1) + torch.arange(M + 1, device=device)).reshape(-1)
        acc = torch.zeros(nb, len(pairs), M + 1, dtype=torch.complex128, device=device)
        for p, (a, b) in enumerate(pairs):
            v = (S[a] * S[b].conj()).reshape(-1)
            for part, src in ((0, v.real), (1, v.imag)):
                t = torch.zeros(nb * (M + 1), dtype=torch.float64, device=device).index_add_(0, idx, src.contiguous())
                torch.view_as_real(acc)[:, p, :, part] = t.view(nb, M + 1)
        return torch.stack([_normalised(acc[b], j, pairs, flagged, total) for b in range(nb)]).cpu().numpy()
    npc = j["n_phase_centers"]
    if npc > 1:
        tint = round(j["integration_time_us"] * 512)
        start = j["start_ticks"] + it * tint
        tfft = M * round(TICKS / j["sample_rate"])
        w = _centre_weights(M, j["window"])
        models = [[_Akima(d, c, start, tint) for c in range(npc)] for d in j["del_bytes"]]
        k = torch.arange(M + 1, dtype=torch.float64, device=device)
        acc = torch.zeros(npc, len(pairs), M + 1, dtype=torch.complex128, device=device)
        cross = range(len(j["streams"]), len(pairs))
        for r0, r1 in _subints(j, nrows):
            g = _gram(S[:, r0:r1], pairs)
            acc[0] += g
            tm = start + round(tfft * (r0 + (r1 - r0) / 2.0))
            for c in range(1, npc):
                phi, delta, amp = np.zeros(len(pairs)), np.zeros(len(pairs)), np.ones(len(pairs))
                for p in cross:
                    m1, m2 = (models[j["streams"][s][10]] for s in pairs[p])
                    dd1, dd2 = m1[c].delay(tm) - m1[0].delay(tm), m2[c].delay(tm) - m2[0].delay(tm)
                    t = dd1 * (1 - m1[0].rate(tm)) - dd2 * (1 - m2[0].rate(tm))
                    lag = abs(int(math.floor(abs(dd1 - dd2) * j["sample_rate"] + 0.5)))
                    if lag < M and w[lag] > 1e-4:
                        amp[p] = 1.0 / w[lag]
                    f = j["channel_freq"] * t
                    phi[p] = 2 * np.pi * (f - math.floor(f))
                    delta[p] = 2 * np.pi * j["sample_rate"] / (2.0 * M) * t
                A, P, D = (torch.from_numpy(v).to(device)[:, None] for v in (amp, phi, delta))
                acc[c] += g * torch.polar(A.expand(-1, M + 1), P + D * k)
        return torch.stack([_normalised(acc[c], j, pairs, flagged, total) for c in range(npc)]).cpu().numpy()
    out = _normalised(_gram(S, pairs), j, pairs, flagged, total)
    n = j["number_channels"]
    if n < M:
        X = out.clone()
        X[:, 0] = X[:, 0].real.to(torch.complex128)
        X[:, M] = X[:, M].real.to(torch.complex128)
        r = torch.fft.irfft(X, n=2 * M, dim=1) * (2 * M)
        lag = torch.cat([r[:, :n], 0.5 * (r[:, n:n + 1] + r[:, 2 * M - n:2 * M - n + 1]), r[:, 2 * M - n + 1:]], dim=1)
        lag = lag * torch.from_numpy(j["lag_window"].astype(np.float64)).to(device)
        out = torch.fft.rfft(lag, dim=1) / (2 * M)
    return out[None].cpu().numpy()


def exact(case, seed):
    if case["kind"] == "frontend":
        return None  # bytes only
    device = "cuda:0" if torch.cuda.is_available() else "cpu"
    alloc, keep = _pinned()
    if case["kind"] == "batch":
        jobs = _batch_jobs(case, seed, alloc)
    else:
        jobs = [_job(case, seed, sb, alloc) for sb in range(case["subbands"])]
    out = []
    for j in jobs:
        vis = np.concatenate([_exact_job(j, it, device) for it in range(j["n_integrations"])])
        out.append({"head": None, "baselines": None, "vis": vis, "tsys": None})
    return out
