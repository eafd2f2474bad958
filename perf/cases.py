"""Performance cases of the search framework: what its users have it do, from
the smallest blocks of the tests to the 4096-channel headline gulp, each run
through the Python package's public classes.

kind      entry point                              stands for
clean     RFICleaner.execute_normalized_device     cleaning one packed gulp that is on the device
search    FDMTBoxcar.execute_device                the dedispersion search of one calibrated waterfall
pipeline  GulpPipeline.execute_device              a beam's gulp from packed samples to candidates
post      CandidatePostprocessPlan.execute_device  clustering a gulp's raw detections
serve     BeamServer.submit_ptr / wait             one gulp of each of several unlike beams
batch     BeamBatch.execute_ptrs / results         the same beams as one batched call

Observations are synthetic (the noise, RFI and pulse recipe of
frost_b200.synth, generated on the GPU): 64 us samples over 1200-1536 MHz
unless a case says otherwise. A pass is the next gulp of a stream: the
objects keep their calibration and histories as a beam's do.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from frost_b200.batch import BeamBatch
from frost_b200.config import (BlockLayout, BoxcarConfig, DataType, FillMode, PeakMode, RfiConfig, Storage,
                               ZeroDMMode)
from frost_b200.dedisp import band_edges, generate_dm_list
from frost_b200.pipeline import GulpPipeline, plan_for
from frost_b200.postprocess import (GIANT_DTYPE, CandidatePostprocessLayout, CandidatePostprocessPlan,
                                    SearchConfig, SubbandDedupMode)
from frost_b200.rfi import RFICleaner
from frost_b200.search import CANDIDATE_DTYPE, FDMTBoxcar
from frost_b200.serve import BeamServer

KDM = 4.148808e3  # s MHz^2 cm^3 / pc
TSAMP = 64e-6
F_LOW, F_HIGH = 1200.0, 1536.0
DTYPES = {"u1": DataType.UINT1, "u2": DataType.UINT2, "u4": DataType.UINT4, "u8": DataType.UINT8,
          "u16": DataType.UINT16, "u32": DataType.UINT32, "f32": DataType.FLOAT32}


# ---- the cases ---------------------------------------------------------------


def listed():
    return [
        # The tests' smallest whole block: latency, not bandwidth.
        dict(name="clean_64x4096_u8", kind="clean", nchans=64, nsamps=4096, dtype="u8", recipe="default"),
        # An older backend's 2-bit data, an odd number of samples and a band that is no power of two.
        dict(name="clean_1536x40001_u2", kind="clean", nchans=1536, nsamps=40001, dtype="u2", recipe="mean"),
        # A float32 beam of the serving mix, every strategy, zero-DM fit and equalisation.
        dict(name="clean_1024x65536_f32", kind="clean", nchans=1024, nsamps=65536, dtype="f32", recipe="zdot"),
        # The headline gulp's cleaning stage.
        dict(name="clean_4096x262144_u8", kind="clean", nchans=4096, nsamps=262144, dtype="u8", recipe="full"),
        # The tests' smallest sub-band search.
        dict(name="search_64x4096_fp32", kind="search", nchans=64, nsamps=4096, dm_max=60.0, depth=2,
             boxcar=32, storage="fp32", peaks="width", trapezoid=False),
        # The 1024-channel, DM 0-500 workload with the default FP32 planes.
        dict(name="search_1024x65536_fp32", kind="search", nchans=1024, nsamps=65536, dm_max=500.0, depth=0,
             boxcar=64, storage="fp32", peaks="width", trapezoid=False),
        # Ragged in every size, trapezoid filters, one peak over all widths, sub-bands.
        dict(name="search_1000x50001_fp16", kind="search", nchans=1000, nsamps=50001, dm_max=900.0, depth=1,
             boxcar=100, storage="fp16", peaks="across", trapezoid=True),
        # The headline band and DM range in short gulps with FP32 planes (11 planes).
        dict(name="search_4096x65536_fp32", kind="search", nchans=4096, nsamps=65536, dm_max=2000.0, depth=2,
             boxcar=256, storage="fp32", peaks="width", trapezoid=False),
        # The 1024-channel workload end to end, frost's default RFI, giants out.
        dict(name="pipe_1024x65536_fp16", kind="pipeline", nchans=1024, nsamps=65536, dm_max=500.0, depth=0,
             boxcar=64, dtype="u8", recipe="default", storage="fp16", post=True),
        # The headline workload: one gulp of a 4096-channel beam, 11 planes.
        dict(name="pipe_4096x262144_fp16", kind="pipeline", nchans=4096, nsamps=262144, dm_max=2000.0, depth=2,
             boxcar=256, dtype="u8", recipe="full", storage="fp16", post=False),
        # The headline gulp's raw detections.
        dict(name="post_220000", kind="post", rows=220000, dedup="transitive"),
        # Four unlike beams of the serving mix, one gulp of each in flight.
        dict(name="serve_4_beams", kind="serve", beams=4, nchans=1024, nsamps=65536, dm_max=1500.0, depth=1,
             boxcar=256),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the listed range, few of them round."""
    kind = rng.choice(["clean", "clean", "search", "search", "pipeline", "post", "serve", "batch"])
    if kind == "post":
        return dict(kind=kind, rows=_logint(rng, 200, 220000), dedup=rng.choice(["transitive", "seeded"]))
    if kind == "clean":
        nchans = 8 * _logint(rng, 8, 512)
        nsamps = _logint(rng, 4096, min(262144, (1 << 28) // nchans))
        dtype = rng.choice(["u1", "u2", "u4", "u8", "u8", "u8", "u16", "f32", "f32"])
        recipes = ["default", "mean"] if dtype in ("u1", "u2", "u4") else ["default", "mean", "noise", "full", "zdot"]
        return dict(kind=kind, nchans=nchans, nsamps=nsamps, dtype=dtype, recipe=rng.choice(recipes))
    if kind in ("serve", "batch"):
        nsamps = _logint(rng, 8192, 65536)
        return dict(kind=kind, beams=rng.randint(2, 4), nchans=_logint(rng, 128, 1024), nsamps=nsamps,
                    dm_max=round(nsamps / 17.6 * rng.uniform(0.05, 0.38), 1), depth=rng.choice([0, 1]),
                    boxcar=rng.choice([32, 64, 128, 256]))
    nchans = _logint(rng, 64, 2048)
    nsamps = _logint(rng, 4096, 65536)
    case = dict(kind=kind, nchans=nchans, nsamps=nsamps,
                dm_max=round(nsamps / 17.6 * rng.uniform(0.05, 0.4), 1), depth=rng.choice([0, 1, 2]),
                boxcar=rng.randint(16, 256), storage=rng.choice(["fp16", "fp32"]))
    if kind == "search":
        case.update(peaks=rng.choice(["width", "width", "across"]), trapezoid=rng.choice([False, False, True]))
    else:
        case.update(dtype=rng.choice(["u8", "u8", "f32"]), recipe=rng.choice(["default", "full"]),
                    post=rng.choice([False, True]))
    return case


# ---- configurations ----------------------------------------------------------


def _rfi(recipe):
    cfg = RfiConfig()
    if recipe == "mean":
        cfg.fill = FillMode.MEAN
    elif recipe == "noise":
        cfg.fill = FillMode.NOISE
        cfg.zero_dm = ZeroDMMode.SUBTRACT
    elif recipe in ("full", "zdot"):
        cfg.moments.enabled = True
        cfg.iqrm.enabled = True
        cfg.kadane_channel.enabled = True
        cfg.kadane_spectrum.enabled = True
        cfg.zero_dm = ZeroDMMode.SUBTRACT
        if recipe == "zdot":
            cfg.dropout.enabled = True
            cfg.zero_dm = ZeroDMMode.ZDOT
            cfg.equalize = True
    return cfg


def _layout(case, dtype=None):
    foff = -(F_HIGH - F_LOW) / case["nchans"]
    return BlockLayout(case["nchans"], case["nsamps"], DTYPES[dtype or case.get("dtype", "f32")], TSAMP,
                       F_HIGH + foff / 2, foff)


def _boxcar(case, storage=None):
    return BoxcarConfig(max_boxcar=case["boxcar"], wtsp=2.0, detect_thresh=6.0,
                        use_trapezoid=bool(case.get("trapezoid", False)),
                        peak_mode=PeakMode.ACROSS_WIDTHS if case.get("peaks") == "across" else PeakMode.PER_WIDTH,
                        storage=Storage.FP16 if (storage or case["storage"]) == "fp16" else Storage.FP32,
                        max_candidates=1 << 20 if case["nchans"] * case["nsamps"] >= 1 << 28 else 1 << 16,
                        max_cands_per_dm=4096)


def _plan(case, lay):
    return plan_for(lay, 0.0, case["dm_max"], case["depth"])


# ---- inputs ------------------------------------------------------------------


def _add_pulses(x, time_major, rng, n, dm_max, amplitude):
    """Dispersed Gaussian pulses added to x ([T][C], highest frequency first,
    or [C][T], lowest first); amplitude(width) per channel and sample."""
    T, C = x.shape if time_major else x.shape[::-1]
    bw = (F_HIGH - F_LOW) / C
    f = (F_HIGH - bw / 2 - bw * np.arange(C)) if time_major else (F_LOW + bw / 2 + bw * np.arange(C))
    flat = x.view(-1)
    for _ in range(n):
        dm, width = rng.uniform(0.05 * dm_max, 0.95 * dm_max), rng.uniform(1.0, 64.0)
        delay = KDM * dm * (f ** -2.0 - F_HIGH ** -2.0) / TSAMP
        centre = rng.uniform(0.0, max(1.0, T - delay.max() - 4 * width)) + delay
        sig = max(width / 2.355, 0.3)
        half = int(math.ceil(4 * sig)) + 1
        t = np.floor(centre)[:, None] + np.arange(-half, half + 1)[None, :]
        prof = np.exp(-0.5 * ((t - centre[:, None]) / sig) ** 2) * amplitude(width)
        ok = (t >= 0) & (t < T)
        c = np.broadcast_to(np.arange(C)[:, None], t.shape)
        at = (t * C + c if time_major else c * T + t)[ok].astype(np.int64)
        part = torch.from_numpy(prof[ok].astype(np.float32)).to(x.device)
        flat.index_add_(0, torch.from_numpy(at).to(x.device), part)


def _pulse_count(nsamps):
    return max(2, min(20, nsamps // 13000))


def _filterbank(nchans, nsamps, dtype, dm_max, seed, rfi=True):
    """Packed time-major samples on the GPU: noise, 5 % noisy channels,
    zero-DM bursts, dropouts and dispersed pulses."""
    g = torch.Generator("cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    bits = DTYPES[dtype].bits if dtype != "f32" else 8
    if dtype == "u16":
        mean, sd = 3000.0, 100.0
    elif dtype == "u32":
        mean, sd = 1.0e6, 300.0
    else:
        mean, sd = ((1 << bits) - 1) / 2.0, max((1 << bits) / 16.0, 0.8)
    x = torch.empty((nsamps, nchans), dtype=torch.float32, device="cuda")
    x.normal_(mean, sd, generator=g)
    if rfi:
        noisy = torch.from_numpy(np.sort(rng.choice(nchans, max(1, nchans // 20), replace=False))).cuda()
        x[:, noisy] += torch.empty((nsamps, noisy.numel()), device="cuda").normal_(0.0, 3.0 * sd, generator=g)
    _add_pulses(x, True, rng, _pulse_count(nsamps), dm_max,
                lambda w: rng.uniform(7.0, 50.0) * sd / math.sqrt(nchans * max(1.0, 1.064 * w)))
    if rfi:
        for _ in range(max(1, nsamps // 13000)):
            at, n = int(rng.integers(0, nsamps - 50)), int(rng.integers(1, 51))
            x[at:at + n] += 40.0 * sd
        for _ in range(max(1, nsamps // 87000)):
            at = int(rng.integers(0, max(1, nsamps - 512)))
            x[at:at + min(512, nsamps // 8)] = mean if dtype == "f32" else 0.0
    if dtype == "f32":
        return x.view(torch.uint8).view(-1)
    x.round_().clamp_(0, float(2 ** bits - 1) if bits < 32 else 4.0e9)
    if dtype in ("u16", "u32"):
        v = x.to(torch.int32)
        return (v.to(torch.int16) if dtype == "u16" else v).view(torch.uint8).view(-1)
    v = x.to(torch.uint8).view(-1)
    if bits < 8:
        v = v.view(-1, 8 // bits)
        packed = torch.zeros(v.shape[0], dtype=torch.uint8, device="cuda")
        for k in range(8 // bits):
            packed |= v[:, k] << (k * bits)
        v = packed
    return v


def _waterfall(case, seed, device="cuda"):
    """A calibrated unit-noise waterfall [channel][time], lowest frequency first, with pulses."""
    g = torch.Generator(device).manual_seed(seed)
    rng = np.random.default_rng(seed)
    x = torch.empty((case["nchans"], case["nsamps"]), dtype=torch.float32, device=device)
    x.normal_(0.0, 1.0, generator=g)
    _add_pulses(x, False, rng, _pulse_count(case["nsamps"]), case["dm_max"],
                lambda w: rng.uniform(9.0, 50.0) / math.sqrt(case["nchans"] * max(1.0, 1.064 * w)))
    return x


def _detections(n, seed):
    """About n raw detections of one 4096-channel, 262144-sample gulp, as the
    11-plane search reports them: pulses over hundreds of DM trials and
    several widths in every plane, and scattered noise peaks."""
    rng = np.random.default_rng(seed)
    gulp, nchans, ndm, nw = 262144, 4096, 3625, 9
    bw = (F_HIGH - F_LOW) / nchans
    planes = [(0, 0, 0, nchans)]
    for level in (1, 2):
        w = nchans >> level
        planes += [(level, i, i * w, (i + 1) * w) for i in range(1 << level)]
        planes += [(level, (1 << level) + i, i * w + w // 2, (i + 1) * w + w // 2) for i in range((1 << level) - 1)]
    pulses = max(1, min(20, n // 500))
    noise = n // 200
    spread = max(2, (n - noise) // (pulses * len(planes) * 6))
    parts = []

    def rows(plane, dm_idx, filt, peak, snr):
        level, idx, cb, ce = plane
        out = np.zeros(dm_idx.size, CANDIDATE_DTYPE)
        out["width"] = 1 << filt
        out["peak_sample"] = peak
        out["begin_sample"] = np.maximum(peak - rng.integers(0, 1 + (1 << filt)), 0)
        out["end_sample"] = peak + rng.integers(0, 1 + (1 << filt))
        out["snr"], out["dm"] = snr, dm_idx * (2000.0 / ndm)
        out["f_low_mhz"], out["f_high_mhz"] = F_LOW + cb * bw, F_LOW + ce * bw
        out["filter_idx"], out["dm_idx"] = filt, dm_idx
        out["chan_begin"], out["chan_end"], out["subband_level"], out["subband_idx"] = cb, ce, level, idx
        return out

    for _ in range(pulses):
        t0, d0 = rng.uniform(1000, gulp - 50000), int(rng.integers(100, ndm - 100))
        f0, snr0 = int(rng.integers(0, nw)), rng.uniform(12.0, 60.0)
        for plane in planes:
            d = np.arange(max(0, d0 - spread // 2), min(ndm, d0 - spread // 2 + spread))
            d, f = (a.ravel() for a in np.meshgrid(d, np.arange(max(0, f0 - 3), min(nw, f0 + 3))))
            arrival = t0 + KDM * d0 * (2000.0 / ndm) * ((F_LOW + plane[2] * bw) ** -2 - F_HIGH ** -2) / TSAMP
            peak = np.clip(arrival + 0.3 * (d - d0) + rng.normal(0, 1 + (1 << f) / 8), 0, gulp - 1024).astype(np.int64)
            snr = 6.0 + snr0 * np.exp(-np.abs(d - d0) / max(1.0, spread / 3)) * rng.uniform(0.5, 1.0, d.size)
            parts.append(rows(plane, d, f, peak, snr))
    which = rng.integers(0, len(planes), noise)
    for k, plane in enumerate(planes):
        m = int((which == k).sum())
        f = rng.integers(0, nw, m)
        parts.append(rows(plane, rng.integers(0, ndm, m), f, rng.integers(0, gulp - 1024, m), rng.uniform(6.0, 7.0, m)))
    out = np.concatenate(parts)
    return out[rng.permutation(out.size)]


class _Device:
    """A float32 device array at an address, for torch.as_tensor: the tensor
    holds this object, and with it the owner of the memory."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False), version=3)


# ---- prepare / run -----------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    torch.cuda.init()
    state = dict(kind=kind)
    if kind == "clean":
        lay = _layout(case)
        state["raw"] = _filterbank(case["nchans"], case["nsamps"], case["dtype"], 100.0, seed)
        state["cleaner"] = RFICleaner(_rfi(case["recipe"]), lay, 2.0)
        state["shape"], state["view"], state["ptr"] = (case["nchans"], case["nsamps"]), None, None
    elif kind == "search":
        lay = _layout(case)
        state["waterfall"] = _waterfall(case, seed)
        state["search"] = FDMTBoxcar(_plan(case, lay), _boxcar(case))
        state["found"] = _Kept(CANDIDATE_DTYPE, _boxcar(case).max_candidates)
        state["nsamps"] = case["nsamps"]
    elif kind == "pipeline":
        lay = _layout(case)
        state["raw"] = _filterbank(case["nchans"], case["nsamps"], case["dtype"], case["dm_max"], seed,
                                   rfi=case["recipe"] == "full")
        torch.cuda.empty_cache()
        bc = _boxcar(case)
        post = SearchConfig(boxcar_max=case["boxcar"], max_candidates=bc.max_candidates) if case["post"] else None
        state["pipe"] = GulpPipeline(_rfi(case["recipe"]), lay, 2.0, _plan(case, lay), bc, postprocess=post)
        state["pipe"].search.autotune()  # once per beam, as the server does when it admits one
        state["found"] = _Kept(CANDIDATE_DTYPE, bc.max_candidates)
        state["giants"] = _Kept(GIANT_DTYPE, 1 << 14, "giant_")
        state["nsamps"] = case["nsamps"]
    elif kind == "post":
        rows = _detections(case["rows"], seed)
        state["gulp"], state["n"], state["step"] = 262144, rows.size, 0
        state["gulps"] = []  # a stream of four gulps, the last one final
        for k in range(4):
            r = rows.copy()
            for f in ("peak_sample", "begin_sample", "end_sample"):
                r[f] += np.uint64(k * state["gulp"])
            state["gulps"].append(torch.from_numpy(r.view(np.uint8)).cuda())
        state["giants"] = _Kept(GIANT_DTYPE, 1 << 16)
        dedup = SubbandDedupMode.SEEDED if case["dedup"] == "seeded" else SubbandDedupMode.TRANSITIVE
        state["plan"] = CandidatePostprocessPlan(
            SearchConfig(boxcar_max=256, max_candidates=1 << 18, subband_dedup=dedup),
            CandidatePostprocessLayout(4096, TSAMP, -(F_HIGH - F_LOW) / 4096))
    else:
        serve = kind == "serve"
        host = BeamServer(slots=case["beams"]) if serve else BeamBatch()
        state["host"], state["blocks"], state["beams"], state["found"] = host, [], [], []
        for b in range(case["beams"]):
            # unlike beams: full and half band, uint8 and float32, shorter DM ranges
            beam = dict(case, nchans=max(16, case["nchans"] >> (b // 2)), dm_max=case["dm_max"] * (1 - 0.15 * b),
                        dtype="f32" if b % 2 else "u8")
            lay = _layout(beam)
            raw = _filterbank(beam["nchans"], beam["nsamps"], beam["dtype"], beam["dm_max"], seed + 101 * b)
            torch.cuda.empty_cache()
            state["beams"].append(host.add_beam(_rfi("full"), lay, 2.0, _plan(beam, lay), _boxcar(beam, "fp16")))
            state["blocks"].append(raw)
            state["found"].append(_Kept(CANDIDATE_DTYPE, _boxcar(beam, "fp16").max_candidates, "b%d_" % b))
        state["nsamps"] = case["nsamps"]
    torch.cuda.synchronize()
    return state


class _Kept:
    """A program's own table of one gulp's rows, `capacity` of them, the ones
    after the last row zero."""

    def __init__(self, dtype, capacity, prefix=""):
        rows = np.zeros(capacity, dtype)
        self.raw, self.size, self.used, self.count = rows.view(np.uint8), dtype.itemsize, 0, prefix + "count"
        self.out = {prefix + f: rows[f] for f in dtype.names}

    def columns(self, rows):
        used = rows.size * self.size
        self.raw[:used] = rows.view(np.uint8)
        if used < self.used:
            self.raw[used:self.used] = 0
        self.used = used
        return dict(self.out, **{self.count: rows.size})


def run(state):
    kind = state["kind"]
    if kind == "clean":
        raw, cleaner = state["raw"], state["cleaner"]
        ptr = cleaner.execute_normalized_device(raw.data_ptr(), raw.numel(), state["shape"][1])
        if ptr != state["ptr"]:  # the cleaner's output buffer: the same one from gulp to gulp
            state["ptr"] = ptr
            state["view"] = torch.as_tensor(_Device(ptr, state["shape"], cleaner), device="cuda")
        return dict(waterfall=state["view"], mask=cleaner.channel_mask())
    if kind == "search":
        res = state["search"].execute_device(state["waterfall"].data_ptr(), state["nsamps"])
        return state["found"].columns(res.candidates)
    if kind == "pipeline":
        pipe = state["pipe"]
        res = pipe.execute_device(state["raw"].data_ptr(), state["nsamps"])
        out = state["found"].columns(res.candidates)
        out["mask"] = pipe.rfi.channel_mask()
        if pipe.post is not None:
            out.update(state["giants"].columns(pipe.postprocessed.candidates))
        return out
    if kind == "post":
        k = state["step"]
        state["step"] = (k + 1) % len(state["gulps"])
        end = (k + 1) * state["gulp"]
        res = state["plan"].execute_device(state["gulps"][k].data_ptr(), state["n"], end, state["gulp"],
                                           k + 1 == len(state["gulps"]), end - 256)
        return dict(state["giants"].columns(res.candidates), pending=res.pending_candidates)
    host, out = state["host"], {}
    if kind == "serve":
        tickets = [host.submit_ptr(b, raw.data_ptr(), raw.numel(), state["nsamps"], True)
                   for b, raw in zip(state["beams"], state["blocks"])]
        found = [host.wait(t)[0] for t in tickets]
    else:
        host.execute_ptrs([raw.data_ptr() for raw in state["blocks"]], [state["nsamps"]] * len(state["blocks"]), True)
        found = [host.results(b) for b in state["beams"]]
    for kept, rows in zip(state["found"], found):
        out.update(kept.columns(rows))
    return out


# ---- bytes, operations and 64-bit values -------------------------------------


class _Tree:
    """The channel tree of the search (balanced halving; a row of delay d
    splits into round(d K(mid, high) / K(low, high)) samples across the upper
    part and the rest across the lower; a single channel is a window of d + 1
    samples), with the rows that the searched planes need of every node."""

    def __init__(self, case):
        lay = _layout(case)
        pc = _plan(case, lay)
        self.nchans = case["nchans"]
        self.f_min, self.f_max = (float(v) for v in band_edges(pc))
        self.tsamp = float(np.float32(TSAMP))
        dms = generate_dm_list(pc)
        self.planes = []  # (level, index, a, mid, b, delays, dms)
        C, by_depth = self.nchans, {}
        todo = [(0, C, 0)]
        while todo:
            a, b, d = todo.pop(0)
            by_depth.setdefault(d, []).append((a, b))
            if b - a > 1 and d <= case["depth"]:
                m = a + (b - a) // 2
                todo += [(a, m, d + 1), (m, b, d + 1)]
        bands = [(0, 0, 0, C // 2, C)]
        for s in range(1, case["depth"] + 1):
            bands += [(s, i, a, a + (b - a) // 2, b) for i, (a, b) in enumerate(by_depth[s])]
            half = by_depth[s + 1]
            bands += [(s, len(by_depth[s]) + i, half[2 * i + 1][0], half[2 * i + 1][1], half[2 * i + 2][1])
                      for i in range(len(by_depth[s]) - 1)]
        self.need = {}  # (a, mid, b) -> delays
        for s, i, a, m, b in bands:
            k = self.K(a, b)
            x = KDM * dms.astype(np.float64) * k / self.tsamp
            d = np.floor(x + 0.5).astype(np.int64)
            keep = np.concatenate([[True], d[1:] != d[:-1]])
            self.planes.append((s, i, a, m, b, d[keep], dms[keep]))
            self.need[a, m, b] = np.union1d(self.need.get((a, m, b), []), d[keep]).astype(np.int64)
        # widest first: a node's parents come before it
        done, queue = set(), sorted(self.need, key=lambda n: n[0] - n[2])
        while queue:
            n = queue.pop(0)
            if n in done:
                continue
            done.add(n)
            a, m, b = n
            if b - a == 1:
                continue
            lo, hi, parts = *self.parts(n), self.split(n, self.need[n])
            for child, d in ((lo, parts[0]), (hi, parts[1])):
                self.need[child] = np.union1d(self.need.get(child, []), d).astype(np.int64)
                if child in done:
                    done.discard(child)
                queue.append(child)
            queue.sort(key=lambda n: n[0] - n[2])
        self.rows = sum(d.size for n, d in self.need.items() if n[2] - n[0] > 1)
        self.searched = sum(p[5].size for p in self.planes)

    def edge(self, c):
        return self.f_min + c * ((self.f_max - self.f_min) / self.nchans)

    def K(self, a, b):
        return 1.0 / self.edge(a) ** 2 - 1.0 / self.edge(b) ** 2

    def parts(self, n):
        a, m, b = n
        return (a, a + (m - a) // 2, m), (m, m + (b - m) // 2, b)

    def split(self, n, d):
        a, m, b = n
        hi = np.floor(d * (self.K(m, b) / self.K(a, b)) + 0.5).astype(np.int64)
        return d - hi, hi

    def lengths(self, n, d):
        """Window length of every channel of node n for the delays d: [len(d)][b - a]."""
        a, m, b = n
        if b - a == 1:
            return d[:, None] + 1
        lo, hi = self.parts(n)
        dl, dh = self.split(n, d)
        return np.concatenate([self.lengths(lo, dl), self.lengths(hi, dh)], axis=1)


def _widths(boxcar):
    w = [1]
    while 2 * w[-1] <= boxcar:
        w.append(2 * w[-1])
    return w


_counts = {}


def _search_work(case):
    """Bytes (the waterfall once, float32) and additions (one per sample of
    every tree row; a difference and a comparison per width of every searched
    one) of a search."""
    key = tuple(case[k] for k in ("nchans", "nsamps", "dm_max", "depth"))
    if key not in _counts:
        if case["nchans"] * case["dm_max"] > 1.0e6:
            # about one row per sample of the largest delay in every level, and the level-1 leaves
            rows = int(17.54 * case["dm_max"] * math.log2(case["nchans"])) + case["nchans"]
            searched = int(17.54 * case["dm_max"])
        else:
            t = _Tree(case)
            rows, searched = t.rows, t.searched
        _counts[key] = rows, searched
    rows, searched = _counts[key]
    T = case["nsamps"]
    return dict(bytes=4.0 * case["nchans"] * T, flops=float(rows + 2 * len(_widths(case["boxcar"])) * searched) * T)


def _clean_work(case):
    """The packed samples read and the float32 waterfall written once; a few
    operations a sample for the mean, the deviation, the clipping test and
    the calibration."""
    n = case["nchans"] * case["nsamps"]
    return dict(bytes=n * (DTYPES[case["dtype"]].bits / 8 + 4.0), flops=10.0 * n)


def work(case):
    kind = case["kind"]
    if kind == "clean":
        return _clean_work(case)
    if kind == "search":
        return _search_work(case)
    if kind == "post":  # each 72-byte detection read once, and a giant's 176 bytes for about 1 % of them
        return dict(bytes=74.0 * case["rows"], flops=100.0 * case["rows"])
    if kind == "pipeline":  # packed samples in; the waterfall need not leave the chip
        c, s = _clean_work(case), _search_work(case)
        return dict(bytes=c["bytes"] - s["bytes"], flops=c["flops"] + s["flops"])
    total = dict(bytes=0.0, flops=0.0)
    for b in range(case["beams"]):
        beam = dict(case, kind="pipeline", nchans=max(16, case["nchans"] >> (b // 2)),
                    dm_max=case["dm_max"] * (1 - 0.15 * b), dtype="f32" if b % 2 else "u8")
        w = work(beam)
        total = {k: total[k] + w[k] for k in total}
    return total


def _box_power(length, w, trapezoid):
    """Sum of squares of a width-w window convolved with a box of `length` samples."""
    win = np.ones(w)
    if trapezoid and w >= 3:
        e = (w + 1) // 4
        win[:e] = win[w - e:] = 0.5
    return float(np.square(np.convolve(win, np.ones(length))).sum())


def exact(case, seed):
    """The search's S/N and DM columns from a float64 restatement of the tree,
    the boxcars and the run peaks (first gulp of a stream, no history). The
    cleaner's output is fixed to the bit by the order of its own sums, and
    clustering computes no new numbers: no separate 64-bit value. With FP16
    planes the list itself follows the planes' rounding at the threshold. The
    headline-sized searches would take minutes."""
    if case["kind"] != "search" or case["storage"] != "fp32" or case["nchans"] * case["nsamps"] > 1 << 26:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = _waterfall(case, seed, dev).double()
    tree, T = _Tree(case), case["nsamps"]
    widths, trap, thresh = _widths(case["boxcar"]), bool(case["trapezoid"]), 6.0
    sums = torch.nn.functional.pad(x.cumsum(1), (1, 0))  # sums[c][i] = x[c][:i]
    del x
    rows = {}

    def later(row, d):
        return row if d == 0 else torch.nn.functional.pad(row[:max(T - d, 0)], (min(d, T), 0))

    uses = {}
    for n in tree.need:
        if n[2] - n[0] > 1:
            for child in tree.parts(n):
                uses[child] = uses.get(child, 0) + 1
    wanted = {(p[2], p[3], p[4]) for p in tree.planes}
    tables = {}
    for n in sorted(tree.need, key=lambda n: n[2] - n[0]):
        a, m, b = n
        if b - a == 1:
            out = []
            for d in tree.need[n].tolist():
                s = sums[a]
                out.append(s[1:] - torch.nn.functional.pad(s, (d, 0))[:T] if d else s[1:] - s[:-1])
        else:
            lo, hi = tree.parts(n)
            dl, dh = tree.split(n, tree.need[n])
            il, ih = np.searchsorted(tree.need[lo], dl), np.searchsorted(tree.need[hi], dh)
            out = [rows[lo][i] + later(rows[hi][j], int(d)) for i, j, d in zip(il, ih, dl)]
            for child in (lo, hi):
                uses[child] -= 1
                if uses[child] == 0 and child not in wanted:
                    rows[child] = None
        rows[n] = out
    snr, dm = [], []
    t = torch.arange(T, device=dev)
    for _, _, a, m, b, delays, dms in tree.planes:
        n = (a, m, b)
        at = np.searchsorted(tree.need[n], delays)
        lens = tree.lengths(n, delays)
        tables = {(L, w): _box_power(L, w, trap) for L in np.unique(lens) for w in widths}
        var = np.array([[sum(cnt * tables[L, w] for L, cnt in zip(*np.unique(ls, return_counts=True))) for w in widths]
                        for ls in lens])
        for r, (i, d) in enumerate(zip(at, delays.tolist())):
            p = torch.nn.functional.pad(rows[n][i].cumsum(0), (1, 0))

            def window(w, p=p):  # sum of the w samples that end at t
                return p[1:] - torch.nn.functional.pad(p, (w - 1, 0))[:T]
            series = []
            for k, w in enumerate(widths):
                s = window(w)
                if trap and w >= 3:
                    e = (w + 1) // 4
                    first = torch.nn.functional.pad(window(e), (w - e, 0))[:T]
                    s = s - 0.5 * (window(e) + first)
                s = s / math.sqrt(var[r, k])
                s[:d + w - 1] = -math.inf
                series.append(s)
            series = torch.stack(series)
            if case["peaks"] == "across":
                best, which = series.max(0)
                series, which = best[None], which[None]
            else:
                which = torch.arange(len(widths), device=dev)[:, None].expand(-1, T)
            found = []
            up = series > thresh
            for k in torch.nonzero(up.any(1)).view(-1).tolist():
                u = up[k].to(torch.int8)
                edge = torch.nn.functional.pad(u, (1, 1)).diff()
                begin, end = torch.nonzero(edge == 1).view(-1).tolist(), torch.nonzero(edge == -1).view(-1).tolist()
                for lo, hi in zip(begin, end):
                    if hi == T:  # still open: reported with the next gulp
                        continue
                    run = series[k, lo:hi]
                    j = int(torch.nonzero(run == run.max())[0])
                    found.append((lo + j, int(which[k, lo + j]), float(run[j])))
            for _, _, v in sorted(found):
                snr.append(v)
                dm.append(float(dms[r]))
    out = dict.fromkeys(CANDIDATE_DTYPE.names)
    capacity = _boxcar(case).max_candidates
    for name, v in (("snr", snr), ("dm", dm)):
        out[name] = torch.nn.functional.pad(torch.tensor(v, dtype=torch.float64), (0, capacity - len(v)))
    return out
