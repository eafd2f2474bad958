"""The per-channel statistics kernels at the sizes where their column
streaming can go wrong (channel groups of less than a warp, rows of any byte
pitch, windows of one sample row to several stages, short last stages),
against the same arithmetic in numpy: sums in row order (np.cumsum), every
operation rounded as the reference's strict IEEE build rounds it. The bar is
bit equality."""

import json

import numpy as np
import pytest

from frost_b200.config import BlockLayout, DataType, RfiConfig, ZeroDMMode
from tests.rfi_cases import CASES, make_case, pack
from tests.test_rfi_gpu import GOLDEN, digest

MAX_ROWS = 3125


def windows(nsamps, window):
    n = max(nsamps // window, 1)
    return [(w * window, nsamps if w + 1 == n else (w + 1) * window) for w in range(n)]


def remedian(v):
    while v.shape[0] > 1:
        v = np.sort(v.reshape(-1, 5, v.shape[1]), axis=1)[:, 2]
    return v[0]


def ordered_sum(v):
    return np.cumsum(v, axis=0)[-1]


def bandpass(x):
    """(level, scale) of each channel of one window x [rows][channels] float32
    (remedian, MAD, two 4.5 sigma clips)."""
    m = 1
    while m * 5 <= min(x.shape[0], MAX_ROWS):
        m *= 5
    v = x[[i * x.shape[0] // m for i in range(m)]]
    level = remedian(v)
    sd = (remedian(np.abs(v - level)) * np.float32(1.4826)).astype(np.float64)
    centre, v = level.astype(np.float64), v.astype(np.float64)
    mean = ordered_sum(v) / m
    sd = np.where(sd > 0, sd, np.sqrt(ordered_sum(np.square(v - mean)) / m))
    live = np.ones(x.shape[1], bool)
    for _ in range(2):
        dv = v - centre
        keep = np.abs(dv) <= 4.5 * sd
        count = keep.sum(0).astype(np.float64)
        live &= count >= 2
        shift = ordered_sum(np.where(keep, dv, 0.0)) / np.maximum(count, 1)
        ss = ordered_sum(np.where(keep, (dv - shift) * (dv - shift), 0.0))
        clipped = np.sqrt(ss / np.maximum(count, 1))
        live &= clipped > 0
        centre, sd = np.where(live, centre + shift, centre), np.where(live, clipped, sd)
    return centre.astype(np.float32), np.where(v.min(0) < v.max(0), sd, 0).astype(np.float32)


def same_measured(got, want, scales):
    """Bit equality of every cell of a measured (window, channel): one whose
    sampled values are all equal has no scale, and its cells are filled."""
    on = np.concatenate([np.repeat(s[:, None] > 0, e - b, axis=1) for (b, e), s in scales], axis=1)
    return np.array_equal(got.view(np.uint32)[on], want.view(np.uint32)[on])


def samples(rng, nsamps, nchans, dtype):
    mean, sd, hi = {DataType.UINT2: (1.5, 0.8, 3), DataType.UINT8: (120.0, 12.0, 255),
                    DataType.UINT16: (3000.0, 100.0, 65535), DataType.FLOAT32: (10.0, 2.0, None)}[dtype]
    x = rng.normal(mean, sd, (nsamps, nchans))
    x[rng.random((nsamps, nchans)) < 0.01] += 6 * sd  # clipped in the refinement
    # a channel whose scale remedian is zero
    x[:, -1] = np.where(rng.random(nsamps) < 0.1, x[:, -1], np.rint(mean))
    if hi is None:
        return x.astype(np.float32)
    return np.clip(np.rint(x), 0, hi).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("nchans,nsamps,window,dtype", [
    (1, 64, 64, DataType.FLOAT32), (31, 127, 127, DataType.UINT8), (33, 640, 130, DataType.FLOAT32),
    (64, 4096, 2000, DataType.UINT8), (100, 9001, 4000, DataType.UINT16), (104, 3300, 3200, DataType.UINT2),
    (161, 6400, 3125, DataType.FLOAT32), (1001, 1300, 130, DataType.UINT8), (1024, 1000, 100, DataType.FLOAT32)])
def test_bandpass_levels_and_scales(nchans, nsamps, window, dtype):
    from frost_b200.rfi import RFICleaner
    rng = np.random.default_rng(nchans * 7919 + nsamps)
    x = samples(rng, nsamps, nchans, dtype)
    gpu = RFICleaner(RfiConfig.quiet(), BlockLayout(nchans, nsamps, dtype, 2.0 ** -10, 1400.0, 1.0), window * 2.0 ** -10)
    got = gpu.execute_normalized(pack(x, dtype))
    want, scales = np.zeros((nchans, nsamps), np.float32), []
    for b, e in windows(nsamps, window):
        level, scale = bandpass(x[b:e])
        scales.append(((b, e), scale))
        with np.errstate(divide="ignore", invalid="ignore"):
            want[:, b:e] = ((x[b:e] - level) * (np.float32(1) / scale)).T
    assert same_measured(got, want, scales)


def welford(x):
    """(mean, std) float32 of each column of x, updated row by row in double."""
    mean, var = np.zeros(x.shape[1]), np.zeros(x.shape[1])
    for n, row in enumerate(x.astype(np.float64), 1):
        delta = row - mean
        mean = mean + delta / n
        var = var + delta * (row - mean)
    return mean.astype(np.float32), np.sqrt(var / x.shape[0]).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("nchans,nsamps,window", [(1, 64, 64), (33, 131, 65), (50, 2100, 1000), (128, 1041, 513),
                                                  (1001, 1300, 130), (1024, 1000, 100)])
def test_welford_remeasure(nchans, nsamps, window):
    """equalize rescales the cleaned cells (0 + 1 * z for float32 input) and
    calibrates them again by their Welford mean and std."""
    from frost_b200.rfi import RFICleaner
    rng = np.random.default_rng(nchans * 131 + nsamps)
    x = samples(rng, nsamps, nchans, DataType.FLOAT32)
    cfg = RfiConfig.quiet()
    cfg.equalize = True
    gpu = RFICleaner(cfg, BlockLayout(nchans, nsamps, DataType.FLOAT32, 2.0 ** -10, 1400.0, 1.0), window * 2.0 ** -10)
    got = gpu.execute_normalized(pack(x, DataType.FLOAT32))
    want, scales = np.zeros((nchans, nsamps), np.float32), []
    for b, e in windows(nsamps, window):
        level, scale = bandpass(x[b:e])
        scales.append(((b, e), scale))
        with np.errstate(divide="ignore", invalid="ignore"):
            y = np.float32(0) + np.float32(1) * ((x[b:e] - level) * (np.float32(1) / scale))
            mean, std = welford(y)
            want[:, b:e] = ((y - mean) * (np.float32(1) / std)).T
    assert same_measured(got, want, scales)


@pytest.mark.gpu
@pytest.mark.parametrize("nchans,nsamps,window", [(9, 200, 100), (41, 2100, 700), (130, 5000, 2500), (1001, 1300, 130),
                                                  (1024, 1000, 100)])
def test_moments_do_not_depend_on_the_sample_type(nchans, nsamps, window):
    """The same values as uint8, uint16 and float32 (other copies, shifts and
    conversions of the moments pass) give the same masks and output."""
    from frost_b200.rfi import RFICleaner
    rng = np.random.default_rng(nchans + nsamps)
    x = samples(rng, nsamps, nchans, DataType.UINT8)
    x[:, nchans // 2] = np.clip(np.rint(rng.normal(120, 40, nsamps)), 0, 255)
    cfg = RfiConfig()
    cfg.moments.enabled = cfg.iqrm.enabled = cfg.kadane_channel.enabled = True
    cfg.zero_dm = ZeroDMMode.SUBTRACT
    out = []
    for dtype in (DataType.UINT8, DataType.UINT16, DataType.FLOAT32):
        gpu = RFICleaner(cfg, BlockLayout(nchans, nsamps, dtype, 2.0 ** -10, 1400.0, 1.0), window * 2.0 ** -10)
        out.append((digest(gpu.execute_normalized(pack(x, dtype))), digest(gpu.channel_mask()),
                    gpu.report()["chans_moments"]))
    assert out[0] == out[1] == out[2]


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_golden_digests(name):
    """The reference cleaner's committed digests of every strategy mix."""
    from frost_b200.rfi import RFICleaner
    golden = json.load(open(GOLDEN))[name]
    cfg, layout, baseline, blocks = make_case(name)
    gpu = RFICleaner(cfg, layout, baseline)
    for step, (block, nsamps) in enumerate(blocks):
        assert digest(gpu.execute_normalized(block, nsamps)) == golden[step]["out_sha256"]
        assert digest(gpu.channel_mask()) == golden[step]["mask_sha256"]


@pytest.mark.gpu
@pytest.mark.parametrize("nchans,capacity,valid", [(64, 256, 256), (64, 257, 131), (65, 320, 320), (67, 321, 65),
                                                   (4, 64, 64), (130, 1023, 1000)])
def test_normalize_writes_every_cell(nchans, capacity, valid):
    """Vector and scalar loads and stores of the transpose; masked channels
    and rows past the valid ones are zero in a buffer that held other data
    (a second, shorter block after a whole one)."""
    from frost_b200.rfi import RFICleaner
    rng = np.random.default_rng(nchans + capacity)
    x = samples(rng, capacity, nchans, DataType.FLOAT32)
    cfg = RfiConfig.quiet()
    cfg.zap_chans = [(1, 1)]
    gpu = RFICleaner(cfg, BlockLayout(nchans, capacity, DataType.FLOAT32, 2.0 ** -10, 1400.0, -1.0), 32.0)
    gpu.execute_normalized(pack(x + 1, DataType.FLOAT32))
    got = gpu.execute_normalized(pack(x, DataType.FLOAT32), valid)
    level, scale = bandpass(x[:valid])
    want = np.zeros((nchans, capacity), np.float32)
    want[:, :valid] = ((x[:valid] - level) * (np.float32(1) / scale)).T
    want[1] = 0
    assert np.array_equal(got.view(np.uint32), want[::-1].view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("nsamps", [64, 1001, 8193, 400001])
def test_dropout_cut_is_the_exact_median(nsamps):
    """Rows whose spread is below 0.97 of the median row spread (one rank of
    a series shorter than a CTA's share to one too long for shared memory),
    and their neighbours, are flagged."""
    from frost_b200.rfi import RFICleaner
    nchans, fraction = 8, 0.97
    rng = np.random.default_rng(nsamps)
    x = np.clip(np.rint(rng.normal(120, 12, (nsamps, nchans))), 0, 255)
    cfg = RfiConfig.quiet()
    cfg.dropout.enabled = True
    cfg.dropout.min_std_fraction = fraction
    gpu = RFICleaner(cfg, BlockLayout(nchans, nsamps, DataType.UINT8, 2.0 ** -10, 1400.0, 1.0), 4096.0)
    gpu.execute_normalized(pack(x, DataType.UINT8))
    mean = x.sum(1) / nchans
    spread = np.sqrt(np.maximum(np.square(x).sum(1) / nchans - mean * mean, 0)).astype(np.float32)
    low = spread < np.float32(fraction) * np.sort(spread)[nsamps // 2]
    want = low | np.append(low[1:], False) | np.insert(low[:-1], 0, False)
    assert np.array_equal(gpu.time_flags(nsamps).astype(bool), want)


@pytest.mark.gpu
@pytest.mark.parametrize("nchans,nsamps", [(7, 300), (35, 1025), (131, 2050), (1501, 1100), (1504, 2049)])
@pytest.mark.parametrize("zdot", [False, True])
def test_scans_do_not_depend_on_the_sample_type(nchans, nsamps, zdot):
    """Kadane across frequency and along time and the zdot sums of the same
    values as uint8, uint16 and float32 (rows of any pitch, shifted and whole
    vectors), with masked channels, an unmeasured one and runs of both signs."""
    from frost_b200.rfi import RFICleaner
    rng = np.random.default_rng(nchans + nsamps)
    x = rng.normal(120, 12, (nsamps, nchans))
    x[nsamps // 3:nsamps // 3 + 4, nchans // 4:nchans // 2 + 1] += 60
    x[nsamps // 2:nsamps // 2 + 4, nchans // 3:] -= 50
    x[nsamps // 4:nsamps // 4 + 120, nchans // 2] += 25
    x[:nsamps // 2, nchans - 1] = 120
    x = np.clip(np.rint(x), 0, 255)
    cfg = RfiConfig()
    cfg.kadane_channel.enabled = cfg.kadane_spectrum.enabled = True
    cfg.kadane_channel.min_duration, cfg.kadane_spectrum.min_bandwidth = 0.02, 2.0
    cfg.zero_dm = ZeroDMMode.ZDOT if zdot else ZeroDMMode.OFF
    cfg.zap_chans = [(2, 2)]
    out = []
    for dtype in (DataType.UINT8, DataType.UINT16, DataType.FLOAT32):
        gpu = RFICleaner(cfg, BlockLayout(nchans, nsamps, dtype, 2.0 ** -10, 1400.0, 1.0), 500 * 2.0 ** -10)
        rep = (digest(gpu.execute_normalized(pack(x, dtype))), gpu.report())
        out.append((rep[0],) + tuple(rep[1][k] for k in ("samps_kadane", "cells_kadane_spectrum",
                                                         "cells_kadane_channel", "samps_broad", "chans_dead")))
    assert out[0] == out[1] == out[2]


@pytest.mark.gpu
@pytest.mark.parametrize("nchans,nsamps", [(8, 200), (56, 131), (1000, 70), (1029, 67), (4104, 66)])
@pytest.mark.parametrize("dtype,bits", [(DataType.UINT1, 1), (DataType.UINT2, 2), (DataType.UINT4, 4), (DataType.UINT8, 8),
                                        (DataType.UINT16, 16), (DataType.UINT32, 24), (DataType.FLOAT32, 0)])
def test_clean_rows_are_written_as_read(nchans, nsamps, dtype, bits):
    """Strips of many rows, of one and of a part of one, whole and partial;
    groups of four samples of each width and single ones."""
    from frost_b200.rfi import RFICleaner
    if nchans * max(bits, 1) % 8 != 0 and bits < 8 and bits != 0:
        pytest.skip("rows are whole bytes")
    rng = np.random.default_rng(nchans + nsamps + bits)
    x = (rng.normal(0, 3, (nsamps, nchans)) if bits == 0 else rng.integers(0, 2 ** bits, (nsamps, nchans))).astype(np.float32)
    gpu = RFICleaner(RfiConfig.quiet(), BlockLayout(nchans, nsamps, dtype, 2.0 ** -10, 1400.0, 1.0), 32.0)
    got = gpu.execute_normalized(pack(x, dtype))
    level, scale = bandpass(x)
    with np.errstate(divide="ignore", invalid="ignore"):
        want = np.ascontiguousarray(((x - level) * (np.float32(1) / scale)).T)
    assert same_measured(got, want, [((0, nsamps), scale)])
