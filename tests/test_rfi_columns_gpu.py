"""The per-channel statistics kernels at the sizes where their column
streaming can go wrong (channel groups of less than a warp, rows of any byte
pitch, windows of one sample row to several stages, short last stages),
against the same arithmetic in numpy: sums in row order (np.cumsum), every
operation rounded as the reference's strict IEEE build rounds it. The bar is
bit equality."""

import numpy as np
import pytest

from frost_b200.config import BlockLayout, DataType, RfiConfig
from tests.rfi_cases import pack

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
    return centre.astype(np.float32), sd.astype(np.float32)


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
    (161, 6400, 3125, DataType.FLOAT32)])
def test_bandpass_levels_and_scales(nchans, nsamps, window, dtype):
    from frost_b200.rfi import RFICleaner
    rng = np.random.default_rng(nchans * 7919 + nsamps)
    x = samples(rng, nsamps, nchans, dtype)
    gpu = RFICleaner(RfiConfig.quiet(), BlockLayout(nchans, nsamps, dtype, 2.0 ** -10, 1400.0, 1.0), window * 2.0 ** -10)
    got = gpu.execute_normalized(pack(x, dtype))
    want = np.zeros((nchans, nsamps), np.float32)
    for b, e in windows(nsamps, window):
        level, scale = bandpass(x[b:e])
        want[:, b:e] = ((x[b:e] - level) * (np.float32(1) / scale)).T
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
