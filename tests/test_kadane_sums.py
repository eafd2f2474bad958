"""The maximum-sum runs of the RFI scans over every float they can meet. A
float32 channel whose scale has no float inverse (below 2^-128) gives NaN
(0 x inf) where a sample equals the channel's level: such a value ends the
open run, as the reference's comparison does, and later runs count."""

import os
import subprocess

import numpy as np
import pytest

from frost_b200.config import BlockLayout, DataType, RfiConfig
from tests.rfi_cases import pack

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_run_forms_match_the_full_state(tmp_path):
    exe = str(tmp_path / "kadane_sums_test")
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-I" + os.path.join(ROOT, "frost_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "kadane_sums_test.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    assert "bad 0" in r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("nchans", [96, 101])
def test_runs_after_a_channel_without_a_float_inverse(nchans):
    """Rows with a run of raised channels above such a channel have the same
    spans whether that channel is used or zapped. Its samples are 0, a, 0, -a
    and so on (level exactly 0); the raised rows are ones where it is 0, and
    the channels below it are lowered there, so the run starts above it."""
    from frost_b200.rfi import RFICleaner
    nsamps, tiny = 3125, 20
    rng = np.random.default_rng(nchans)
    x = rng.normal(100, 10, (nsamps, nchans)).astype(np.float32)
    x[:, tiny] = np.float32(1e-39) * np.array([0, 1, 0, -1], np.float32)[np.arange(nsamps) % 4]
    rows = np.arange(400, 2400, 200)
    x[rows, :tiny] = 80
    x[rows, tiny + 5:tiny + 45] = 135
    cells = []
    for zap in ([], [(tiny, tiny)]):
        cfg = RfiConfig.quiet()
        cfg.kadane_spectrum.enabled = True
        cfg.kadane_spectrum.threshold, cfg.kadane_spectrum.min_bandwidth = 15.0, 8.0
        cfg.kadane_spectrum.whole_band_fraction = 0.9
        cfg.zap_chans = zap
        gpu = RFICleaner(cfg, BlockLayout(nchans, nsamps, DataType.FLOAT32, 2.0 ** -10, 1400.0, -1.0), 64.0)
        gpu.execute_normalized(pack(x, DataType.FLOAT32))
        cells.append(gpu.report()["cells_kadane_spectrum"])
    assert cells[0] == cells[1] >= 40 * rows.size
