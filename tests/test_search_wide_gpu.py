"""Boxcars and trapezoids wider than a search chunk, whose halo every chunk
scans for itself, up to the widest that a launch's shared memory holds;
several chunks a gulp and a ragged last one, against the FP64 oracle with the
search tests' criteria. FP16 planes get whole samples: their sums are exact
there (far below 2048), so the same criteria hold."""

import numpy as np
import pytest

from frost_b200.config import BoxcarConfig, PeakMode, Storage
from tests.search_cases import compare, make_stream, plan_config, run_engine
from tests.test_search_gpu import PULSES, oracle_for

pytestmark = pytest.mark.gpu

WIDE = ((9000, 12.0, 3000.0, 0.04), (26000, 25.0, 1500.0, 0.06))


@pytest.mark.parametrize("gulp,max_boxcar,wtsp,trapezoid,mode,storage,chunk", [
    (24001, 8192, 2.0, True, PeakMode.PER_WIDTH, Storage.FP16, 4096),
    (24001, 6300, 1.6, True, PeakMode.ACROSS_WIDTHS, Storage.FP32, 4096),  # widest 5938
    (12290, 3000, 2.2, True, PeakMode.PER_WIDTH, Storage.FP32, 2048),
    (12290, 5400, 1.5, False, PeakMode.ACROSS_WIDTHS, Storage.FP32, 4096),
    (11000, 2500, 1.7, False, PeakMode.ALL, Storage.FP16, 2048)])
def test_halos_wider_than_a_chunk_match_the_oracle(gulp, max_boxcar, wtsp, trapezoid, mode, storage, chunk):
    from frost_b200.search import FDMTBoxcar
    pc = plan_config(nchans=48, depth=1, gulp=gulp, dm_max=30.0)
    bc = BoxcarConfig(max_boxcar=max_boxcar, wtsp=wtsp, use_trapezoid=trapezoid, detect_thresh=5.5, peak_mode=mode,
                      storage=storage, max_candidates=1 << 22, max_cands_per_dm=0)
    stream = make_stream(pc, 3, seed=gulp + max_boxcar, pulses=PULSES + WIDE)
    if storage == Storage.FP16:
        stream = np.rint(stream)
    eng = FDMTBoxcar(pc, bc)
    eng.set_launch_shape(search_chunk=chunk)
    cands = run_engine(eng, stream, gulp)
    ref = oracle_for(pc, bc).search(stream, gulp, [np.ones(pc.nchans, np.uint8)] * 3)
    n, missing, extra, bad = compare(cands, ref, bc.detect_thresh)
    assert n > 0 and not missing and not extra and not bad, (missing[:3], extra[:3], bad[:3])
