"""The search's bounds where they are tight or special: trapezoids of every
small width (one and two 4-sample groups for each of their four prefix
values), chunks that are not steady (a gulp's partial last chunk of one
sample to almost a whole chunk, a mask change, a threshold near the noise),
peaks across widths, halos wider than a chunk's carried part; against the
FP64 oracle with the search tests' criteria."""

import numpy as np
import pytest

from frost_b200.config import BoxcarConfig, PeakMode, Storage
from tests.search_cases import compare, make_stream, plan_config, run_engine
from tests.test_search_gpu import PULSES, oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gulp,max_boxcar,wtsp,trapezoid,mode,thresh", [
    (4096, 7, 1.1, True, PeakMode.PER_WIDTH, 5.0),       # widths 1, 2, 3, ... 7
    (4097, 16, 2.0, True, PeakMode.ACROSS_WIDTHS, 5.0),  # one column in the last chunk
    (8190, 33, 1.3, True, PeakMode.PER_WIDTH, 4.5),      # all but two
    (5000, 300, 2.0, True, PeakMode.ACROSS_WIDTHS, 5.0),
    (5001, 24, 1.5, False, PeakMode.ACROSS_WIDTHS, 4.5),
    (6003, 64, 2.0, False, PeakMode.PER_WIDTH, 4.5),
    (12289, 32, 2.0, False, PeakMode.ALL, 5.5)])
def test_bounds_match_the_oracle(gulp, max_boxcar, wtsp, trapezoid, mode, thresh):
    from frost_b200.search import FDMTBoxcar
    pc = plan_config(nchans=48, depth=1, gulp=gulp, dm_max=30.0)
    bc = BoxcarConfig(max_boxcar=max_boxcar, wtsp=wtsp, use_trapezoid=trapezoid, detect_thresh=thresh, peak_mode=mode,
                      max_candidates=1 << 20, max_cands_per_dm=1 << 16)
    stream = make_stream(pc, 3, seed=gulp + max_boxcar, pulses=PULSES)
    rng = np.random.default_rng(gulp)
    masks = [np.ones(pc.nchans, np.uint8), np.ones(pc.nchans, np.uint8), (rng.random(pc.nchans) > 0.2).astype(np.uint8)]
    masked = stream.copy()
    for g, m in enumerate(masks):
        masked[:, g * gulp:(g + 1) * gulp] *= m[:, None]
    cands = run_engine(FDMTBoxcar(pc, bc), stream, gulp, masks=masks)
    ref = oracle_for(pc, bc).search(masked, gulp, masks)
    n, missing, extra, bad = compare(cands, ref, bc.detect_thresh)
    assert n > 0 and not missing and not extra and not bad, (missing[:3], extra[:3], bad[:3])


@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP16])
@pytest.mark.parametrize("gulp,tile,depth", [(3001, 0, 0), (5003, 4096, 2), (8200, 0, 1)])
def test_histories_of_ragged_gulps(gulp, tile, depth, storage):
    """Every row keeps the columns its readers shift into, for gulps that end
    at any column: the third gulp's planes against the oracle's rows over the
    whole stream (the storage precisions' bounds of the search tests)."""
    from frost_b200.search import FDMTBoxcar
    pc = plan_config(nchans=50, depth=depth, gulp=gulp, dm_max=45.0)
    bc = BoxcarConfig(max_boxcar=40, detect_thresh=8.0, storage=storage, max_candidates=1 << 18)
    stream = make_stream(pc, 3, seed=gulp, pulses=PULSES)
    eng = FDMTBoxcar(pc, bc, tile_nsamps=tile)
    eng.capture_planes(True)
    run_engine(eng, stream, gulp, drain=False)
    bound = 1e-5 if storage == Storage.FP32 else 1e-2
    for p, band in enumerate(oracle_for(pc, bc).bands):
        rows = oracle_for(pc, bc).dedisperse(stream, band)[:, -gulp:]
        rms = np.sqrt(np.mean(rows ** 2, axis=1, keepdims=True)) + 1e-12
        assert np.max(np.abs(eng.plane_data(p, gulp) - rows) / rms) < bound, p
