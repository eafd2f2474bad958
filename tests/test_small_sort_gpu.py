"""The order of detections at the sizes where the sort changes form: one CTA
up to 8192 rows (a warp's share of one to eight rounds), tiles above. Without
clustering the post-processing plan returns every row in (plane, DM index,
width index, sample) order, which numpy gives too."""

import numpy as np
import pytest

from frost_b200.postprocess import CandidatePostprocessLayout, CandidatePostprocessPlan, SearchConfig
from frost_b200.search import CANDIDATE_DTYPE


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1025, 4097, 8191, 8192, 8193, 20000])
def test_rows_come_back_in_order(n):
    rng = np.random.default_rng(n)
    rows = np.zeros(n, CANDIDATE_DTYPE)
    rows["peak_sample"] = rng.permutation(4 * n)[:n]  # no two rows alike
    rows["begin_sample"] = rows["end_sample"] = rows["peak_sample"]
    rows["dm_idx"] = rng.integers(0, 300, n)
    rows["filter_idx"] = rng.integers(0, 5, n)
    rows["width"] = 1 << rows["filter_idx"]
    rows["snr"] = rng.uniform(6, 30, n).astype(np.float32)
    half = rng.integers(0, 2, n)
    rows["subband_level"], rows["subband_idx"] = 1, half
    rows["chan_begin"], rows["chan_end"] = 32 * half, 32 * half + 32
    plan = CandidatePostprocessPlan(SearchConfig(max_candidates=1 << 16, cluster=False),
                                    CandidatePostprocessLayout(64, 1e-3, -1.0))
    got = plan.execute(rows, 4 * n, 4 * n, True, 4 * n).candidates
    planes = got["plane"].astype(np.int64)
    keys = np.stack([planes, got["dm_idx"], got["filter_idx"], got["samp_idx"]]).astype(np.int64)
    order = np.lexsort(keys[::-1])
    assert got.size == n and np.array_equal(order, np.arange(n))
    want = np.sort(rows["peak_sample"])
    assert np.array_equal(np.sort(got["samp_idx"]), want)
    by_sample = {int(r["peak_sample"]): float(r["snr"]) for r in rows}
    assert all(by_sample[int(g["samp_idx"])] == float(g["snr"]) for g in got)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["TRANSITIVE", "SEEDED"])
@pytest.mark.parametrize("n", [2, 17, 128, 129, 700, 4097])
def test_pair_tiles_match_the_oracle(n, mode):
    """Sub-band dedup at the edges of the pair tiles (chunks of 16 and of 128
    rows) equals the oracle's plan, row for row."""
    from frost_b200.postprocess import ClusterTolerances, SubbandDedupMode, SubbandDedupPlan
    from oracle import postprocess as op
    from tests.postprocess_cases import random_giants, same_giants
    g = random_giants(n, n, spread=20 * n)
    tol = ClusterTolerances(3, 3, 200, 8.0, 1e-3, 6.0)
    m = SubbandDedupMode[mode]
    want = op.backend("oracle").subband_dedup(g, tol, 1e-3, m)
    assert same_giants(SubbandDedupPlan(m).execute(g, tol, 1e-3), want)
