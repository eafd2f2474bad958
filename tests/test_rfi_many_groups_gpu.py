"""The column kernels where a CTA holds four 32-channel groups side by side
(more groups an SM than any line of rfi_columns.cuh: 960 groups), with 16- and
4-byte copies: the bars of the kernels' own tests."""

import pytest

from frost_b200.config import DataType
from tests import test_rfi_columns_gpu as columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchans,nsamps,window", [(1024, 3000, 100), (1001, 3900, 130)])
@pytest.mark.parametrize("dtype", [DataType.UINT8, DataType.FLOAT32])
def test_four_groups_a_cta(nchans, nsamps, window, dtype):
    columns.test_bandpass_levels_and_scales(nchans, nsamps, window, dtype)
    columns.test_welford_remeasure(nchans, nsamps, window)
    columns.test_moments_do_not_depend_on_the_sample_type(nchans, nsamps, window)
