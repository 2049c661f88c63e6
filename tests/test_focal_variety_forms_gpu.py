"""The two forms of the focal variety count alike: a raster of few blocks compares pairs, the same
raster many times in a stack ORs one-hot words; both against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16])
@pytest.mark.parametrize("r,shape", [(1, (5, 7)), (1, (35, 485)), (2, (17, 130)), (2, (16, 500))])
@pytest.mark.parametrize("values", [12, 250])
def test_few_blocks_and_many_agree(vsr, dtype, r, shape, values):
    rng = np.random.default_rng(values + shape[1])
    d = rng.integers(0, values, shape).astype(dtype)
    d[:, : shape[1] // 3] = 3
    for nodata in (3, None):
        ref = oracle.focal_stat(d, r, r, nodata, "variety")
        one = vsr.raster_focal_variety(vsr.from_numpy(d, nodata=nodata), r).to_numpy()
        many = vsr.raster_focal_variety(vsr.from_numpy(np.repeat(d[None], 700, 0), nodata=nodata), r).to_numpy()
        np.testing.assert_array_equal(one, ref)
        np.testing.assert_array_equal(many, np.repeat(ref[None], 700, 0))
