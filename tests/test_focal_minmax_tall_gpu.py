"""Focal min, max and range of 8/16-bit rasters in strips of every height (32 to 256 rows: as tall as
leaves the GPU enough of them), against numpy on slices of rows."""

from __future__ import annotations

import numpy as np
import pytest
from numpy.lib.stride_tricks import sliding_window_view

pytestmark = pytest.mark.gpu


def _reference(d, r, nd, y0, y1):
    a, b = max(0, y0 - r), min(d.shape[0], y1 + r)
    pad = ((r - (y0 - a), r - (b - y1)), (r, r))
    z, valid = d[a:b].astype(np.float64), d[a:b] != nd
    win = lambda fill: sliding_window_view(np.pad(np.where(valid, z, fill), pad, constant_values=fill),  # noqa: E731
                                           (2 * r + 1, 2 * r + 1))
    lo, hi = win(np.inf).min((-2, -1)), win(-np.inf).max((-2, -1))
    out = {"min": lo, "max": hi, "range": hi - lo}
    for v in out.values():
        v[d[y0:y1] == nd] = nd
    return out


@pytest.mark.parametrize("r,height", [(1, 90_001), (3, 170_002), (4, 340_003), (2, 640_004)])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16])
def test_tall_strips(vsr, dtype, r, height):
    rng = np.random.default_rng(r)
    info = np.iinfo(dtype)
    d = rng.integers(info.min, info.max, (height, 16), endpoint=True).astype(dtype)
    d[rng.random(d.shape) < 0.05] = 9
    ras = vsr.from_numpy(d, nodata=9)
    got = {"min": vsr.raster_focal_min(ras, r), "max": vsr.raster_focal_max(ras, r), "range": vsr.raster_focal_range(ras, r)}
    for y0 in (0, height // 3, height - 600):
        ref = _reference(d, r, 9, y0, y0 + 600)
        for k, v in got.items():
            np.testing.assert_array_equal(v.to_numpy()[y0 : y0 + 600], ref[k])
