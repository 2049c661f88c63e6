"""Focal std in strips of every height (16 to 128 rows: as tall as leaves the GPU enough of them) and
of rasters of too few strips.  The reference is extended precision on slices of rows; a float64
result lies within one ulp of it (the sums are exact, root and quotient within 0.52 ulp)."""

from __future__ import annotations

import numpy as np
import pytest
from numpy.lib.stride_tricks import sliding_window_view

pytestmark = pytest.mark.gpu
ND = 7


def _reference(d, r, y0, y1):
    """Rows y0 .. y1 of the std of ``d``."""
    a, b = max(0, y0 - r), min(d.shape[0], y1 + r)
    top, bottom = r - (y0 - a), r - (b - y1)
    z = d[a:b].astype(np.longdouble)
    valid = d[a:b] != ND
    pad = ((top, bottom), (r, r))
    win = sliding_window_view(np.pad(np.where(valid, z, 0), pad), (2 * r + 1, 2 * r + 1))
    ok = sliding_window_view(np.pad(valid, pad), (2 * r + 1, 2 * r + 1))
    n = np.maximum(ok.sum((-2, -1)), 1)
    mean = win.sum((-2, -1)) / n
    dev = np.where(ok, win - mean[..., None, None], 0)
    out = np.sqrt((dev * dev).sum((-2, -1)) / n)
    out[d[y0:y1] == ND] = ND
    return out


def _data(dtype, height, rng, width=13):
    base = 120 + 60 * np.sin(np.arange(height) / 40.0)[:, None]
    d = (base + rng.normal(0, 4, (height, width))).astype(dtype)
    d[rng.random(d.shape) < 0.02] = ND
    return d


@pytest.mark.parametrize("r,height", [(1, 80_001), (3, 160_002), (5, 320_003), (3, 640_004)])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16, np.float32])
def test_tall_strips(vsr, dtype, r, height):
    rng = np.random.default_rng(r)
    d = _data(dtype, height, rng)
    out = vsr.raster_focal_std(vsr.from_numpy(d, nodata=ND), r).to_numpy()
    o32 = vsr.raster_focal_std(vsr.from_numpy(d, nodata=ND), r, out_dtype=np.float32).to_numpy()
    for y0 in (0, height // 3, height // 2 + 77, height - 700):
        ref = _reference(d, r, y0, y0 + 700)
        got = out[y0 : y0 + 700]
        assert (np.abs(got - ref) <= 2.0**-52 * np.abs(ref)).all()
        if dtype != np.float32:  # rounded once from the exact sums
            np.testing.assert_array_equal(o32[y0 : y0 + 700], ref.astype(np.float32))


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16])
@pytest.mark.parametrize("r,shape", [(1, (5, 7)), (3, (60, 130)), (5, (61, 131)), (7, (80, 116))])
def test_few_strips_and_many_agree(vsr, dtype, r, shape):
    """One raster alone (shared-memory kernel) and many of them in a stack (strips): the same bits."""
    rng = np.random.default_rng(r)
    d = _data(dtype, shape[0], rng, shape[1])
    for out_dtype in (np.float64, np.float32):
        one = vsr.raster_focal_std(vsr.from_numpy(d, nodata=ND), r, out_dtype=out_dtype).to_numpy()
        many = vsr.raster_focal_std(vsr.from_numpy(np.repeat(d[None], 400, 0), nodata=ND), r,
                                    out_dtype=out_dtype).to_numpy()
        np.testing.assert_array_equal(many, np.repeat(one[None], 400, 0))


@pytest.mark.parametrize("r", [1, 3, 7])
def test_strips_without_integers(vsr, r):
    """Values 80 binades apart, edges and gaps: two float64 passes (1e-12, as in the other tests)."""
    rng = np.random.default_rng(r)
    d = np.exp(rng.uniform(-40, 40, (90, 300))).astype(np.float32)
    d[rng.random(d.shape) < 0.05] = ND
    d[20:40, 30:60] = ND
    out = vsr.raster_focal_std(vsr.from_numpy(d, nodata=ND), r).to_numpy()
    ref = _reference(d, r, 0, 90)
    assert (np.abs(out - ref) <= 1e-12 * np.abs(ref)).all()
