"""Focal std of float32 and of unaligned or wide-window 8/16-bit rasters (integer-sum warp strips).

The sums are exact and the square root and division are rounded within 0.52 ulp, so a float64
output lies within one ulp (2^-52 relative) of the same formula in extended precision; rasters whose
values span more binades than the integers hold take two float64 passes (1e-12, as in the other
tests).  Shapes: narrower than a strip, one column more than 120 (R <= 4) or 112 (R >= 5) per warp,
more than one 64-row strip.
"""

from __future__ import annotations

import numpy as np
import pytest
from numpy.lib.stride_tricks import sliding_window_view

pytestmark = pytest.mark.gpu


def _reference(data, nodata, r):
    z = data.astype(np.longdouble)
    nd = np.isnan(data) if nodata is not None and nodata != nodata else (data == nodata if nodata is not None else data != data)
    valid = ~nd & ~np.isnan(z)
    if nodata is None:
        nd = np.zeros(data.shape, bool)
    k = 2 * r + 1
    win = sliding_window_view(np.pad(np.where(valid, z, 0), r), (k, k))
    ok = sliding_window_view(np.pad(valid, r), (k, k))
    n = ok.sum((-2, -1))
    with np.errstate(invalid="ignore", divide="ignore"):
        mean = win.sum((-2, -1)) / n
        d = np.where(ok, win - mean[..., None, None], 0)
        out = np.where(n > 0, np.sqrt((d * d).sum((-2, -1)) / np.maximum(n, 1)), 0)
    out[nd] = nodata if nodata is not None else 0
    return out


def _f32(kind, shape, rng):
    base = np.linspace(20.0, 400.0, shape[0] * shape[1]).reshape(shape)
    if kind == "dem":
        d = base + rng.normal(0, 2, shape)
    elif kind == "coast":  # zeros, both signs, small magnitudes beside large ones
        d = np.where(base < 150, np.round(rng.normal(0, 3, shape), 2), base)
    elif kind == "unit":  # 1e-6 .. 1
        d = rng.random(shape) ** 4 + 1e-6
    else:  # "wide": more binades than the integers hold
        d = np.exp(rng.uniform(-40, 40, shape))
    return d.astype(np.float32)


@pytest.mark.parametrize("kind", ["dem", "coast", "unit", "wide"])
@pytest.mark.parametrize("r,shape", [(1, (5, 7)), (2, (67, 121)), (3, (70, 240)), (4, (129, 481)), (5, (66, 113)),
                                     (7, (40, 460))])
def test_std_float32(vsr, kind, r, shape):
    rng = np.random.default_rng(r * 100 + shape[1])
    d = _f32(kind, shape, rng)
    d[rng.random(shape) < 0.03] = np.nan
    d[rng.random(shape) < 0.05] = -9999.0
    d[: shape[0] // 3, : shape[1] // 4] = -9999.0
    tol = 1e-12 if kind == "wide" else 2.0**-52
    for nd in (-9999.0, float("nan"), None):
        ref = _reference(d, nd, r)
        if nd is None or nd != nd:
            # -9999 counts as a value here: a wide span in the "coast" and "unit" rasters
            bound = 1e-12 * np.abs(ref) + 1e-12
        else:
            bound = tol * np.abs(ref) + (1e-12 if kind == "wide" else 0)
        out = vsr.raster_focal_std(vsr.from_numpy(d, nodata=nd), r).to_numpy()
        m = ~np.isnan(ref.astype(np.float64))
        np.testing.assert_array_equal(np.isnan(out), ~m)
        assert (np.abs(out[m] - ref[m]) <= bound[m]).all(), f"{kind} nd={nd}"
        o32 = vsr.raster_focal_std(vsr.from_numpy(d, nodata=nd), r, out_dtype=np.float32).to_numpy()
        np.testing.assert_array_equal(o32, out.astype(np.float32))


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16])
@pytest.mark.parametrize("r,shape", [(1, (5, 7)), (3, (66, 123)), (4, (70, 241)), (5, (67, 224)), (7, (130, 113)),
                                     (2, (40, 244))])
def test_std_integers(vsr, dtype, r, shape):
    rng = np.random.default_rng(r)
    info = np.iinfo(dtype)
    d = rng.integers(info.min, info.max, shape, endpoint=True).astype(dtype)
    d[: shape[0] // 2] = info.max - (d[: shape[0] // 2] & 3)
    d[rng.random(shape) < 0.1] = 7
    for nd in (7, None):
        ref = _reference(d, nd, r)
        out = vsr.raster_focal_std(vsr.from_numpy(d, nodata=nd), r).to_numpy()
        assert (np.abs(out - ref) <= 2.0**-52 * np.abs(ref)).all()
        o32 = vsr.raster_focal_std(vsr.from_numpy(d, nodata=nd), r, out_dtype=np.float32).to_numpy()
        np.testing.assert_array_equal(o32, ref.astype(np.float32))


def test_std_float32_infinities_and_bands(vsr):
    rng = np.random.default_rng(3)
    d = rng.normal(100, 5, (3, 70, 130)).astype(np.float32)
    d[1, 20, 60] = np.inf
    out = vsr.raster_focal_std(vsr.from_numpy(d), 2).to_numpy()
    near = np.zeros((70, 130), bool)
    near[18:23, 58:63] = True
    np.testing.assert_array_equal(np.isnan(out[1]), near)
    for b in range(3):
        ok = np.ones((70, 130), bool) if b != 1 else ~near
        with np.errstate(invalid="ignore"):
            ref = _reference(d[b], None, 2)
        assert (np.abs(out[b] - ref)[ok] <= 1e-12 * np.abs(ref)[ok]).all()
