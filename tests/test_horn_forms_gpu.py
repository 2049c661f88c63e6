"""The Horn kernels give one and the same result: TMA tiles (float32, aligned rows), strips (float32,
odd rows; 8/16-bit) and one thread per pixel (int32, float64).  On whole elevations every gradient
is exact, so slope, aspect and hillshade are equal bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AFF = (30.0, 0.0, 0.0, 0.0, -20.0, 0.0)


def _dem(shape, rng):
    yy, xx = np.mgrid[0 : shape[0], 0 : shape[1]]
    d = np.round(700 + 400 * np.sin(yy / 13.0) * np.cos(xx / 11.0) + rng.normal(0, 40, shape))
    d[rng.random(shape) < 0.01] = 9
    return d


@pytest.mark.parametrize("shape", [(66, 128), (66, 127), (300, 1000), (300, 1001)])
@pytest.mark.parametrize("nodata", [9, None])
def test_float32_equals_scalar_form(vsr, shape, nodata):
    d = _dem(shape, np.random.default_rng(shape[1]))
    a = vsr.raster_terrain(vsr.from_numpy(d.astype(np.float32), nodata=nodata, affine=AFF))
    b = vsr.raster_terrain(vsr.from_numpy(d.astype(np.int32), nodata=nodata, affine=AFF))
    for k in ("slope", "aspect", "hillshade"):
        np.testing.assert_array_equal(a[k].to_numpy(), b[k].to_numpy())


@pytest.mark.parametrize("height", [80_001, 160_002, 313_003])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16, np.float32])
def test_tall_strips_equal_scalar_form(vsr, dtype, height):
    """Strips of 16, 32 and 64 rows (a strip is as tall as leaves the GPU enough of them)."""
    rng = np.random.default_rng(height)
    d = np.round(120 + 60 * np.sin(np.arange(height) / 13.0)[:, None] + rng.normal(0, 20, (height, 13))).clip(0, 255)
    d[rng.random(d.shape) < 0.01] = 9
    for nodata in (9, None):
        a = vsr.raster_terrain(vsr.from_numpy(d.astype(dtype), nodata=nodata, affine=AFF))
        b = vsr.raster_terrain(vsr.from_numpy(d.astype(np.int32), nodata=nodata, affine=AFF))
        for k in ("slope", "aspect", "hillshade"):
            np.testing.assert_array_equal(a[k].to_numpy(), b[k].to_numpy())


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32])
@pytest.mark.parametrize("shape", [(1, 1), (3, 126), (700, 601), (1100, 1201)])
def test_few_strips_and_many_agree(vsr, dtype, shape):
    """Rasters of too few strips take one thread per pixel; beside one another in a stack they do not."""
    rng = np.random.default_rng(shape[0])
    d = _dem(shape, rng)
    d = d.clip(0, 255) if dtype == np.uint8 else d
    stack = np.repeat(d.astype(dtype)[None], 8 if shape[0] > 500 else 1500, 0)
    a = vsr.raster_terrain(vsr.from_numpy(stack[0], nodata=9, affine=AFF))
    b = vsr.raster_terrain(vsr.from_numpy(stack, nodata=9, affine=AFF))
    for k in ("slope", "aspect", "hillshade"):
        np.testing.assert_array_equal(np.repeat(a[k].to_numpy()[None], len(stack), 0), b[k].to_numpy())
