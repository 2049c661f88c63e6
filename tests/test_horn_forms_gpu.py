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
