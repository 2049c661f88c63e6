"""Focal variety against the oracle (exact counts): class maps (one pass of 32 values), maps with
hundreds of values (several passes), noise with more values than the set form takes (the pairs form
per tile), every dtype and unequal radii.  Shapes: narrower than a strip, one column more than a
warp's 120 or 112, wider than a block's 480, more than one 64-row strip."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _map(classes, dtype, shape, rng):
    ids = rng.choice(np.iinfo(dtype).max if classes > 200 else 200, classes, replace=False)
    patch = rng.integers(0, classes, (shape[0] // 3 + 1, shape[1] // 5 + 1))
    d = np.kron(patch, np.ones((3, 5), int))[: shape[0], : shape[1]]
    salt = rng.random(shape) < 0.1
    d[salt] = rng.integers(0, classes, int(salt.sum()))
    d = ids[d]
    if np.iinfo(dtype).min < 0:
        d = d - 100
    return d.astype(dtype)


@pytest.mark.parametrize("dtype,classes", [(np.uint8, 5), (np.uint8, 33), (np.uint8, 200), (np.int16, 12),
                                           (np.uint16, 65), (np.int16, 700), (np.uint16, 20000)])
@pytest.mark.parametrize("r,shape", [(1, (3, 5)), (2, (67, 121)), (3, (65, 483)), (4, (70, 128)), (5, (64, 113)),
                                     (7, (81, 225))])
def test_variety_maps(vsr, dtype, classes, r, shape):
    rng = np.random.default_rng(r + classes)
    d = _map(classes, dtype, shape, rng)
    nd = int(d[0, 0])
    d[: shape[0] // 4, : shape[1] // 3] = nd
    for nodata in (nd, None):
        ref = oracle.focal_stat(d, r, r, nodata, "variety")
        out = vsr.raster_focal_variety(vsr.from_numpy(d, nodata=nodata), r).to_numpy()
        np.testing.assert_array_equal(out, ref)
    o32 = vsr.raster_focal_variety(vsr.from_numpy(d), r, out_dtype=np.float32).to_numpy()
    np.testing.assert_array_equal(o32, ref.astype(np.float32))


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int32, np.float32, np.float64])
@pytest.mark.parametrize("radius", [1, 3, (0, 2), (3, 1), (7, 6), 7])
def test_variety_pairs(vsr, dtype, radius):
    rng = np.random.default_rng(9)
    shape = (2, 37, 131)
    d = rng.integers(0, 9, shape).astype(dtype)
    if np.dtype(dtype).kind == "f":
        d = d * dtype(0.5) - dtype(1)
        d[rng.random(shape) < 0.05] = np.nan
        d[rng.random(shape) < 0.05] *= -1  # -0.0 equals 0.0
    elif np.dtype(dtype).itemsize == 4:
        d = d - 4
    ry, rx = (radius, radius) if isinstance(radius, int) else radius
    out = vsr.raster_focal_variety(vsr.from_numpy(d, nodata=3), radius).to_numpy()
    for b in range(2):
        np.testing.assert_array_equal(out[b], oracle.focal_stat(d[b], ry, rx, 3, "variety"))
