"""The register Gaussian (3 to 17 taps) and the strip kernel's small sizes against the float64 oracle.

Tolerance 1e-5 relative, that of the other Gaussian tests: FP32 sums of at most 17 + 17 positive
terms round to below 40 * 2^-24 = 2.4e-6.  Shapes: narrower than a warp's 120 or 112 columns, one
column more, several strips; gaps (nodata) that enter and leave the weight sums, rows without gaps
between them, a NaN and an infinity in the data."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _data(dtype, shape, rng):
    base = 300 + 40 * np.sin(np.arange(shape[0]) / 9.0)[:, None] + 25 * np.cos(np.arange(shape[1]) / 7.0)[None]
    return (base + rng.uniform(0, 5, shape)).astype(dtype) if dtype != np.uint8 else rng.integers(1, 255, shape).astype(dtype)


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16, np.float32, np.int32, np.float64])
@pytest.mark.parametrize("k,shape", [(1, (9, 30)), (3, (2, 5)), (3, (70, 121)), (5, (131, 240)), (9, (64, 360)),
                                     (11, (65, 113)), (13, (150, 225)), (17, (200, 130)), (19, (140, 150))])
def test_gaussian_small_kernels(vsr, dtype, k, shape):
    rng = np.random.default_rng(k + shape[1])
    d = _data(dtype, shape, rng)
    nd = 7
    h = shape[0]
    d[h // 2, shape[1] // 3] = nd  # one gap between clean rows
    if h > 100:
        d[-20:][rng.random((20, shape[1])) < 0.2] = nd
        d[5:9, 3:60] = nd
    sigma = k / 6.0
    w = oracle.gaussian_weights(sigma, k)
    for nodata in (nd, None):
        ref = oracle.convolve_normalized(d, w, nodata)
        for out_dtype in (np.float64, np.float32):
            out = vsr.raster_gaussian_filter(vsr.from_numpy(d, nodata=nodata), sigma, kernel_size=k, precision="fp32",
                                             out_dtype=out_dtype).to_numpy()
            assert out.dtype == out_dtype
            np.testing.assert_allclose(out, ref, rtol=1e-5, atol=0)


def test_gaussian_nan_inf_and_bands(vsr):
    rng = np.random.default_rng(2)
    d = _data(np.float32, (3, 90, 250)[1:], rng)[None].repeat(3, 0)
    d[1, 40, 100] = np.nan
    d[2, 50, 130] = np.inf
    for nodata in (None, float("nan"), 12345.0):
        out = vsr.raster_gaussian_filter(vsr.from_numpy(d, nodata=nodata), 1.5, kernel_size=9).to_numpy()
        w = oracle.gaussian_weights(1.5, 9)
        for b in range(3):
            z = np.where(np.isinf(d[b]), np.float32(1e30), d[b])
            ref = oracle.convolve_normalized(z, w, nodata)
            far = ref > 1e20  # windows that hold the infinity
            if nodata is not None and np.isnan(nodata):
                np.testing.assert_array_equal(np.isnan(out[b]), np.isnan(ref))
            m = np.isfinite(ref) & ~far
            assert np.isinf(out[b][far]).all()
            np.testing.assert_allclose(out[b][m], ref[m], rtol=1e-5)
            np.testing.assert_array_equal(np.isnan(out[b]), np.isnan(ref))
