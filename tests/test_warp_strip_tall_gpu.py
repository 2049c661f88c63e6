"""The register Gaussian and convolution in strips of 16, 32 and 64 rows (as tall as leaves the GPU
enough of them): gaps that leave the window and come back within a strip, rows without any between.

Against the float64 oracle on slices (1e-5, as the other tests of these kernels: FP32 sums of positive
terms with at most 17 + 17 roundings each, numerator and weight sum together below 70 * 2^-24 =
4.2e-6), and bit for bit against the same rows cut out as a small raster, whose strips have 16 rows:
every window sees the same rows."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ND = 7


def _data(dtype, height, rng):
    d = (300 + 40 * np.sin(np.arange(height) / 9.0)[:, None] + rng.uniform(0, 5, (height, 250))).astype(dtype)
    lone = rng.integers(0, height, height // 40)  # single gaps, some 40 rows apart: two or none in a window
    d[lone, rng.integers(0, 250, lone.size)] = ND
    d[height // 2 : height // 2 + 30][rng.random((30, 250)) < 0.2] = ND
    return d


def _compare(run, weights, d, r):
    h = d.shape[0]
    out = run(d)
    for y0 in (0, 1000, h // 2 - 60, h - 300):
        a, b = max(0, y0 - r), min(h, y0 + 300 + r)
        ref = oracle.convolve_normalized(d[a:b], weights, ND)
        cut = run(np.ascontiguousarray(d[a:b]))
        rows = slice(y0 - a, y0 - a + 300)
        np.testing.assert_allclose(out[y0 : y0 + 300], ref[rows], rtol=1e-5, atol=0)
        np.testing.assert_array_equal(out[y0 : y0 + 300], cut[rows])


@pytest.mark.parametrize("height", [27_001, 54_002, 105_003])
@pytest.mark.parametrize("dtype,k", [(np.float32, 3), (np.uint16, 9), (np.float32, 17)])
def test_gaussian(vsr, dtype, k, height):
    d = _data(dtype, height, np.random.default_rng(k))
    _compare(lambda x: vsr.raster_gaussian_filter(vsr.from_numpy(x, nodata=ND), k / 6.0, kernel_size=k, precision="fp32",
                                                  out_dtype=np.float32).to_numpy(),
             oracle.gaussian_weights(k / 6.0, k), d, k // 2)


@pytest.mark.parametrize("height", [27_001, 54_002, 105_003])
@pytest.mark.parametrize("dtype,k", [(np.float32, 3), (np.uint16, 7), (np.float32, 13)])
def test_convolution(vsr, dtype, k, height):
    rng = np.random.default_rng(k)
    w = rng.random((k, k))
    w /= w.sum()
    _compare(lambda x: vsr.raster_convolve(vsr.from_numpy(x, nodata=ND), w, precision="fp32", out_dtype=np.float32).to_numpy(),
             w, _data(dtype, height, rng), k // 2)
