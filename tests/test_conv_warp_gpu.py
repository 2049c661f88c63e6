"""The register convolution (odd square kernels of 3 to 13) against the float64 oracle.

Tolerance 1e-5 relative, that of the other convolution tests: FP32 sums of at most 169 terms with
one sign round to below 180 * 2^-24 = 1.1e-5 in the worst case and near 1e-6 in practice; the sums
here are of positive weights.  A kernel with weights of both signs is held to 1e-5 of sum |w v|.
Shapes: narrower than a warp's 120 or 112 columns, one column more, several strips; gaps that enter
and leave the weight sums with clean rows between them."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _data(dtype, shape, rng):
    base = 150 + 40 * np.sin(np.arange(shape[0]) / 9.0)[:, None] + 25 * np.cos(np.arange(shape[1]) / 7.0)[None]
    return (base + rng.uniform(0, 5, shape)).astype(dtype)


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16, np.float32])
@pytest.mark.parametrize("k,shape", [(3, (2, 5)), (3, (70, 121)), (5, (131, 240)), (7, (64, 360)), (9, (65, 113)),
                                     (11, (150, 225)), (13, (140, 130))])
def test_convolve_small_kernels(vsr, dtype, k, shape):
    rng = np.random.default_rng(k + shape[1])
    d = _data(dtype, shape, rng)
    nd = 7
    h = shape[0]
    d[h // 2, shape[1] // 3] = nd  # one gap between clean rows
    if h > 100:
        d[-20:][rng.random((20, shape[1])) < 0.2] = nd
        d[5:9, 3:60] = nd
    w = rng.random((k, k))
    w[0, 0] = 0.0
    for nodata in (nd, None):
        ref = oracle.convolve_normalized(d, w, nodata)
        for out_dtype in (np.float64, np.float32):
            out = vsr.raster_convolve(vsr.from_numpy(d, nodata=nodata), w, precision="fp32", out_dtype=out_dtype).to_numpy()
            assert out.dtype == out_dtype
            np.testing.assert_allclose(out, ref, rtol=1e-5, atol=0)


def test_convolve_signed_zero_sum_nan_and_bands(vsr):
    rng = np.random.default_rng(4)
    d = _data(np.float32, (90, 250), rng)[None].repeat(2, 0)
    d[1, 40, 100] = np.nan
    w = rng.random((5, 5)) - 0.2
    for nodata in (None, float("nan"), 12345.0):
        out = vsr.raster_convolve(vsr.from_numpy(d, nodata=nodata), w).to_numpy()
        for b in range(2):
            ref = oracle.convolve_normalized(d[b], w, nodata)
            np.testing.assert_array_equal(np.isnan(out[b]), np.isnan(ref))
            m = np.isfinite(ref)
            den = w.sum()
            bound = 1e-5 * np.abs(w).sum() * 260.0 / den
            inner = np.zeros_like(m)
            inner[2:-2, 2:-2] = True
            assert (np.abs(out[b] - ref)[m & inner] <= bound).all()
    lap = np.array([[0.0, 1, 0], [1, -4, 1], [0, 1, 0]])  # weight sum 0: nodata inside
    out = vsr.raster_convolve(vsr.from_numpy(d[0], nodata=-1.0), lap).to_numpy()
    np.testing.assert_array_equal(out[1:-1, 1:-1], -1.0)
