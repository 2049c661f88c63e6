"""TRI, TPI and curvature on integers: units that change along a strip, rows that share none, sizes
around the 126-column strips, every 8/16-bit type, float32 outputs.

TRI and TPI of windows within four binades are the float64 formula's results bit for bit; the
curvature rounds once where the formula rounds five times, so the two differ by at most 2.5 ulp of
the larger of the terms (2^-51 of |a| / cx^2 + |b| / cy^2, times 100)."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

AFF = (12.5, 0.0, 0.0, 0.0, -7.5, 0.0)


def _check(vsr, d, nodata, aff, exact=True):
    res = vsr.raster_terrain_derivatives(vsr.from_numpy(d, nodata=nodata, affine=aff))
    z = np.pad(d.astype(np.float64), 1, mode="edge")
    terms = 100 * (np.abs(z[1:-1, :-2]) + np.abs(z[1:-1, 2:]) + 2 * np.abs(z[1:-1, 1:-1])) / aff[0] ** 2
    terms += 100 * (np.abs(z[:-2, 1:-1]) + np.abs(z[2:, 1:-1]) + 2 * np.abs(z[1:-1, 1:-1])) / aff[4] ** 2
    for k in ("tri", "tpi", "curvature"):
        ref, _ = oracle.terrain_derivative(d, aff, nodata, k)
        out = res[k].to_numpy()
        assert out.dtype == np.float64
        if k != "curvature" and exact:
            np.testing.assert_array_equal(out, ref, err_msg=k)
        else:
            bound = 2.0**-51 * terms if exact else 1e-12 * (np.abs(ref) + np.abs(d).max())
            assert (np.abs(out - ref) <= bound + 1e-300).all(), k
        # a float32 result is the float64 one rounded
        from vsr_gb300 import algebra

        r = vsr.from_numpy(d, nodata=nodata, affine=aff)
        o32 = algebra.terrain_derivatives(r, tri=k == "tri", tpi=k == "tpi", curvature=k == "curvature",
                                          out_dtype=np.float32)
        got = next(t for t in o32 if t is not None)[0].cpu().numpy()
        if exact:
            np.testing.assert_array_equal(got, out.astype(np.float32), err_msg=k)


@pytest.mark.parametrize("shape", [(1, 1), (2, 300), (3, 126), (70, 127), (129, 253), (67, 504)])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16, np.float32])
def test_integer_strips(vsr, dtype, shape):
    rng = np.random.default_rng(shape[1])
    yy, xx = np.mgrid[0 : shape[0], 0 : shape[1]]
    z = 120 + 60 * np.sin(yy / 21.0) * np.cos(xx / 17.0) + rng.normal(0, 3, shape)
    d = z.astype(dtype)
    d[rng.random(shape) < 0.01] = 9
    for nodata in (9, None):
        _check(vsr, d, nodata, AFF)
    _check(vsr, d, 9, (10.0, 0.0, 0.0, 0.0, -10.0, 0.0))


def test_units_change_down_the_strip(vsr):
    """From 1e-3 to 1e4 along the rows, zeros and signs: each row triple within four binades is exact."""
    rng = np.random.default_rng(1)
    h, w = 400, 260
    base = 10.0 ** np.linspace(-3, 4, h)[:, None]
    d = (base * (1 + 0.01 * rng.random((h, w)))).astype(np.float32)
    d[200:, 100:] *= -1
    d[50:60] = 0.0
    _check(vsr, d, None, AFF, exact=False)
    _check(vsr, d[60:200].copy(), None, AFF)


def test_far_cells_and_wide_values(vsr):
    rng = np.random.default_rng(2)
    d = np.exp(rng.uniform(-20, 20, (90, 140))).astype(np.float32)
    _check(vsr, d, None, AFF, exact=False)
    e = rng.uniform(100, 200, (70, 130)).astype(np.float32)
    _check(vsr, e, None, (1.0, 0.0, 0.0, 0.0, -1000.0, 0.0), exact=False)
