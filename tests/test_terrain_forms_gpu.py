"""Terrain derivatives in every form they take: strips and one pixel per thread, values that share a
32-bit unit, a 64-bit unit or none, strips of 8 to 64 rows.

TRI and TPI are exact integers rounded once wherever a unit of 35 binades holds the window, so they
equal the exact value rounded to float64 (formed here in extended precision).  The curvature rounds
once (32-bit units) or after FP64 products of exact sums: factors, products and sum off by half an
ulp each, below 2^-51 of |a| / cx^2 + |b| / cy^2, times 100.  The bound here is in terms of a and b
themselves, the window's second differences."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AFF = (12.5, 0.0, 0.0, 0.0, -7.5, 0.0)
ND = -9999.0


def _check(vsr, d, aff=AFF, nodata=None):
    res = vsr.raster_terrain_derivatives(vsr.from_numpy(d, nodata=nodata, affine=aff))
    got = {k: r.to_numpy() for k, r in res.items()}
    z = d.astype(np.longdouble)
    c = z[1:-1, 1:-1]
    around = [z[i : i + c.shape[0], j : j + c.shape[1]] for i in range(3) for j in range(3) if (i, j) != (1, 1)]
    tri, tot = np.zeros_like(c), np.zeros_like(c)
    hit = d[1:-1, 1:-1] == nodata
    for v in around:
        tri += np.abs(v - c)
        tot += v - c
        hit = hit | (v == nodata)
    cx2, cy2 = (np.longdouble(abs(aff[i])) ** 2 for i in (0, 4))
    a, b = around[3] + around[4] - 2 * c, around[1] + around[6] - 2 * c
    curv = -100 * (a / cx2 + b / cy2)
    bound = 100 * 2.0**-51 * (np.abs(a) / cx2 + np.abs(b) / cy2)
    for k, ref in (("tri", tri / 8), ("tpi", -tot / 8), ("curvature", curv)):
        out = got[k]
        assert (out[[0, -1]] == ND).all() and (out[:, [0, -1]] == ND).all() if nodata is None else True
        inner = out[1:-1, 1:-1]
        assert (inner[hit] == nodata).all() if nodata is not None else True
        if k == "curvature":
            assert (np.abs(inner - ref)[~hit] <= bound[~hit]).all()
        else:
            np.testing.assert_array_equal(inner[~hit], ref.astype(np.float64)[~hit], err_msg=k)
    return got


def _dem(kind, shape, rng):
    yy, xx = np.mgrid[0 : shape[0], 0 : shape[1]]
    wave = np.sin(yy / 21.0) * np.cos(xx / 17.0)
    if kind == "land":  # one unit
        d = 1200 + 300 * wave + rng.normal(0, 3, shape)
    elif kind == "coast":  # through zero, zeros
        d = np.where(wave > 0.1, 0.0, 500 * wave + rng.normal(0, 1, shape))
    elif kind == "noise":
        d = rng.normal(0, 1, shape)
    else:  # "ramp": 2^-3 .. 2^12 and back within some 60 rows, signs by column
        d = np.exp2(4.5 + 7.5 * np.sin(yy / 10.0)) * (1 + 0.01 * rng.random(shape)) * np.where(xx % 90 < 45, 1, -1)
    return d.astype(np.float32)


@pytest.mark.parametrize("kind", ["land", "coast", "noise", "ramp"])
@pytest.mark.parametrize("shape", [(3, 3), (70, 127), (129, 253)])
def test_few_strips_and_many_agree(vsr, kind, shape):
    rng = np.random.default_rng(shape[1])
    d = _dem(kind, shape, rng)
    one = _check(vsr, d)
    n = 1 + 6000 // (((shape[0] + 7) // 8) * ((shape[1] + 125) // 126))
    many = vsr.raster_terrain_derivatives(vsr.from_numpy(np.repeat(d[None], n, 0), affine=AFF))
    for k in ("tri", "tpi"):
        np.testing.assert_array_equal(many[k].to_numpy(), np.repeat(one[k][None], n, 0))
    d[rng.random(shape) < 0.01] = -77.0
    _check(vsr, d, nodata=-77.0)


@pytest.mark.parametrize("kind", ["coast", "noise", "ramp"])
@pytest.mark.parametrize("shape", [(1300, 1201), (900, 2000)])
def test_strips_of_wide_values(vsr, kind, shape):
    rng = np.random.default_rng(shape[1])
    d = _dem(kind, shape, rng)
    _check(vsr, d)
    d[rng.random(shape) < 0.01] = -77.0
    _check(vsr, d, (30.0, 0, 0, 0, -30.0, 0), nodata=-77.0)


@pytest.mark.parametrize("kind", ["land", "ramp"])
@pytest.mark.parametrize("height", [80_001, 160_002, 313_003])
def test_tall_strips(vsr, kind, height):
    """Strips of 16, 32 and 64 rows: units change many times on the way down."""
    _check(vsr, _dem(kind, (height, 13), np.random.default_rng(height)))


@pytest.mark.parametrize("dtype", [np.int16, np.float32])
@pytest.mark.parametrize("shape", [(90, 100), (1300, 1201)])
def test_cells_far_apart(vsr, dtype, shape):
    """Curvature factors that no common integer unit holds."""
    d = np.round(_dem("land", shape, np.random.default_rng(1))).astype(dtype)
    _check(vsr, d, (1.0, 0, 0, 0, -1000.0, 0))
    _check(vsr, d, (500.0, 0, 0, 0, -0.5, 0))


def test_values_no_unit_holds(vsr):
    """Infinities, NaN and magnitudes 60 binades apart stay where they are; the rest of the raster is exact."""
    for shape in ((80, 130), (1300, 1201)):
        d = _dem("land", shape, np.random.default_rng(4))
        ref = vsr.raster_terrain_derivatives(vsr.from_numpy(d, affine=AFF))
        d[40, 60], d[50, 70], d[60, 80], d[70, 20] = np.inf, np.nan, 1e-20, 1e25
        far = np.zeros(shape, bool)
        for y, x in ((40, 60), (50, 70), (60, 80), (70, 20)):
            far[y - 1 : y + 2, x - 1 : x + 2] = True
        got = vsr.raster_terrain_derivatives(vsr.from_numpy(d, affine=AFF))
        for k in ("tri", "tpi"):
            np.testing.assert_array_equal(got[k].to_numpy()[~far], ref[k].to_numpy()[~far])
            assert not np.isfinite(got[k].to_numpy()[39:42, 59:62]).any()
            assert np.isnan(got[k].to_numpy()[49:52, 69:72]).all()
