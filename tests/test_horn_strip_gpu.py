"""Slope, aspect and hillshade of 8/16-bit DEMs and of float32 DEMs with odd rows, around the
126-column strips: against the oracle (1e-4 degrees, 1 DN, nodata exact, as the other Horn tests)
and bit for bit against the TMA kernel on the same float32 values with padded rows."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

AFF = (30.0, 0.0, 0.0, 0.0, -20.0, 0.0)


def _dem(dtype, shape, rng):
    yy, xx = np.mgrid[0 : shape[0], 0 : shape[1]]
    z = 120 + 60 * np.sin(yy / 13.0) * np.cos(xx / 11.0) + rng.normal(0, 6, shape)
    return z.astype(dtype)


@pytest.mark.parametrize("shape", [(1, 1), (1, 7), (5, 1), (3, 126), (66, 127), (130, 253), (64, 505)])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16, np.float32])
def test_strips_match_oracle(vsr, dtype, shape):
    rng = np.random.default_rng(shape[1])
    d = _dem(dtype, shape, rng)
    d[rng.random(shape) < 0.02] = 9
    for nd in (9, None):
        out = vsr.raster_terrain(vsr.from_numpy(d, nodata=nd, affine=AFF))
        rs, ra = oracle.slope_aspect(d, AFF, nd)
        rh, _ = oracle.hillshade(d, AFF, nd)
        s, a, h = (out[k].to_numpy() for k in ("slope", "aspect", "hillshade"))
        assert s.dtype == (np.float32 if dtype == np.float32 else np.float64)
        np.testing.assert_allclose(s, rs, atol=1e-4, rtol=0)
        da = np.abs(a.astype(np.float64) - ra)
        assert np.minimum(da, 360 - da).max() <= 1e-4
        assert np.abs(h.astype(int) - rh.astype(int)).max() <= 1
        if nd is not None:
            ring = oracle.nodata_ring(d, nd)
            assert (s[ring] == nd).all() and (a[ring] == nd).all() and (h[ring] == 0).all()


@pytest.mark.parametrize("nodata", [-9999.0, float("nan"), None])
@pytest.mark.parametrize("mode", ["window", "center"])
def test_odd_rows_equal_padded_rows(vsr, nodata, mode):
    """The same pixels with a pitch of 255 (strips) and of 256 (TMA), near 0 m and with holes."""
    import torch

    from vsr_gb300 import _lib

    rng = np.random.default_rng(5)
    h, w = 150, 255
    d = (_dem(np.float32, (h, w), rng) - 110).astype(np.float32)
    if nodata is not None:
        d[rng.random((h, w)) < 0.01] = nodata
    lib = _lib.load()
    flags = _lib.VSR_HORN_CENTER_ONLY if mode == "center" else _lib.VSR_HORN_SA_NAN_UNMASKED
    kind = 0 if nodata is None else (2 if np.isnan(nodata) else 1)
    got = []
    for pitch in (255, 256):
        src = torch.zeros((h, pitch), dtype=torch.float32, device="cuda")
        src[:, :w] = torch.from_numpy(d).cuda()
        s, a = (torch.zeros((h, pitch), dtype=torch.float32, device="cuda") for _ in range(2))
        hs = torch.zeros((h, pitch), dtype=torch.uint8, device="cuda")
        rc = lib.vsr_horn_fused(src.data_ptr(), 5, h, w, pitch, 30.0, 20.0, 0.0 if nodata is None else nodata, kind,
                                flags, s.data_ptr(), a.data_ptr(), 5, pitch, hs.data_ptr(), pitch, 1.5, 0.7, 5.0,
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        got.append([t[:, :w].cpu().numpy() for t in (s, a, hs)])
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("shape", [(3, 126), (66, 127), (130, 253), (257, 505)])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16])
def test_integer_strips_equal_generic(vsr, dtype, shape):
    """The same whole elevations as 8/16-bit (strips) and as int32 (one thread per pixel):
    exact gradients, so every output is equal bit for bit."""
    rng = np.random.default_rng(shape[0])
    d = _dem(dtype, shape, rng)
    d[rng.random(shape) < 0.01] = 9
    for nd in (9, None):
        a = vsr.raster_terrain(vsr.from_numpy(d, nodata=nd, affine=AFF))
        b = vsr.raster_terrain(vsr.from_numpy(d.astype(np.int32), nodata=nd, affine=AFF))
        for k in ("slope", "aspect", "hillshade"):
            np.testing.assert_array_equal(a[k].to_numpy(), b[k].to_numpy())
