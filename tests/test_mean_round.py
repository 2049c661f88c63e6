"""csrc/mean_round.h: the focal mean's float64 quotient of a sum of 8/16-bit values by its count is the
division's.  Host: every count up to 81 and every sum.  GPU: window means against numpy's division,
radius 1 to 4, strips of 32 to 256 rows (as tall as leaves the GPU enough of them)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest
from numpy.lib.stride_tricks import sliding_window_view

CSRC = Path(__file__).resolve().parents[1] / "vibespatial-raster_gb300" / "csrc"


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
def test_every_quotient(tmp_path):
    exe = tmp_path / "check"
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-ffp-contract=off", "-I", str(CSRC), "-o", str(exe),
                    str(Path(__file__).with_name("mean_round_check.c")), "-lm"], check=True)
    n, bad = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert n > 300_000_000 and bad == 0


def _means(d, r, nd, y0, y1):
    a, b = max(0, y0 - r), min(d.shape[0], y1 + r)
    pad = ((r - (y0 - a), r - (b - y1)), (r, r))
    valid = np.ones(d[a:b].shape, bool) if nd is None else d[a:b] != nd
    s = sliding_window_view(np.pad(np.where(valid, d[a:b], 0).astype(np.int64), pad), (2 * r + 1, 2 * r + 1)).sum((-2, -1))
    n = sliding_window_view(np.pad(valid, pad), (2 * r + 1, 2 * r + 1)).sum((-2, -1))
    out = s / np.maximum(n, 1)
    if nd is not None:
        out[d[y0:y1] == nd] = nd
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint16])
@pytest.mark.parametrize("r,shape", [(1, (5, 8)), (2, (33, 484)), (3, (300, 120)), (4, (150, 124)), (3, (20_001, 16)),
                                     (1, (170_002, 16)), (4, (340_003, 16)), (3, (640_004, 16))])
def test_window_means(vsr, dtype, r, shape):
    rng = np.random.default_rng(r)
    info = np.iinfo(dtype)
    d = rng.integers(info.min, info.max, shape, endpoint=True).astype(dtype)
    d[rng.random(shape) < 0.05] = 9
    for nd in (9, None):
        out = vsr.raster_focal_mean(vsr.from_numpy(d, nodata=nd), r).to_numpy()
        o32 = vsr.raster_focal_mean(vsr.from_numpy(d, nodata=nd), r, out_dtype=np.float32).to_numpy()
        h = shape[0]
        for y0 in (0, h // 3, max(0, h - 600)):
            y1 = min(h, y0 + 600)
            ref = _means(d, r, nd, y0, y1)
            np.testing.assert_array_equal(out[y0:y1], ref)
            np.testing.assert_array_equal(o32[y0:y1], ref.astype(np.float32))
