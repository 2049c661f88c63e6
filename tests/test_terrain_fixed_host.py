"""Host check of csrc/terrain_fixed.h: curvature factors and their product with integer sums against
128-bit floating point, 64-bit integers as float64 bits against the compiler's conversion.

Bound of the curvature: half an ulp for the result, half a unit of 2^-s for each factor, one unit for
the ones' complement of negative values."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "vibespatial-raster_gb300" / "csrc"


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
def test_fixed_point_curvature(tmp_path):
    exe = tmp_path / "check"
    built = subprocess.run(["gcc", "-O2", "-std=gnu11", "-I", str(CSRC), "-o", str(exe),
                            str(Path(__file__).with_name("terrain_fixed_check.c")), "-lm"], capture_output=True, text=True)
    if "_Float128" in built.stderr:
        pytest.skip("gcc without _Float128")
    assert built.returncode == 0, built.stderr
    out = subprocess.run([str(exe), "200000"], capture_output=True, text=True, check=True).stdout
    n, bad, refused, undue, scaled, wrong = map(int, out.split())
    assert n > 1_000_000 and bad == 0
    assert refused > 1000 and undue == 0  # factors more than 2^14 apart only
    assert scaled == 2_000_000 and wrong == 0
