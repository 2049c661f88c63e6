"""Host check of csrc/std_round64.h: sqrt(N) / n as a float64 with integer arithmetic, against a
__float128 reference over random and edge values; the bound is 0.52 ulp (0.5 for the final rounding,
2^-58 before it; perfect squares exact), whatever the last bits of the reciprocal root estimate."""

import platform
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "vibespatial-raster_gb300" / "csrc"

pytestmark = pytest.mark.skipif(shutil.which("gcc") is None or platform.machine() != "x86_64",
                                reason="gcc with __float128 not available")


def test_std_f64_within_half_an_ulp(tmp_path):
    exe = tmp_path / "check"
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-I", str(CSRC), "-o", str(exe),
                    str(Path(__file__).with_name("std_round64_check.c")), "-lm"], check=True)
    n, worst, bad = map(int, subprocess.run([str(exe), "2000000"], capture_output=True, text=True, check=True).stdout.split())
    assert n > 1900000 and bad == 0
    assert worst <= 520  # thousandths of an ulp
