"""csrc/div_round.h: a quotient from an estimated reciprocal, a Newton step and one residual correction
is within 0.5 + 2^-21 ulp of n / w (2.5 ulp times the correction's relative error, 1.5 2^-23, beyond the
last rounding).

Host: every quotient near a halfway case (only there can it differ from the rounded one) and random
ones.  GPU: the convolution with one-tap kernels, whose numerator w v and weight sum w are known
exactly, over the divisors for which an estimate one ulp off leaves the reciprocal off as well."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "vibespatial-raster_gb300" / "csrc"


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
def test_quotients_near_halfway_cases(tmp_path):
    exe = tmp_path / "check"
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-ffp-contract=off", "-I", str(CSRC), "-o", str(exe),
                    str(Path(__file__).with_name("div_round_check.c")), "-lm"], check=True)
    n, differ, wrong, beyond = map(int, subprocess.run([str(exe)], capture_output=True, text=True,
                                                       check=True).stdout.split())
    assert n > 60_000_000
    assert wrong == 0  # a rounded reciprocal gives the rounded quotient
    assert differ < 100 and beyond <= 8  # 2^-21 ulp


def _hard_divisors():
    """Mantissas in [1, 2) whose reciprocal, one ulp up, does not come back in one Newton step."""
    w = (np.arange(1 << 23, dtype=np.uint32) | 0x3F800000).view(np.float32)
    t = (1.0 / w.astype(np.float64)).astype(np.float32)
    bad = np.zeros(w.shape, bool)
    for r0 in (np.nextafter(t, np.float32(4)), np.nextafter(t, np.float32(0))):
        wd, rd = w.astype(np.longdouble), r0.astype(np.longdouble)
        e = (1 - wd * rd).astype(np.float32).astype(np.longdouble)
        bad |= (e * rd + rd).astype(np.float32) != t
    return w[bad]


@pytest.mark.gpu
@pytest.mark.parametrize("holes", [False, True])
def test_one_tap_kernels(vsr, holes):
    rng = np.random.default_rng(3)
    divisors = _hard_divisors()
    assert 20 < len(divisors) < 200
    for w in divisors:
        d = (rng.integers(1 << 23, 1 << 24, (64, 257)) / w).astype(np.float32)
        if holes:
            d[rng.random(d.shape) < 0.05] = -1.0
        k = np.zeros((3, 3))
        k[1, 1] = w
        out = vsr.raster_convolve(vsr.from_numpy(d, nodata=-1.0), k, out_dtype=np.float32).to_numpy()
        hole = d == -1.0
        assert (out[hole] == -1.0).all()
        exact = (d * w).astype(np.float32)[~hole].astype(np.float64) / float(w)
        ulp = np.ldexp(1.0, np.frexp(exact)[1] - 24)
        assert (np.abs(out[~hole] - exact) <= (0.5 + 2.0**-21) * ulp).all()
