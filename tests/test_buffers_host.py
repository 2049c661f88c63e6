"""Host state behind device-resident rasters (no GPU: CPU tensors stand in for device ones)."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from vsr_gb300 import buffers

PKG = Path(__file__).resolve().parents[1] / "vibespatial-raster_gb300"

# every trial starts from a freshly executed module, as a process's first use does
FIRST_USE = """
import importlib, sys, threading
import torch
import vsr_gb300.buffers as buffers
sys.setswitchinterval(1e-6)
t, errors = torch.zeros((2, 3)), []
for _ in range(150):
    buffers = importlib.reload(buffers)
    buffers.as_device_tensor = lambda x: x
    gate = threading.Barrier(6)
    def first(b=buffers, gate=gate):
        gate.wait()
        try:
            assert b.from_device(t).dtype == b.np.float32 and b.torch_dtype("int16") is torch.int16
        except Exception as e:
            errors.append(repr(e))
    threads = [threading.Thread(target=first) for _ in range(6)]
    [x.start() for x in threads]
    [x.join() for x in threads]
print(len(errors), errors[:3])
"""


def test_first_use_from_several_threads():
    out = subprocess.run([sys.executable, "-c", FIRST_USE], cwd=PKG, capture_output=True, text=True, check=True).stdout
    assert out.startswith("0 "), out


def test_unfetched_pixels_cannot_be_written(monkeypatch):
    """``data`` of a raster on the device is a placeholder that all such rasters share."""
    import torch

    monkeypatch.setattr(buffers, "as_device_tensor", lambda t: t)
    a, b = (buffers.from_device(torch.zeros(shape)) for shape in ((4, 5), (2, 4, 5)))
    assert a.data.shape == (4, 5) and b.data.dtype == np.float32 and b.data.nbytes == 160
    with pytest.raises(ValueError):
        a.data[1, 2] = 7.0
    assert not b.data.any()
    got = a.to_numpy()  # fetched: the raster's own buffer
    got[1, 2] = 7.0
    assert a.data[1, 2] == 7.0 and not b.to_numpy().any()


def test_events_built_without_init_are_whole():
    kind, where = buffers.RasterDiagnosticKind.RUNTIME, buffers.Residency.DEVICE
    for given in ({}, {"visible_to_user": True, "elapsed_seconds": 0.5}):
        made, ref = (f(kind=kind, detail="d", residency=where, **given)
                     for f in (buffers.diagnostic_event, buffers.RasterDiagnosticEvent))
        assert made == ref and vars(made) == vars(ref)
