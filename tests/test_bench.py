"""The benchmark's host-side parts."""
import json
import os
import sys

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if REPO not in sys.path:
    sys.path.insert(0, REPO)

import bench  # noqa: E402


def test_a_missing_reference_library_does_not_cost_the_line(monkeypatch):
    """The reference's sources may not be at hand: the line then says why its CPU baseline
    is missing.  Any other failure of that baseline is still an error."""
    def missing(*args, **kwargs):
        raise OSError("libhsi_ref.so: cannot open shared object file")

    monkeypatch.setattr(bench, "cpu_reference", missing)
    cpu = bench.cpu_baseline("sam_cem")
    assert list(cpu) == ["unavailable"] and "libhsi_ref.so" in cpu["unavailable"]
    json.dumps(cpu)

    def broken(*args, **kwargs):
        raise ValueError("shape")

    monkeypatch.setattr(bench, "cpu_reference", broken)
    with pytest.raises(ValueError):
        bench.cpu_baseline("sam_cem")
    monkeypatch.setattr(bench, "cpu_reference", lambda *a, **k: (np.array([0.5, 1.5]), 4, 250000))
    cpu = bench.cpu_baseline("rx_ace", " (all of it)")
    assert cpu["value"] == 1.0 and cpu["cores"] == 4 and "(all of it)" in cpu["sample"]
