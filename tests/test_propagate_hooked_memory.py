"""A run with the launch hook set is chunked by the free memory, whatever its size."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

from chaos_b200 import MGS, QRSpectrum, StandardMap, _abi

P = importlib.import_module("chaos_b200.propagate")   # the package exports a function of that name


class _Library:
    def cl_b200_check(self, run):
        return 0


@pytest.mark.parametrize("free_orbits,chunks", [(12, [12, 12, 12, 4]), (40, [40])])
def test_hooked_run_asks_for_the_free_memory(monkeypatch, free_orbits, chunks):
    per = P.bytes_per_orbit(2, 2) + _abi.state_bytes(_abi.RED_QR, 2)
    sizes = []

    def hooked(L, run, n, *rest):
        sizes.append(n)
        return 0.0, 1

    monkeypatch.setattr(P, "lib", lambda: _Library())
    monkeypatch.setattr(P, "probe", lambda: dict(free_bytes=2 * free_orbits * per))
    monkeypatch.setattr(P, "_hooked_chunk", hooked)
    monkeypatch.setattr(P.launch_plan, "device_record", lambda precision: (1.0, 1 << 20))
    monkeypatch.setattr(P.launch_plan, "BEFORE_LAUNCH", lambda *a: None)
    P.propagate(StandardMap(1.0), np.zeros((40, 2)), 10, k=2, reducers=(QRSpectrum(MGS()),), finals=False)
    assert sizes == chunks
