"""A run that was not sized by the free memory beforehand is chunked by it once its allocation fails."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

from chaos_b200 import MGS, QRSpectrum, StandardMap, _abi
from chaos_b200.foundation import DeviceError

P = importlib.import_module("chaos_b200.propagate")   # the package exports a function of that name


class _Library:
    """The calls propagate_frames makes, with room for `room` orbits at a time."""

    def __init__(self, room):
        self.room, self.asked = room, []

    def cl_b200_check(self, run):
        return 0

    def cl_b200_propagate(self, run, n, bufs, prov):
        self.asked.append(n)
        return 0 if n <= self.room else _abi.ENOMEM


@pytest.mark.parametrize("room,free_orbits,calls", [(40, 40, [40]), (12, 12, [40, 12, 12, 12, 4]), (0, 100, [40])])
def test_chunks_after_a_failed_allocation(monkeypatch, room, free_orbits, calls):
    L = _Library(room)
    per = P.bytes_per_orbit(2, 2) + _abi.state_bytes(_abi.RED_QR, 2)
    monkeypatch.setattr(P, "lib", lambda: L)
    monkeypatch.setattr(P, "last_error", lambda: "out of memory")
    monkeypatch.setattr(P, "probe", lambda: dict(free_bytes=2 * free_orbits * per))
    monkeypatch.setattr(P.launch_plan, "device_record", lambda precision: (1.0, 1 << 20))
    run = lambda: P.propagate(StandardMap(1.0), np.zeros((40, 2)), 10, k=2, reducers=(QRSpectrum(MGS()),), finals=False)  # noqa: E731
    if room == 0:
        with pytest.raises(DeviceError):
            run()
    else:
        run()
    assert L.asked == calls
