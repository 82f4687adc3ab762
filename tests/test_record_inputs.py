"""The recorders leave the caller's start frames alone, whatever their memory order: the library writes the final frames
into the array that it is handed."""
from __future__ import annotations

import ctypes as C
import importlib

import numpy as np
import pytest

from chaos_b200 import MGS, Benettin, QRSpectrum, StandardMap

M = importlib.import_module("chaos_b200.record")


class _Library:
    """Answers the calls of the three recorders; a run overwrites its frames (`nbytes`)."""

    def __init__(self, nbytes):
        self.nbytes = nbytes

    def __getattr__(self, name):
        if name.endswith("_columns"):
            return lambda *a: 4
        if name.endswith("_state_bytes"):
            return lambda *a: 8
        return self._run

    def _run(self, run, n, *rest):
        Wc = [p for p in rest if isinstance(p, int) and p > 1 << 16][1]   # after the points
        C.memset(Wc, 0, self.nbytes)
        return 0


def _frames(n, d, k, order):
    W = np.random.default_rng(1).normal(size=(n, d, k))
    return np.ascontiguousarray(W.transpose(0, 2, 1)).transpose(0, 2, 1) if order == "columns" else W


@pytest.mark.parametrize("order", ["rows", "columns"])
@pytest.mark.parametrize("call", ["benettin", "mgs", "indicators", "pairs"])
def test_start_frames_are_not_written(monkeypatch, call, order):
    n, d = 5, 4 if call == "pairs" else 2
    W0 = _frames(n, d, 1 if call == "benettin" else 2, order)
    monkeypatch.setattr(M, "lib", lambda: _Library(W0.nbytes))
    x0, before = np.zeros((n, d)), W0.copy()
    if call == "indicators":
        r = M.record_indicators(StandardMap(1.0), x0, 10, 1, ["SALI"], [5, 10], W0=W0)
    elif call == "pairs":
        r = M.record_indicator_pairs(StandardMap(1.0), x0, W0, 10, 1, ["RLI"], [5, 10])
    else:
        r = M.record(StandardMap(1.0), x0, 10, 1, Benettin() if call == "benettin" else QRSpectrum(MGS()), [5, 10], W0=W0)
    assert not r.W.any() and np.array_equal(W0, before)
