"""An allocation that fails leaves nothing behind: the run that follows it, and the chunks of a run that met it, are the
ordinary ones bit for bit. The failure is a request of 1 TiB, which no device has: the library returns its error before
it reads a buffer or launches anything."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

from chaos_b200 import MGS, QRSpectrum, StandardMap, _abi
from chaos_b200._lib import lib
from helpers import identity_frames, same_bits, states_equal, uniform_starts

P = importlib.import_module("chaos_b200.propagate")   # the package exports a function of that name
pytestmark = pytest.mark.gpu

N = 40
TOO_MANY = 1 << 36   # orbits of two doubles each


class _FirstCallFails:
    def __init__(self):
        self.asked = []

    def __getattr__(self, name):
        return getattr(lib(), name)

    def cl_b200_propagate(self, run, n, bufs, prov):
        self.asked.append(n)
        return lib().cl_b200_propagate(run, TOO_MANY if len(self.asked) == 1 else n, bufs, prov)


def _run():
    return P.propagate(StandardMap(6.0), uniform_starts(N, 2, 1), 50, k=2, W0=identity_frames(N, 2, 2),
                       reducers=(QRSpectrum(MGS()),), finals=False)


@pytest.mark.parametrize("room,calls", [(12, [N, 12, 12, 12, 4]), (100, [N])])
def test_run_goes_on_after_a_failed_allocation(monkeypatch, room, calls):
    want = _run()
    per = P.bytes_per_orbit(2, 2) + _abi.state_bytes(_abi.RED_QR, 2)
    L = _FirstCallFails()
    with monkeypatch.context() as m:
        m.setattr(P, "lib", lambda: L)
        m.setattr(P, "probe", lambda: dict(free_bytes=2 * room * per))
        if room < N:
            got = _run()
        else:   # memory enough for the run as it is: the failure is the caller's
            with pytest.raises(P.DeviceError):
                _run()
    assert L.asked == calls
    if room >= N:
        got = _run()   # the next call on this thread
    assert same_bits(got.x, want.x) and same_bits(got.W, want.W) and states_equal(got.states, want.states)
    assert np.array_equal(got.code, want.code) and not want.code.any()
