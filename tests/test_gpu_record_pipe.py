"""The recorder's pipeline of warps (at most 9472 orbits of the standard maps, tau <= 4) against its one-thread kernel
(larger ensembles), bit for bit: the same orbits once in one call of 9600 and once in smaller calls. Failing orbits
stand at block edges; grid steps fall inside, at the ends of and between the pipeline's blocks of four steps."""
from __future__ import annotations

import numpy as np
import pytest

from chaos_b200 import CGS, MGS, HouseholderQR, QRSpectrum, StandardMap, WrappedStandardMap, record, torus_state
from helpers import same_bits

pytestmark = pytest.mark.gpu

N_ALL = 9600


def _starts(name):
    z = np.random.default_rng(41).uniform(0, 2 * np.pi, (N_ALL, 2))
    if name == "wrapped":
        return WrappedStandardMap(6.0), np.array([torus_state(v) for v in z])
    z[[0, 31, 64, 9471, 9472]] = [[np.nan, 1.0], [1.0, np.inf], [1.0, 1e306], [np.nan, 1.0], [1.0, 1e306]]
    return StandardMap(2.5), z


@pytest.mark.parametrize("est", [QRSpectrum(CGS()), QRSpectrum(MGS()), QRSpectrum(HouseholderQR())], ids=repr)
@pytest.mark.parametrize("name", ["standard", "wrapped"])
@pytest.mark.parametrize("tau, N, L", [(1, 61, None), (1, 62, 31), (2, 62, None), (2, 60, 6), (3, 63, None), (4, 64, 20)])
def test_pipeline_equals_one_thread(est, name, tau, N, L):
    sys, x0 = _starts(name)
    W0 = np.broadcast_to(np.eye(2), (N_ALL, 2, 2)).copy()
    W0[70] = [[1e300, 0.0], [0.0, 1e300]]      # out of the straight-line range
    W0[71] = 0.0                               # zero columns
    grid = sorted({tau, 2 * tau, 5 * tau, 8 * tau, 9 * tau, N // tau * tau})
    whole = record(sys, x0, N, tau, est, grid, W0=W0, launch_steps=L)
    for lo, hi in ((0, 9472), (0, 33), (64, 96), (9471, 9472), (9472, N_ALL)):
        part = record(sys, x0[lo:hi], N, tau, est, grid, W0=W0[lo:hi], launch_steps=L)
        for key in ("R", "x", "W"):
            assert same_bits(np.ascontiguousarray(getattr(part, key)), np.ascontiguousarray(getattr(whole, key)[lo:hi])), key
        assert same_bits(part.states.view(np.float64), whole.states[lo:hi].view(np.float64)), "states"
        for key in ("fail", "code", "hstep"):
            assert np.array_equal(getattr(part, key), getattr(whole, key)[lo:hi]), key
