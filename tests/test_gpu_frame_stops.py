"""Two frames on one orbit that stop at different handoffs.

The origin of FroeschleMap(-1/2, -1/2, 0) is a fixed point whose tangent doubles (1, 1) and halves (2, -1) of each
degree of freedom, both without rounding. Over tau = 1023 steps a unit column along (2, -1) shrinks below the smallest
normal number, where GALI stops, while no entry of the orthonormal frame overflows; started 2^1000 long, it passes the
first handoff and stops the indicator frame at the second. The record then keeps the first handoff's values, whatever the
other frame does afterwards. Compared bit for bit (tolerance: none)."""
from __future__ import annotations

import numpy as np
import pytest

from chaos_b200 import GALI, SALI, FroeschleMap, HouseholderQR, QRSpectrum, propagate_frames
from chaos_b200.propagate import FrameSpec
from helpers import haar_frames, same_bits, states_equal

pytestmark = pytest.mark.gpu

N, TAU = 33, 1023


def _frames():
    W = np.zeros((N, 4, 4))
    W[:, [0, 2], 0] = W[:, [1, 3], 1] = 1.0
    W[:, [1, 3], 2] = W[:, [0, 2], 3] = np.array([2.0, -1.0]) * 2.0 ** 1000
    return [FrameSpec(4, (QRSpectrum(HouseholderQR()),), haar_frames(N, 4, 4, 3)), FrameSpec(4, (GALI(), SALI()), W)]


@pytest.mark.parametrize("windows,launch", [(1, None), (2, None), (3, None), (5, None), (5, 2 * TAU), (5, 3 * TAU)])
def test_indicator_frame_stops_first(oracle, windows, launch):
    sysm, x0, frames = FroeschleMap(-0.5, -0.5, 0.0), np.zeros((N, 4)), _frames()
    dev = propagate_frames(sysm, x0, windows * TAU, frames, tau=TAU, launch_steps=launch, finals=False, throw=False)
    ref = oracle.oracle_frames(sysm, x0, windows * TAU, frames, tau=TAU, math="portable")
    first = oracle.oracle_frames(sysm, x0, TAU, frames, tau=TAU, math="portable")[1]["states"]
    for d, r in zip(dev, ref):
        assert np.array_equal(d.code, r["code"]) and np.array_equal(d.hstep, r["hstep"])
        assert same_bits(d.x, r["x"]) and same_bits(d.W, r["W"])
    assert states_equal(dev[0].states, ref[0]["states"])
    assert states_equal(dev[1].states[["r0"]], ref[1]["states"][["r0"]])
    # the fused (GALI, SALI) record stops with the frame, so SALI's is the first handoff's
    assert states_equal(dev[1].states[["r1"]], first[["r1"]])
    if windows > 1:
        assert np.all(dev[1].code == 3) and np.all(dev[1].hstep == 2 * TAU)
        assert np.count_nonzero(dev[0].hstep > 2 * TAU) > N // 2 or windows == 2
        assert np.all(dev[1].states["r0"]["gali"][:, 0] == 1.0)
