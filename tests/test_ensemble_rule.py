"""The variant an untuned ensemble class takes (chaos_b200/csrc/cl_ensemble_rule.h), compiled for the host."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from chaos_b200 import MGS, HouseholderQR, QRSpectrum, StandardMap, StandardMapChain, _abi
from chaos_b200.ensemble import EnsembleClass, make_class_struct
from chaos_b200.propagate import FrameSpec

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148
SOURCE = r"""
#include "cl_ensemble_rule.h"
extern "C" void variant(const cl_ensemble_class* c, int sms, int beside, int* out) {
    const cl::ETune t = cl::asked_variant(*c, cl::untuned_variant(*c, sms, beside != 0));
    out[0] = t.lanes; out[1] = t.minb; out[2] = t.unroll;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(SOURCE)
    gxx = shutil.which("g++")
    r = subprocess.run([gxx, "-std=c++17", "-O1", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "chaos_b200", "csrc"),
                        "-o", str(d / "rule.so"), str(d / "rule.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(str(d / "rule.so"))

    def variant(d, n, precision, beside, alg=HouseholderQR, **asked):
        sysm = StandardMap(1.0) if d == 2 else StandardMapChain(d // 2, 1.0, 0.05)
        tau, k = {2: 5, 4: 10, 8: 10, 16: 20}[d], min(d, 8)
        c = EnsembleClass(sysm, np.zeros((1, d)), FrameSpec(k, (QRSpectrum(alg()),), np.zeros((1, d, k))), tau,
                          100 * tau, precision=precision, **asked)
        keep: list = []
        cs = make_class_struct(c, keep)
        cs.n_orbits = n
        out = (C.c_int * 3)()
        L.variant(C.byref(cs), SMS, int(beside), out)
        return tuple(out)

    return variant


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2500, 18944, 18945, 100000])
@pytest.mark.parametrize("d", [2, 4, 8, 16])
def test_one_thread_kernel_has_its_own_settings(rule, d, n, precision, beside):
    lanes, minb, unroll = rule(d, n, precision, beside, lanes=1)
    assert (lanes, unroll) == (1, 1) and minb == (1 if d >= 8 and n <= (18944 if d == 16 or precision == "mixed" else 37888) else 2)
    assert rule(d, n, precision, beside, lanes=1, minb=4, unroll=10 if d in (4, 8) else 1)[1] == 4
    if d < 8:
        assert rule(d, n, precision, beside) == (1, 2, 1)
    assert rule(d, n, precision, beside, alg=MGS) == (1, 2, 1)


@pytest.mark.parametrize("d,precision,unroll", [(16, "mixed", 20), (16, "fp64", 1), (8, "fp64", 1)])
def test_blocks_an_sm(rule, d, precision, unroll):
    lanes, threads = d // 2, 128 * SMS
    for rounds, alone, beside in ((1, 1, 1), (5, 1, 1), (5.01, 2, 1), (8, 2, 1), (8.01, 2, 2)):
        n = int(np.ceil(rounds * threads / lanes)) if rounds % 1 else int(rounds) * threads // lanes
        assert rule(d, n, precision, False) == (lanes, alone, unroll), rounds
        assert rule(d, n, precision, True) == (lanes, beside, unroll), rounds
        assert rule(d, n, precision, False, minb=4) == (lanes, 4, unroll)


def test_mixed_lattice_of_four_sites(rule):
    assert rule(8, 18944, "mixed", True) == (4, 1, 10)
    assert rule(8, 18945, "mixed", True) == (1, 2, 1)
    assert rule(8, 18945, "mixed", True, lanes=4) == (4, 2, 1)
