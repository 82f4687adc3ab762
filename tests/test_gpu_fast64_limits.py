"""The straight-line Float64 operations at the limits of the range they accept (chaos_b200/csrc/cl_fast64.cuh).

Wherever `Ok` accepts a divisor and a dividend the quotient must be the IEEE one, and the reciprocal and the root over
exponents within +-900, bit for bit (tolerance: none). Frames whose columns hold entries so far apart that a quotient is
subnormal must take the general code: the map with K = 0 leaves such a column as it is."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from chaos_b200 import CGS, FLI, GALI, MEGNO, MGS, SALI, Benettin, FroeschleMap, QRSpectrum, StandardMap, StandardMapChain
from chaos_b200.propagate import FrameSpec
from helpers import haar_frames
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "chaoslab_b200.h"
#include "cl_fast64.cuh"
using namespace cl;
typedef unsigned long long u64;
__device__ u64 out_[5];
__device__ u64 rnd(u64& s) { s += 0x9e3779b97f4a7c15ULL; return mix64(s); }
__device__ double mk(u64 r, int e) {   // exponent e, subnormal below -1022
    const double m = __longlong_as_double((long long)((r & 0xfffffffffffffULL) | (1023ULL << 52)));
    return ldexp(m, e);
}
__device__ bool ne(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }
__global__ void operands(u64 seed, int iters) {
    u64 s = mix64(seed * 1000003 + blockIdx.x * (u64)blockDim.x + threadIdx.x);
    for (int it = 0; it < iters; ++it) {
        u64 r1 = rnd(s), r2 = rnd(s), r3 = rnd(s);
        if ((r3 & 15) == 1) r1 |= 0xfffffffff0000ULL;
        if ((r3 & 15) == 2) r1 &= 0xff;
        if ((r3 & 15) == 3) r2 &= 0xfff;
        const int eb = (int)((r3 >> 8) % 1030) - 810;
        const int ea = eb + 40 - (int)((r3 >> 24) % (eb + 860));   // down to 2^-820, past both limits
        double b = mk(r1, eb), a = mk(r2, ea > 1020 ? 1020 : ea);
        if (it == 0) { b = 3 * 0x1p600; a = 9.225598902603729e-143; }
        if (r3 >> 63) a = -a;
        Ok ok;
        ok.divisor(b);
        ok.dividend(a);
        const double ref = a / b;
        if (ok.ok && fabs(ref) < 0x1p1000) {
            atomicAdd(&out_[0], 1);
            if (fabs(ref) < 0x1p-900) atomicAdd(&out_[1], 1);
            if (ne(quo64(a, b, rcp64(b)), ref)) atomicAdd(&out_[2], 1);
        }
        const double c = mk(r2, (int)((r3 >> 40) % 1800) - 900);
        if (ne(rcp64(c), 1.0 / c)) atomicAdd(&out_[3], 1);
        if (ne(root64(c), sqrt(c))) atomicAdd(&out_[4], 1);
    }
}
extern "C" int run(unsigned long long* out) {
    operands<<<148 * 8, 256>>>(3, 400);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    return cudaMemcpyFromSymbol(out, out_, sizeof out_) == cudaSuccess ? 0 : 2;
}
"""


def test_accepted_operands_give_the_ieee_results(tmp_path):
    src, so = tmp_path / "limits.cu", tmp_path / "limits.so"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                        "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                        "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "chaos_b200", "csrc"),
                        "-o", str(so), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = (C.c_uint64 * 5)()
    assert C.CDLL(str(so)).run(out) == 0
    accepted, low, quotient, reciprocal, root = list(out)
    # of 121e6 draws; quotients below 2^-900 come from divisors above 2^100 alone: (110 / 1030) (55 / 1000) of them, 7e5
    assert accepted > 50_000_000 and low > 500_000
    assert (quotient, reciprocal, root) == (0, 0, 0)


CASES = [(2, 2, (SALI(),)), (2, 2, (MEGNO(),)), (2, 2, (FLI(),)), (2, 1, (Benettin(),)),
         (2, 2, (MEGNO(replace=False), FLI(replace=False), SALI())), (2, 2, (QRSpectrum(MGS()),)),
         (2, 2, (QRSpectrum(CGS()),)), (4, 4, (GALI(), SALI())), (4, 2, (SALI(),)), (16, 8, (GALI(),)),
         (8, 8, (QRSpectrum(MGS()),))]


@pytest.mark.parametrize("tau", [1, 5])
@pytest.mark.parametrize("d,k,chain", CASES, ids=repr)
def test_entries_far_apart_in_one_column(oracle, d, k, chain, tau):
    """Column 0 holds b at a position and a at a momentum, which K = 0 keeps. With b = 3 2^600 and a = 9.2e-143 their
    quotient is a subnormal next to a tie; the other two lie on either side of the accepted range's end."""
    n, half = 33, d // 2
    W0 = haar_frames(n, d, k, 4)
    W0[:, :, 0] = 0.0
    W0[:, 0, 0] = 3 * 2.0 ** 600
    W0[:, half, 0] = 9.225598902603729e-143
    W0[1::3, 0, 0], W0[1::3, half, 0] = 1.9 * 2.0 ** 209, 1.3 * 2.0 ** -800
    W0[2::3, 0, 0], W0[2::3, half, 0] = 1.9 * 2.0 ** 210, 1.3 * 2.0 ** -801
    W0[::2, half, 0] *= -1.0
    sysm = StandardMap(0.0) if d == 2 else FroeschleMap(0.0, 0.0, 0.0) if d == 4 else StandardMapChain(half, 0.0, 0.0)
    x0 = np.random.default_rng(8).uniform(0, 6, (n, d))
    _compare(sysm, x0, 2 * tau, [FrameSpec(k, chain, W0)], tau, oracle)
