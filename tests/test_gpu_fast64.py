"""The straight-line Float64 operations of the handoffs (chaos_b200/csrc/cl_fast64.cuh) and the steps built on them.

The operations must give the IEEE quotient, root and the portable logarithm bit for bit (tolerance: none), on random
operands and on the operands whose exact result lies nearest a rounding tie, where a wrong last bit would show. The
steps must leave their range for the general code whenever an entry, norm or pivot is outside it: frames scaled to the
ends of the Float64 range, tiny and zero entries, and orbits that fail after successful handoffs (whose records keep the
values of the last successful one) are compared with the oracle bit for bit.
"""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from chaos_b200 import (CGS, FLI, GALI, MEGNO, MGS, SALI, Benettin, FroeschleMap, GivensQR, HenonHeilesFlow,
                        HouseholderQR, IntegratorMap, KahanLi, QRSpectrum, StandardMap)
from chaos_b200 import propagate_frames
from chaos_b200.propagate import FrameSpec
from helpers import haar_frames, same_bits, states_equal, uniform_starts
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "chaoslab_b200.h"
#include "cl_fast64.cuh"
#include "cl_split_frames.cuh"
using namespace cl;
typedef unsigned long long u64;
__device__ u64 bad[11];
__device__ u64 rnd(u64& s) { s += 0x9e3779b97f4a7c15ULL; return mix64(s); }
__device__ double mk(u64 r, int e) { return __longlong_as_double((long long)((r & 0xfffffffffffffULL) | ((u64)(1023 + e) << 52))); }
__device__ bool ne(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }
__device__ u64 inv64(u64 b) { u64 x = b; for (int i = 0; i < 6; ++i) x *= 2 - b * x; return x; }
__global__ void operands(u64 seed, int iters) {
    u64 s = mix64(seed * 1000003 + blockIdx.x * (u64)blockDim.x + threadIdx.x);
    for (int it = 0; it < iters; ++it) {
        u64 r1 = rnd(s), r2 = rnd(s), r3 = rnd(s);
        const int kind = r3 & 63;   // significands at the ends of a binade, all ones among them
        if (kind == 1) r1 |= 0xfffffffff0000ULL;
        if (kind == 2) r1 &= 0xff;
        if (kind == 3) r1 = ~0ULL;
        if (kind == 4) r2 &= 0xfff;
        const int e1 = (int)((r3 >> 8) % 1400) - 700, e2 = (int)((r3 >> 24) % 200) - 100;
        const double b = mk(r1, e1), c = mk(r1, (int)(r3 % 3) - 1);
        double a = mk(r2, e1 / 2 + e2);
        if (r3 >> 63) a = -a;
        if (kind == 5) a = r3 >> 63 ? -0.0 : 0.0;
        const double y = rcp64(b), ref = a / b;
        if (ne(y, 1.0 / b)) atomicAdd(&bad[0], 1);
        if ((a == 0.0 || (fabs(ref) > 1e-290 && fabs(ref) < 1e290)) && ne(quo64(a, b, y), ref)) atomicAdd(&bad[1], 1);
        if (ne(root64(b), sqrt(b))) atomicAdd(&bad[2], 1);
        if (ne(log64(b), cl_log(b)) || ne(log64(c), cl_log(c))) atomicAdd(&bad[3], 1);
        // a norm with its reciprocal, of two and of four entries
        Ok okn;
        const double v[4] = {b, mk(r2, e1 + (int)((r3 >> 33) % 5) - 2), mk(r1 ^ r2, e1 - (int)((r3 >> 36) % 60)), mk(r2 >> 3, e1)};
        double y2, y4;
        const double n2 = norm64r<2>(v, okn, y2), n4 = norm64r<4>(v, okn, y4);
        if (e1 > -600 && e1 < 600 && (!okn.ok || ne(n2, safe_norm<2>(v)) || ne(n4, safe_norm<4>(v)) || ne(y2, 1.0 / n2) || ne(y4, 1.0 / n4))) atomicAdd(&bad[8], 1);
        // quotients nearest a tie: A 2^t - B m = k with m odd, k small
        u64 B = (r1 & 0xfffffffffffffULL) | (1ULL << 52) | 1;
        if (r3 & 1) B |= 0xff00000000000ULL;
        const long long k = (long long)((r3 >> 40) % 9) * 2 - 7;
        const int t = (r3 >> 50) & 1 ? 53 : 54;
        const u64 mask = (1ULL << t) - 1;
        u64 m = ((u64)(-k) * inv64(B)) & mask;
        if (t == 53) m |= 1ULL << 53;
        const unsigned __int128 P = (unsigned __int128)B * m + (unsigned __int128)(__int128)k;
        const u64 A = (u64)(P >> t);
        if (m >> 53 == 1 && (m & 1) && ((u64)P & mask) == 0 && A >> 52 == 1) {
            atomicAdd(&bad[6], 1);
            if (ne(quo64((double)A, (double)B, rcp64((double)B)), (double)A / (double)B)) atomicAdd(&bad[4], 1);
        }
    }
}
// roots nearest a tie: m^2 = S 2^t + k with m odd, k = 1 mod 8, by lifting the root of k modulo 2^t
__global__ void roots() {
    const long long k = ((long long)(blockIdx.x * blockDim.x + threadIdx.x) - 4096) * 8 + 1;
    for (int t = 54; t <= 55; ++t) {
        u64 r = 1;
        for (int j = 3; j < t; ++j)
            if (((r * r - (u64)k) & ((1ULL << (j + 1)) - 1)) != 0) r += 1ULL << (j - 1);
        const u64 mask = (1ULL << t) - 1;
        for (int v = 0; v < 8; ++v) {
            u64 m = (((v & 1 ? 0 - r : r) + (v & 2 ? 1ULL << (t - 1) : 0)) & mask) + (v & 4 ? 1ULL << 53 : 0);
            if (m >> 53 != 1 || !(m & 1)) continue;
            const unsigned __int128 sq = (unsigned __int128)m * m - (unsigned __int128)(__int128)k;
            const u64 S = (u64)(sq >> t);
            if (((u64)sq & mask) != 0 || S >> 52 != 1) continue;
            for (int e = -600; e <= 600; e += 200) {
                const double s = ldexp((double)S, (t == 54 ? -52 : -51) + e);
                atomicAdd(&bad[7], 1);
                if (ne(root64(s), sqrt(s))) atomicAdd(&bad[5], 1);
            }
        }
    }
}
// the Float32 reciprocal and root of the split kernel, every significand, at the ends and the middle of their range
__global__ void all32() {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = -100; e <= 100; e += 50)
        for (int odd = 0; odd < 2; ++odd) {
            const float v = __uint_as_float(m | static_cast<unsigned>(127 + e + odd) << 23);
            if (__float_as_uint(split::rcp32(v)) != __float_as_uint(1.0f / v)) atomicAdd(&bad[9], 1);
            if (__float_as_uint(split::root32(v)) != __float_as_uint(sqrtf(v))) atomicAdd(&bad[10], 1);
        }
}
extern "C" int run(unsigned long long* out) {
    operands<<<148 * 8, 256>>>(1, 400);
    roots<<<32, 256>>>();
    all32<<<(1 << 23) / 256, 256>>>();
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    return cudaMemcpyFromSymbol(out, bad, sizeof bad) == cudaSuccess ? 0 : 2;
}
"""


def test_operations_are_the_ieee_ones(tmp_path):
    src, so = tmp_path / "ops.cu", tmp_path / "ops.so"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                        "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                        "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "chaos_b200", "csrc"),
                        "-o", str(so), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = (C.c_uint64 * 11)()
    assert C.CDLL(str(so)).run(out) == 0
    reciprocal, quotient, root, log, hard_quotient, hard_root, n_quotient, n_root, norm, rcp32, root32 = list(out)
    assert n_quotient > 1_000_000 and n_root > 10_000
    assert (reciprocal, quotient, root, log, norm, hard_quotient, hard_root, rcp32, root32) == (0,) * 9


CHAINS = [(2, (QRSpectrum(MGS()),)), (2, (QRSpectrum(CGS()),)), (2, (QRSpectrum(HouseholderQR()),)),
          (2, (QRSpectrum(GivensQR()),)), (1, (Benettin(),)), (2, (SALI(),)),
          (2, (MEGNO(replace=False), FLI(replace=False), SALI())), (2, (MEGNO(),)), (2, (FLI(),)),
          (4, (QRSpectrum(HouseholderQR()),)), (4, (GALI(), SALI()))]


@pytest.mark.parametrize("scale", [1e-315, 1e-250, 1e-150, 1e-20, 1.0, 1e150, 1e250, 1e300], ids=repr)
@pytest.mark.parametrize("k,chain", CHAINS, ids=repr)
def test_frames_at_the_ends_of_the_range(oracle, k, chain, scale):
    n, d = 96, 4 if k == 4 else 2
    sysm = FroeschleMap(1.5, 1.5, 0.05) if d == 4 else StandardMap(6.0)
    W0 = haar_frames(n, d, k, 5) * scale
    W0[1::4, 0, 0] = 0.0            # exact zeros, of both signs, and entries far below their column's norm
    W0[2::4, 1, 0] = -0.0
    W0[3::4, d - 1, k - 1] *= 1e-290
    x0, frame = uniform_starts(n, d, 6), FrameSpec(k, chain, W0)
    if len(chain) == 2 and scale < 2.3e-308:
        # GALI rejects a subnormal norm that SALI would accept, and the fused (GALI, SALI) record stops with the frame,
        # where two separate reducers would run SALI once more: the GALI record and the stop are the oracle's
        dev = propagate_frames(sysm, x0, 60, [frame], tau=3, seed=7, finals=False, throw=False)[0]
        ref = oracle.oracle_frames(sysm, x0, 60, [frame], tau=3, seed=7, math="portable")[0]
        assert np.all(dev.code == 3) and np.array_equal(dev.code, ref["code"]) and same_bits(dev.W, ref["W"])
        assert states_equal(dev.states[["r0"]], ref["states"][["r0"]])
        return
    _compare(sysm, x0, 60, [frame], 3, oracle)


def test_uncoupled_frames_keep_their_zeros(oracle):
    """mu = 0 decouples the two maps: half of a frame's entries are zeros of either sign in every window."""
    n = 64
    W0 = np.broadcast_to(np.eye(4), (n, 4, 4)).copy()
    W0[::2, 2, 2] = -1.0
    frames = [FrameSpec(4, (QRSpectrum(HouseholderQR()),), W0), FrameSpec(4, (GALI(), SALI()), W0)]
    _compare(FroeschleMap(1.5, 0.7, 0.0), uniform_starts(n, 4, 8), 200, frames, 10, oracle)


@pytest.mark.parametrize("k,chain", [(2, (SALI(),)), (2, (GALI(),)), (4, (GALI(),)),
                                     (2, (MEGNO(replace=False), FLI(replace=False), QRSpectrum(GivensQR())))], ids=repr)
def test_orbits_that_fail_after_good_handoffs(oracle, k, chain):
    """Starts above the escape energy leave the well and overflow after some windows; the record keeps the values of
    the last handoff that succeeded. Relaunched windows carry them."""
    n = 200
    x0 = uniform_starts(n, 4, 9, lo=-0.9, hi=0.9)
    sysm = IntegratorMap(KahanLi(8), HenonHeilesFlow(), 0.05)
    fr = [FrameSpec(k, chain, haar_frames(n, 4, k, 10))]
    for launch in (None, 20):
        dev, _ = _compare(sysm, x0, 400, fr, 5, oracle, launch_steps=launch)
        assert 0 < np.count_nonzero(dev[0].code) < n
        assert np.any((dev[0].code != 0) & (dev[0].hstep > 10))


@pytest.mark.parametrize("chain", [(QRSpectrum(MGS()),), (QRSpectrum(GivensQR()),), (SALI(),), (MEGNO(),),
                                   (MEGNO(replace=False), FLI(replace=False), SALI())], ids=repr)
@pytest.mark.parametrize("n,N,tau", [(1, 1, 1), (31, 7, 1), (33, 12, 3), (65, 20, 4), (40, 9, 3), (9473, 10, 2)])
def test_pipelined_small_ensembles(oracle, n, N, tau, chain):
    """The pipeline of warps at the edges of its blocks (one step, part of a block, windows that do not fill one, spare
    lanes), one orbit past its range, and with orbits that stop on the way: huge starts overflow, a frame of zeros and a
    non-finite one fail at the first handoff, and a kicked map of 1e300 overflows later. Relaunched windows too."""
    W0 = haar_frames(n, 2, 2, 14)
    x0 = uniform_starts(n, 2, 15)
    if n >= 31:
        W0[3] = 0.0
        W0[5, 1, 1] = np.inf
        W0[7] *= 1e250
        x0[9, 0] = np.nan
    for K in (6.0, 1e300):
        for launch in (None, tau):
            _compare(StandardMap(K), x0, N, [FrameSpec(2, chain, W0)], tau, oracle, launch_steps=launch)
