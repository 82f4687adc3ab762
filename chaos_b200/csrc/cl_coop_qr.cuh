// cl_coop_qr.cuh -- QRSpectrum's factorisation and checks over a group of G lanes, shared by the cooperative kernels
// (cl_coop.cuh, cl_coop_orbit.cuh). The frame is staged column-major in shared memory; lane j owns columns j, j + G, ...
//
// A handoff is bound by the latency of its dependent chains, one warp holding 32 / G orbits. So everything that is
// independent runs in different lanes, in straight-line code: the columns of R^{-1} (window_Gw) one per lane instead
// of all on the first, its two Frobenius sums on two lanes side by side, the maxima as trees, the norms' quotients by a
// shared reciprocal (cl_fast64.cuh). What stays serial is what the reference's rounding order makes so: the left-folded
// sums. The loops over the reflectors are not unrolled: eight copies of a reflector's code did not stay in the
// instruction cache (1.4 of 6.7 stall cycles per instruction).
// Every entry is computed by the operations of cl_qr.cuh in their order and type, so the results are bit-identical to
// the one-thread kernel's; operands outside the straight-line range take the general operations.
// d = 16, k = 8, tau = 10, Float64, 2048 orbits x 2000 steps: 14.6 -> 5.3 ms of kernel (Float32 frames 4.2 -> 2.3 ms; d = 8 9.1 -> 4.3 ms, mixed 4.0 -> 2.3 ms).
#pragma once

#include "cl_fast64.cuh"
#include "cl_kernel.cuh"

namespace cl {

template <int G>
__device__ __forceinline__ unsigned group_mask(int lane) {
    return G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
}

template <int G>
__device__ __forceinline__ bool group_all(unsigned mask, bool p) {
    return (__ballot_sync(mask, p) & mask) == mask;
}

// Norm of a D-vector and the vector over it: the straight-line forms in Float64 where they are exact
template <int D, typename Real>
__device__ __forceinline__ Real coop_norm(const Real* v) {
    if constexpr (sizeof(Real) == 8) {
        Ok ok;
        const double r = norm64<D>(v, ok);
        if (ok.ok) return r;
    }
    return nrm<D>(v);
}
template <int D, typename Real>
__device__ __forceinline__ void coop_divide(const Real* v, Real by, Real* out) {
    if constexpr (sizeof(Real) == 8) {
        Ok ok;
        ok.divisor(by);
        const double y = rcp64(by);
        double q[D];
#pragma unroll
        for (int l = 0; l < D; ++l) { ok.dividend(v[l]); q[l] = quo64(v[l], by, y); }
        if (ok.ok) {
#pragma unroll
            for (int l = 0; l < D; ++l) out[l] = q[l];
            return;
        }
    }
#pragma unroll
    for (int l = 0; l < D; ++l) out[l] = dv(v[l], by);
}
template <typename Real>
__device__ __forceinline__ double coop_log(Real a) {
    if constexpr (sizeof(Real) == 8) {
        Ok ok;
        ok.positive<800>(a);
        if (ok.ok) return log64(a);
    }
    return lnr(a);
}

// _reflector (householder.jl:19-28) of rows jj.. of a column, written to u (zeros above); rho the column's new
// diagonal entry. False (u zero) when the norm is zero or not finite.
template <int D, typename Real>
__device__ __forceinline__ bool coop_reflector(const Real* col, int jj, Real* u, Real& rho) {
    Real a[D], ajj = Real(0);
#pragma unroll
    for (int r = 0; r < D; ++r) {
        a[r] = r >= jj ? col[r] : Real(0);
        ajj = r == jj ? col[r] : ajj;
    }
    const Real cn = coop_norm<D>(a);
    if (!(isfin(cn) && cn > Real(0))) {
#pragma unroll
        for (int r = 0; r < D; ++r) u[r] = Real(0);
        rho = cn;
        return false;
    }
    const bool neg = ajj < Real(0);
    ajj = ajj + (neg ? -cn : cn);
#pragma unroll
    for (int r = 0; r < D; ++r) a[r] = r == jj ? ajj : a[r];
    coop_divide<D>(a, coop_norm<D>(a), a);
#pragma unroll
    for (int r = 0; r < D; ++r) u[r] = a[r];
    rho = neg ? cn : -cn;
    return true;
}

struct CoopFactor { int count, status, column; };

// HouseholderQR (householder.jl:19-80) of the columns in A (column j + m G in A[m]): R's upper triangle with its
// positive diagonal in sR (K x K, zeros below), Q's columns in sQ and in A, the reflectors in sU (D x NREF).
template <int D, int K, int G, typename Real>
__device__ __forceinline__ CoopFactor coop_householder(Real (&A)[(K + G - 1) / G][D], Real* sQ, Real* sU, Real* sR,
                                                       unsigned gm, int j) {
    constexpr int KPL = (K + G - 1) / G, NREF = K < D ? K : K - 1;
    CoopFactor f{0, QR_OK, 0};
#pragma unroll 1
    for (int jj = 0; jj < NREF; ++jj) {
        const int owner = jj % G, mj = jj / G;
        Real* u = sU + jj * D;
        int okv = 0;
        Real rho = Real(0);
        if (j == owner) {
            Real col[D];
#pragma unroll
            for (int r = 0; r < D; ++r) {
                col[r] = A[0][r];
#pragma unroll
                for (int m = 1; m < KPL; ++m) col[r] = m == mj ? A[m][r] : col[r];
            }
            okv = coop_reflector<D>(col, jj, u, rho) ? 1 : 0;
        }
        __syncwarp(gm);
        if (__shfl_sync(gm, okv, owner, G)) {
            Real ur[D];
#pragma unroll
            for (int r = 0; r < D; ++r) ur[r] = u[r];
#pragma unroll
            for (int m = 0; m < KPL; ++m) {
                const Real w = dotv<D>(ur, A[m]);
#pragma unroll
                for (int r = 0; r < D; ++r) A[m][r] = A[m][r] - (Real(2) * ur[r]) * w;
            }
            f.count += 1;
        }
        if (j == owner) {
#pragma unroll
            for (int m = 0; m < KPL; ++m)
#pragma unroll
                for (int r = 0; r < D; ++r)
                    if (m == mj && r == jj) A[m][r] = rho;
        }
    }
    // _finish (householder.jl:66-75): the signs of the diagonal (a bit mask every lane reads), then R with its signs
#pragma unroll
    for (int m = 0; m < KPL; ++m)
#pragma unroll
        for (int r = 0; r < K; ++r)
            if (r == j + m * G) sR[r + r * K] = A[m][r];
    __syncwarp(gm);
    unsigned neg = 0;
#pragma unroll
    for (int r = 0; r < K; ++r) neg |= (sR[r + r * K] < Real(0) ? 1u : 0u) << r;
    __syncwarp(gm);
#pragma unroll
    for (int m = 0; m < KPL; ++m) {
        const int cc = j + m * G;
        if (cc >= K) continue;
#pragma unroll
        for (int r = 0; r < K; ++r) {
            const Real sgr = (neg >> r) & 1u ? Real(-1) : Real(1);
            sR[r + cc * K] = r > cc ? Real(0) : sgr * A[m][r];
        }
#pragma unroll
        for (int r = 0; r < D; ++r) A[m][r] = r == cc ? Real(1) : Real(0);
    }
    // Q = the reflectors applied to I[:, 1:K] in reverse (householder.jl:77-80), then the signs
#pragma unroll 1
    for (int jj = NREF - 1; jj >= 0; --jj) {
        Real ur[D];
#pragma unroll
        for (int r = 0; r < D; ++r) ur[r] = sU[jj * D + r];
#pragma unroll
        for (int m = 0; m < KPL; ++m) {
            const Real w = dotv<D>(ur, A[m]);
#pragma unroll
            for (int r = 0; r < D; ++r) A[m][r] = A[m][r] - (Real(2) * ur[r]) * w;
        }
    }
#pragma unroll
    for (int m = 0; m < KPL; ++m) {
        const int cc = j + m * G;
        if (cc >= K) continue;
        const Real sgc = (neg >> cc) & 1u ? Real(-1) : Real(1);
#pragma unroll
        for (int r = 0; r < D; ++r) { A[m][r] = A[m][r] * sgc; sQ[cc * D + r] = A[m][r]; }
    }
    __syncwarp(gm);
#pragma unroll
    for (int jj = K - 1; jj >= 0; --jj) {   // the first failing pivot wins
        const Real pv = sR[jj + jj * K];
        if (!(isfin(pv) && pv > Real(0))) { f.status = QR_PIVOT; f.column = jj + 1; }
    }
    return f;
}

// window_Gw (orthonormalize.jl:112-127) of the R in sR, the same in every lane; `tri` is K (K + 1) / 2 words of scratch.
// Lane j solves columns j, j + G, ... of R^{-1}; then lane 0 folds R's squares and lane 1 those of R^{-1}, column by
// column (the zeros below the diagonal add nothing to either sum). Pivots are finite and positive.
template <int K, int G, typename Real>
__device__ __forceinline__ Real coop_window_Gw(const Real* sR, Real* tri, unsigned gm, int j) {
    constexpr int KPL = (K + G - 1) / G;
    constexpr bool f64 = sizeof(Real) == 8;
    Real rin[K], rd[K];
    Ok ok;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        rd[i] = sR[i + i * K];
        if constexpr (f64) { ok.positive<100>(rd[i]); rin[i] = rcp64(rd[i]); }
        else rin[i] = dv(Real(1), rd[i]);
    }
#pragma unroll
    for (int m = 0; m < KPL; ++m) {
        const int cc = j + m * G;
        Real ri[K];
#pragma unroll
        for (int i = K - 1; i >= 0; --i) {
            // s = sum over l = i + 1 .. cc of R[i, l] ri[l] in that order; ri[l] is 0 for l > cc
            Real s = Real(0);
#pragma unroll
            for (int l = i + 1; l < K; ++l) {
                const Real t = s + sR[i + l * K] * ri[l];
                s = l <= cc ? t : s;
            }
            if constexpr (f64) {
                if (i <= cc) ok.ok = ok.ok && (static_cast<unsigned>(__double2hiint(sR[i + (cc < K ? cc : 0) * K])) & 0x7fffffffu) < (1023u + 100u) << 20;
                ri[i] = i == cc ? rin[i] : (i < cc ? quo64z(-s, rd[i], rin[i]) : 0.0);
            } else {
                ri[i] = i == cc ? rin[i] : (i < cc ? dv(-s, rd[i]) : Real(0));
            }
            if (i <= cc && cc < K) tri[cc * (cc + 1) / 2 + i] = ri[i];
        }
    }
    __syncwarp(gm);
    const bool first = j == 0;
    const Real* from = first ? sR : tri;
    Real v = from[0], s = v * v;
#pragma unroll
    for (int c = 1; c < K; ++c)
#pragma unroll
        for (int i = 0; i <= c; ++i) {
            v = from[first ? i + c * K : c * (c + 1) / 2 + i];
            s = s + v * v;
        }
    Real root;
    if constexpr (f64) {
        if (j <= 1) ok.positive<700>(s);
        root = root64(s);
        if (!group_all<G>(gm, ok.ok)) {   // some entry outside the range: the general operations, on the first lane
            Real g = Real(0);
            if (j == 0) {
                Real R[K * K];
#pragma unroll
                for (int l = 0; l < K * K; ++l) R[l] = sR[l];
                g = window_Gw<K>(R);
            }
            return __shfl_sync(gm, g, 0, G);
        }
    } else {
        root = sqt(s);
    }
    return __shfl_sync(gm, root, 0, G) * __shfl_sync(gm, root, 1, G);
}

// orth_loss (qr_spectrum.jl:4): each lane its own columns (in A) of the upper triangle of Q'Q, then the maximum over the
// group, which does not depend on the order it is combined in
template <int D, int K, int G, typename Real>
__device__ __forceinline__ Real coop_orth(const Real (&A)[(K + G - 1) / G][D], const Real* sQ, unsigned gm, int j) {
    constexpr int KPL = (K + G - 1) / G;
    Real om = Real(0);
    bool first = true;
#pragma unroll
    for (int m = 0; m < KPL; ++m) {
        const int cc = j + m * G;
#pragma unroll
        for (int r = 0; r < K; ++r) {
            if (r > cc || cc >= K) continue;
            const Real* qi = sQ + r * D;
            Real acc = qi[0] * A[m][0];
#pragma unroll
            for (int l = 1; l < D; ++l) acc = fma(qi[l], A[m][l], acc);
            if (r == cc) acc = acc - Real(1);
            const Real av = fabs(acc);
            om = first ? av : mx(om, av);
            first = false;
        }
    }
#pragma unroll
    for (int off = G / 2; off >= 1; off >>= 1) om = mx(om, __shfl_xor_sync(gm, om, off, G));
    return om;
}

}  // namespace cl
