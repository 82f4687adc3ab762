// cl_fast64.cuh -- correctly rounded Float64 division, square root and the portable logarithm as straight-line code.
//
// The reducers' handoffs are chains of norms, quotients by a common norm, square roots and logarithms. The operators
// `/` and sqrt() carry a branch to a general routine each, so the compiler can neither overlap two of them nor share
// the reciprocal of a common divisor: one handoff of QRSpectrum(MGS) at k = 2 (13 quotients, 5 roots, 2 logarithms)
// cost ~1100 instructions and 5300 cycles of dependent latency. Here every operation is branch-free on operands whose
// exponents lie well inside the Float64 range, gives the IEEE result bit for bit there, and records in `Ok` when an
// operand left that range; a caller that finds the record set repeats the handoff with the operators.
//
//   reciprocal  a hardware estimate (rcp.approx.ftz.f64, about 2^-20) refined once cubically and once by Newton:
//               the last step rounds 1/b correctly unless b's significand is all ones (P. Markstein, "Computation of
//               elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), and that
//               one significand is set by its value, 2^-e (1 + 2^-52).
//   quotient    one product and two fmas by the rounded reciprocal of a shared divisor (Markstein 1990; N. Brisebarre,
//               J.-M. Muller, S. K. Raina, "Accelerating correctly rounded floating-point division when the divisor
//               is known in advance", IEEE Trans. Comput. 53, 2004). The sign of a zero dividend is restored.
//   root        the estimate rsqrt.approx.ftz.f64 refined cubically, then one residual correction (Markstein 1990).
// Dependent latencies on a B200 (cycles): `/` 114, sqrt 182, cl_log 399; rcp64 76, a further quotient 30, root64 77,
// log64 297, and independent ones overlap. What bounds a handoff of a small ensemble is the chain of these; of a large
// one, the instructions. Whole kernels before and after, one orbit a thread: wrapped standard map, MGS, tau = 1, 65536
// orbits x 1000 steps 3.70 -> 2.09 ms (4096 x 4000 11.09 -> 4.35, before the pipeline of cl_pipe.cuh took that size, now
// 2.49); standard map, MEGNO + FLI + SALI, 20001 x 1000 4.73 -> 1.43 ms; Froeschle map, Householder | GALI + SALI, tau =
// 10, 65536 x 1000 6.60 -> 2.29 ms.
// tests/test_gpu_fast64.py holds each to the operators on random operands and on the operands nearest a tie,
// tests/test_gpu_fast64_limits.py over the whole range that `Ok` accepts.
#pragma once

#include "cl_math.cuh"
#include "cl_qr.cuh"

namespace cl {

// Whether every operand so far was inside the range the straight-line forms are exact on.
struct Ok {
    bool ok = true;
    // a divisor, radicand or logarithm argument: positive, normal, exponent within +-E of 0
    template <int E>
    __device__ __forceinline__ void positive(double b) {
        constexpr unsigned lo = static_cast<unsigned>(1023 - E) << 20, span = static_cast<unsigned>(2 * E) << 20;
        ok = ok && static_cast<unsigned>(__double2hiint(b)) - lo < span;
    }
    // The divisor of `dividend`s: positive, exponent from -800 to 209, so that no accepted quotient is below 2^-1010. (A
    // bound relative to each divisor, for divisors up to 2^700, cost the lattices' handoffs 2-4 % of the kernel.)
    __device__ __forceinline__ void divisor(double b) {
        constexpr unsigned lo = static_cast<unsigned>(1023 - 800) << 20, span = static_cast<unsigned>(800 + 210) << 20;
        ok = ok && static_cast<unsigned>(__double2hiint(b)) - lo < span;
    }
    // a dividend: zero, or large enough that the quotient's residual is exact
    __device__ __forceinline__ void dividend(double a) {
        constexpr unsigned lo = static_cast<unsigned>(1023 - 800) << 20;
        const unsigned h = static_cast<unsigned>(__double2hiint(a)) & 0x7fffffffu;
        ok = ok && (h >= lo || (h | static_cast<unsigned>(__double2loint(a))) == 0u);
    }
};

// RN(1 / b) from y within an ulp of it (the last step of rcp64)
__device__ __forceinline__ double rcp64_last(double b, double y) {
    y = fma(fma(-b, y, 1.0), y, y);
    const int hb = __double2hiint(b);
    const bool ones = __double2loint(b) == -1 && (hb & 0xfffff) == 0xfffff;
    return ones ? __hiloint2double((2046 << 20) - (hb & 0x7ff00000) - (1 << 20), 1) : y;
}
// RN(1 / b) for a positive b with an exponent within +-900.
__device__ __forceinline__ double rcp64(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return rcp64_last(b, fma(fma(e, e, e), y, y));
}
// RN(a / b), y = rcp64(b), b > 0; quo64z may give a zero quotient of a zero dividend the other sign
__device__ __forceinline__ double quo64z(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-q, b, a), y, q);
}
__device__ __forceinline__ double quo64(double a, double b, double y) {
    const double r = quo64z(a, b, y);
    return __hiloint2double(__double2hiint(r) | (__double2hiint(a) & 0x80000000), __double2loint(r));
}
// RN(sqrt(s)) for a positive s with an exponent within +-900; h: 1 / (2 sqrt(s)) to about an ulp
__device__ __forceinline__ double root64(double s, double& h) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    double g = s * y;
    h = 0.5 * y;
    const double r = fma(-g, h, 0.5);
    const double t = fma(1.5 * r, r, r);
    g = fma(t, g, g);
    h = fma(t, h, h);
    return fma(fma(-g, g, s), h, g);
}
__device__ __forceinline__ double root64(double s) { double h; return root64(s, h); }
// cl_log of a positive normal x, bit for bit, without its special cases
__device__ __forceinline__ double log64(double x) {
    const int hx = __double2hiint(x);
    const int lx = __double2loint(x);
    const int hm = (hx & 0x000fffff) | 0x3ff00000;
    const double m1 = __hiloint2double(hm, lx);
    const bool big = m1 > CL_SQRT2;
    const double f = (big ? __hiloint2double(hm - 0x00100000, lx) : m1) - 1.0;
    // the exponent as a double: exact through 2^52 + 2^31 + e
    const int ei = (hx >> 20) - 1023 + (big ? 1 : 0);
    const double e = __hiloint2double(0x43300000, ei ^ static_cast<int>(0x80000000)) - 4503601774854144.0;
    const double d = 2.0 + f;
    const double s = quo64(f, d, rcp64(d));
    const double z = s * s;
    double R = CL_LOG_T9;
    R = fma(R, z, CL_LOG_T8);
    R = fma(R, z, CL_LOG_T7);
    R = fma(R, z, CL_LOG_T6);
    R = fma(R, z, CL_LOG_T5);
    R = fma(R, z, CL_LOG_T4);
    R = fma(R, z, CL_LOG_T3);
    R = fma(R, z, CL_LOG_T2);
    R = fma(R, z, CL_LOG_T1);
    R = R * z;
    const double hfsq = 0.5 * f * f;
    return e * CL_LN2_HI - ((hfsq - (s * (hfsq + R) + e * CL_LN2_LO)) - f);
}

// safe_norm<N> of v[0], v[stride], ...: max, quotients by it, the root of their squares' sum. A quotient below 2^-100
// need not be exact: its square is absorbed by the sum, which holds a 1 when it is complete, whatever its bits.
// Only the first n <= N entries count (n a constant of the caller's unrolled loop).
// norm64r also gives the norm's rounded reciprocal: the product of the two reciprocals at hand, 1/m and 1/sqrt of the
// sum, is within some ulps of it, so one Newton step replaces the hardware estimate and its cubic refinement (30 of 85
// cycles of the chain).
template <int N>
__device__ __forceinline__ double norm64r(const double* v, Ok& ok, double& rcp, int n = N) {
    double t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = i < n ? fabs(v[i]) : 0.0;
#pragma unroll
    for (int w = 8; w >= 1; w >>= 1)   // the maximum as a tree (a compare and select cost 19 cycles of latency)
#pragma unroll
        for (int i = 0; i < N && i < w; ++i)
            if (i + w < N && i + w < n) t[i] = t[i + w] > t[i] ? t[i + w] : t[i];
    const double m = t[0];
    ok.positive<700>(m);
    const double y = rcp64(m);
    double q = quo64z(v[0], m, y);
    double s = q * q;
#pragma unroll
    for (int i = 1; i < N; ++i) if (i < n) { q = quo64z(v[i], m, y); s = s + q * q; }
    ok.positive<10>(s);   // in [1, N (1 + eps)]; a NaN among the entries shows here
    double h;
    const double r = m * root64(s, h);
    const double e = y * (h + h);
    rcp = rcp64_last(r, fma(fma(-r, e, 1.0), e, e));
    return r;
}
template <int N>
__device__ __forceinline__ double norm64(const double* v, Ok& ok, int n = N) {
    double rcp;   // not used: the compiler drops it
    return norm64r<N>(v, ok, rcp, n);
}

// ---- the orthonormalisations of cl_qr.cuh in the straight-line operations ------------------------------------------
// The same operations in the same order, with the products by the structural zeros of a reflector, of an identity
// column or of a triangle left out: each such term adds +-0 to a sum, which changes at most the sign of a zero. Zeros
// of R reach no output, Householder's Q cannot differ (its zero entries are +0 times a column sign in both forms), and
// a Givens Q that holds a zero is left to the general form. Only a factorisation that succeeds, with every column
// and pivot in range, is returned as ok.
template <int D, int K>
struct QRFast {
    double Q[D * K];
    double rd[K], lg[K];   // R's diagonal and its logarithms
    double Gw, orth;
    int count;
    bool ok;
};

// The quotients' dividends are not checked: one too small to be exact belongs to an entry of R^{-1} so small that b, which
// holds the pivots' inverse squares (at least 2^-200) and is at most 2^700, is the same with any such value in its place.
template <int K>
__device__ __forceinline__ double window_Gw64(const double* R, const double* rin, Ok& ok) {
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int i = 0; i <= j; ++i) { const double a = fabs(R[i + j * K]); m = a > m ? a : m; }
    ok.positive<100>(m);
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        double Ri[K];
        Ri[j] = rin[j];
#pragma unroll
        for (int i = j - 1; i >= 0; --i) {
            double s = R[i + (i + 1) * K] * Ri[i + 1];
#pragma unroll
            for (int l = i + 2; l <= j; ++l) s = s + R[i + l * K] * Ri[l];
            Ri[i] = quo64z(-s, R[i + i * K], rin[i]);
        }
#pragma unroll
        for (int i = 0; i <= j; ++i) {
            a = i + j == 0 ? R[0] * R[0] : a + R[i + j * K] * R[i + j * K];
            b = i + j == 0 ? Ri[0] * Ri[0] : b + Ri[i] * Ri[i];
        }
    }
    ok.positive<700>(a);
    ok.positive<700>(b);
    return root64(a) * root64(b);
}

template <int D, int K>
__device__ __forceinline__ double orth_loss64(const double* Q) {
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int i = 0; i <= j; ++i) {
            double acc = Q[i * D] * Q[j * D];
#pragma unroll
            for (int q = 1; q < D; ++q) acc = fma(Q[q + i * D], Q[q + j * D], acc);
            if (i == j) acc = acc - 1.0;
            const double a = fabs(acc);
            m = a > m ? a : m;
        }
    return m;
}

// CGS / MGS (orth_gs)
template <int ALG, int D, int K>
__device__ __forceinline__ void gs64(const double* W, double* Q, double* R, double* rin, Ok& ok) {
#pragma unroll
    for (int m = 0; m < K; ++m) {
        const double* w = W + m * D;
        double u[D];
#pragma unroll
        for (int i = 0; i < D; ++i) u[i] = w[i];
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const double* qi = Q + i * D;
            const double* from = ALG == CL_QR_CGS ? w : u;
            double c = qi[0] * from[0];
#pragma unroll
            for (int l = 1; l < D; ++l) c = c + qi[l] * from[l];
            R[i + m * K] = c;
#pragma unroll
            for (int l = 0; l < D; ++l) u[l] = u[l] - c * qi[l];
        }
        double y;
        const double gamma = norm64r<D>(u, ok, y);
        ok.positive<100>(gamma);   // as every pivot; the other two factorisations divide by at most twice one
        R[m + m * K] = gamma;
        rin[m] = y;
#pragma unroll
        for (int l = 0; l < D; ++l) {
            ok.dividend(u[l]);
            Q[l + m * D] = quo64(u[l], gamma, y);
        }
    }
}

// Householder (orth_householder): reflector j holds rows j.. only, and touches rows j.. of the columns right of it;
// column l of Q is I's column until reflector l.
template <int D, int K>
__device__ __forceinline__ int householder64(const double* W, double* Q, double* R, double* rin, Ok& ok) {
    constexpr int NREF = K < D ? K : K - 1;
    double A[D * K], U[D * K];
#pragma unroll
    for (int l = 0; l < D * K; ++l) A[l] = W[l];
#pragma unroll
    for (int j = 0; j < NREF; ++j) {
        double a[D];
#pragma unroll
        for (int i = 0; i < D; ++i) a[i] = i + j < D ? A[i + j + j * D] : 0.0;
        const double c = norm64<D>(a, ok, D - j);
        const bool neg = a[0] < 0.0;
        a[0] = a[0] + (neg ? -c : c);
        double y;
        const double nv = norm64r<D>(a, ok, y, D - j);
#pragma unroll
        for (int i = 0; i < D; ++i)
            if (i + j < D) {
                ok.dividend(a[i]);
                U[i + j + j * D] = quo64(a[i], nv, y);
            }
        A[j + j * D] = neg ? c : -c;
#pragma unroll
        for (int l = j + 1; l < K; ++l) {
            double w = U[j + j * D] * A[j + l * D];
#pragma unroll
            for (int i = j + 1; i < D; ++i) w = w + U[i + j * D] * A[i + l * D];
#pragma unroll
            for (int i = j; i < D; ++i) A[i + l * D] = A[i + l * D] - (2.0 * U[i + j * D]) * w;
        }
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const double p = A[j + j * D];
        const bool neg = p < 0.0;
        const double r = fabs(p);
        ok.positive<100>(r);
        rin[j] = rcp64(r);
#pragma unroll
        for (int i = 0; i < K; ++i)
            if (i < j) R[i + j * K] = A[i + i * D] < 0.0 ? -A[i + j * D] : A[i + j * D];
        R[j + j * K] = r;
        const int j0 = j < NREF ? j : NREF - 1;
        double* q = Q + j * D;
        double w = U[j + j0 * D];
#pragma unroll
        for (int i = 0; i < D; ++i) q[i] = i < j0 ? 0.0 : (i == j ? 1.0 : 0.0) - (2.0 * U[i + j0 * D]) * w;
#pragma unroll
        for (int k = NREF - 2; k >= 0; --k) {
            if (k >= j0) continue;
            w = U[k + 1 + k * D] * q[k + 1];
#pragma unroll
            for (int i = 0; i < D; ++i)
                if (i > k + 1) w = w + U[i + k * D] * q[i];
#pragma unroll
            for (int i = 0; i < D; ++i)
                if (i >= k) q[i] = q[i] - (2.0 * U[i + k * D]) * w;
        }
#pragma unroll
        for (int i = 0; i < D; ++i) q[i] = neg ? -q[i] : q[i];
    }
    return NREF;
}

// Givens (orth_givens): rows of [W | I]; an entry of I's part that no rotation has filled is known to be zero
template <int D, int K>
__device__ __forceinline__ int givens64(const double* W, double* Q, double* R, double* rin, Ok& ok) {
    constexpr int WD = K + D, J = K < D - 1 ? K : D - 1;
    double rows[D][WD];
    bool nz[D][WD];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int l = 0; l < WD; ++l) {
            nz[i][l] = l < K || l - K == i;
            rows[i][l] = l < K ? W[i + l * D] : (l - K == i ? 1.0 : 0.0);
        }
    int count = 0;
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int i = D - 1; i >= 1; --i) {
            if (i < j + 1) continue;
            const double ab[2] = {rows[i - 1][j], rows[i][j]};
            double y;
            const double rho = norm64r<2>(ab, ok, y);
            ok.dividend(ab[0]);
            ok.dividend(ab[1]);
            const double c = quo64(ab[0], rho, y), s = quo64(ab[1], rho, y);
#pragma unroll
            for (int l = 0; l < WD; ++l) {
                if (l <= j) continue;
                const bool na = nz[i - 1][l], nb = nz[i][l];
                const double ra = rows[i - 1][l], rb = rows[i][l];
                if (na && nb) {
                    rows[i - 1][l] = c * ra + s * rb;
                    rows[i][l] = c * rb - s * ra;
                } else if (na) {
                    rows[i - 1][l] = c * ra;
                    rows[i][l] = -(s * ra);
                } else if (nb) {
                    rows[i - 1][l] = s * rb;
                    rows[i][l] = c * rb;
                }
                nz[i - 1][l] = nz[i][l] = na || nb;
            }
            rows[i - 1][j] = rho;
            count += 1;
        }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const double p = rows[j][j];
        const bool neg = p < 0.0;
        const double r = fabs(p);
        ok.positive<100>(r);
        rin[j] = rcp64(r);
        R[j + j * K] = r;
#pragma unroll
        for (int i = 0; i < K; ++i)
            if (i < j) R[i + j * K] = rows[i][i] < 0.0 ? -rows[i][j] : rows[i][j];
#pragma unroll
        for (int a = 0; a < D; ++a) {
            const double q = rows[j][K + a];
            ok.ok = ok.ok && q != 0.0;
            Q[a + j * D] = neg ? -q : q;
        }
    }
    return count;
}

// Which factorisations have a straight-line form (RGS repeats its passes and the augmented sweep carries D more
// columns: they keep the general form, and so do frames whose arrays would not fit one thread's registers).
template <int ALG, int D, int K>
constexpr bool qr_fast_v = (ALG == CL_QR_CGS || ALG == CL_QR_MGS || ALG == CL_QR_HOUSEHOLDER || ALG == CL_QR_GIVENS) &&
                           D * K <= 16;

// The whole of QRSpectrum's handoff before its state changes (qr_spectrum.jl:50-70)
template <int ALG, int D, int K>
__device__ __forceinline__ void qr64(const double* W, double tol, QRFast<D, K>& f) {
    Ok ok;
    double R[K * K], rin[K];
    f.count = 1;
    if constexpr (ALG == CL_QR_HOUSEHOLDER) f.count = householder64<D, K>(W, f.Q, R, rin, ok);
    else if constexpr (ALG == CL_QR_GIVENS) f.count = givens64<D, K>(W, f.Q, R, rin, ok);
    else gs64<ALG, D, K>(W, f.Q, R, rin, ok);
#pragma unroll
    for (int j = 0; j < K; ++j) {
        f.rd[j] = R[j + j * K];
        ok.positive<100>(f.rd[j]);
        f.lg[j] = log64(f.rd[j]);
    }
    const double eps = Eps<double>::eps();
    f.Gw = window_Gw64<K>(R, rin, ok);
    ok.positive<400>(f.Gw);
    constexpr bool gs = ALG == CL_QR_CGS || ALG == CL_QR_MGS;
    if (gs) ok.ok = ok.ok && f.Gw * eps < 0.5;
    f.orth = K >= 2 ? orth_loss64<D, K>(f.Q) : 0.0;
    const double thr = tol * eps * static_cast<double>(K) * (gs ? f.Gw : 1.0);
    if (K >= 2) ok.ok = ok.ok && f.orth <= thr;
    f.ok = ok.ok;
}
// _G_from_Gw
template <int K>
__device__ __forceinline__ double G_from_Gw64(double Gw) {
    if (K == 1) return 1.0;
    if (K == 2) {
        const double z = Gw * Gw - 4.0;
        return (Gw + (z > 0.0 ? root64(z > 0.0 ? z : 1.0) : 0.0)) * 0.5;
    }
    return Gw;
}

// ---- the column norms that SALI, MEGNO and FLI take of one frame ---------------------------------------------------
struct Pair64 { double a[2], y[2], lg[2]; bool ok; };
template <int D>
__device__ __forceinline__ void pair64(const double* W, Pair64& m) {
    Ok ok;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        m.a[j] = norm64r<D>(W + j * D, ok, m.y[j]);
        ok.divisor(m.a[j]);
        m.lg[j] = log64(m.a[j]);
#pragma unroll
        for (int i = 0; i < D; ++i) ok.dividend(W[i + j * D]);
    }
    m.ok = ok.ok;
}

}  // namespace cl
