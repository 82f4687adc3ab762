// cl_reducers.cuh -- the reducers fused into the orbit kernel: QRSpectrum (all six orthonormalisers), Benettin,
// SALI, GALI, MEGNO and FLI, and RLI for the pair streams of the indicator recorder. Each is a tag type with
//   State<D, K>                the isbits layout of the reference's state struct with T = Float64
//   step(st, n, W, prm, pend)  `reducer_step` (src/Tangent/Tangent.jl:44-49): never throws, records failures
//   failed(st)                 `reducer_failed`
// In Float64 a step runs on measures taken ahead in straight-line code (cl_fast64.cuh: the column norms that SALI,
// MEGNO and FLI share, the factorisation of QRSpectrum): the same bits wherever `ok` holds; otherwise, and whenever a
// reducer is about to fail, the general code below decides. DEFER leaves the values that only the last handoff's
// record keeps (SALI's distance, GALI's volumes) to one evaluation on that handoff's unit columns (`value`), and
// marks them in `pend`.
// and its own `replace` semantics on the frame W (d x K, column-major, registers). With Real = double every
// operation is the reference's, in its order; with Real = float (mixed kernels) the frame, norms and QR are
// Float32 while the logarithms and their Neumaier sums stay Float64.
#pragma once

#include <type_traits>

#include "cl_fast64.cuh"
#include "cl_math.cuh"
#include "cl_qr.cuh"

namespace cl {

typedef int64_t i64;

struct RedParams { double orthogonality_tol; };

// ---- QRSpectrum (src/Lyapunov/qr_spectrum.jl:14-96) -------------------------------------------------------------------
template <int K> struct QRState {
    CS sums[K]; i64 n; double G_max, orth_max; i64 count_max; int8_t code; i64 column; double value, threshold; i64 step;
};
static_assert(sizeof(QRState<2>) == 16 * 2 + 72 && sizeof(QRState<8>) == 16 * 8 + 72, "QRState layout");

template <int ALG>
struct RQR {
    static constexpr int kind = CL_RED_QR, alg = ALG;
    static constexpr bool pair = false, replaces = true, defers = false;
    template <int D, int K> using State = QRState<K>;
    // the straight-line factorisation f of this W (st.code is 0)
    template <int D, int K>
    static __device__ __forceinline__ void step_fast(State<D, K>& st, i64 n, double* W, const RedParams& prm,
                                                     const QRFast<D, K>& f) {
        if (!f.ok) {   // by copies, so that only this branch keeps the arrays in memory
            State<D, K> s2 = st;
            double W2[D * K];
#pragma unroll
            for (int l = 0; l < D * K; ++l) W2[l] = W[l];
            general_out<D, K>(&s2, n, W2, prm.orthogonality_tol);
            st = s2;
#pragma unroll
            for (int l = 0; l < D * K; ++l) W[l] = W2[l];
            return;
        }
#pragma unroll
        for (int i = 0; i < K; ++i) cs_add(st.sums[i], f.lg[i]);
        const double G = G_from_Gw64<K>(f.Gw);
        st.n = n;
        st.G_max = G > st.G_max ? G : st.G_max;
        st.orth_max = f.orth > st.orth_max ? f.orth : st.orth_max;
        st.count_max = st.count_max > f.count ? st.count_max : f.count;
        st.column = 0;
#pragma unroll
        for (int l = 0; l < D * K; ++l) W[l] = f.Q[l];
    }
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& st, i64 n, T* W, const RedParams& prm, int&) {
        if (st.code != 0) return;
        if constexpr (sizeof(T) == 8 && qr_fast_v<ALG, D, K>) {
            QRFast<D, K> f;
            qr64<ALG, D, K>(W, prm.orthogonality_tol, f);
            step_fast<D, K>(st, n, W, prm, f);
        } else {
            general<D, K>(st, n, W, prm);
        }
    }
    template <int D, int K>
    static __device__ __noinline__ void general_out(State<D, K>* st, i64 n, double* W, double tol) {
        general<D, K>(*st, n, W, RedParams{tol});
    }
    template <int D, int K, typename T>
    static __device__ __forceinline__ void general(State<D, K>& st, i64 n, T* W, const RedParams& prm) {
        T Q[D * K], R[K * K];
        const QRRes f = orthonormalize<ALG, D, K>(W, Q, R);
        if (f.status != QR_OK) {   // _factor_failure, qr_spectrum.jl:43-48
            if (f.status == QR_PASSES) {
                st.code = 2; st.column = f.column; st.value = MAX_PASSES + 1; st.threshold = MAX_PASSES;
            } else {
                T pv = R[0];
#pragma unroll
                for (int j = 0; j < K; ++j) if (j + 1 == f.column) pv = R[j + j * K];
                st.code = 1; st.column = f.column; st.value = static_cast<double>(pv);
                st.threshold = isfin(pv) ? 0.0 : __longlong_as_double(0x7ff0000000000000LL);
            }
            st.step = n;
            return;
        }
        const T eps = Eps<T>::eps();
        const T Gw = window_Gw<K>(R);
        constexpr bool gs = ALG == CL_QR_CGS || ALG == CL_QR_MGS || ALG == CL_QR_RGS;
        if (gs && !(static_cast<double>(Gw * eps) < 0.5)) {   // conditioning (GS family only)
            st.code = 3; st.column = 0; st.value = static_cast<double>(Gw * eps); st.threshold = 0.5; st.step = n;
            return;
        }
        const T orth = K >= 2 ? orth_loss<D, K>(Q) : T(0);
        const T g = (ALG == CL_QR_CGS || ALG == CL_QR_MGS) ? Gw : T(1);
        const T thr = static_cast<T>(prm.orthogonality_tol) * eps * static_cast<T>(K) * g;
        if (K >= 2 && !(orth <= thr)) {
            st.code = 4; st.column = 0; st.value = static_cast<double>(orth); st.threshold = static_cast<double>(thr);
            st.step = n;
            return;
        }
#pragma unroll
        for (int i = 0; i < K; ++i) cs_add(st.sums[i], lnr(R[i + i * K]));
        const T G = G_from_Gw<K>(Gw);
        st.n = n;
        st.G_max = jl_max(st.G_max, static_cast<double>(G));
        st.orth_max = jl_max(st.orth_max, static_cast<double>(orth));
        st.count_max = st.count_max > f.count ? st.count_max : f.count;
        st.column = 0;
#pragma unroll
        for (int l = 0; l < D * K; ++l) W[l] = Q[l];
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& st) { return st.code != 0; }
};

// ---- Benettin (src/Lyapunov/benettin.jl:11-53) --------------------------------------------------------------------
struct BenettinState { CS sum; i64 n; int8_t code; double value; i64 step; };
static_assert(sizeof(BenettinState) == 48, "BenettinState layout");

struct RBenettin {
    static constexpr int kind = CL_RED_BENETTIN, alg = 0;
    static constexpr bool pair = false, replaces = true, defers = false;
    template <int D, int K> using State = BenettinState;
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& st, i64 n, T* W, const RedParams&, int&) {
        if (st.code != 0) return;
        if constexpr (sizeof(T) == 8) {
            Ok ok;
            double y;
            const double a = norm64r<D>(W, ok, y), lg = log64(a);
            ok.divisor(a);
            double u[D];
#pragma unroll
            for (int l = 0; l < D; ++l) { ok.dividend(W[l]); u[l] = quo64(W[l], a, y); }
            if (ok.ok) {
                cs_add(st.sum, lg);
                st.n = n;
#pragma unroll
                for (int l = 0; l < D; ++l) W[l] = u[l];
                return;
            }
        }
        const T alpha = nrm<D>(W);
        if (!(isfin(alpha) && alpha > T(0))) { st.code = 1; st.value = static_cast<double>(alpha); st.step = n; return; }
        cs_add(st.sum, lnr(alpha));
        st.n = n;
#pragma unroll
        for (int l = 0; l < D * K; ++l) W[l] = dv(W[l], alpha);
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& st) { return st.code != 0; }
};

// ---- SALI (src/Indicators/sali.jl:14-68) ---------------------------------------------------------------------------
struct SALIState { CS s1, s2; double sali, value; i64 n, step; int8_t code, column; };
static_assert(sizeof(SALIState) == 72, "SALIState layout");

// Column-norm failure record shared by SALI, MEGNO and FLI (sali.jl:102-106): column 1 unless only column 2 fails.
template <typename St, typename T>
__device__ __forceinline__ bool pair_norms(St& st, i64 n, T a1, T a2) {
    const bool ok1 = isfin(a1) && a1 > T(0), ok2 = isfin(a2) && a2 > T(0);
    if (ok1 && ok2) return true;
    st.column = ok1 ? 2 : 1; st.value = static_cast<double>(ok1 ? a2 : a1); st.step = n; st.code = 1;
    return false;
}

// The frame's norms and their logarithms as the general code takes them (Float32, or Float64 out of the fast range):
// false after recording a failure.
template <int D, typename St, typename T>
__device__ __forceinline__ bool pair_general(St& st, i64 n, const T* W, T* a, double* lg) {
    a[0] = nrm<D>(W);
    a[1] = nrm<D>(W + D);
    if (!pair_norms(st, n, a[0], a[1])) return false;
    lg[0] = lnr(a[0]);
    lg[1] = lnr(a[1]);
    return true;
}
// W's two columns over their norms
template <int D>
__device__ __forceinline__ void pair_unit(double* W, const Pair64& m, const double* a) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < D; ++i) W[i + j * D] = m.ok ? quo64(W[i + j * D], m.a[j], m.y[j]) : W[i + j * D] / a[j];
}
// min(|u1 - u2|, |u1 + u2|) of unit columns (sali.jl:107-110)
template <int D, typename T>
__device__ __forceinline__ double sali_value(const T* W) {
    T dm[D], dp[D];
#pragma unroll
    for (int i = 0; i < D; ++i) { dm[i] = W[i] - W[D + i]; dp[i] = W[i] + W[D + i]; }
    if constexpr (sizeof(T) == 8) {
        Ok ok;
        const double a = norm64<D>(dm, ok), b = norm64<D>(dp, ok);
        if (ok.ok) return a < b ? a : b;
    }
    return static_cast<double>(jl_min(nrm<D>(dm), nrm<D>(dp)));
}

struct RSALI {
    static constexpr int kind = CL_RED_SALI, alg = 0;
    static constexpr bool pair = true, replaces = true, defers = true;
    template <int D, int K> using State = SALIState;
    template <int D, int K, bool DEFER>
    static __device__ __forceinline__ void step_pair(State<D, K>& st, i64 n, double* W, const Pair64& m, int& pend) {
        double a[2] = {m.a[0], m.a[1]}, lg[2] = {m.lg[0], m.lg[1]};
        if (!m.ok && !pair_general<D>(st, n, W, a, lg)) return;
        pair_unit<D>(W, m, a);
        cs_add(st.s1, lg[0]);
        cs_add(st.s2, lg[1]);
        if (DEFER) pend = 1;
        else st.sali = sali_value<D>(W);
        st.n = n;
    }
    template <int D, int K>
    static __device__ __forceinline__ void value(State<D, K>& st, const double* U, int) { st.sali = sali_value<D>(U); }
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& st, i64 n, T* W, const RedParams&, int& pend) {
        if (st.code != 0) return;
        if constexpr (sizeof(T) == 8) {
            Pair64 m;
            pair64<D>(W, m);
            step_pair<D, K, DEFER>(st, n, W, m, pend);
        } else {
            T a[2];
            double lg[2];
            if (!pair_general<D>(st, n, W, a, lg)) return;
#pragma unroll
            for (int i = 0; i < D; ++i) { W[i] = dv(W[i], a[0]); W[D + i] = dv(W[D + i], a[1]); }
            cs_add(st.s1, lg[0]);
            cs_add(st.s2, lg[1]);
            st.sali = sali_value<D>(W);
            st.n = n;
        }
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& st) { return st.code != 0; }
};

// ---- GALI (src/Indicators/gali.jl:17-201) --------------------------------------------------------------------------
template <int K> struct GALIState { double s[K], c[K], gali[K - 1]; double value; i64 n, step; int8_t code; i64 column; };
static_assert(sizeof(GALIState<4>) == 24 * 4 + 32, "GALIState layout");

template <int K, bool WITH_SALI> struct GALIFrameState { GALIState<K> g; };
template <int K> struct GALIFrameState<K, true> { GALIState<K> g; SALIState s; };

// GALI; with WITH_SALI also the SALI of the frame's first two columns. A separate SALI run (k = 2) on the same orbit
// and W0 is bitwise GALI's columns 1-2 (test/gali/ga_ac05_08.jl:356-397): same norms, same Neumaier sums, same unit
// columns. So the chain (GALI, SALI) of one frame gives both records, laid out as the tuple (GALIState, SALIState);
// the SALI record stops with the frame when GALI fails on a column SALI does not read.
template <bool WITH_SALI>
struct RGALI {
    static constexpr int kind = CL_RED_GALI, alg = 0;
    static constexpr bool pair = false, replaces = true, defers = true;
    template <int D, int K> using State = GALIFrameState<K, WITH_SALI>;
    // Bits of `pend`: 1 the volumes, 2 SALI's distance too. A handoff's values depend on its unit columns alone, and
    // every later successful handoff overwrites them, so the record needs only the last one's (gali.jl:156,
    // sali.jl:108).
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& S, i64 n, T* W, const RedParams&, int& pend) {
        GALIState<K>& st = S.g;
        if (st.code != 0) return;
        T a[K];
        double lg[K];
        bool fast = false;
        if constexpr (sizeof(T) == 8) {
            Ok ok;
            double y[K];
#pragma unroll
            for (int j = 0; j < K; ++j) {
                a[j] = norm64r<D>(W + j * D, ok, y[j]);
                ok.divisor(a[j]);
                lg[j] = log64(a[j]);
#pragma unroll
                for (int i = 0; i < D; ++i) ok.dividend(W[i + j * D]);
            }
            fast = ok.ok;
            if (fast) {
#pragma unroll
                for (int j = 0; j < K; ++j)
#pragma unroll
                    for (int i = 0; i < D; ++i) W[i + j * D] = quo64(W[i + j * D], a[j], y[j]);
            }
        }
        if (!fast) {
#pragma unroll
            for (int j = 0; j < K; ++j) a[j] = nrm<D>(W + j * D);   // _norm_col
        }
        bool sali_ok = true;
        if constexpr (WITH_SALI) sali_ok = S.s.code == 0 && (fast || pair_norms(S.s, n, a[0], a[1]));
        if (!fast) {
            int bad = 0;
#pragma unroll
            for (int j = K - 1; j >= 0; --j)
                if (!(isfin(a[j]) && a[j] >= Eps<T>::floatmin())) bad = j + 1;
            if (bad != 0) {
                T v = a[0];
#pragma unroll
                for (int j = 0; j < K; ++j) if (j + 1 == bad) v = a[j];
                st.value = static_cast<double>(v); st.step = n; st.code = 1; st.column = bad;
                return;
            }
#pragma unroll
            for (int j = 0; j < K; ++j) {
                lg[j] = lnr(a[j]);
#pragma unroll
                for (int i = 0; i < D; ++i) W[i + j * D] = dv(W[i + j * D], a[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < K; ++j) {
            CS acc{st.s[j], st.c[j]};
            cs_add(acc, lg[j]);
            st.s[j] = acc.s; st.c[j] = acc.c;
        }
        if constexpr (WITH_SALI) {
            if (sali_ok) {
                S.s.s1 = CS{st.s[0], st.c[0]};
                S.s.s2 = CS{st.s[1], st.c[1]};
                S.s.n = n;
            }
        }
        if (DEFER) pend = sali_ok ? 3 : 1;
        else value<D, K>(S, W, sali_ok ? 3 : 1);
        st.n = n;
    }
    template <int D, int K, typename T>
    static __device__ __forceinline__ void value(State<D, K>& S, const T* U, int pend) {
        GALIState<K>& st = S.g;
        if constexpr (WITH_SALI) {
            if (pend & 2) S.s.sali = sali_value<D>(U);
        }
        T Q[D * K];
#pragma unroll
        for (int l = 0; l < D * K; ++l) Q[l] = U[l];
        T g = T(1);   // _gram_core!, gali.jl:81-100
#pragma unroll
        for (int j = 0; j < K; ++j) {
#pragma unroll
            for (int pass = 0; pass < 2; ++pass)
#pragma unroll
                for (int p = 0; p < j; ++p) {
                    T cc = T(0);
#pragma unroll
                    for (int i = 0; i < D; ++i) cc = cc + Q[i + p * D] * Q[i + j * D];
#pragma unroll
                    for (int i = 0; i < D; ++i) Q[i + j * D] = Q[i + j * D] - cc * Q[i + p * D];
                }
            const T r = nrm<D>(Q + j * D);
            const T sc = r == T(0) ? T(1) : r;
#pragma unroll
            for (int i = 0; i < D; ++i) Q[i + j * D] = dv(Q[i + j * D], sc);
            if (j > 0) { g = g * r; st.gali[j - 1] = static_cast<double>(g); }
        }
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& S) {
        if constexpr (WITH_SALI) return S.g.code != 0 || S.s.code != 0;
        return S.g.code != 0;
    }
};

// ---- MEGNO (src/Indicators/megno.jl:29-113) -------------------------------------------------------------------------
struct MegnoSums { CS s, R1, R2, Q, Q2; };
struct MEGNOState { MegnoSums c1, c2; double value; i64 n, K, step; int8_t code, column; };
static_assert(sizeof(MEGNOState) == 200, "MEGNOState layout");

__device__ __forceinline__ void megno_add(MegnoSums& m, double a, double tn, double yn) {   // megno.jl:63-67
    cs_add(m.R1, tn * a);
    cs_add(m.R2, tn * tn * a);
    cs_add(m.s, a);
    const double t = 2 * cs_total(m.R1);
    Ok ok;
    ok.dividend(t);
    cs_add(m.Q, ok.ok ? quo64(t, tn, yn) : t / tn);   // tn a step count, yn = rcp64(tn)
    cs_add(m.Q2, 3 * cs_total(m.R2));
}

template <bool REPLACE>
struct RMEGNO {
    static constexpr int kind = CL_RED_MEGNO, alg = 0;
    static constexpr bool pair = true, replaces = REPLACE, defers = false;
    template <int D, int K> using State = MEGNOState;
    static __device__ __forceinline__ void sums(MEGNOState& st, i64 n, const double* lg) {
        const double tn = static_cast<double>(n), yn = rcp64(tn);
        megno_add(st.c1, lg[0], tn, yn);
        megno_add(st.c2, lg[1], tn, yn);
        st.n = n; st.K = st.K + 1;
    }
    template <int D, int K, bool DEFER>
    static __device__ __forceinline__ void step_pair(State<D, K>& st, i64 n, double* W, const Pair64& m, int&) {
        double a[2] = {m.a[0], m.a[1]}, lg[2] = {m.lg[0], m.lg[1]};
        if (!m.ok && !pair_general<D>(st, n, W, a, lg)) return;
        sums(st, n, lg);
        if (REPLACE) pair_unit<D>(W, m, a);
    }
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& st, i64 n, T* W, const RedParams&, int& pend) {
        if (st.code != 0) return;
        if constexpr (sizeof(T) == 8) {
            Pair64 m;
            pair64<D>(W, m);
            step_pair<D, K, DEFER>(st, n, W, m, pend);
        } else {
            T a[2];
            double lg[2];
            if (!pair_general<D>(st, n, W, a, lg)) return;
            sums(st, n, lg);
            if (REPLACE) {
#pragma unroll
                for (int i = 0; i < D; ++i) { W[i] = dv(W[i], a[0]); W[D + i] = dv(W[D + i], a[1]); }
            }
        }
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& st) { return st.code != 0; }
};

// ---- FLI (src/Indicators/fli.jl:26-96) -------------------------------------------------------------------------------
struct FLIState { CS s1, s2; double f1, fB, value; i64 n, step, step1, stepB; int8_t code, column, colB; };
static_assert(sizeof(FLIState) == 96, "FLIState layout");

template <bool REPLACE>
struct RFLI {
    static constexpr int kind = CL_RED_FLI, alg = 0;
    static constexpr bool pair = true, replaces = REPLACE, defers = false;
    template <int D, int K> using State = FLIState;
    static __device__ __forceinline__ void sums(FLIState& st, i64 n, const double* lg) {
        cs_add(st.s1, lg[0]);
        cs_add(st.s2, lg[1]);
        const double S1 = cs_total(st.s1), S2 = cs_total(st.s2);   // fli_maxima, fli.jl:54-60
        if (S1 > st.f1) { st.f1 = S1; st.step1 = n; }
        if (S1 > st.fB) { st.fB = S1; st.stepB = n; st.colB = 1; }
        if (S2 > st.fB) { st.fB = S2; st.stepB = n; st.colB = 2; }
        st.n = n;
    }
    template <int D, int K, bool DEFER>
    static __device__ __forceinline__ void step_pair(State<D, K>& st, i64 n, double* W, const Pair64& m, int&) {
        double a[2] = {m.a[0], m.a[1]}, lg[2] = {m.lg[0], m.lg[1]};
        if (!m.ok && !pair_general<D>(st, n, W, a, lg)) return;
        sums(st, n, lg);
        if (REPLACE) pair_unit<D>(W, m, a);
    }
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& st, i64 n, T* W, const RedParams&, int& pend) {
        if (st.code != 0) return;
        if constexpr (sizeof(T) == 8) {
            Pair64 m;
            pair64<D>(W, m);
            step_pair<D, K, DEFER>(st, n, W, m, pend);
        } else {
            T a[2];
            double lg[2];
            if (!pair_general<D>(st, n, W, a, lg)) return;
            sums(st, n, lg);
            if (REPLACE) {
#pragma unroll
                for (int i = 0; i < D; ++i) { W[i] = dv(W[i], a[0]); W[D + i] = dv(W[D + i], a[1]); }
            }
        }
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& st) { return st.code != 0; }
};

// ---- RLI (src/Indicators/rli.jl:24-114) -------------------------------------------------------------------------
// On a pair stream (PairMap, d = 2h): the two arriving columns, (xi; 0) of orbit A and (0; xi) of orbit B, Benettin's
// log sums per column, DL = |S_B - S_A| / n with the correction terms split out, and the compensated sum Q of the DL
// series; the off-block entries must stay exactly 0 (code 2, "pairing").
struct RLIState { CS sA, sB, Q; double value; i64 n, K, step; int8_t code, column; };
static_assert(sizeof(RLIState) == 88, "RLIState layout");

template <bool REPLACE>
struct RRLI {
    static constexpr int kind = CL_RED_RLI, alg = 0;
    static constexpr bool pair = false, replaces = REPLACE, defers = false;
    template <int D, int K> using State = RLIState;
    template <int D, int K, bool DEFER = false, typename T>
    static __device__ __forceinline__ void step(State<D, K>& st, i64 n, T* W, const RedParams&, int&) {
        if (st.code != 0) return;
        const T a1 = nrm<D>(W), a2 = nrm<D>(W + D);
        if (!pair_norms(st, n, a1, a2)) return;
        constexpr int h = D / 2;
        T m1 = T(0), m2 = T(0);   // _offblock, rli.jl:58-65
#pragma unroll
        for (int i = 0; i < h; ++i) { m1 = jl_max(m1, fabs(W[h + i])); m2 = jl_max(m2, fabs(W[D + i])); }
        if (!(m1 == T(0) && m2 == T(0))) {
            const bool first_clean = m1 == T(0);
            st.column = first_clean ? 2 : 1; st.value = static_cast<double>(first_clean ? m2 : m1); st.step = n; st.code = 2;
            return;
        }
        cs_add(st.sA, lnr(a1));
        cs_add(st.sB, lnr(a2));
        cs_add(st.Q, fabs((st.sB.s - st.sA.s) + (st.sB.c - st.sA.c)) / static_cast<double>(n));   // rli_dl, rli.jl:53
        st.n = n;
        st.K = st.K + 1;
        if (REPLACE) {
#pragma unroll
            for (int i = 0; i < D; ++i) { W[i] = dv(W[i], a1); W[D + i] = dv(W[D + i], a2); }
        }
    }
    template <int D, int K>
    static __device__ __forceinline__ bool failed(const State<D, K>& st) { return st.code != 0; }
};

}  // namespace cl
