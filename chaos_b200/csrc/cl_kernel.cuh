// cl_kernel.cuh -- the fused orbit kernel: one orbit per thread, the point in Float64 registers, every tangent
// frame (D x K) and every reducer state in registers, handoffs every tau steps, only final records written to HBM.
//
// It is the device body of the reference's `_orbit_kernel!` (src/Tangent/propagate.jl:32-50) running
// `_orbit_body` (src/Tangent/orbit.jl:44-60): tangent at the old point, frame product, forward; every tau steps the
// status check (`_status`, orbit.jl:3) and the reducer chain (`_apply`, orbit.jl:23-28: every reducer runs, each
// on the W the previous one returned, then `_any_failed`); the final status check only at step N; a launch of
// `steps` steps from global step n0 that carries x, W, states, code and hstep (D44 relaunch), with an orbit that
// failed in an earlier launch frozen.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/chaoslab_b200.h"
#include "cl_math.cuh"
#include "cl_reducers.cuh"
#include "cl_systems.cuh"

namespace cl {

constexpr int8_t STATUS_OK = 0, STATUS_STATE = 1, STATUS_W = 2, STATUS_REDUCER = 3;

struct KArgs {
    i64 n;                       // orbits in this launch
    i64 n0, steps, N;            // launch window and run length
    int tau;
    int soa;                     // x / W layout: 1 component-major, 0 orbit-major
    const double* x_in;          // n0 == 0: x0; else carried x (may equal x_out)
    double* x_out;
    const double* W_in[CL_MAX_FRAMES];   // n0 == 0: W0 or NULL (seeded); else carried W
    double* W_out[CL_MAX_FRAMES];
    uint64_t* states[CL_MAX_FRAMES];     // orbit-major, Julia layout
    int8_t* code[CL_MAX_FRAMES];
    i64* hstep[CL_MAX_FRAMES];
    uint64_t seed;
    i64 orbit_base;
    RedParams prm[CL_MAX_FRAMES][CL_MAX_REDUCERS];
};

// ---- what a frame's chain measures of the arriving W before any reducer runs --------------------------------------
// Float64 only: one evaluation of the column norms for all of SALI, MEGNO and FLI that see the arriving frame, and
// the factorisation of a QRSpectrum that does, in straight-line code (cl_fast64.cuh) that overlaps with the next
// step's sines.
struct NoMeasure {};
template <int I, class... Rs> struct FirstQR { static constexpr int alg = 0, at = 0; };
template <int I, class R, class... Rs> struct FirstQR<I, R, Rs...> {
    using Tail = FirstQR<I + 1, Rs...>;   // only a reducer that sees the arriving frame
    static constexpr int alg = R::alg ? R::alg : (R::replaces ? 0 : Tail::alg);
    static constexpr int at = R::alg ? I : Tail::at;
};
template <class... Rs> struct FirstPair { static constexpr bool value = false; };
template <class R, class... Rs> struct FirstPair<R, Rs...> {
    static constexpr bool value = R::pair || (!R::replaces && FirstPair<Rs...>::value);
};
template <class... Rs> struct LastOf { static constexpr bool defers = false; };
template <class R> struct LastOf<R> { static constexpr bool defers = R::defers; };
template <class R, class R2, class... Rs> struct LastOf<R, R2, Rs...> : LastOf<R2, Rs...> {};

template <int D, int K, typename T, class... Rs>
struct Measure {
    static constexpr bool f64 = sizeof(T) == 8;
    static constexpr bool pair = f64 && K == 2 && FirstPair<Rs...>::value;
    static constexpr int alg = FirstQR<0, Rs...>::alg;
    static constexpr bool qr = f64 && alg != 0 && qr_fast_v<alg, D, K>;
    typename std::conditional<pair, Pair64, NoMeasure>::type p;
    typename std::conditional<qr, QRFast<D, K>, NoMeasure>::type q;
    __device__ __forceinline__ void take(const T* W, const RedParams* prm) {
        if constexpr (pair) pair64<D>(W, p);
        if constexpr (qr) qr64<alg, D, K>(W, prm[FirstQR<0, Rs...>::at].orthogonality_tol, q);
    }
};

// ---- the reducer chain of one frame as a recursive aggregate --------------------------------------------------------
template <int D, int K, class... Rs> struct Chain;
template <int D, int K> struct Chain<D, K> {
    static constexpr int bytes = 0;
    template <bool FRESH, bool DEFER, typename T, class M>
    __device__ __forceinline__ void run(i64, T*, const RedParams*, const M&, int&) {}
    template <typename T> __device__ __forceinline__ void value(const T*, int) {}
    __device__ __forceinline__ bool failed() const { return false; }
    __device__ __forceinline__ void load(const uint64_t*) {}
    __device__ __forceinline__ void store(uint64_t*) const {}
    __device__ __forceinline__ void zero() {}
};
template <int D, int K, class R, class... Rs> struct Chain<D, K, R, Rs...> {
    using Head = typename R::template State<D, K>;
    static_assert(sizeof(Head) % 8 == 0, "state size");
    static constexpr int hwords = static_cast<int>(sizeof(Head) / 8);
    static constexpr int bytes = static_cast<int>(sizeof(Head)) + Chain<D, K, Rs...>::bytes;
    Head head;
    Chain<D, K, Rs...> tail;
    // FRESH: W is the frame that m measured. DEFER: the last reducer's values are left to `value`.
    template <bool FRESH, bool DEFER, typename T, class M>
    __device__ __forceinline__ void run(i64 n, T* W, const RedParams* p, const M& m, int& pend) {
        constexpr bool defer = DEFER && sizeof...(Rs) == 0;
        if constexpr (FRESH && R::pair && M::pair) {
            if (!failed_head()) R::template step_pair<D, K, defer>(head, n, W, m.p, pend);
        } else if constexpr (FRESH && R::alg != 0 && M::qr) {
            if (!failed_head()) R::template step_fast<D, K>(head, n, W, p[0], m.q);
        } else {
            R::template step<D, K, defer>(head, n, W, p[0], pend);
        }
        tail.template run<FRESH && !R::replaces, DEFER>(n, W, p + 1, m, pend);
    }
    template <typename T>
    __device__ __forceinline__ void step(i64 n, T* W, const RedParams* p) {
        Measure<D, K, T, R, Rs...> m;
        m.take(W, p);
        int pend = 0;
        run<true, false>(n, W, p, m, pend);
    }
    template <typename T> __device__ __forceinline__ void value(const T* U, int pend) {
        if constexpr (sizeof...(Rs) == 0) R::template value<D, K>(head, U, pend);
        else tail.value(U, pend);
    }
    __device__ __forceinline__ bool failed_head() const { return R::template failed<D, K>(head); }
    __device__ __forceinline__ bool failed() const { return R::template failed<D, K>(head) || tail.failed(); }
    __device__ __forceinline__ void load(const uint64_t* src) {
        uint64_t* h = reinterpret_cast<uint64_t*>(&head);
#pragma unroll
        for (int w = 0; w < hwords; ++w) h[w] = src[w];
        tail.load(src + hwords);
    }
    __device__ __forceinline__ void store(uint64_t* dst) const {
        const uint64_t* h = reinterpret_cast<const uint64_t*>(&head);
#pragma unroll
        for (int w = 0; w < hwords; ++w) dst[w] = h[w];
        tail.store(dst + hwords);
    }
    __device__ __forceinline__ void zero() {
        uint64_t* h = reinterpret_cast<uint64_t*>(&head);
#pragma unroll
        for (int w = 0; w < hwords; ++w) h[w] = 0;
        tail.zero();
    }
};

template <int KK, class... Rs> struct Frame {
    static constexpr int K = KK;
    static constexpr bool defers = LastOf<Rs...>::defers;
    template <int D> using Chain_ = Chain<D, KK, Rs...>;
    template <int D, typename T> using Measure_ = Measure<D, KK, T, Rs...>;
};

// ---- seeded Haar frames --------------------------------------------------------------------------------------------
// Key derivation of `initial_deviations` (src/Tangent/initial.jl:27-28): key = _mix(_mix(seed) + orbit); the
// normal variates are this library's own counter stream (Box-Muller on u_t = ((_mix(key + t) >> 11) + 1/2) 2^-53),
// not StableRNGs.jl, then two Gram-Schmidt passes per column. The oracle restates the same stream.
template <int D, int K, typename T>
__device__ __forceinline__ void seeded_frame(uint64_t seed, i64 orbit, T* W) {
    const uint64_t key = mix64(mix64(seed) + static_cast<uint64_t>(orbit));
    double G[D * D];
#pragma unroll
    for (int t = 0; t < D * D; t += 2) {
        const double u1 = (static_cast<double>(mix64(key + static_cast<uint64_t>(t)) >> 11) + 0.5) * 0x1p-53;
        const double u2 = (static_cast<double>(mix64(key + static_cast<uint64_t>(t) + 1) >> 11) + 0.5) * 0x1p-53;
        const double r = sqrt(-2.0 * cl_log(u1));
        double sn, cs; cl_sincos((2 * 3.141592653589793) * u2, &sn, &cs);
        G[t] = r * cs;
        if (t + 1 < D * D) G[t + 1] = r * sn;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
#pragma unroll
        for (int pass = 0; pass < 2; ++pass)
#pragma unroll
            for (int i = 0; i < j; ++i) {
                const double c = dotv<D>(G + i * D, G + j * D);
#pragma unroll
                for (int l = 0; l < D; ++l) G[l + j * D] = G[l + j * D] - c * G[l + i * D];
            }
        double s = G[j * D] * G[j * D];
#pragma unroll
        for (int l = 1; l < D; ++l) s = s + G[l + j * D] * G[l + j * D];
        const double nr = sqrt(s);
#pragma unroll
        for (int l = 0; l < D; ++l) G[l + j * D] = G[l + j * D] / nr;
    }
#pragma unroll
    for (int l = 0; l < D * K; ++l) W[l] = static_cast<T>(G[l]);
}

// ---- per-frame register state ---------------------------------------------------------------------------------------
template <int D, typename Real, class F>
struct FrameRegs {
    static constexpr int K = F::K;
    Real W[D * K];
    typename F::template Chain_<D> st;
    int8_t code;
    i64 hstep;
    bool alive;
    int pend;        // values the chain left to the end of the launch (0: none) ...
    bool pend_here;  // ... and whether W holds their unit columns (else the copy taken at the window's start)
};

template <int D, int S>
__device__ __forceinline__ bool all_finite_x(const double* x) {
    unsigned m = 0;
#pragma unroll
    for (int i = 0; i < S; ++i) m = max(m, static_cast<unsigned>(__double2hiint(x[i])) & 0x7ff00000u);
    return m != 0x7ff00000u;
}
template <int N, typename Real>
__device__ __forceinline__ bool all_finite(const Real* W) {
    if constexpr (sizeof(Real) == 8) {   // the largest exponent field, on the integer pipe
        unsigned m = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) m = max(m, static_cast<unsigned>(__double2hiint(W[i])) & 0x7ff00000u);
        return m != 0x7ff00000u;
    } else {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; ++i) ok = ok && isfin(W[i]);
        return ok;
    }
}

template <int D, int S, typename Real, class F>
__device__ __forceinline__ void frame_load(FrameRegs<D, Real, F>& fr, int f, const KArgs& a, i64 i, bool fresh) {
    constexpr int K = F::K;
    const i64 so = a.soa ? 1 : D * K, sc = a.soa ? a.n : 1;
    fr.pend = 0;
    fr.pend_here = true;
    if (fresh) {
        if (a.W_in[f]) {
#pragma unroll
            for (int l = 0; l < D * K; ++l) fr.W[l] = static_cast<Real>(a.W_in[f][i * so + l * sc]);
        } else {
            seeded_frame<D, K>(a.seed, a.orbit_base + i + 1, fr.W);
        }
        fr.st.zero();
        fr.code = STATUS_OK;
        fr.hstep = 0;
        fr.alive = true;
    } else {
#pragma unroll
        for (int l = 0; l < D * K; ++l) fr.W[l] = static_cast<Real>(a.W_in[f][i * so + l * sc]);
        constexpr int words = F::template Chain_<D>::bytes / 8;
        if (words > 0) fr.st.load(a.states[f] + i * words);
        fr.code = a.code[f][i];
        fr.hstep = a.hstep[f] ? a.hstep[f][i] : 0;
        fr.alive = fr.code == STATUS_OK;
    }
}

template <int D, int S, typename Real, class F>
__device__ __forceinline__ void frame_store(const FrameRegs<D, Real, F>& fr, int f, const KArgs& a, i64 i) {
    constexpr int K = F::K;
    const i64 so = a.soa ? 1 : D * K, sc = a.soa ? a.n : 1;
#pragma unroll
    for (int l = 0; l < D * K; ++l) a.W_out[f][i * so + l * sc] = static_cast<double>(fr.W[l]);
    constexpr int words = F::template Chain_<D>::bytes / 8;
    if (words > 0) fr.st.store(a.states[f] + i * words);
    a.code[f][i] = fr.code;
    if (a.hstep[f]) a.hstep[f][i] = fr.hstep;
}

// At a handoff: _status, then the chain, then _any_failed (orbit.jl:54-57). m: the measures of fr.W.
template <int D, int S, bool DEFER, typename Real, class F, class M>
__device__ __forceinline__ void frame_handoff(FrameRegs<D, Real, F>& fr, const double* x, i64 n, const RedParams* prm,
                                              const M& m) {
    if (!fr.alive) return;
    constexpr int K = F::K;
    int8_t c = all_finite_x<D, S>(x) ? (all_finite<D * K>(fr.W) ? STATUS_OK : STATUS_W) : STATUS_STATE;
    int pend = 0;
    if (c == STATUS_OK) {
        fr.st.template run<true, DEFER>(n, fr.W, prm, m, pend);
        if (fr.st.failed()) c = STATUS_REDUCER;
    }
    if (DEFER) {
        if (pend) { fr.pend = pend; fr.pend_here = true; }
        else fr.pend_here = false;
    }
    if (c != STATUS_OK) { fr.code = c; fr.hstep = n; fr.alive = false; }
}
template <int D, int S, typename Real, class F>
__device__ __forceinline__ void frame_handoff(FrameRegs<D, Real, F>& fr, const double* x, i64 n, const RedParams* prm) {
    typename F::template Measure_<D, Real> m;
    m.take(fr.W, prm);
    frame_handoff<D, S, false>(fr, x, n, prm, m);
}

// The unit columns that a deferring frame's pending values belong to, kept while a window advances W: read again
// only when the window fails. Frames of more than four entries keep them in local memory, out of the registers.
template <bool DEFER, int N, typename Real> struct Kept {
    __device__ __forceinline__ void take(const Real*) {}
};
template <int N, typename Real> struct Kept<true, N, Real> {
    Real U[N];
    __device__ __forceinline__ void take(const Real* W) {
#pragma unroll
        for (int l = 0; l < N; ++l) U[l] = W[l];
        if (N > 4) asm volatile("" ::"l"(U) : "memory");
    }
};
template <bool DEFER, class FR, class KE>
__device__ __forceinline__ void frame_values(FR& fr, const KE& kept) {
    if constexpr (DEFER) {
        if (fr.pend) {
            constexpr int N = sizeof(fr.W) / sizeof(fr.W[0]);
            double V[N];
#pragma unroll
            for (int l = 0; l < N; ++l) V[l] = fr.pend_here ? fr.W[l] : kept.U[l];
            fr.st.value(V, fr.pend);
        }
    }
}

// ---- the kernel ------------------------------------------------------------------------------------------------------
// MINB is the register budget as resident blocks of 128 threads per SM (1: no cap); the tuner picks it per run.
template <class Sys, typename Real, class F0, class F1, class F2, int NF, int MINB>
__global__ void __launch_bounds__(128, MINB) orbit_kernel(const KArgs a, const Sys sys) {
    constexpr int D = Sys::D, S = Sys::S;
    const i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const bool fresh = a.n0 == 0;
    const i64 xso = a.soa ? 1 : S, xsc = a.soa ? a.n : 1;

    double x[S];
    const double* xin = a.x_in;
#pragma unroll
    for (int c = 0; c < S; ++c) x[c] = xin[i * xso + c * xsc];

    FrameRegs<D, Real, F0> fr0;
    FrameRegs<D, Real, F1> fr1;
    FrameRegs<D, Real, F2> fr2;
    frame_load<D, S>(fr0, 0, a, i, fresh);
    if (NF > 1) frame_load<D, S>(fr1, 1, a, i, fresh);
    if (NF > 2) frame_load<D, S>(fr2, 2, a, i, fresh);
    const bool any0 = fr0.alive || (NF > 1 && fr1.alive) || (NF > 2 && fr2.alive);
    if (!any0) return;   // frozen since an earlier launch: nothing is rewritten

    // Float64 frames leave SALI's and GALI's values to the last handoff; maps of dimension 2 evaluate the next step's
    // sine and cosine beside the handoff, whose quotients and roots it does not depend on (one block of straight-line
    // code, so the two chains of dependent operations overlap).
    constexpr bool f64 = sizeof(Real) == 8;
    constexpr bool D0 = f64 && F0::defers, D1 = f64 && NF > 1 && F1::defers, D2 = f64 && NF > 2 && F2::defers;
    constexpr bool AHEAD = D == 2 && NF == 1;
    Kept<D0, D * F0::K, Real> k0;
    Kept<D1, D * F1::K, Real> k1;
    Kept<D2, D * F2::K, Real> k2;
    typename Sys::template JacR<Real> J;
    auto advance = [&]() {
        if (NF == 1 || fr0.alive) sys.template apply<F0::K>(J, fr0.W);
        if (NF > 1 && fr1.alive) sys.template apply<F1::K>(J, fr1.W);
        if (NF > 2 && fr2.alive) sys.template apply<F2::K>(J, fr2.W);
        sys.forward(x, J);
    };
    if (AHEAD) sys.jac(x, J);
    i64 n = a.n0;
    const i64 handoffs = a.steps / a.tau;
    for (i64 h = 0; h < handoffs; ++h) {
        // a stopped frame's W no longer holds unit columns: its last ones stay kept while the other frames run on
        if (NF == 1 || fr0.alive) k0.take(fr0.W);
        if (NF > 1 && fr1.alive) k1.take(fr1.W);
        if (NF > 2 && fr2.alive) k2.take(fr2.W);
        for (int t = AHEAD ? 1 : 0; t < a.tau; ++t) {
            if (!AHEAD) sys.jac(x, J);
            advance();
            if (AHEAD) sys.jac(x, J);
        }
        if (AHEAD) { advance(); sys.jac(x, J); }
        n += a.tau;
        {
            typename F0::template Measure_<D, Real> m0;
            m0.take(fr0.W, a.prm[0]);
            frame_handoff<D, S, D0>(fr0, x, n, a.prm[0], m0);
        }
        if (NF > 1) {
            typename F1::template Measure_<D, Real> m1;
            m1.take(fr1.W, a.prm[1]);
            frame_handoff<D, S, D1>(fr1, x, n, a.prm[1], m1);
        }
        if (NF > 2) {
            typename F2::template Measure_<D, Real> m2;
            m2.take(fr2.W, a.prm[2]);
            frame_handoff<D, S, D2>(fr2, x, n, a.prm[2], m2);
        }
        const bool any = fr0.alive || (NF > 1 && fr1.alive) || (NF > 2 && fr2.alive);
        if (!any) break;
    }
    frame_values<D0>(fr0, k0);
    if (NF > 1) frame_values<D1>(fr1, k1);
    if (NF > 2) frame_values<D2>(fr2, k2);
    // orbit.jl:58: the final status check runs only at step N
    if (fr0.alive) { fr0.code = n == a.N ? (all_finite_x<D, S>(x) ? (all_finite<D * F0::K>(fr0.W) ? STATUS_OK : STATUS_W) : STATUS_STATE) : STATUS_OK; fr0.hstep = n; }
    if (NF > 1 && fr1.alive) { fr1.code = n == a.N ? (all_finite_x<D, S>(x) ? (all_finite<D * F1::K>(fr1.W) ? STATUS_OK : STATUS_W) : STATUS_STATE) : STATUS_OK; fr1.hstep = n; }
    if (NF > 2 && fr2.alive) { fr2.code = n == a.N ? (all_finite_x<D, S>(x) ? (all_finite<D * F2::K>(fr2.W) ? STATUS_OK : STATUS_W) : STATUS_STATE) : STATUS_OK; fr2.hstep = n; }

#pragma unroll
    for (int c = 0; c < S; ++c) a.x_out[i * xso + c * xsc] = x[c];
    const bool was0 = fresh || a.code[0][i] == STATUS_OK;
    if (was0) frame_store<D, S>(fr0, 0, a, i);
    if (NF > 1) { const bool was = fresh || a.code[1][i] == STATUS_OK; if (was) frame_store<D, S>(fr1, 1, a, i); }
    if (NF > 2) { const bool was = fresh || a.code[2][i] == STATUS_OK; if (was) frame_store<D, S>(fr2, 2, a, i); }
}

// A placeholder frame for unused slots (never loaded, stepped or stored).
using NoFrame = Frame<1>;

}  // namespace cl
