// cl_pipe.cuh -- the orbit kernel of small ensembles of the two-dimensional maps as a pipeline of five warps per 32
// orbits. One thread per orbit leaves most schedulers without a warp when there are few orbits (4096 orbits are 128
// warps for 592 schedulers), and a step's time is then one thread's instruction stream: the map (about 130
// instructions), the frame's way to the next step (250) and everything that only the records need (300). Here each part
// is a warp's, and an SM's four schedulers share them:
//   warp 0     the point: sine and cosine, forward; hands on the tangent entry of every step and the point at handoffs
//   warp 1     the frame: tangent product and, at a handoff, only what the frame continues as (the orthonormal factor,
//              the unit columns); hands on the frame as it arrives at each handoff
//   warps 2, 3 the measures (Measure: factorisation, norms, logarithms) of the arriving frames, alternate handoffs
//   warp 4     the records: frame_handoff, the one-thread kernel's code, on the arriving frame and its measures; owns the
//              status, the reducer states, the final frame and the stores
// Warp 1 continues a frame by the very operations warps 2-4 perform on it, so they agree bit for bit while an orbit
// runs; once warp 4 has stopped an orbit, what the others compute for it is not looked at. The warps work on blocks of
// PIPE_STEPS steps, each one block behind the one before it, and meet at a barrier after each block.
// Wrapped standard map, MGS, tau = 1, 4736 orbits x 1000 steps: 0.96 -> 0.63 ms; standard map, Householder, tau = 4 0.31 ->
// 0.21, MEGNO + FLI + SALI 1.21 -> 0.97 (there warp 4's sums are the longest). The line is two blocks an SM, which its
// registers hold: 9472 orbits 0.96 -> 0.70 ms, 14208 orbits 0.97 against 1.41 the other way. Every chain gains at the line
// (standard map, 9472 x 1000, one orbit a thread / pipeline, tau = 1 | tau = 4): MGS .94/.70 | .33/.26, CGS .94/.70 |
// .32/.25, Householder .91/.64 | .32/.25, Givens .75/.50 | .28/.20, SALI .85/.57 | .30/.22, MEGNO 1.00/.73 | .34/.27, FLI
// .81/.59 | .29/.22, MEGNO + SALI 1.11/.90 | .37/.31, FLI + SALI .95/.69 | .33/.25, MEGNO + FLI + SALI 1.22/1.05 | .40/.38.
// Above tau = PIPE_STEPS the handoffs are too few for the split to pay.
#pragma once

#include <type_traits>

#include "cl_kernel.cuh"

namespace cl {

constexpr i64 PIPE_ORBITS = 9472;   // 2 x 148 x 32
constexpr int PIPE_STEPS = 4;   // steps a block at most: whole handoffs

// What a chain leaves as the frame: its last reducer's, when the earlier ones replace nothing and the last has a
// straight-line form here.
template <class... Rs> struct PipeLast { static constexpr bool ok = false; using R = void; };
template <class R_> struct PipeLast<R_> {
    using R = R_;
    template <int D, int K> static constexpr bool fits() {
        return R_::replaces && ((R_::pair && K == 2) || (R_::alg != 0 && qr_fast_v<R_::alg, D, K>));
    }
};
template <class R1, class R2, class... Rs> struct PipeLast<R1, R2, Rs...> {
    using R = typename PipeLast<R2, Rs...>::R;
    template <int D, int K> static constexpr bool fits() { return !R1::replaces && PipeLast<R2, Rs...>::template fits<D, K>(); }
};
template <class F> struct PipeFrame { static constexpr bool ok = false; };
template <int KK, class R1, class... Rs> struct PipeFrame<Frame<KK, R1, Rs...>> {
    using Last = PipeLast<R1, Rs...>;
    using R = typename Last::R;
    static constexpr int at = sizeof...(Rs);   // its place in the chain
    using M = Measure<2, KK, double, R1, Rs...>;
    static constexpr bool ok = Last::template fits<2, KK>() && M::qr != M::pair;   // one kind of measure between the warps
};
template <class Sys, typename Real, class F, int NF> struct PipeOf {
    static constexpr bool sys = std::is_same<Sys, SysStandard>::value || std::is_same<Sys, SysWrapped>::value;
    static constexpr bool ok = sys && sizeof(Real) == 8 && NF == 1 && PipeFrame<F>::ok;
};

// The frame after a handoff
template <class R, int D, int K>
__device__ __forceinline__ void pipe_next(double* W, double tol) {
    Ok ok;
    double V[D * K];
    if constexpr (R::pair) {
        double a[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            double y;
            a[j] = norm64r<D>(W + j * D, ok, y);
            ok.divisor(a[j]);
#pragma unroll
            for (int i = 0; i < D; ++i) { ok.dividend(W[i + j * D]); V[i + j * D] = quo64(W[i + j * D], a[j], y); }
        }
        if (!ok.ok) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                a[j] = nrm<D>(W + j * D);
#pragma unroll
                for (int i = 0; i < D; ++i) V[i + j * D] = W[i + j * D] / a[j];
            }
        }
    } else {
        double RR[K * K], rin[K];
        if constexpr (R::alg == CL_QR_HOUSEHOLDER) householder64<D, K>(W, V, RR, rin, ok);
        else if constexpr (R::alg == CL_QR_GIVENS) givens64<D, K>(W, V, RR, rin, ok);
        else gs64<R::alg, D, K>(W, V, RR, rin, ok);
        if (!ok.ok) {   // the general step on a state and a frame of its own (only this branch keeps them in memory)
            typename R::template State<D, K> st;
            uint64_t* w = reinterpret_cast<uint64_t*>(&st);
#pragma unroll
            for (int l = 0; l < static_cast<int>(sizeof(st) / 8); ++l) w[l] = 0;
            double V2[D * K];
#pragma unroll
            for (int l = 0; l < D * K; ++l) V2[l] = W[l];
            R::template general_out<D, K>(&st, 1, V2, tol);
#pragma unroll
            for (int l = 0; l < D * K; ++l) V[l] = V2[l];
        }
    }
#pragma unroll
    for (int l = 0; l < D * K; ++l) W[l] = V[l];
}

// A measure as Float64 words and a flag between the warps
template <class M, int D, int K>
struct PipeWords {
    static constexpr int n = M::qr ? D * K + K + 2 : 6;
    template <class Put> static __device__ __forceinline__ bool put(const M& m, Put&& to) {
        if constexpr (M::qr) {
#pragma unroll
            for (int l = 0; l < D * K; ++l) to(l, m.q.Q[l]);
#pragma unroll
            for (int j = 0; j < K; ++j) to(D * K + j, m.q.lg[j]);
            to(D * K + K, m.q.Gw);
            to(D * K + K + 1, m.q.orth);
            return m.q.ok;
        } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) { to(j, m.p.a[j]); to(2 + j, m.p.y[j]); to(4 + j, m.p.lg[j]); }
            return m.p.ok;
        }
    }
    template <class Get> static __device__ __forceinline__ void get(M& m, bool ok, Get&& from) {
        if constexpr (M::qr) {
#pragma unroll
            for (int l = 0; l < D * K; ++l) m.q.Q[l] = from(l);
#pragma unroll
            for (int j = 0; j < K; ++j) m.q.lg[j] = from(D * K + j);
            m.q.Gw = from(D * K + K);
            m.q.orth = from(D * K + K + 1);
            m.q.count = 1;   // one pass, one reflector or one rotation at D = 2
            m.q.ok = ok;
        } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) { m.p.a[j] = from(j); m.p.y[j] = from(2 + j); m.p.lg[j] = from(4 + j); }
            m.p.ok = ok;
        }
    }
};

// What the warps hand on, and the parts of warps 0 to 3 for one block of steps. JACS: the tangent entries at the handoffs'
// points go along with them (the recorder's monitor).
template <int D, int S, int K, int MN, bool JACS>
struct PipeShared {
    static constexpr int B = PIPE_STEPS;
    double sc[2][B][32];             // the tangent entry of each step: warp 0 -> 1
    double sx[4][B][S][32];          // the point at each handoff: warp 0 -> 4, three blocks later
    double sw[3][B][D * K][32];      // the arriving frame at each handoff: warp 1 -> 2, 3 and 4
    double sm[2][B][MN][32];         // its measures: warps 2, 3 -> 4
    double sj[JACS ? 4 : 1][JACS ? B : 1][JACS ? 32 : 1];   // the tangent entry at each handoff's point: warp 0 -> 4
    int sok[2][B][32];
    int running;
};

template <class Sys, class R, class M, int K, bool JACS>
struct PipeParts {
    static constexpr int D = Sys::D, S = Sys::S;
    using MW = PipeWords<M, D, K>;
    using Shared = PipeShared<D, S, K, MW::n, JACS>;
    // warp 0: the points of block p
    static __device__ __forceinline__ void points(Shared& sh, const Sys& sys, double* x, StdJac& J, i64 p, int hs, int tau, int lane) {
        int t = 0;
        for (int h = 0; h < hs; ++h) {
            for (int q = 0; q < tau; ++q, ++t) {
                sh.sc[p & 1][t][lane] = J.c;
                sys.forward(x, J);
                sys.jac(x, J);
            }
#pragma unroll
            for (int q = 0; q < S; ++q) sh.sx[p & 3][h][q][lane] = x[q];
            if constexpr (JACS) sh.sj[p & 3][h][lane] = J.c;
        }
    }
    // warp 1: the frames of block b
    static __device__ __forceinline__ void frames(Shared& sh, const Sys& sys, double* W, double tol, i64 b, int hs, int tau, int lane) {
        int t = 0;
        for (int h = 0; h < hs; ++h) {
            for (int q = 0; q < tau; ++q, ++t) {
                StdJac Jt;
                Jt.s = 0.0;
                Jt.c = sh.sc[b & 1][t][lane];
                sys.template apply<K>(Jt, W);
            }
#pragma unroll
            for (int l = 0; l < D * K; ++l) sh.sw[b % 3][h][l][lane] = W[l];
            pipe_next<R, D, K>(W, tol);
        }
    }
    // warps 2 and 3: the measures of block b's handoffs h0 and h0 + 2
    static __device__ __forceinline__ void measures(Shared& sh, const RedParams* prm, i64 b, int hs, int h0, int lane) {
        auto take = [&](int h, M& m) {
            double W[D * K];
#pragma unroll
            for (int l = 0; l < D * K; ++l) W[l] = sh.sw[b % 3][h][l][lane];
            m.take(W, prm);
        };
        auto put = [&](int h, const M& m) {
            sh.sok[b & 1][h][lane] = MW::put(m, [&](int l, double v) { sh.sm[b & 1][h][l][lane] = v; });
        };
        M m0, m1;
        if (h0 + 2 < hs) {   // both of this warp's handoffs side by side
            take(h0, m0);
            take(h0 + 2, m1);
            put(h0, m0);
            put(h0 + 2, m1);
        } else if (h0 < hs) {
            take(h0, m0);
            put(h0, m0);
        }
    }
    // warp 4: what arrives at handoff h of block b
    static __device__ __forceinline__ void arrive(const Shared& sh, double* W, double* x, M& m, i64 b, int h, int lane) {
#pragma unroll
        for (int l = 0; l < D * K; ++l) W[l] = sh.sw[b % 3][h][l][lane];
#pragma unroll
        for (int q = 0; q < S; ++q) x[q] = sh.sx[b & 3][h][q][lane];
        MW::get(m, sh.sok[b & 1][h][lane] != 0, [&](int l) { return sh.sm[b & 1][h][l][lane]; });
    }
};

template <class Sys, class F>
__global__ void __launch_bounds__(160, 2) pipe_kernel(const KArgs a, const Sys sys) {
    constexpr int D = Sys::D, S = Sys::S, K = F::K, B = PIPE_STEPS;
    using R = typename PipeFrame<F>::R;
    using M = typename F::template Measure_<D, double>;
    using P = PipeParts<Sys, R, M, K, false>;
    static_assert(M::qr != M::pair, "one kind of measure");
    constexpr bool DEFER = F::defers;
    __shared__ typename P::Shared sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const i64 orbit = static_cast<i64>(blockIdx.x) * 32 + lane;
    const bool mine = orbit < a.n;
    const i64 i = mine ? orbit : a.n - 1;       // spare lanes follow the last orbit and store nothing
    const bool fresh = a.n0 == 0;
    const i64 xso = a.soa ? 1 : S, xsc = a.soa ? a.n : 1;

    // handoffs a block (B tau <= PIPE_STEPS steps, or one handoff), blocks of the launch
    const int H = a.tau < B ? B / a.tau : 1;
    const i64 handoffs = a.steps / a.tau, blocks = (handoffs + H - 1) / H;
    auto in_block = [&](i64 b) { return static_cast<int>(min(static_cast<i64>(H), handoffs - b * H)); };

    double x[S];
    StdJac J;
#pragma unroll
    for (int q = 0; q < S; ++q) x[q] = a.x_in[i * xso + q * xsc];
    FrameRegs<D, double, F> fr;
    if (warp == 1 || warp == 4) frame_load<D, S>(fr, 0, a, i, fresh);
    const bool was = warp == 4 && mine && (fresh || fr.alive);   // not frozen since an earlier launch
    Kept<DEFER, D * K, double> kept;
    if (warp == 0) sys.jac(x, J);
    if (threadIdx.x == 0) sh.running = 1;
    i64 n = a.n0;
    __syncthreads();

    for (i64 p = 0; p < blocks + 3; ++p) {
        if (warp == 0) {
            if (p < blocks) P::points(sh, sys, x, J, p, in_block(p), a.tau, lane);
        } else if (warp == 1) {
            const i64 b = p - 1;
            if (b >= 0 && b < blocks)
                P::frames(sh, sys, fr.W, a.prm[0][PipeFrame<F>::at].orthogonality_tol, b, in_block(b), a.tau, lane);
        } else if (warp < 4) {
            const i64 b = p - 2;
            if (b >= 0 && b < blocks) P::measures(sh, a.prm[0], b, in_block(b), warp - 2, lane);
        } else {
            const i64 b = p - 3;
            if (b >= 0) {
                const int hs = in_block(b);
                for (int h = 0; h < hs; ++h) {
                    n += a.tau;
                    if (!fr.alive) continue;
                    kept.take(fr.W);
                    M m;
                    P::arrive(sh, fr.W, x, m, b, h, lane);
                    frame_handoff<D, S, DEFER>(fr, x, n, a.prm[0], m);
                }
                const bool any = __any_sync(0xffffffffu, fr.alive);
                if (lane == 0) sh.running = any;
            }
        }
        __syncthreads();
        if (!sh.running) break;
        __syncthreads();   // `running` is read before the next block may write it
    }
    if (!was) return;
    frame_values<DEFER>(fr, kept);
    // orbit.jl:58: the final status check runs only at step N
    if (fr.alive) {
        fr.code = n == a.N ? (all_finite_x<D, S>(x) ? (all_finite<D * K>(fr.W) ? STATUS_OK : STATUS_W) : STATUS_STATE) : STATUS_OK;
        fr.hstep = n;
    }
#pragma unroll
    for (int q = 0; q < S; ++q) a.x_out[i * xso + q * xsc] = x[q];
    frame_store<D, S>(fr, 0, a, i);
}

}  // namespace cl
