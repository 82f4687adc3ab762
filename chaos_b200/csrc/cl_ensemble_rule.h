// cl_ensemble_rule.h -- which variant of its kernels an ensemble class takes: host code without CUDA, so that the rule can
// be tested anywhere.
#pragma once

#include <cstdint>

#include "../../include/chaoslab_b200.h"

namespace cl {

struct ETune { int block, minb, unroll, lanes; };   // lanes: per orbit (1 = one orbit per thread)

// Lanes per orbit of the cooperative form of a run (the lattice's site count), or 1 when it has none.
inline int coop_lanes(const cl_run& r) {
    if (r.sys.kind != CL_SYS_CHAIN || r.n_frames != 1) return 1;
    const cl_frame& f = r.frames[0];
    if (f.n_reducers != 1 || f.reducers[0].kind != CL_RED_QR || f.reducers[0].alg != CL_QR_HOUSEHOLDER) return 1;
    const int ns = r.d / 2;
    if ((ns != 2 && ns != 4 && ns != 8) || f.k % ns != 0) return 1;
    return ns;
}

// An untuned class of 4 or 8 sites takes the cooperative kernel (one orbit per 4 or 8 lanes), whose longest orbit
// finishes several times sooner: at 10000 orbits a class and lengths to 1e5 (ms, one orbit per thread / cooperative)
// d = 16 Float64 807 / 146, mixed 390 / 69; d = 8 Float64 602 / 197, mixed 127 / 115; the four classes together 415 / 145
// mixed and 1043 / 249 Float64. It also carries the larger load of 65536 orbits a class, lengths to 2e4 (d = 16 Float64
// 301 / 179, mixed 93 / 74; d = 8 Float64 137 / 103), but for d = 8 in mixed precision (31 / 40), whose frame fits one
// thread's registers: that one goes back to a thread per orbit when those fill a block of every SM.
inline bool coop_by_default(const cl_ensemble_class& c, int sms) {
    const int lanes = coop_lanes(c.run);
    if (lanes < 4 || !c.buf.W0[0]) return false;
    return lanes > 4 || c.run.precision == CL_PREC_FP64 || c.n_orbits <= 128 * static_cast<int64_t>(sms);
}

// The settings of a class nobody tuned, in the form that runs it: such a class may ask for the one-thread kernel (lanes = 1).
inline ETune untuned_variant(const cl_ensemble_class& c, int sms, bool beside) {
    ETune t{128, 2, 1, 1};
    if (!coop_by_default(c, sms)) return t;
    const int lanes = coop_lanes(c.run);
    const bool coop = c.lanes != 1;
    if (coop) {
        t.lanes = lanes;
        // the window unrolled at the compiled tau: mixed d = 16 80 -> 69 ms, Float64 146 -> 184 (one orbit per thread, 2500
        // orbits to 2e4, mixed d = 8 26 -> 76, d = 16 77 -> 95)
        if (c.run.precision != CL_PREC_FP64) t.unroll = c.run.tau;
    }
    // One block an SM while the class is a few rounds of them: the longest orbits set its time, and a second block beside
    // theirs slows them. Up to 8 rounds beside other classes, which take the room (two blocks of these kernels fill an
    // SM's registers; 10000 orbits a class 142 against 145 ms; 65536 a class 209 against 131), and for one orbit per
    // thread (18000 orbits to 2e4, ms at one / two blocks: mixed d = 8 25 / 32, d = 16 78 / 85, Float64 120 / 121, 169 /
    // 250). A cooperative class alone up to 5 (d = 16, lengths to 1e5: 4.6 rounds mixed 71 / 79, Float64 147 / 174; 5.5 85 /
    // 81, 176 / 176; 6.3 98 / 80, 202 / 177; lengths to 2e4: 3.0 14.5 / 16.7, 29.8 / 35.3; 3.8 18.1 / 16.8, 36.2 / 35.4;
    // 6.3 29.6 / 18.1, 61.6 / 38.9).
    if (c.n_orbits * lanes <= (coop && !beside ? 5 : 8) * 128 * static_cast<int64_t>(sms)) t.minb = 1;
    return t;
}

// t (tuned or not) with what the class itself asks for, as far as its kernels have it
inline ETune asked_variant(const cl_ensemble_class& c, ETune t) {
    if (c.minb > 0) t.minb = c.minb;
    if (c.unroll > 0) t.unroll = c.unroll;
    if (c.lanes > 0) t.lanes = c.lanes;
    if (t.unroll != 1 && t.unroll != c.run.tau) t.unroll = 1;
    if (t.lanes > 1 && (t.lanes != coop_lanes(c.run) || !c.buf.W0[0])) t.lanes = 1;
    return t;
}

}  // namespace cl
