// cl_monitor.cuh -- the recorders' non-raising monitor, RunMonitor (src/Experiments/run_record.jl:24-43): at each
// handoff the tangent M of the map at the orbit point and the running maxima of |det M - 1|, max|M' Omega M - Omega|
// and max|M|; never fails. Shared by the study recorder and the indicator recorder's kernels.
#pragma once

#include <type_traits>

#include "cl_registry.cuh"

namespace cl {

struct MonState { double det_max, symp_max, M_max; };
static_assert(sizeof(MonState) == 24, "MonState layout");

// The tangent M of the map at x, column-major 2 x 2: standard maps [[1 + K cos x, 1], [K cos x, 1]]
// (standard_map.jl:24-27 as the kernels build it), linear maps A.
template <class Sys>
__device__ __forceinline__ void dense_tangent(const Sys& sys, const double* x, double* M) {
    if constexpr (std::is_same<Sys, SysLinear<2>>::value) {
#pragma unroll
        for (int l = 0; l < 4; ++l) M[l] = sys.A[l];
    } else {
        StdJac J;
        sys.jac(x, J);
        const double o = 1.0;
        M[0] = o + J.c; M[1] = J.c; M[2] = o; M[3] = o;
    }
}

// Julia's max of two non-negative values, without a branch: NaN if either is NaN (two zeros are both +0)
__device__ __forceinline__ double max_nonneg(double x, double y) { return x >= y || x != x ? x : y; }

// RunMonitor's step (run_record.jl:37-40) on the tangent M: det of a 2 x 2 static matrix M[1] M[4] - M[3] M[2]; M' Omega
// M by the StaticArrays products (the fused chain; Omega's zeros and ones leave M' Omega = [-M[2] M[1]; -M[4] M[3]] for a
// finite M, and the point is finite here); Julia's NaN-propagating max.
__device__ __forceinline__ void monitor_tangent(const double* M, MonState& m) {
    const double edet = fabs((M[0] * M[3] - M[2] * M[1]) - 1.0);
    const double P[4] = {-M[1], -M[3], M[0], M[2]};
    const double Om[4] = {0.0, -1.0, 1.0, 0.0};
    double es = 0.0, mm = 0.0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            es = max_nonneg(es, fabs(fma(P[i + 2], M[1 + 2 * j], P[i] * M[2 * j]) - Om[i + 2 * j]));
            mm = max_nonneg(mm, fabs(M[i + 2 * j]));
        }
    m.det_max = max_nonneg(m.det_max, edet);
    m.symp_max = max_nonneg(m.symp_max, es);
    m.M_max = max_nonneg(m.M_max, mm);
}
template <class Sys>
__device__ __forceinline__ void monitor_step(const Sys& sys, const double* x, MonState& m) {
    double M[4];
    dense_tangent(sys, x, M);
    monitor_tangent(M, m);
}
// The same from the tangent entries J of the next step, which the recorders evaluate at this very point: a standard
// map's sine and cosine are taken once, not twice (mixed kernels hold a Float32 J and take their own).
template <class Sys, class J>
__device__ __forceinline__ void monitor_ahead(const Sys& sys, const double* x, const J& Jn, MonState& m) {
    if constexpr (std::is_same<J, StdJac>::value) {
        const double M[4] = {1.0 + Jn.c, Jn.c, 1.0, 1.0};
        monitor_tangent(M, m);
    } else {
        monitor_step(sys, x, m);
    }
}

}  // namespace cl
