// A lower bound of the Johnson-Cook thermal factor that takes no power: a
// particle whose equivalent stress lies below ylo times it cannot yield,
// where ylo bounds (A + B eps^n)(1 + C ln es) from below.
//
// tt = 1 - Ts^m with Ts in [0, 1]: Ts^m lies below its chord (m >= 1) or its
// tangent at Ts = 1 (m < 1), so tt >= c (1 - Ts) with c = min(m, 1).  The
// factor that the step computes, 1 - pow(Ts, m) in R, can be smaller than tt
// by an absolute error: pow is within 4 ulp (FP32) or 2 ulp (FP64) of a
// number of at most 1, and the subtraction rounds once more.  Near Ts = 1,
// where tt itself is of that size, no relative margin covers it, so the bound
// gives up 4 eps(R) of ylo; the relative margin (1e-4) is for the roundings
// that are relative to the result: of c, of the bound and of ylo tt.
#pragma once

#include <algorithm>
#include <cmath>
#include <limits>

#ifdef __CUDACC__
#define MPMB_HD __host__ __device__ __forceinline__
#else
#define MPMB_HD inline
#endif

namespace mpmb {

// ylo tt >= scale (1 - Ts) - slack; scale = slack = 0: no bound (m <= 0).
template <typename R> struct FlowBound {
    R scale, slack;
};

template <typename R> inline FlowBound<R> flow_bound(R ylo, double m) {
    if (!(m > 0.0)) return {R(0), R(0)};
    return {(R)((double)ylo * std::min(m, 1.0) * (1.0 - 1e-4)),
            (R)(4.0 * (double)std::numeric_limits<R>::epsilon() * (double)ylo)};
}

template <typename R> MPMB_HD R flow_bound_at(R scale, R slack, R Ts) {
    using std::fma;
    return fma(scale, R(1) - Ts, -slack);
}

}  // namespace mpmb
