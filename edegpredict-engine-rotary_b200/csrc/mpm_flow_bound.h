// A lower bound of the Johnson-Cook thermal factor that takes no power: a
// particle whose equivalent stress lies below ylo times it cannot yield,
// where ylo bounds (A + B eps^n)(1 + C ln es) from below.
//
// tt = 1 - Ts^m with Ts in [0, 1]: Ts^m lies below its chord (m >= 1) or its
// tangent at Ts = 1 (m < 1), so tt >= c (1 - Ts) with c = min(m, 1).  The
// factor that the step computes, 1 - pow(Ts, m) in R, can be smaller than tt
// by an absolute error: pow is within 4 ulp (FP32) or 2 ulp (FP64) of a
// number of at most 1, and the subtraction rounds once more, 4 eps(R) in all.
// Near Ts = 1, where tt itself is of that size, no relative margin covers it:
// the bound is c (kFlowTs - Ts) with kFlowTs = 1 - 2^-16, which gives up
// c 2^-16, at least 4 eps(FP32) for m >= 1/32 (no bound below that).  The
// relative margin (1e-4) is for the roundings that are relative to the result:
// of c, of the bound and of ylo tt.
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define MPMB_HD __host__ __device__ __forceinline__
#else
#define MPMB_HD inline
#endif

namespace mpmb {

constexpr double kFlowTs = 1.0 - 1.0 / 65536.0;

// ylo c with the margin: times kFlowTs - Ts it lies below ylo tt (0: no bound).
template <typename R> inline R flow_scale(R ylo, double m) {
    return m >= 1.0 / 32.0 ? (R)((double)ylo * std::min(m, 1.0) * (1.0 - 1e-4)) : R(0);
}

template <typename R> MPMB_HD R flow_bound(R scale, R Ts) { return scale * (R(kFlowTs) - Ts); }

}  // namespace mpmb
