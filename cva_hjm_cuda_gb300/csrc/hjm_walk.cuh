// hjm_walk.cuh -- the convection step as a random walk: the operand tables'
// closed form (hjm_contract.cu, hjm_mresp.cu).
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "hjm_device.cuh"

namespace hjm {

// The step as a walk.  One step moves the curve by h[t] <- a0 h[t] + a1 h[t+1]
// + a2 h[t+2] (Euler: 1 - c, c, 0; the predictor-corrector: 1 - c + c^2/2,
// c - c^2, c^2/2) up to the last tenors, whose rows use the backward difference
// d = h[L] - h[L-1].  That slope does not change over a step, so the rows are
// the same walk on the curve extended beyond L along d, and with D_t the
// loading's deviation from that line (zero from L - 1 on)
//     (A^m S)[j] = S_L + (j - L + m c) d + sum_i f_m(i) D_{j+i},
// f_m(i) the probability that m steps move i tenors.  Every lag is then
// independent of the others: a few launches of thousands of threads instead of
// a recursion over the lags, which is serial and bound by the FP64 pipe's
// latency (2,450 lags of the 25y swap: 1.2 ms by one CTA; 40 us this way).
struct WalkParams {
    double a1, a2;          // r = a / a0 of the recurrence: see below
    double log_hi, log_lo;  // log a0
    double b2, inv;         // a2 / (a1 + a2), 1 / (a1 + a2)
    double rcp[kMaxTenor];  // 1 / (i + 1)
};

inline WalkParams walk_params(double c, bool pc)
{
    WalkParams K;
    const double a0 = pc ? 1.0 - c + 0.5 * c * c : 1.0 - c, a1 = pc ? c - c * c : c, a2 = pc ? 0.5 * c * c : 0.0;
    const long double cl = c, log_a0 = pc ? log1pl(-cl + 0.5L * cl * cl) : log1pl(-cl);
    K.log_hi = (double)log_a0;
    K.log_lo = (double)(log_a0 - (long double)K.log_hi);
    K.a1 = a1 / a0;
    K.a2 = a2 / a0;
    K.b2 = a2 / (a1 + a2);
    K.inv = 1.0 / (a1 + a2);
    for (int i = 0; i < kMaxTenor; ++i) K.rcp[i] = 1.0 / (double)(i + 1);
    return K;
}

// a0^e: the exponent's rounding would cost e log a0 2^-53
__device__ __forceinline__ double walk_power(const WalkParams& K, double e)
{
    const double x = e * K.log_hi;
    return exp(x) * (1.0 + fma(e, K.log_lo, fma(e, K.log_hi, -x)));
}

}  // namespace hjm
