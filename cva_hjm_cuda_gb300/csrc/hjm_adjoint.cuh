// hjm_adjoint.cuh -- what the adjoint's kernels share (hjm_adjoint.cu,
// hjm_adjoint_run.cu).
#pragma once

#include <cuda_runtime.h>

#include "hjm_device.cuh"

namespace hjm {

constexpr int kAdjCta = 64;  // paths per CTA

__host__ __device__ inline size_t align128(size_t x) { return (x + 127) & ~(size_t)127; }

// Seeds of date i from its sampled forward x, discount factor D and cfbar.
__device__ __forceinline__ void date_seeds(const PathParams<float>& P, int i, double x, float D, float cfbar,
                                           float& xbar, float& abar)
{
    const float mm = (float)P.m;
    const float xf = (float)x;
    const float e = expf(xf / mm);
    const float L = mm * expm1f(xf / mm);
    const float pa = (float)P.payA[i], pbk = (float)P.payB[i];
    xbar = cfbar * D * pa * e;
    abar = -(float)P.dt * D * cfbar * (pa * L - pbk);
}

}  // namespace hjm
