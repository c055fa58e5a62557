// fp32_fast.cuh -- FP32 exponential and logarithm of the step loops, straight from
// the GPU's ex2 and lg2 with flushed subnormals: without the scaling that serves
// subnormal arguments and results, which cost 1 to 2 % of every FP32 kernel (a
// logarithm's argument here is a normal number; of a growth factor below 2^-126
// a path's sums see nothing).  What is evaluated once per path takes __expf,
// whose subnormal results count: a bumped state may multiply them by as much.
// Flushing whole files by --ftz=true was no faster, and took spots and strikes
// below 1.2e-38 for zero.
#pragma once

#include <cuda_runtime.h>

namespace mcdg {

__device__ __forceinline__ float fast_log2(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float fast_log(float x) { return fast_log2(x) * 0.693147181f; }  // ln 2

__device__ __forceinline__ float fast_exp(float x) {  // 2^(x / ln 2)
    const float y = x * 1.442695041f;
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return r;
}

}  // namespace mcdg
