// Pointwise functions of the Gated DeltaNet kernels.
#pragma once

#include <cuda_runtime.h>

namespace b200 {

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
// SiLU on the special-function unit (ex2.approx + rcp.approx, about 2 ulp): the sequence-form conv kernel evaluates it
// 6144 times per token and is otherwise bound by these instructions, not by memory.
__device__ __forceinline__ float silu_fast(float x) { return __fdividef(x, 1.0f + __expf(-x)); }
// The same in five instructions (subnormal operands flushed, the quotient as a product with the reciprocal).
__device__ __forceinline__ float silu_sfu(float x) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return x * r;
}
__device__ __forceinline__ float softplus_f(float x) { return x > 20.0f ? x : logf(1.0f + expf(x)); }

}  // namespace b200
