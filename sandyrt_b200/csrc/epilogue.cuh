// Epilogue arithmetic shared by the matrix-product kernels: bias, activation, residual.
#pragma once

#include "common.cuh"

enum SandyAct : int { SANDY_ACT_NONE = 0, SANDY_ACT_GELU_TANH = 1, SANDY_ACT_GELU_ERF = 2, SANDY_ACT_RELU_SQUARED = 3 };

// gelu_new, in the reference's order of operations (src/ir/BuiltinLowering.cpp:116-140):
//   x2 = u*u; x3 = x2*u; inner = u + 0.044715*x3; t = tanh(0.7978845608028654*inner);
//   (0.5*u) * (1 + t)
__device__ __forceinline__ float gelu_tanh(float u) {
    const float x2 = u * u;
    const float x3 = x2 * u;
    const float inner = u + 0.044715f * x3;
    const float t = tanhf(0.7978845608028654f * inner);
    return (0.5f * u) * (1.0f + t);
}

// Exact gelu: 0.5*u*(1 + erf(u / sqrt(2))).  The reference has no erf op
// (ScalarOp list, src/ir/KernelIR.h:317-337); this follows the formula.
__device__ __forceinline__ float gelu_erf(float u) {
    return 0.5f * u * (1.0f + erff(u * 0.70710678118654752440f));
}

// gelu_new as u / (1 + exp(-2 y)), y = 0.79788456 (u + 0.044715 u^3), which is the formula above with tanh written out: two
// special-function instructions and five others (with 1 - 2 / (exp(2 y) + 1) for tanh, __expf and __fdividef, twice as many, a
// product of 2,048 x 3,072 x 768 took 16.2 us, with this 14.2).  The absolute error stays below 6e-7.  The relative
// one is that of the exponential's argument, rounded to a float, times the argument: below 1e-6 down to u = -4, 2e-6 to -5, 4e-6 to -7,
// 1e-5 to -10, below which the result is less than 1e-22.  For write-backs that round to bfloat16 or sit in a
// tensor-core kernel's critical path; the 32-bit path keeps tanhf.
__device__ __forceinline__ float gelu_tanh_fast(float u) {
    // exp(-2 y) = 2^(u (c1 + c3 u^2)), c1 = -2 * 0.79788456 * log2(e), c3 = 0.044715 c1
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(u * fmaf(-0.10294324f, u * u, -2.3022082f)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return u * r;
}

// relu(u)^2
__device__ __forceinline__ float relu_squared(float u) {
    u = fmaxf(u, 0.0f);
    return u * u;
}

__device__ __forceinline__ float apply_act_fast(float v, int act) {
    if (act == SANDY_ACT_GELU_TANH) return gelu_tanh_fast(v);
    if (act == SANDY_ACT_GELU_ERF) return gelu_erf(v);
    if (act == SANDY_ACT_RELU_SQUARED) return relu_squared(v);
    return v;
}

__device__ __forceinline__ float apply_act(float v, int act) {
    if (act == SANDY_ACT_GELU_TANH) return gelu_tanh(v);
    if (act == SANDY_ACT_GELU_ERF) return gelu_erf(v);
    if (act == SANDY_ACT_RELU_SQUARED) return relu_squared(v);
    return v;
}
