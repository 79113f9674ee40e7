// The gated activations of feed-forwards, float32 arithmetic.
#pragma once

#include "common.cuh"

__device__ __forceinline__ float silu_mul(float g, float u) { return g / (1.0f + expf(-g)) * u; }
// 1 / x in one instruction (and the scaling of the ends of its range), within one unit of the last place
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 1 / (1 + e^-z) for results of type T: rounded to bfloat16, from the hardware exponential and reciprocal
template <typename T> __device__ __forceinline__ float sigmoid_for(float z) {
    return sizeof(T) == 2 ? rcp_approx(1.0f + __expf(-z)) : 1.0f / (1.0f + expf(-z));
}
// For results that are rounded to bfloat16: the hardware exponential and reciprocal (errors of
// a few 1e-7 relative, a thousand times below the rounding).  The correctly rounded reciprocal is a call a value:
// half of the time of a product's epilogue with it (13,200 cycles a tile of 256 tokens, tanh-GELU 6,500).
__device__ __forceinline__ float silu_mul_fast(float g, float u) {
    return g * rcp_approx(1.0f + __expf(-g)) * u;
}

// the tanh form of GELU: 0.5 z (1 + tanh(sqrt(2 / pi) (z + 0.044715 z^3)))
__device__ __forceinline__ float gelu_tanh_mul(float g, float u) {
    return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
}
// the clamped form: g = min(gate, limit), u = clamp(up, -limit, limit), g sigmoid(alpha g) (u + 1)
__device__ __forceinline__ float swish_clamped_mul(float g, float u, float limit, float alpha) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
}
// ACT 0: SiLU; 1: GELU (tanh form); 2: the clamped form with p0 = limit, p1 = alpha
template <int ACT> __device__ __forceinline__ float act_mul(float g, float u, float p0, float p1) {
    return ACT == 2 ? swish_clamped_mul(g, u, p0, p1) : ACT == 1 ? gelu_tanh_mul(g, u) : silu_mul(g, u);
}
template <int ACT> __device__ __forceinline__ float act_mul_fast(float g, float u, float p0, float p1) {
    return ACT == 2 ? swish_clamped_mul(g, u, p0, p1) : ACT == 1 ? gelu_tanh_mul(g, u) : silu_mul_fast(g, u);
}
// the same with the form as an argument
__device__ __forceinline__ float act_mul_of(int act, float g, float u, float p0, float p1) {
    return act == 2 ? swish_clamped_mul(g, u, p0, p1) : act == 1 ? gelu_tanh_mul(g, u) : silu_mul(g, u);
}
