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
// 1 / (1 + e^-z) for a result of type T that is rounded at once (a value that enters a float32 sum takes the other form):
// for bfloat16 from the hardware exponential and reciprocal.  The exponential's bound grows with its argument, 2 + 1.16 |z|
// units of the last place: 3e-7 at |z| = 1, 1.5e-6 at a z of -20, where a rounding to bfloat16 is 2e-3.  Errors of the rounded
// results against 64 bits, gates with a spread of 1, 6 and 20, with the full exponential and division / with this: sigmoid
// gates, norm then gate and convolutions with SiLU 1.654e-3 to 1.667e-3, the same to seven digits in every case.
template <typename T> __device__ __forceinline__ float sigmoid_for(float z) {
    return sizeof(T) == 2 ? rcp_approx(1.0f + __expf(-z)) : 1.0f / (1.0f + expf(-z));
}
template <typename T> __device__ __forceinline__ float silu_for(float z) {
    return sizeof(T) == 2 ? z * sigmoid_for<T>(z) : silu_mul(z, 1.0f);
}
// For results that are rounded to bfloat16: the hardware exponential and a correctly rounded reciprocal.
__device__ __forceinline__ float silu_mul_fast(float g, float u) {
    return g * __frcp_rn(1.0f + __expf(-g)) * u;
}
// The same with the hardware's reciprocal, for gate and up as float32 sums leave them (a product's result is rounded to
// bfloat16 before the form above sees it, 2e-3 of its value).  An epilogue of 256 tokens takes 13,200 cycles with the rounded
// reciprocal, 6,500 with tanh-GELU.
__device__ __forceinline__ float silu_mul_sums(float g, float u) {
    return g * sigmoid_for<bf16>(g) * u;
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
template <int ACT> __device__ __forceinline__ float act_mul_sums(float g, float u, float p0, float p1) {
    return ACT == 0 ? silu_mul_sums(g, u) : act_mul<ACT>(g, u, p0, p1);
}
// the same with the form as an argument
__device__ __forceinline__ float act_mul_of(int act, float g, float u, float p0, float p1) {
    return act == 2 ? swish_clamped_mul(g, u, p0, p1) : act == 1 ? gelu_tanh_mul(g, u) : silu_mul(g, u);
}
