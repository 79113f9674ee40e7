// What the softmax warps of the tcgen05 attention kernels share.  A tile of 64 scores a thread is bound by its 64
// exponentials (four a cycle and scheduler: 512 cycles), so everything else is done two values or three operands an
// instruction: 32 maxima, 32 multiply-adds, 32 additions, 32 conversions.  (One value each, a tile took 1,175 cycles for a
// block alone on its SM and 1,400 for two; with this 2,048 tokens of 28 / 4 heads of 128 went from 43.6 to 38.9 us, the
// other changes of the attention kernel among them.)
#pragma once

#include "common.cuh"

namespace slb_softmax {

__device__ __forceinline__ uint64_t pair_bits(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 pair_of(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// 2^x in one instruction (exp2f adds a range fix-up around it; the probabilities here are rounded to bfloat16 anyway,
// and -inf gives 0)
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}

// scores outside [lo, hi) become -inf; all of the warp's threads call it
__device__ __forceinline__ void mask_keys(float (&s)[64], int lo, int hi) {
#pragma unroll
    for (int i = 0; i < 64; ++i) s[i] = i < hi ? s[i] : -INFINITY;
    if (__any_sync(0xffffffffu, lo > 0)) {
#pragma unroll
        for (int i = 0; i < 64; ++i) s[i] = i >= lo ? s[i] : -INFINITY;
    }
}
__device__ __forceinline__ float max_of(const float (&s)[64]) {
    float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};       // four chains, not one
#pragma unroll
    for (int i = 0; i < 64; i += 2) m[(i >> 1) & 3] = max3(m[(i >> 1) & 3], s[i], s[i + 1]);
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}
// packed[i] = bfloat16 of 2^(s scale - ref) for two neighbouring scores; their float32 sum is returned
__device__ __forceinline__ float exponentials(const float (&s)[64], float scale, float ref, uint32_t (&packed)[32]) {
    const uint64_t sc = pair_bits(scale, scale), off = pair_bits(-ref, -ref);
    uint64_t sum[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const float2 x = pair_of(fma2(pair_bits(s[2 * i], s[2 * i + 1]), sc, off));
        const float p0 = fast_exp2(x.x), p1 = fast_exp2(x.y);
        sum[i & 3] = add2(sum[i & 3], pair_bits(p0, p1));
        packed[i] = pack2(p0, p1);
    }
    const float2 t = pair_of(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])));
    return t.x + t.y;
}

}  // namespace slb_softmax
