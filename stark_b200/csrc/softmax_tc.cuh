// What the softmax warps of the two prompt-attention kernels do with a piece of 32 scores of one row (prefill_attention_tc.cu,
// layered_attention_tc.cu).
#pragma once
#include "device_math.cuh"

namespace sb {

__device__ inline float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Two f32 operations in one instruction, each rounded as the single one.
__device__ inline float2 fma_pair(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)), "l"(*reinterpret_cast<uint64_t *>(&c)));
    return *reinterpret_cast<float2 *>(&d);
}
__device__ inline float2 add_pair(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)));
    return *reinterpret_cast<float2 *>(&d);
}

// Scores of keys past `pos` become -inf: probabilities of exactly zero.  Only steps on the diagonal have any; the others pay one branch.
__device__ __forceinline__ void hide_keys(uint32_t (&v)[32], uint32_t key0, uint32_t pos) {
    if (key0 + 31u <= pos) return;
#pragma unroll
    for (uint32_t i = 0; i < 32u; ++i)
        if (key0 + i > pos) v[i] = 0xff800000u;
}

__device__ __forceinline__ float largest(const uint32_t (&v)[32]) {
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four chains
#pragma unroll
    for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
    return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}

// exp2(v * scale - top), as pairs of bf16 terms hi + lo (two roundings to nearest), and added to the row's sums.  exp2 of a non-positive
// argument: the hardware approximation is good to two units of an f32's last place, far inside what the bf16 pair keeps.
__device__ __forceinline__ void probabilities(const uint32_t (&v)[32], float scale, float top, float2 (&sums)[2], uint32_t (&hi)[16],
                                              uint32_t (&lo)[16]) {
    const float2 scale2 = make_float2(scale, scale), shift2 = make_float2(-top, -top), minus1 = make_float2(-1.0f, -1.0f);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 x = fma_pair(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), scale2, shift2);
        const float2 e = make_float2(ex2_approx(x.x), ex2_approx(x.y));
        sums[i & 1] = add_pair(sums[i & 1], e);
        hi[i] = f32x2_to_bf16x2(e.x, e.y);
        const float2 rest = fma_pair(make_float2(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u)), minus1, e);
        lo[i] = f32x2_to_bf16x2(rest.x, rest.y);
    }
}

}  // namespace sb
