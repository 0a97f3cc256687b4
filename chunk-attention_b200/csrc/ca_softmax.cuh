// One thread's row of a 64-token score tile, as tcgen05.ld leaves it (two halves of 32 columns): its maximum and its weights.
//
// The tcgen05 attention kernels keep two softmax warps on a scheduler, too few to hide a chain of dependent operations or to issue
// every cycle, so what counts is the length of a tile's chain and its instructions: maxima and sums go in four chains of 3-operand
// maxima and of pairs, products and differences in pairs of fp32 (two results per instruction, each rounded as the scalar one).
// 8192 tokens of one prompt, 32 heads on 8 of 128: 601 -> 586 us; the kernel of wide shared runs is as fast either way.
#pragma once
#include "ca_ptx.cuh"
#include "ca_types.cuh"

namespace ca {

__device__ __forceinline__ uint64_t pair_u32(uint32_t lo, uint32_t hi) { return pair_f32(__uint_as_float(lo), __uint_as_float(hi)); }

__device__ __forceinline__ float tile_max(const uint32_t (&s0)[32], const uint32_t (&s1)[32]) {
    float m[4];
#pragma unroll
    for (int k = 0; k < 4; k++) m[k] = fmaxf(__uint_as_float(s0[k]), __uint_as_float(s1[k]));
#pragma unroll
    for (int i = 4; i < 32; i++) m[i & 3] = fmaxf(fmaxf(m[i & 3], __uint_as_float(s0[i])), __uint_as_float(s1[i]));
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// s <- 2^(s * scale - m); the sum of the weights comes back
__device__ __forceinline__ float tile_weights(uint32_t (&s0)[32], uint32_t (&s1)[32], float scale, float m) {
    const uint64_t scale2 = pair_f32(scale, scale), minus_m = pair_f32(-m, -m);
    uint64_t sum[4];
#pragma unroll
    for (int i = 0; i < 32; i++) {
        uint32_t& a = i < 16 ? s0[2 * (i & 15)] : s1[2 * (i & 15)];
        uint32_t& b = i < 16 ? s0[2 * (i & 15) + 1] : s1[2 * (i & 15) + 1];
        float x, y;
        unpair_f32(fma_f32x2(pair_u32(a, b), scale2, minus_m), x, y);
        x = ptx::fast_exp2(x);
        y = ptx::fast_exp2(y);
        a = __float_as_uint(x);
        b = __float_as_uint(y);
        sum[i & 3] = i < 4 ? pair_f32(x, y) : add_f32x2(sum[i & 3], pair_f32(x, y));
    }
    float x, y;
    unpair_f32(add_f32x2(add_f32x2(sum[0], sum[1]), add_f32x2(sum[2], sum[3])), x, y);
    return x + y;
}

// 32 weights as bf16 pairs, and what their rounding left out
__device__ __forceinline__ void split_weights(const uint32_t (&s)[32], uint32_t* hi, uint32_t* lo) {
    const uint64_t minus_one = pair_f32(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
        hi[i] = *reinterpret_cast<const uint32_t*>(&h);
        float x, y;
        unpair_f32(fma_f32x2(pair_u32(hi[i] << 16, hi[i] & 0xffff0000u), minus_one, pair_u32(s[2 * i], s[2 * i + 1])), x, y);
        const __nv_bfloat162 l = __floats2bfloat162_rn(x, y);
        lo[i] = *reinterpret_cast<const uint32_t*>(&l);
    }
}

}  // namespace ca
