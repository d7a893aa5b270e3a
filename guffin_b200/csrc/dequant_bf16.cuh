// Quantised weights to bf16 operands of the tensor core (shared memory of prefill.cu, HBM tiles of prompt.cu).
#pragma once

#include "common.cuh"

#include <cuda_bf16.h>

namespace gf {

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// Four consecutive K elements of column n of the B stage, starting at k (a multiple of four).
__device__ __forceinline__ void store_b4(uint8_t* stage, uint32_t n, uint32_t k, const float (&v)[4]) {
    uint8_t* dst = stage + (n >> 3) * 1024u + (k >> 3) * 128u + (n & 7u) * 16u + (k & 7u) * 2u;
    *reinterpret_cast<uint2*>(dst) = make_uint2(bf16_pair(v[0], v[1]), bf16_pair(v[2], v[3]));
}
__device__ __forceinline__ float half_bits(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }
__device__ __forceinline__ uint32_t byte_of(uint32_t word, uint32_t i) { return (word >> (8u * i)) & 0xffu; }

// ---- dequantisation of one column of one lane slot (column g + 8 * col of a column pair) for one block of
// 64 K elements: the reference's values exactly (quantization.cpp:457,517,590), then rounded to bf16.  `row`
// is the pair row (streaming layout, common.cuh), `n` the column inside the CTA tile.  A code byte becomes
// a float by a byte permute into the mantissa of 2^23 and one exact subtraction.

__device__ __forceinline__ float code_float(uint32_t word, uint32_t i, float bias) {      // byte i of word, minus (bias - 2^23)
    return __fsub_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u + i)), bias);
}

// The same two values at a time with the packed f32x2 instructions (each half rounds like the scalar
// instruction, so the values are bit for bit those of the scalar form): typedef and helpers as in gemv.cuh.
typedef unsigned long long pf2;
__device__ __forceinline__ pf2 pf2_make(float lo, float hi) {
    pf2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
    return r;
}
__device__ __forceinline__ pf2 pf2_mul(pf2 a, pf2 b) { pf2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ pf2 pf2_add(pf2 a, pf2 b) { pf2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint32_t pf2_bf16(pf2 v) {              // both halves rounded to bf16, low half in the low 16 bits
    uint32_t lo, hi, r;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "r"(hi), "r"(lo));
    return r;
}
// Bytes i and i + 1 of `word` as floats, minus (bias - 2^23) each; neg_bias = {-bias, -bias}.
__device__ __forceinline__ pf2 code_pair(uint32_t word, uint32_t i, pf2 neg_bias) {
    pf2 raw;
    asm("mov.b64 %0, {%1, %2};" : "=l"(raw) : "r"(__byte_perm(word, 0x4B000000u, 0x7540u + i)), "r"(__byte_perm(word, 0x4B000000u, 0x7541u + i)));
    return pf2_add(raw, neg_bias);
}
// Four consecutive K elements of column n of the B stage from two packed pairs.
__device__ __forceinline__ void store_b4_pairs(uint8_t* stage, uint32_t n, uint32_t k, pf2 v01, pf2 v23) {
    uint8_t* dst = stage + (n >> 3) * 1024u + (k >> 3) * 128u + (n & 7u) * 16u + (k & 7u) * 2u;
    *reinterpret_cast<uint2*>(dst) = make_uint2(pf2_bf16(v01), pf2_bf16(v23));
}

__device__ __forceinline__ void dequant_q4k(const uint8_t* row, uint32_t sub, uint32_t lane, uint32_t col, uint32_t n, uint8_t* stage) {
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint2 words = *reinterpret_cast<const uint2*>(row + sub * 512u + lane * 16u + col * 8u);      // this column's {w0, w1}
    const uint4 h = *reinterpret_cast<const uint4*>(row + 2048u + (g + 8u * col) * 16u);
    const float d = half_bits(h.x & 0xffffu), dmin = half_bits(h.x >> 16);
    // 6-bit scales and minima of groups 2 * sub (low nibbles) and 2 * sub + 1 (high nibbles).
    const uint32_t scales = sub < 2u ? (h.y & 0x3f3f3f3fu) : ((h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u));
    const uint32_t minima = sub < 2u ? (h.z & 0x3f3f3f3fu) : (((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u));
    const uint32_t first = (sub & 1u) * 2u;
    const pf2 neg_bias = pf2_make(-8388608.0f, -8388608.0f);
#pragma unroll
    for (uint32_t nib = 0; nib < 2u; ++nib) {
        const float ds = __fmul_rn(d, (float)byte_of(scales, first + nib));
        const float dm = __fmul_rn(dmin, (float)byte_of(minima, first + nib));
        const pf2 ds2 = pf2_make(ds, ds), neg_dm2 = pf2_make(-dm, -dm);       // d * sc * q - dmin * mn, each step rounded once
#pragma unroll
        for (uint32_t w = 0; w < 2u; ++w) {
            const uint32_t codes = ((w == 0u ? words.x : words.y) >> (4u * nib)) & 0x0f0f0f0fu;
            const pf2 v01 = pf2_add(pf2_mul(ds2, code_pair(codes, 0u, neg_bias)), neg_dm2);
            const pf2 v23 = pf2_add(pf2_mul(ds2, code_pair(codes, 2u, neg_bias)), neg_dm2);
            store_b4_pairs(stage, n, 32u * nib + 16u * w + 4u * t, v01, v23);
        }
    }
}

__device__ __forceinline__ void dequant_q6k(const uint8_t* row, uint32_t sub, uint32_t lane, uint32_t col, uint32_t n, uint8_t* stage) {
    const uint32_t g = lane >> 2, t = lane & 3u, half = sub >> 1, upper = sub & 1u;       // quarters 2 * upper, 2 * upper + 1 of the half
    const uint32_t column = g + 8u * col;
    const uint4 ql = *reinterpret_cast<const uint4*>(row + half * 1536u + col * 512u + lane * 16u);      // {s0 even, s0 odd, s1 even, s1 odd}
    const uint2 qh = *reinterpret_cast<const uint2*>(row + half * 1536u + 1024u + lane * 16u + col * 8u);      // {s0, s1}
    const float d = half_bits(*reinterpret_cast<const unsigned short*>(row + 3328u + column * 2u));
    const uint8_t* scale_bytes = row + 3072u + column * 16u;
#pragma unroll
    for (uint32_t s = 0; s < 2u; ++s) {
        const uint32_t even = s ? ql.z : ql.x, odd = s ? ql.w : ql.y, high = s ? qh.y : qh.x;
#pragma unroll
        for (uint32_t qq = 0; qq < 2u; ++qq) {
            const uint32_t quarter = 2u * upper + qq;
            const float ds = __fmul_rn(d, (float)(int)(signed char)scale_bytes[8u * half + 2u * quarter + s]);
            const uint32_t codes = (((qq ? odd : even) >> (4u * upper)) & 0x0f0f0f0fu) | (((high >> (2u * quarter)) & 0x03030303u) << 4);
            const pf2 ds2 = pf2_make(ds, ds), neg_bias = pf2_make(-(8388608.0f + 32.0f), -(8388608.0f + 32.0f));
            store_b4_pairs(stage, n, 32u * qq + 16u * s + 4u * t, pf2_mul(ds2, code_pair(codes, 0u, neg_bias)),
                           pf2_mul(ds2, code_pair(codes, 2u, neg_bias)));
        }
    }
}

__device__ __forceinline__ void dequant_q80(const uint8_t* row, uint32_t sub, uint32_t lane, uint32_t col, uint32_t n, uint8_t* stage) {
    const uint32_t g = lane >> 2, t = lane & 3u, column = g + 8u * col;
#pragma unroll
    for (uint32_t bb = 0; bb < 2u; ++bb) {
        const uint32_t block = 2u * sub + bb;
        const uint2 words = *reinterpret_cast<const uint2*>(row + block * 512u + lane * 16u + col * 8u);      // this column's {w0, w1}
        const float d = half_bits(*reinterpret_cast<const unsigned short*>(row + 2048u + column * 8u + block * 2u));
#pragma unroll
        for (uint32_t w = 0; w < 2u; ++w) {
            const uint32_t codes = (w == 0u ? words.x : words.y) ^ 0x80808080u;        // int8 + 128
            const pf2 d2 = pf2_make(d, d), neg_bias = pf2_make(-(8388608.0f + 128.0f), -(8388608.0f + 128.0f));
            store_b4_pairs(stage, n, 32u * bb + 16u * w + 4u * t, pf2_mul(d2, code_pair(codes, 0u, neg_bias)),
                           pf2_mul(d2, code_pair(codes, 2u, neg_bias)));
        }
    }
}

}  // namespace gf
