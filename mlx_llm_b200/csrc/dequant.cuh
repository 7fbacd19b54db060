// Group-quantized codes to bf16 weights without a conversion.
//
// An unsigned byte c in the low bits of a bf16, with nothing above it, IS the number c 2^-133 (up to 127 a subnormal, from 128 on the
// exponent's lowest bit takes over where they end).  One fma with scale 2^93 and bias 2^-40 then gives bf16(c scale + bias) 2^-40 with
// the one rounding that the format asks for; the f32 sums are scaled back at the end.  A nibble in bits 4-7 counts 2^4 times as much.
// (A Q8 weight that an f32 fma and a second rounding to bf16 give can differ in its last bit where the scale is 2^14 or more below the
// bias, a handful in a billion.)  Exact for scales below 2^33 and weights above 2^-86; a matrix with a larger scale gets no table (b2_gemm_build_sbt) and stays with
// the kernels that mask into 128 + c and subtract.
#pragma once
#include "common.cuh"

constexpr uint32_t kByteUnit = 0x2b806e00u;    // (2^93, 2^-40) for a table word (scale, bias)
constexpr uint32_t kNibbleUnit = 0x2b806c00u;  // (2^89, 2^-40)
constexpr float kUnscale = 1099511627776.f;    // 2^40

__device__ __forceinline__ uint32_t fma_bf2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t mul_bf2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// 8 Q4 codes in natural order: scales (scale 2^93, scale 2^89), three instructions a pair
__device__ __forceinline__ void scaled_q4(uint32_t w, uint32_t scales, uint32_t b2, uint32_t (&out)[4]) {
    out[0] = fma_bf2(prmt(w, 0u, 0x4040u) & 0x00f0000fu, scales, b2);
    out[1] = fma_bf2(prmt(w, 0u, 0x4141u) & 0x00f0000fu, scales, b2);
    out[2] = fma_bf2(prmt(w, 0u, 0x4242u) & 0x00f0000fu, scales, b2);
    out[3] = fma_bf2(prmt(w, 0u, 0x4343u) & 0x00f0000fu, scales, b2);
}
// the same codes as (c0,c4) (c1,c5) (c2,c6) (c3,c7), nine instructions for the eight
__device__ __forceinline__ void scaled_q4_paired(uint32_t w, uint32_t s_lo, uint32_t s_hi, uint32_t b2, uint32_t (&out)[4]) {
    const uint32_t v = w >> 8;
    out[0] = fma_bf2(w & 0x000f000fu, s_lo, b2);
    out[1] = fma_bf2(w & 0x00f000f0u, s_hi, b2);
    out[2] = fma_bf2(v & 0x000f000fu, s_lo, b2);
    out[3] = fma_bf2(v & 0x00f000f0u, s_hi, b2);
}
// 4 Q8 codes
__device__ __forceinline__ void scaled_q8(uint32_t w, uint32_t s2, uint32_t b2, uint32_t& lo, uint32_t& hi) {
    lo = fma_bf2(prmt(w, 0u, 0x4140u), s2, b2);
    hi = fma_bf2(prmt(w, 0u, 0x4342u), s2, b2);
}
