// Group-quantized codes to bf16 weights without a conversion.
//
// An unsigned byte c in the low bits of a bf16, with nothing above it, IS the number c 2^-133 (up to 127 a subnormal, from 128 on the
// exponent's lowest bit takes over where they end).  With scale 2^(133 - shift) and bias 2^-shift one fma gives the weight times 2^-shift;
// the f32 sums are scaled back at the end.  A nibble in bits 4-7 counts 2^4 times as much.  Q4 weights are rounded once in every
// projection kernel; Q8 weights are an f32 fma, then rounded to bf16 (b2_dequantize, the kernels without a table), and so they are here.
//
// The table of scales and biases holds them scaled.  A matrix's shift is the least with which its scales stay finite: 0 while all are
// below 2^-5, which those of ordinary weights are, and then nothing is lost anywhere.  Up to 2^11 it is at most 16; every weight is
// still exact (b2_gemm_table_shift refuses what is not), and f32 sums keep all their bits down to 2^-110.  A matrix that is refused
// stays with the kernels that mask into 128 + c and subtract.
#pragma once
#include "common.cuh"

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
// 8 Q4 codes in natural order: scales (scale, scale 2^-4), three instructions a pair
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
// 4 Q8 codes: a byte two bytes up is the same number in f32, and two of them are one fma
__device__ __forceinline__ void scaled_q8(uint32_t w, float scale, float bias, uint32_t& lo, uint32_t& hi) {
    auto pair = [&](uint32_t c0, uint32_t c1) {
        uint64_t r;
        asm("{\n.reg .b64 c, s, b;\nmov.b64 c, {%1, %2};\nmov.b64 s, {%3, %3};\nmov.b64 b, {%4, %4};\nfma.rn.f32x2 %0, c, s, b;\n}\n"
            : "=l"(r)
            : "r"(c0), "r"(c1), "f"(scale), "f"(bias));
        return pack_bf2(__uint_as_float((uint32_t)r), __uint_as_float((uint32_t)(r >> 32)));
    };
    lo = pair(prmt(w, 0u, 0x4044u), prmt(w, 0u, 0x4144u));
    hi = pair(prmt(w, 0u, 0x4244u), prmt(w, 0u, 0x4344u));
}
// The same weights by half the instructions, where one_rounding() holds.
__device__ __forceinline__ void scaled_q8_once(uint32_t w, uint32_t s2, uint32_t b2, uint32_t& lo, uint32_t& hi) {
    lo = fma_bf2(prmt(w, 0u, 0x4140u), s2, b2);
    hi = fma_bf2(prmt(w, 0u, 0x4342u), s2, b2);
}
// One fma in bf16 gives the bits of the two roundings unless the first drops a bias so small that code scale alone is a tie of the
// second: never where the scale's exponent is at most 15 above the bias's (all mantissas, codes and signs tried; from 16 on 1 weight
// in 70 000 differs, and more).  Taken where the fields differ by at most 8, since a subnormal bias lies up to 6 below its field.  For
// a table word: the difference of its exponents, 133 apart already, times 2^23, less at most 2^15.
__device__ __forceinline__ bool one_rounding(uint32_t sb) { return (int)((sb & 0x7f807f80u) * 0xffffu) < ((133 + 9) << 23) - (1 << 15); }
