// Bit-exact float epilogue and prologue arithmetic shared by all convolution kernels.
//
// Every rounding step of the reference's x86 code is written out with an explicit intrinsic so that
// the compiler neither fuses nor splits anything (the library is also compiled with -fmad=false):
//   dequantize  v = fma((float)acc, scale_in, bias)      Tensor/QuantizeX86.cpp:851-903 as built with the
//                                                         reference's -Ofast -mfma flags (one FMA);
//               without bias: (float)acc * scale_in       Tensor/QuantizeX86.cpp:864-880
//   activation  ReLU / LeakyReLU / clip[0,6]              Tensor/QuantizeX86.hpp:72-106
//   requantize  q = float2int8(v * scale_out)             Tensor/QuantizeX86.cpp:1723-1870
//   float2int8  trunc(v + copysign(0.5, v)), clamp ±127   Tensor/VecIntrinsic.hpp:71-95   (rounding 0)
//               round half away from zero, clamp ±127     Tensor/QuantizeX86.cpp:18-23    (rounding 1)
//   no bias     fma(a, s, -0.0) is a * s to the last bit, the sign of zero included: bias_or_neutral below
//   quantize    q = float2int8(x * scale)                 Tensor/QuantizeX86.cpp:396-549
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ottk {

enum : int { ACT_NONE = 0, ACT_RELU = 1, ACT_LRELU = 2, ACT_RELU6 = 3 };
constexpr int ACT_POS = 4;  // kernel builds only: int8 output whose activation the clamp to [0, 127] carries out, see EpilogueParams
enum : int { ROUND_ADD_HALF_TRUNC = 0, ROUND_HALF_AWAY = 1 };

// Per-layer epilogue parameters. Arrays are device pointers with one entry per (padded) output channel;
// entries of padding channels are zero so those channels come out as 0.
struct EpilogueParams {
    const float* scale_in;   // [cout_pad]
    const float* bias;       // [cout_pad] (zeros when the layer has no bias)
    const float* scale_out;  // [cout_pad] (per-tensor scale replicated); unused for fp32 output
    int has_bias;
    int act_type;
    float act_param0;
    int rounding;
    int one_scale_out;       // every channel's scale_out is scale_out0, and finite (padding channels, which hold 0, take it too)
    float scale_out0;
    // ReLU, or ReLU6 where f(6) is 127 in every channel, and |v * scale_out| + 1 stays below 2^15 in every channel whatever the int8
    // input is, and not signed_rounding: float2int8(act(v) * scale_out) is trunc(v * scale_out + h) clamped to [0, 127], see requant4_pos
    int int8_pos;
    // ReLU or ReLU6, and some channel's scale_out is below zero, or some sum gives a product so close to 0.5 that one rounding would not do
    // for two (round2_nonneg)
    int signed_rounding;
};

__device__ __forceinline__ float dequant(int acc, float scale_in, float bias, int has_bias) {
    const float a = __int2float_rn(acc);
    return has_bias ? __fmaf_rn(a, scale_in, bias) : __fmul_rn(a, scale_in);
}

// the bias of a channel, or the value that makes the fma a plain product in a layer without bias
__device__ __forceinline__ float bias_or_neutral(const EpilogueParams& ep, int c) { return ep.has_bias ? ep.bias[c] : -0.0f; }

template <int ACT>
__device__ __forceinline__ float activate_t(float v, float p0) {
    if (ACT == ACT_RELU) return v > 0.f ? v : 0.f;
    if (ACT == ACT_LRELU) return v > 0.f ? v : __fmul_rn(v, p0);
    if (ACT == ACT_RELU6) return fminf(fmaxf(v, 0.f), 6.f);
    return v;
}

__device__ __forceinline__ float activate(float v, int act, float p0) {
    switch (act) {
        case ACT_RELU: return activate_t<ACT_RELU>(v, p0);
        case ACT_LRELU: return activate_t<ACT_LRELU>(v, p0);
        case ACT_RELU6: return activate_t<ACT_RELU6>(v, p0);
        default: return v;
    }
}

// Both int8 rounding rules are trunc(v + copysign(h, v)): h = 0.5 is the packed path's rule as it stands; with h = 0.5 - 2^-25,
// the largest fp32 below one half, the same sum rounds half away from zero. (frac(v) >= 0.5: the exact sum lies at most 2^-25
// below the next integer n and rounds to n, at n = 1 by ties-to-even; frac(v) < 0.5: it lies below n by more than half a step of
// fp32 there. Checked for every fp32 value up to 2^23 in magnitude.) So the rule is a constant, not code of its own.
constexpr uint32_t kHalfTrunc = 0x3F000000u, kHalfAway = 0x3EFFFFFFu;
__host__ __device__ __forceinline__ uint32_t half_bits(int rounding) { return rounding == ROUND_HALF_AWAY ? kHalfAway : kHalfTrunc; }

// copysign(h, v) as one logic instruction: (bits(v) & 0x80000000) | bits(h). Written as lop3 with both constants in
// registers; the compiler's own form takes two instructions per value (a logic instruction carries one immediate).
__device__ __forceinline__ float half_signed(float v, uint32_t h) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(__float_as_uint(v)), "r"(0x80000000u), "r"(h));
    return __uint_as_float(r);
}

// float -> int in [-127,127], kept as int so four of them can be packed by the caller.
__device__ __forceinline__ int float2int8(float v, uint32_t h) { return max(-127, min(127, __float2int_rz(__fadd_rn(v, half_signed(v, h))))); }

__device__ __forceinline__ int requant(int acc, float scale_in, float bias, float scale_out, const EpilogueParams& ep) {
    float v = dequant(acc, scale_in, bias, ep.has_bias);
    v = activate(v, ep.act_type, ep.act_param0);
    return float2int8(__fmul_rn(v, scale_out), half_bits(ep.rounding));
}

__device__ __forceinline__ float dequant_act(int acc, float scale_in, float bias, const EpilogueParams& ep) {
    return activate(dequant(acc, scale_in, bias, ep.has_bias), ep.act_type, ep.act_param0);
}

__device__ __forceinline__ int quantize1(float x, float scale, uint32_t h) {
    return float2int8(__fmul_rn(x, scale), h);
}

// ---- fast forms used by the hot loops (same results as the functions above) ----

// two s32 -> two saturated s8 in the low half of d, upper half taken from c (cvt.pack)
__device__ __forceinline__ uint32_t pack_sat_s8x2(int hi, int lo, uint32_t c) {
    uint32_t d;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(c));
    return d;
}

// four s32 -> four saturated s8, a in byte 0
__device__ __forceinline__ uint32_t pack_sat_s8x4(int a, int b, int c, int d) {
    return pack_sat_s8x2(b, a, pack_sat_s8x2(d, c, 0));
}

// two values -> trunc(v + copysign(h, v)), clamped below at -127 only (trunc(max(adj, -127.5)) == max(trunc(adj), -127)); the
// clamp at +127 is left to pack_sat_s8x4
__device__ __forceinline__ int2 round2(float2 v, uint32_t h) {
    const float2 r = __fadd2_rn(v, make_float2(half_signed(v.x, h), half_signed(v.y, h)));
    return make_int2(__float2int_rz(fmaxf(r.x, -127.5f)), __float2int_rz(fmaxf(r.y, -127.5f)));
}

// Behind ReLU / ReLU6 and a scale that is not negative the product and the rounding are one fused multiply-add: trunc(fma(y, s, 0.5)). For
// every integer n >= 1 that passes n + 0.5 at the same product as BOTH rules with their two roundings: RN(p) >= n + 0.5 and RN(p + 0.5) >= n + 1
// each ask for p >= n + 0.5 - half a step of fp32, the steps below n + 0.5 and n + 1 being equal, ties going up in both (n + 0.5 and n + 1 have even
// significands). Only below 0.5, where the steps differ, do they part, for products within 2^-25 of it; which sums give such a
// product is known when the layer is created (EpilogueParams::signed_rounding), and a layer that has one does not come here.
// The two roundings cannot be written as a product and a sum: the compiler contracts mul.rn.f32x2 with an add.rn.f32x2 that is its only
// reader (it does, with -fmad=false and .rn alike), and with h = 0.5 - 2^-25 that moved one product in some millions across
// n + 0.5. round2 is safe from that: the product has a second reader, half_signed.
constexpr uint32_t kHalfFused = 0x3F000000u;

__device__ __forceinline__ int2 round2_nonneg(float2 y, float2 s) {
    const float2 r = __ffma2_rn(y, s, make_float2(__uint_as_float(kHalfFused), __uint_as_float(kHalfFused)));
    return make_int2(__float2int_rz(r.x), __float2int_rz(r.y));
}

// float2int8(y * s), the clamp at +127 left to pack_sat_s8x4. SIGNED: EpilogueParams::signed_rounding
template <int ACT, bool SIGNED = false>
__device__ __forceinline__ int2 round2_act(float2 y, float2 s, uint32_t h) {
    if (!SIGNED && (ACT == ACT_RELU || ACT == ACT_RELU6)) return round2_nonneg(y, s);
    return round2(__fmul2_rn(y, s), h);
}

// Four sums v and scales s of an int8_pos layer -> four int8 of the activated values, va.x in byte 0. Adding 1.5 * 2^23 with rounding
// toward zero leaves trunc(u) in the low bits of the sum (a floor below zero, which the clamp drops), so that neither the activation nor
// a conversion to integer is an instruction of its own, and two values are clamped at a time: 2.3 logic instructions per value
// less. Exact while |u| < 2^15, where the low 16 bits carry the sign.
__device__ __forceinline__ uint32_t requant4_pos(float2 va, float2 sa, float2 vb, float2 sb) {
    const float2 hh = make_float2(__uint_as_float(kHalfFused), __uint_as_float(kHalfFused)), magic = make_float2(12582912.f, 12582912.f);
    const float2 ra = __fadd2_rz(__ffma2_rn(va, sa, hh), magic), rb = __fadd2_rz(__ffma2_rn(vb, sb, hh), magic);
    uint32_t pa = __byte_perm(__float_as_uint(ra.x), __float_as_uint(ra.y), 0x5410), pb = __byte_perm(__float_as_uint(rb.x), __float_as_uint(rb.y), 0x5410);
    asm("min.relu.s16x2 %0, %0, %1;" : "+r"(pa) : "r"(0x007F007Fu));
    asm("min.relu.s16x2 %0, %0, %1;" : "+r"(pb) : "r"(0x007F007Fu));
    return __byte_perm(pa, pb, 0x6420);
}

// quantize 4 floats with one scale and pack them, x in byte 0
__device__ __forceinline__ uint32_t quantize4_pack(float x, float y, float z, float w, float scale, uint32_t h) {
    // the multiplies and the additions of +-h as packed pairs (same IEEE operations, half the instructions)
    const float2 sc = make_float2(scale, scale);
    const int2 a = round2(__fmul2_rn(make_float2(x, y), sc), h), b = round2(__fmul2_rn(make_float2(z, w), sc), h);
    return pack_sat_s8x4(a.x, a.y, b.x, b.y);
}

// 4x4 byte transpose: inputs are 4 words of 4 bytes; o[i] byte j = input j byte i
__device__ __forceinline__ void transpose4x4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t o[4]) {
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(c, d, 0x5140);
    const uint32_t t2 = __byte_perm(a, b, 0x7362), t3 = __byte_perm(c, d, 0x7362);
    o[0] = __byte_perm(t0, t1, 0x5410);
    o[1] = __byte_perm(t0, t1, 0x7632);
    o[2] = __byte_perm(t2, t3, 0x5410);
    o[3] = __byte_perm(t2, t3, 0x7632);
}

__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
    return (uint32_t)(a & 0xff) | ((uint32_t)(b & 0xff) << 8) | ((uint32_t)(c & 0xff) << 16) | ((uint32_t)(d & 0xff) << 24);
}

}  // namespace ottk
