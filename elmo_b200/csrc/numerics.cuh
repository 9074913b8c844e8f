// Element arithmetic shared by the epilogues: bf16/e4m3 conversions with the reference's
// intermediate roundings, sigmoid / BCE terms, the Philox4x32 stream and rounding of the updated weight.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace xmc {

__device__ __forceinline__ float bf16_round(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_bits_to_float(uint32_t b16) { return __uint_as_float(b16 << 16); }

// larger of two bf16 values, two at a time; a NaN loses against a number
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// bf16 bit patterns as 16-bit keys in the order of their values, -0 below +0
__device__ __forceinline__ unsigned int topk_ord16(unsigned int b) { return (b & 0x8000u) ? (~b & 0xFFFFu) : (b | 0x8000u); }

// two e4m3 bytes (low byte first) -> two floats, exact
__device__ __forceinline__ float2 e4m3x2_to_float2(uint16_t v) {
  __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)v, __NV_E4M3);
  return __half22float2(*reinterpret_cast<__half2*>(&h));
}
// two floats -> two e4m3 bytes (x in the low byte), round-to-nearest-even, saturating at +-448
__device__ __forceinline__ uint16_t float2_to_e4m3x2(float x, float y) {
  return (uint16_t)__nv_cvt_float2_to_fp8x2(make_float2(x, y), __NV_SATFINITE, __NV_E4M3);
}

// two f16 -> two floats, exact.  MIXED: as h * 1 - 0 with the mixed-precision multiply-add, which issues every cycle on either
// half of the multiplier-add pipe; the conversion takes two cycles of the half that the wide multiplies of Philox need.
// (Without Philox beside it it is the better one: one-kernel step rounded to nearest, 300 000 x 768 at batch 32, 157 and 161 us.)
template <bool MIXED>
__device__ __forceinline__ void f16x2_to_float2(uint32_t h2, float& lo, float& hi) {
  if constexpr (MIXED)
    asm("{.reg .b16 l, h, one; mov.b32 {l, h}, %2; mov.b16 one, 0x3C00; fma.rn.f32.f16 %0, l, one, %3; fma.rn.f32.f16 %1, h, one, %3;}"
        : "=f"(lo), "=f"(hi) : "r"(h2), "f"(-0.0f));
  else
    asm("{.reg .b16 l, h; mov.b32 {l, h}, %2; cvt.f32.f16 %0, l; cvt.f32.f16 %1, h;}" : "=f"(lo), "=f"(hi) : "r"(h2));
}
// four e4m3 bytes (one word, low byte first) -> four floats, exact; and back, to nearest even, saturating
template <bool MIXED = false>
__device__ __forceinline__ void e4m3x4_to_float4(uint32_t w, float (&f)[4]) {
  uint32_t a, b;
  asm("{.reg .b16 l, h; mov.b32 {l, h}, %2; cvt.rn.f16x2.e4m3x2 %0, l; cvt.rn.f16x2.e4m3x2 %1, h;}" : "=r"(a), "=r"(b) : "r"(w));
  f16x2_to_float2<MIXED>(a, f[0], f[1]);
  f16x2_to_float2<MIXED>(b, f[2], f[3]);
}
__device__ __forceinline__ uint32_t float4_to_e4m3x4(float f0, float f1, float f2, float f3) {
  uint32_t r;
  asm("{.reg .b16 l, h; cvt.rn.satfinite.e4m3x2.f32 l, %2, %1; cvt.rn.satfinite.e4m3x2.f32 h, %4, %3; mov.b32 %0, {l, h};}"
      : "=r"(r) : "f"(f0), "f"(f1), "f"(f2), "f"(f3));
  return r;
}
// four e5m2 bytes (the upper halves of f16) -> four floats, exact; and back, to nearest even: for magnitudes up to kE5m2Max
constexpr float kE5m2Max = 57344.0f;
__device__ __forceinline__ void e5m2x4_to_float4(uint32_t w, float (&f)[4]) {
  f16x2_to_float2<false>(__byte_perm(w, 0u, 0x1404), f[0], f[1]);
  f16x2_to_float2<false>(__byte_perm(w, 0u, 0x3424), f[2], f[3]);
}
__device__ __forceinline__ uint32_t float4_to_e5m2x4(float f0, float f1, float f2, float f3) {
  uint32_t r;
  asm("{.reg .b16 l, h; cvt.rn.satfinite.e5m2x2.f32 l, %2, %1; cvt.rn.satfinite.e5m2x2.f32 h, %4, %3; mov.b32 %0, {l, h};}"
      : "=r"(r) : "f"(f0), "f"(f1), "f"(f2), "f"(f3));
  return r;
}
// four floats -> four e4m3 bytes, towards zero, saturating, a NaN stays one: the stochastic conversion with no random bits
__device__ __forceinline__ uint32_t float4_to_e4m3x4_rz(float f0, float f1, float f2, float f3) {
  uint32_t r;
  asm("cvt.rs.satfinite.e4m3x4.f32 %0, {%4, %3, %2, %1}, %5;" : "=r"(r) : "f"(f0), "f"(f1), "f"(f2), "f"(f3), "r"(0u));
  return r;
}
// two floats -> two bf16 (x in the low half), stochastically: 16 bits of r each, added below the kept mantissa
__device__ __forceinline__ uint32_t float2_to_bf16x2_rs(float x, float y, uint32_t r) {
  uint32_t o;
  asm("cvt.rs.bf16x2.f32 %0, %2, %1, %3;" : "=r"(o) : "f"(x), "f"(y), "r"(r));
  return o;
}
// x + 16 * (low / high half of r), one instruction each (the 16-bit dot product with one weight zero)
__device__ __forceinline__ uint32_t add_low16x16(uint32_t x, uint32_t r) {
  uint32_t y;
  asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(y) : "r"(r), "r"(0x10u), "r"(x));
  return y;
}
__device__ __forceinline__ uint32_t add_high16x16(uint32_t x, uint32_t r) {
  uint32_t y;
  asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(y) : "r"(r), "r"(0x1000u), "r"(x));
  return y;
}
// max(m, |a|, |b|), NaN if any of them is
__device__ __forceinline__ float max3_abs_nan(float m, float a, float b) {
  asm("{.reg .f32 x, y; abs.f32 x, %1; abs.f32 y, %2; max.NaN.f32 %0, %0, x, y;}" : "+f"(m) : "f"(a), "f"(b));
  return m;
}

// Two fp32 operations per instruction (sm_100 packed fp32): same rounding per half as the scalar forms.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// sigmoid(z) = 1 / (1 + 2^(-z log2 e)) with the two approximate special-function ops (relative error
// ~2^-22, far below the bf16 rounding that follows).
__device__ __forceinline__ float fast_sigmoid(float z) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return r;
}
// Sum over logits of max(z,0) + log(1 + exp(-|z|)), the label-independent part of BCE-with-logits (chunked.py:57-72),
// with one logarithm for all of them: log of the product of the 1 + e, e = exp(-|z|) in (0, 1].  What is kept is the
// product MINUS ONE, q' = q + e + q e, a sum of positive terms: it stays accurate to 2^-24 a step also where all e are
// tiny (logits of -20), as log1p of each one would.  Good for 126 logits of either half (2^126).  Two chains, for the
// halves of a pair: five packed or special-function operations where exp and log1p of each logit take over twenty:
// forward of 670 091 x 768 FP8 at batch 512 with loss 906 -> 590 us (without: 400).
struct SoftplusSum {
  uint64_t lin = 0ull, q = 0ull;
  __device__ __forceinline__ void add(float z0, float z1) {
    float e0, e1;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(fabsf(z0) * -1.4426950408889634f));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(fabsf(z1) * -1.4426950408889634f));
    const uint64_t e = pack_f32x2(e0, e1);
    lin = add_f32x2(lin, pack_f32x2(fmaxf(z0, 0.0f), fmaxf(z1, 0.0f)));
    q = fma_f32x2(q, e, add_f32x2(q, e));
  }
  __device__ __forceinline__ void add(float z0) { add(z0, -INFINITY); }      // exp(-inf) = 0: adds nothing
  __device__ __forceinline__ float value() const {
    float l0, l1, q0, q1;
    unpack_f32x2(lin, l0, l1);
    unpack_f32x2(q, q0, q1);
    return (l0 + l1) + (log1pf(q0) + log1pf(q1));
  }
};

// ---------------------------------------------------------------------------------------------
// Philox4x32 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3", SC'11) with kSrRounds = 7
// rounds: the round function and key schedule of Philox4x32-10, stopped after the seventh round -- the
// smallest round count its authors report as passing BigCrush (ten is their default margin; the rounds
// are over a third of the update epilogue's issue cycles, and the bits only dither a rounding).  One call
// serves 8 consecutive weight elements with 16 bits each: counter = (q_lo, q_hi, step_lo, step_hi),
// q = global element index / 8, key = (seed_lo, seed_hi); element j takes half (j & 1) of output word
// (j >> 1).
// ---------------------------------------------------------------------------------------------
constexpr int kSrRounds = 7;
__device__ __forceinline__ uint4 philox4x32_sr(uint4 c, uint2 k) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < kSrRounds; ++r) {
    const unsigned long long p0 = (unsigned long long)M0 * c.x;
    const unsigned long long p1 = (unsigned long long)M1 * c.z;
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ k.x, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ k.y, (uint32_t)p0);
    k.x += W0;
    k.y += W1;
  }
  return c;
}

// Exact stochastic rounding of fp32 w onto the e4m3 grid (subnormals included) with 16 random
// bits; returns a float that lies on the grid (or beyond +-448: the saturating e4m3 conversion
// that follows clamps it).  The sign is kept, also for a zero result; NaN propagates.
//
// The reference's bit trick (fuse_kernel.py:28-36) adds the random bits into the 20 mantissa bits
// an e4m3 normal discards and truncates; below 2^-6 the e4m3 grid is uniform (step 2^-9) and the
// trick no longer sees it.  Scaling by 2^-120 first maps e4m3's smallest normal onto fp32's
// (2^-126): e4m3 subnormals become fp32 subnormals, whose bit pattern is fixed point with bit 20
// worth exactly one e4m3 step, so ONE add-and-mask is exact stochastic rounding on the whole grid,
// carries from the subnormal into the normal range included.  Both scalings are exact (the first
// rounds only below 2^-149, i.e. 2^-29 before scaling).  Needs fp32 denormals (no -ftz).
constexpr float kSrDown = 7.52316384526264005e-37f;   // 2^-120
constexpr float kSrUp = 1.32922799578491587e+36f;     // 2^120
__device__ __forceinline__ float sr_e4m3_finite(float w, uint32_t r16) {
  const uint32_t b = (__float_as_uint(w * kSrDown) + (r16 << 4)) & 0xFFF00000u;
  return __uint_as_float(b) * kSrUp;
}
__device__ __forceinline__ float sr_e4m3(float w, uint32_t r16) {
  const float y = sr_e4m3_finite(w, r16);               // +-Inf stays +-Inf; a NaN pattern may wrap
  return w != w ? w : y;
}
// four e4m3 bytes -> four bf16 (two packed words), exact.  Through the hardware's conversions: four cycles of the
// integer pipe and four of the FMA pipe per pair.  (Shifting and masking the bytes into place and multiplying by 2^120
// takes eight of the integer pipe, which the epilogues beside the converter warps want too.)
__device__ __forceinline__ void e4m3x4_to_bf16x4(uint32_t w, uint32_t& lo, uint32_t& hi) {
  float f[4];
  e4m3x4_to_float4(w, f);
  lo = pack_bf16x2(f[0], f[1]);
  hi = pack_bf16x2(f[2], f[3]);
}

}  // namespace xmc
