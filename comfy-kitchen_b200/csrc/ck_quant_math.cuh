// Arithmetic of one NVFP4 / MXFP8 scale block, shared by the stand-alone quantizers and the
// re-quantizing GEMM epilogue.  Results are bit-identical to the reference's eager path
// (comfy_kitchen/backends/eager/quantization.py:115-160); translation units that include
// this header must not be compiled with fast-math.
#pragma once

#include "ck_common.cuh"

#include <type_traits>

namespace ck {
namespace quant {

// ---------------------------------------------------------------------------
// small-float converts (hardware cvt; rounding = nearest-even, saturating)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t f32_to_e4m3_byte(float v) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.0f), "f"(v));
  return r & 0xFFu;
}

__device__ __forceinline__ float e4m3_byte_to_f32(uint32_t b) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(b)));
  return __half2float(__ushort_as_half(static_cast<unsigned short>(h2 & 0xFFFFu)));
}

// byte = e2m1(hi) << 4 | e2m1(lo)
__device__ __forceinline__ uint32_t f32x2_to_e2m1_byte(float hi, float lo) {
  uint16_t r;
  asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; mov.b16 %0, {t, 0}; }" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}

// 16-bit = e4m3(hi) << 8 | e4m3(lo)
__device__ __forceinline__ uint32_t f32x2_to_e4m3x2(float hi, float lo) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}

// ---------------------------------------------------------------------------
// a / b, correctly rounded, from y = RN(1/b) with five FMA-class operations.
//
// q0 = RN(a*y) is within 2 ulp of a/b; one residual correction makes q1 a faithful
// quotient (error of q0 + r0*y against a/b is below 2^-46 relative), and by Markstein's
// theorem a second correction from a faithful quotient with a correctly rounded
// reciprocal yields RN(a/b), provided every residual is exact.  The caller guarantees
// the exponent window in which that holds (see nvfp4_block) and falls back to
// __fdiv_rn outside it.  The sign of `a` is re-applied at the end because an all-zero
// FMA chain loses a negative zero.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float div_markstein(float a, float b, float y) {
  float q = __fmul_rn(a, y);
  float r = __fmaf_rn(-b, q, a);
  q = __fmaf_rn(r, y, q);
  r = __fmaf_rn(-b, q, a);
  q = __fmaf_rn(r, y, q);
  return copysignf(q, a);
}

__device__ __forceinline__ float amax16(const float (&v)[16]) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(v[i]));
  return m;
}

// Merge the scale bytes of the 4 lanes that share one 4-byte group of the scale tile and
// store them with one 32-bit store from the first of the four lanes.
// ---------------------------------------------------------------------------
// NVFP4
// ---------------------------------------------------------------------------
// One 16-element block -> 8 code bytes (returned as two words) and one E4M3 scale byte.
// Steps follow comfy_kitchen/backends/eager/quantization.py:137-158 one to one.
template <bool kFastDiv>
__device__ __forceinline__ void nvfp4_block(const float (&v)[16], float g, bool hi_first, uint32_t& lo_word,
                                            uint32_t& hi_word, uint32_t& scale_byte) {
  const float amax = amax16(v);
  float s = __fdiv_rn(__fdiv_rn(amax, 6.0f), g);  // :139-140, two true divisions
  s = fminf(s, 448.0f);                           // :141
  scale_byte = f32_to_e4m3_byte(s);               // :142
  const float total = __fmul_rn(g, e4m3_byte_to_f32(scale_byte));  // :143
  const bool dead = (total == 0.0f);              // :146
  const float safe = dead ? 1.0f : total;         // :147

  float q[16];
  // The reciprocal-FMA quotient is exact while no residual can underflow and no
  // quotient can overflow: divisor within 2^+-60 and amax no more than 2^20 divisors.
  // Elements so small that their residual would underflow (|x| < 2^-90) have a
  // quotient below 2^-30 and encode as (signed) zero under either formula.
  const bool window = kFastDiv && (safe >= 0x1p-60f) && (safe <= 0x1p60f);
  // :154-158 clamp to +-6, round to E2M1 (satfinite does the clamp), pack two per byte.
  auto pack = [&](const float (&e)[16]) {
    uint32_t b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      b[i] = hi_first ? f32x2_to_e2m1_byte(e[2 * i], e[2 * i + 1]) : f32x2_to_e2m1_byte(e[2 * i + 1], e[2 * i]);
    }
    lo_word = b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24);
    hi_word = b[4] | (b[5] << 8) | (b[6] << 16) | (b[7] << 24);
  };
  bool done = false;
  if (window) {
    // Codes from the two products that bracket the exact quotient (see nvfp4_blocks);
    // accepted when they agree, which is the rule for all but a few blocks in ten thousand.
    const float y = __frcp_rn(safe);
    const float y_hi = __fmul_rn(y, 0x1.000008p0f), y_lo = __fmul_rn(y, 0x1.fffffp-1f);
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = v[i] * y_hi;
    pack(q);
    const uint32_t lo_a = lo_word, hi_a = hi_word;
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = v[i] * y_lo;
    pack(q);
    done = ((lo_a ^ lo_word) | (hi_a ^ hi_word)) == 0u;
    if (!done && amax <= safe * 0x1p20f) {
#pragma unroll
      for (int i = 0; i < 16; ++i) q[i] = div_markstein(v[i], safe, y);
      pack(q);
      done = true;
    }
  }
  if (!done) {
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = __fdiv_rn(v[i], safe);  // :149
    pack(q);
  }
  if (dead) {  // :150 (positive zeros, signs dropped)
    lo_word = 0;
    hi_word = 0;
  }
}

// ---------------------------------------------------------------------------
// NVFP4 block for the streaming quantizer: 16 elements of a 16-bit type as eight packed
// words.  Same arithmetic as nvfp4_block, arranged for a low instruction count: packed
// abs-max, the two per-block divisions (by 6, by the tensor scale) as reciprocal-FMA
// quotients with reciprocals prepared once per thread, the zero-scale case resolved on the
// packed words, four E2M1 converts packed per 32-bit word, and the nibble order a
// template parameter.
// ---------------------------------------------------------------------------

// word = bytes {e2m1x2(f0,f1), e2m1x2(f2,f3), e2m1x2(f4,f5), e2m1x2(f6,f7)}, lowest byte first;
// within a byte the first argument goes to the high nibble.
__device__ __forceinline__ uint32_t f32x8_to_e2m1_word(float f0, float f1, float f2, float f3, float f4, float f5,
                                                       float f6, float f7) {
  uint32_t r;
  asm("{ .reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %1, %2;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %3, %4;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %5, %6;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %7, %8;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3}; }"
      : "=r"(r)
      : "f"(f0), "f"(f1), "f"(f2), "f"(f3), "f"(f4), "f"(f5), "f"(f6), "f"(f7));
  return r;
}

// a / b for a >= 0 (no sign to restore) with y = RN(1/b); see div_markstein.
__device__ __forceinline__ float div_markstein_nonneg(float a, float b, float y) {
  float q = __fmul_rn(a, y);
  float r = __fmaf_rn(-b, q, a);
  q = __fmaf_rn(r, y, q);
  r = __fmaf_rn(-b, q, a);
  return __fmaf_rn(r, y, q);
}

// max |.| over the 16 values packed in eight words, as a float
template <typename T>
__device__ __forceinline__ float amax16_packed(const uint32_t (&w)[8]) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
    for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
    const uint32_t b = *reinterpret_cast<uint32_t*>(&m);
    return fmaxf(__uint_as_float(b << 16), __uint_as_float(b & 0xFFFF0000u));
  } else {
    __half2 m = __habs2(*reinterpret_cast<const __half2*>(&w[0]));
#pragma unroll
    for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __half2*>(&w[i])));
    const float2 f = __half22float2(m);
    return fmaxf(f.x, f.y);
  }
}

// Per-thread constants of the tensor scale g: its reciprocal and whether g lies in the
// range where the reciprocal-FMA quotients below are exact.
struct TensorScale {
  float g, rcp;
  float s_hi, s_lo;  // bracket 1 / (6 g) by 2^-21 (see nvfp4_blocks)
  bool in_window;
};
__device__ __forceinline__ TensorScale make_tensor_scale(float g) {
  TensorScale t;
  t.g = g;
  t.in_window = (g >= 0x1p-40f) && (g <= 0x1p40f);
  t.rcp = __frcp_rn(t.in_window ? g : 1.0f);
  const float sixth = __frcp_rn(__fmul_rn(6.0f, t.in_window ? g : 1.0f));
  t.s_hi = __fmul_rn(sixth, 0x1.000008p0f);
  t.s_lo = __fmul_rn(sixth, 0x1.fffffp-1f);
  return t;
}

template <typename T>
__device__ __forceinline__ void widen16(const uint32_t (&w)[8], float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
}

// The IEEE-division path of a packed block, out of line: it is taken only outside the
// exactness window (tiny or huge scales), and keeping it out of the caller's body keeps the
// caller's register allocation that of the common path.  Arguments and result travel in
// registers (words by value, a small struct back).
struct BlockCodes {
  uint32_t lo, hi, scale_byte;
};
template <typename T, bool kHiFirst>
__device__ __noinline__ BlockCodes nvfp4_block_packed_ieee(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t w4,
                                                           uint32_t w5, uint32_t w6, uint32_t w7, float g) {
  const uint32_t w[8] = {w0, w1, w2, w3, w4, w5, w6, w7};
  float v[16];
  widen16<T>(w, v);
  BlockCodes r;
  nvfp4_block<false>(v, g, kHiFirst, r.lo, r.hi, r.scale_byte);
  return r;
}

// 8 products v[i] * y -> one word of codes (nibble order as requested)
template <bool kHiFirst>
__device__ __forceinline__ uint32_t scaled_e2m1_word(const float* v, float y) {
  float q[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 p = mul_x2(make_float2(v[2 * i], v[2 * i + 1]), make_float2(y, y));
    q[2 * i] = p.x;
    q[2 * i + 1] = p.y;
  }
  if constexpr (kHiFirst) {
    return f32x8_to_e2m1_word(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7]);
  } else {
    return f32x8_to_e2m1_word(q[1], q[0], q[3], q[2], q[5], q[4], q[7], q[6]);
  }
}

// 1 / t for a positive normal t, one unit in the last place at most off.
__device__ __forceinline__ float approximate_reciprocal(float t) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(t));
  return y;
}

// Codes of sixteen 16-bit values divided by t: p = x y, then one correction by the residual, q = p - (t p - x) y.  With a y that is
// off by e, p is off by up to e + 2^-24, and q, beside its own rounding, by that times e and the residual's rounding: (e + 2^-24)^2 at most, 1.13 x 2^-45
// for one unit in the last place (e = 2^-23), 1.57 x 2^-44 for two.  For an x of at most eleven significant bits the code of q is the code
// of RN(x / t): the two can only part where x / t lies that close to the middle between a rounding boundary and its neighbour, and x and the
// boundary times t are then integers a few units apart; the cases there are have been gone through one by one (test_corrected_quotient_cpu),
// with reciprocals up to two units off.  Only a significand of all ones fails, which the caller sends elsewhere.
// The residual carries the sign opposite to x, so that the sum keeps a negative zero.  Per element one and a half packed
// multiply-adds and half a conversion; two bracketing products took one multiply and one conversion, and the conversions' bytes twice.
template <typename T, bool kHiFirst>
__device__ __forceinline__ void nvfp4_codes_corrected(const uint32_t (&w)[8], float t, float y, uint32_t& lo_word, uint32_t& hi_word) {
  const float2 t2 = make_float2(t, t), minus_y = make_float2(-y, -y);
  float q[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float2 minus_x;
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      minus_x.x = __uint_as_float(w[i] * 0x10000u + 0x80000000u);
      minus_x.y = __uint_as_float((w[i] & 0xFFFF0000u) ^ 0x80000000u);
    } else {
      minus_x = __half22float2(__hneg2(*reinterpret_cast<const __half2*>(&w[i])));
    }
    const float2 p = mul_x2(minus_x, minus_y);
    const float2 r = fma_x2(t2, p, minus_x);
    const float2 c = fma_x2(r, minus_y, p);
    q[2 * i] = c.x;
    q[2 * i + 1] = c.y;
  }
  if constexpr (kHiFirst) {
    lo_word = f32x8_to_e2m1_word(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7]);
    hi_word = f32x8_to_e2m1_word(q[8], q[9], q[10], q[11], q[12], q[13], q[14], q[15]);
  } else {
    lo_word = f32x8_to_e2m1_word(q[1], q[0], q[3], q[2], q[5], q[4], q[7], q[6]);
    hi_word = f32x8_to_e2m1_word(q[9], q[8], q[11], q[10], q[13], q[12], q[15], q[14]);
  }
}

// Whether the significand of t is all ones (see nvfp4_codes_corrected).
__device__ __forceinline__ bool all_ones(float t) { return (__float_as_uint(t) << 9) == 0xFFFFFE00u; }

// Window: tensor scale within 2^+-40, amax zero or within 2^+-60; total = g * scale is then a normal number within 2^+-50 and no
// residual matters that underflows (its quotient encodes as a signed zero).  Everything else takes the IEEE divisions.  The E4M3 scale
// comes from two products that bracket amax / (6 g) by 2^-21 (see nvfp4_blocks) and, when those round apart, from the quotients themselves.
//
// The quantizer of 16-bit inputs was bound by its instructions (issue slots 77 % busy at 24576 x 3072): with bracketing products
// and Markstein's scale / so, static scale, us: bf16 1024 x 3072 3.65 / 3.26, 4096 x 3072 7.90 / 7.35, 16384 x 3072 26.9 / 23.8, 24576 x 3072
// 46.7 / 33.7 (0.88 of the copy rate), 36864 x 3072 50.0 / 49.2, 16384 x 12288 96.0 / 82; behind its reduction 16384 x 3072 44.8 / 39.5.
template <typename T, bool kHiFirst>
__device__ __forceinline__ void nvfp4_block_packed(const uint32_t (&w)[8], const TensorScale& ts, uint32_t& lo_word,
                                                   uint32_t& hi_word, uint32_t& scale_byte) {
  static_assert(sizeof(T) == 2, "packed 16-bit inputs");
  const float amax = amax16_packed<T>(w);
  const uint32_t both = f32x2_to_e4m3x2(__fmul_rn(amax, ts.s_hi), __fmul_rn(amax, ts.s_lo));
  scale_byte = both & 0xFFu;
  const bool in_window = ts.in_window && (amax <= 0x1p60f) && (amax >= 0x1p-60f || amax == 0.0f);
  if ((both >> 8) != scale_byte && in_window) {
    const float s = div_markstein_nonneg(div_markstein_nonneg(amax, 6.0f, 0x1.555556p-3f /* RN(1/6) */), ts.g, ts.rcp);
    scale_byte = f32_to_e4m3_byte(fminf(s, 448.0f));
  }
  const float total = __fmul_rn(ts.g, e4m3_byte_to_f32(scale_byte));
  if (in_window && !all_ones(total)) {
    const bool dead = (total == 0.0f);  // zero scale: every code is +0
    const float t = dead ? 1.0f : total;
    nvfp4_codes_corrected<T, kHiFirst>(w, t, approximate_reciprocal(t), lo_word, hi_word);
    if (dead) {
      lo_word = 0;
      hi_word = 0;
    }
    return;
  }
  const BlockCodes r = nvfp4_block_packed_ieee<T, kHiFirst>(w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], ts.g);
  lo_word = r.lo;
  hi_word = r.hi;
  scale_byte = r.scale_byte;
}

// The same out of line, for callers whose registers are needed elsewhere.
template <typename T, bool kHiFirst>
__device__ __noinline__ BlockCodes nvfp4_block_packed_call(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t w4, uint32_t w5,
                                                           uint32_t w6, uint32_t w7, TensorScale ts) {
  const uint32_t w[8] = {w0, w1, w2, w3, w4, w5, w6, w7};
  BlockCodes r;
  nvfp4_block_packed<T, kHiFirst>(w, ts, r.lo, r.hi, r.scale_byte);
  return r;
}

// ---------------------------------------------------------------------------
// NVFP4 blocks of one thread without a branch in the common case
// ---------------------------------------------------------------------------
// Codes of fp32 inputs and of the fused epilogue: no quotient is computed.  The code of x / total is a monotone step function of the
// quotient, and RN(x / total) lies strictly between x y_lo and x y_hi with y_lo = y (1 - 2^-21) and y_hi = y (1 + 2^-21), y close to
// 1 / total: y is off by 2^-23 at most (nvfp4_block rounds it correctly, 2^-24), y_lo or y_hi, the product and the quotient itself are rounded by up to 2^-24
// each, 1.25 x 2^-22 in all.  So where both products convert to the same codes for a whole block, two multiplies and one convert
// an element, those are the codes of the exact quotients, and only a block in which some product straddles a rounding boundary is
// done again with quotients.  A zero keeps its sign through the multiplication, as the reference's cast keeps it.
// The E4M3 scale is bracketed like those codes: s = RN(RN(amax / 6) / g) deviates from amax / (6 g) by at most 2^-23, and
// amax * s_hi and amax * s_lo lie 2^-21 on either side of it less the 2^-22 of their own four roundings; when both
// round to the same E4M3 byte, that is the byte of s.
// Everything is computed for all of a thread's blocks before one test asks whether some bracket was split or some
// operand lies outside the window; those blocks are done again, out of line.  Straight code lets the blocks' serial
// chains (maximum, scale, conversion there and back, reciprocal) overlap, and has no Markstein chains in it.
// kCorrected: 16-bit codes by nvfp4_codes_corrected, which no bracket can split.  The few-row linear gains by it (8 x 3072 x 3072 6.56 us
// against 6.12, 8 x 18432 x 3072 with a dynamic scale 9.23 / 9.03); the fused epilogue, which waits for a thread's chains, does not: bf16 4608 x
// 12288 x 3072 79.7 us with brackets, 80.7 with the correction.

// Sixteen elements in registers: packed pairs of a 16-bit type, or floats.
template <typename T>
struct Sixteen {
  uint32_t w[4 * sizeof(T)];
  __device__ __forceinline__ void widen(float (&v)[16]) const {
    if constexpr (sizeof(T) == 2) {
      widen16<T>(w, v);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(w[i]);
    }
  }
  __device__ __forceinline__ float amax() const {
    if constexpr (sizeof(T) == 2) {
      return amax16_packed<T>(w);
    } else {
      float v[16];
      widen(v);
      return amax16(v);
    }
  }
};

// A block that the straight code could not settle.  `total` is its scale times g where that much is certain, else negative.
template <typename T, bool kHiFirst>
__device__ __noinline__ BlockCodes nvfp4_block_exact(Sixteen<T> x, float g, float total) {
  float v[16];
  x.widen(v);
  BlockCodes r;
  r.scale_byte = 0;
  if (total > 0.0f && x.amax() <= total * 0x1p20f) {  // residuals of the exact chain representable
    const float y = __frcp_rn(total);
    float q[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = div_markstein(v[i], total, y);
    r.lo = scaled_e2m1_word<kHiFirst>(q, 1.0f);
    r.hi = scaled_e2m1_word<kHiFirst>(q + 8, 1.0f);
    return r;
  }
  nvfp4_block<false>(v, g, kHiFirst, r.lo, r.hi, r.scale_byte);
  return r;
}

template <typename T, bool kHiFirst, int kBlocks, bool kCorrected = sizeof(T) == 2>
__device__ __forceinline__ void nvfp4_blocks(const Sixteen<T> (&x)[kBlocks], const TensorScale& ts, uint32_t (&codes)[kBlocks][2],
                                             uint32_t (&scale_byte)[kBlocks]) {
  float total[kBlocks];
  bool ok[kBlocks], sure[kBlocks];
  bool all = true;
#pragma unroll
  for (int b = 0; b < kBlocks; ++b) {
    const float amax = x[b].amax();
    const uint32_t both = f32x2_to_e4m3x2(__fmul_rn(amax, ts.s_hi), __fmul_rn(amax, ts.s_lo));
    scale_byte[b] = both & 0xFFu;
    total[b] = __fmul_rn(ts.g, e4m3_byte_to_f32(scale_byte[b]));
    const bool dead = total[b] == 0.0f;
    const float t = dead ? 1.0f : total[b], y = approximate_reciprocal(t);
    sure[b] = (both >> 8) == scale_byte[b] && ts.in_window && amax <= 0x1p60f && (amax >= 0x1p-60f || amax == 0.0f);
    uint32_t lo, hi;
    if constexpr (kCorrected) {
      nvfp4_codes_corrected<T, kHiFirst>(x[b].w, t, y, lo, hi);
      sure[b] = sure[b] && !all_ones(total[b]);
      ok[b] = sure[b];
    } else {
      const float y_hi = __fmul_rn(y, 0x1.000008p0f), y_lo = __fmul_rn(y, 0x1.fffffp-1f);
      float v[16];
      x[b].widen(v);
      lo = scaled_e2m1_word<kHiFirst>(v, y_hi);
      hi = scaled_e2m1_word<kHiFirst>(v + 8, y_hi);
      const uint32_t split = (lo ^ scaled_e2m1_word<kHiFirst>(v, y_lo)) | (hi ^ scaled_e2m1_word<kHiFirst>(v + 8, y_lo));
      ok[b] = sure[b] && (split == 0u || dead);
    }
    codes[b][0] = dead ? 0u : lo;  // zero scale: every code is +0
    codes[b][1] = dead ? 0u : hi;
    all = all && ok[b];
  }
  if (!all) {
#pragma unroll
    for (int b = 0; b < kBlocks; ++b) {
      if (!ok[b]) {
        const BlockCodes r = nvfp4_block_exact<T, kHiFirst>(x[b], ts.g, sure[b] ? total[b] : -1.0f);
        codes[b][0] = r.lo;
        codes[b][1] = r.hi;
        if (!sure[b]) scale_byte[b] = r.scale_byte;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// MXFP8 (comfy_kitchen/backends/eager/quantization.py:292-318)
// ---------------------------------------------------------------------------
// clamp(ceil(log2(r)) + 127, 0, 254) for r >= 2^-127, from the bits of r
// (comfy_kitchen/backends/eager/quantization.py:295-300).  r = amax/448 with amax an
// f16/bf16 number is either an exact power of two or far enough from one that the
// reference's float32 log2 cannot round across an integer, so this integer form is
// bit-identical for those input types.
__device__ __forceinline__ uint32_t e8m0_ceil_exponent(float r) {
  const uint32_t bits = __float_as_uint(r);
  const uint32_t e = bits >> 23;  // r > 0
  const uint32_t frac = bits & 0x7FFFFFu;
  uint32_t biased;
  if (e == 0) {
    biased = frac > 0x400000u ? 1u : 0u;  // [2^-127, 2^-126): exactly 2^-127 -> 0
  } else {
    biased = e + (frac != 0u);
  }
  return min(biased, 254u);
}

// What a block of 32 elements with the largest magnitude `amax` is multiplied by, and its scale byte.
struct Mxfp8Scale {
  float inv;
  uint32_t byte;
  bool dead;  // an all-zero block
};
__device__ __forceinline__ Mxfp8Scale mxfp8_scale(float amax) {
  const float need = fmaxf(__fdiv_rn(amax, 448.0f), 0x1p-127f);  // :294-295
  const uint32_t e = e8m0_ceil_exponent(need);                   // :298-302
  Mxfp8Scale s;
  s.dead = (amax == 0.0f);  // :306
  // :303-310: divide by 2^(e-127).  For e in [1, 253] that is an exact multiplication by
  // 2^(127-e); e == 254 needs the subnormal 2^-127; e == 0 decodes to a zero scale and
  // the reference divides by zero (inputs below 448 * 2^-127, outside the pinned domain).
  if (e == 0) {
    s.inv = __int_as_float(0x7F800000);
  } else if (e == 254) {
    s.inv = 0x1p-127f;
  } else {
    s.inv = __uint_as_float((254u - e) << 23);
  }
  if (s.dead) s.inv = 0.0f;  // :307,311 -> all zeros (positive)
  s.byte = s.dead ? 0u : e;  // :318
  return s;
}

// Four elements -> four E4M3 bytes; :314-315 clamp to +-448 and round to E4M3: satfinite performs the clamp
__device__ __forceinline__ uint32_t mxfp8_four(const float* v, const Mxfp8Scale& s) {
  const uint32_t lo = f32x2_to_e4m3x2(s.dead ? 0.0f : v[1] * s.inv, s.dead ? 0.0f : v[0] * s.inv);
  const uint32_t hi = f32x2_to_e4m3x2(s.dead ? 0.0f : v[3] * s.inv, s.dead ? 0.0f : v[2] * s.inv);
  return lo | (hi << 16);
}

// ---------------------------------------------------------------------------
// dynamic per-tensor scale
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float round_to_input_dtype(float v) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    return __bfloat162float(__float2bfloat16_rn(v));
  } else if constexpr (std::is_same<T, __half>::value) {
    return __half2float(__float2half_rn(v));
  } else {
    return v;
  }
}

template <typename T>
__device__ __forceinline__ float abs_max_of_vec(const Vec256& raw) {
  float m = 0.0f;
  if constexpr (sizeof(T) == 2) {
    // |x| of a 16-bit float is its bit pattern without the sign, and for non-negative
    // floats of one format the integer order of the bit patterns is the numeric order:
    // reduce the eight packed pairs as unsigned 16-bit integers, convert once.
    uint32_t p = raw.w[0] & 0x7FFF7FFFu;
#pragma unroll
    for (int i = 1; i < 8; ++i) p = __vmaxu2(p, raw.w[i] & 0x7FFF7FFFu);
    const uint32_t top = max(p & 0xFFFFu, p >> 16);
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      m = __uint_as_float(top << 16);
    } else {
      m = __half2float(__ushort_as_half(static_cast<unsigned short>(top)));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(__uint_as_float(raw.w[i])));
  }
  return m;
}

// The dynamic per-tensor scale: amax / (448 * 6) in the input dtype (a true division, then rounded), then float32.
template <typename T>
__device__ __forceinline__ float nvfp4_scale_of_amax(float amax) {
  return round_to_input_dtype<T>(__fdiv_rn(amax, 2688.0f));
}

}  // namespace quant
}  // namespace ck
