// The NVFP4 block quantizer (one 16-element block -> 8 code bytes + one E4M3 scale, "four over six" scale
// selection), bit-exact against the reference's PyTorch quantizer
// (fouroversix/src/fouroversix/quantize/pytorch/reference.py:242-368).  Shared by the standalone quantizer
// (quantize.cu) and the GEMM epilogue that requantizes its output (gemm_nvfp4.cu).  The arithmetic notes at the
// top of quantize.cu apply to everything here.
#pragma once

#include <cuda_fp4.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace llnv {
namespace quant {

// ---- exact division by a constant -------------------------------------------------------------
template <int D>
__device__ __forceinline__ float div_const(float x) {
  constexpr float d = (float)D;
  constexpr float r = 1.0f / d;                    // correctly rounded at compile time
  const float q = __fmul_rn(x, r);
  const float rem = __fmaf_rn(-d, q, x);
  return __fmaf_rn(rem, r, q);
}

template <int D>
__device__ __forceinline__ F2 div_const2(F2 x) {
  constexpr float d = (float)D;
  constexpr float r = 1.0f / d;
  const F2 q = f2_mul(x, f2_splat(r));
  const F2 rem = f2_fma(f2_splat(-d), q, x);
  return f2_fma(rem, f2_splat(r), q);
}

// ---- hardware conversions ---------------------------------------------------------------------
// two fp32 -> two E2M1 codes (lo in bits 0-3, hi in bits 4-7), round to nearest even, saturating
__device__ __forceinline__ uint32_t cvt_e2m1x2(float lo, float hi) {
  return (uint32_t)__nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
}
// two E2M1 codes -> two fp32 (x = low nibble)
__device__ __forceinline__ float2 e2m1x2_to_float2(uint32_t byte) {
  const __half2_raw h = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)byte, __NV_E2M1);
  return __half22float2(*reinterpret_cast<const __half2*>(&h));
}
// two E2M1 codes minus two fp32 values (mixed-precision subtraction: the fp16 forms of the codes are exact and need no conversion)
__device__ __forceinline__ F2 e2m1x2_minus(uint32_t byte, F2 t) {
  const __half2_raw h = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)byte, __NV_E2M1);
  F2 d;
  asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d.x) : "h"(h.x), "f"(t.x));
  asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d.y) : "h"(h.y), "f"(t.y));
  return d;
}
// two fp32 -> two E4M3 bytes (lo in bits 0-7), round to nearest even, saturating
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {
  return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float2 e4m3x2_to_float2(uint32_t two) {
  const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)two, __NV_E4M3);
  return __half22float2(*reinterpret_cast<const __half2*>(&h));
}

// ---- reference-faithful scalar pieces (slow path) ---------------------------------------------
// Round |xs| onto {0,.5,1,1.5,2,3,4,6,(8)} with ties to even (reference.py:13-34).
__device__ __forceinline__ float e2m1_round_mag(float a) {
  const float k = a < 2.f ? 2.f : (a < 4.f ? 1.f : 0.5f);
  const float kinv = a < 2.f ? 0.5f : (a < 4.f ? 1.f : 2.f);
  return __fmul_rn(rintf(__fmul_rn(a, k)), kinv);
}
// 4-bit code of a rounded magnitude with the sign of xs (reference.py:37-63); magnitude 8 -> 0b1000
__device__ __forceinline__ uint32_t e2m1_code(float mag, bool neg) {
  const int t = (int)(mag * 2.f);               // 0,1,2,3,4,6,8,12,16
  const uint32_t idx = t < 4 ? (uint32_t)t : (t == 4 ? 4u : (t == 6 ? 5u : (t == 8 ? 6u : (t == 12 ? 7u : 8u))));
  return idx == 8u ? 8u : (idx | (neg ? 8u : 0u));
}

template <int RULE>
__device__ __forceinline__ float err_term(float d) {
  if (RULE == LLNV_RULE_MSE) return __fmul_rn(d, d);
  return fabsf(d);
}

struct QuantConsts {
  float amax, enc, dec;
  bool fast;       // amax has <= 8 significant bits and is large enough that no error term is denormal
};

// Slow path for one candidate scale: the reference's arithmetic operation by operation.
template <int RULE>
__device__ __noinline__ void candidate_slow(const float (&x)[16], float s, float inv, float amax, uint32_t& lo, uint32_t& hi,
                                            float& err) {
  lo = hi = 0u;
  err = 0.f;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    float t[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float xv = x[i + 8 * h];
      const float xs = s != 0.f ? __fmul_rn(xv, inv) : 0.f;
      const float m = e2m1_round_mag(fabsf(xs));
      const uint32_t c = e2m1_code(m, xs < 0.f) << (4 * i);
      if (h == 0) lo |= c; else hi |= c;
      const float q = xs < 0.f ? -m : m;
      const float d = __fsub_rn(__fdiv_rn(__fmul_rn(__fmul_rn(q, s), amax), 1536.f), xv);
      t[h] = err_term<RULE>(d);
    }
    if (RULE == LLNV_RULE_ABS_MAX) err = fmaxf(err, fmaxf(t[0], t[1]));
    else {
      const float a = __fadd_rn(t[0], t[1]);
      err = i == 0 ? a : __fadd_rn(err, a);
    }
  }
}

// The reference's arithmetic on 16 fp32 values (whatever type they were loaded from), operation by operation.
template <int RULE>
__device__ __forceinline__ void quant_block_slow_f(const float (&x)[16], const QuantConsts& qc, float hp, uint32_t& c_lo,
                                                   uint32_t& c_hi, uint32_t& sf_out) {
  const uint32_t sc6 = float_to_e4m3(hp);
  const float s6 = e4m3_to_float(sc6);
  const float inv6 = s6 != 0.f ? __fdiv_rn(1.f, __fmul_rn(qc.dec, s6)) : 0.f;
  uint32_t l6, h6;
  float e6;
  candidate_slow<RULE>(x, s6, inv6, qc.amax, l6, h6, e6);
  if (RULE == LLNV_RULE_STATIC_6 || RULE == LLNV_RULE_STATIC_4) {
    c_lo = l6; c_hi = h6; sf_out = sc6;
    return;
  }
  const uint32_t sc4 = float_to_e4m3(__fmul_rn(hp, 1.5f));
  const float s4 = e4m3_to_float(sc4);
  const float inv4 = s4 != 0.f ? __fdiv_rn(1.f, __fmul_rn(qc.dec, s4)) : 0.f;
  uint32_t l4, h4;
  float e4;
  candidate_slow<RULE>(x, s4, inv4, qc.amax, l4, h4, e4);
  const bool sel4 = e4 < e6;
  c_lo = sel4 ? l4 : l6;
  c_hi = sel4 ? h4 : h6;
  sf_out = sel4 ? sc4 : sc6;
}

// x[16] is indexed with run-time i in candidate_slow: keep it out of the fast path's registers
template <int RULE>
__device__ __noinline__ void quant_block_slow(const uint32_t (&w)[8], const QuantConsts& qc, float hp, uint32_t& c_lo,
                                              uint32_t& c_hi, uint32_t& sf_out) {
  float x[16];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    x[2 * j] = bf16_lo(w[j]);
    x[2 * j + 1] = bf16_hi(w[j]);
  }
  quant_block_slow_f<RULE>(x, qc, hp, c_lo, c_hi, sf_out);
}

// One 16-element block of fp16 input (w: 8 words of packed halves): the values go through the reference's arithmetic as
// fp32, one operation at a time (the packed fast path below relies on bf16 inputs: a tensor amax of at most 8 significant
// bits makes several of its products exact, which an fp16 tensor does not give).  The reference's CUDA backend takes
// fp16 activations as well as bf16 (fouroversix/src/fouroversix/quantize/cuda/backend.py:45-51).
template <int RULE>
__device__ __noinline__ void quant_block_f16(const uint32_t (&w)[8], const QuantConsts& qc, uint32_t& c_lo, uint32_t& c_hi,
                                             uint32_t& sf_out) {
  float x[16];
  float bmax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
    x[2 * j] = f.x;
    x[2 * j + 1] = f.y;
    bmax = fmaxf(bmax, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
  if (bmax == 0.f || qc.amax == 0.f) { c_lo = c_hi = 0u; sf_out = 0u; return; }
  const float hp = RULE == LLNV_RULE_STATIC_4 ? __fmul_rn(__fmul_rn(bmax, 0.25f), qc.enc) : __fmul_rn(__fdiv_rn(bmax, 6.f), qc.enc);
  quant_block_slow_f<RULE>(x, qc, hp, c_lo, c_hi, sf_out);
}

// Whether candidate 4 has the smaller error, with the reference's rounding of every operation (the packed form: each lane
// rounds as the scalar operation does).  sa6, sa4: scale * amax, exact (4 + 8 significant bits).
template <int RULE>
__device__ __forceinline__ bool four_is_better(const uint32_t (&w)[8], float inv6, float inv4, float sa6, float sa4) {
  float e6 = 0.f, e4 = 0.f;
  // pair j holds elements (2j, 2j+1) in w[j] and (2j+8, 2j+9) in w[j+4]; the error sum adds
  // element i to element i+8 first, then the eight lane sums left to right
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const F2 xa = {bf16_lo(w[j]), bf16_hi(w[j])};                    // elements 2j, 2j+1
    const F2 xb = {bf16_lo(w[j + 4]), bf16_hi(w[j + 4])};            // elements 2j+8, 2j+9
    const F2 zero = f2_splat(0.f);
    const F2 sa6v = f2_fma(xa, f2_splat(inv6), zero), sb6v = f2_fma(xb, f2_splat(inv6), zero);
    const F2 sa4v = f2_fma(xa, f2_splat(inv4), zero), sb4v = f2_fma(xb, f2_splat(inv4), zero);
    const uint32_t ca6 = cvt_e2m1x2(sa6v.x, sa6v.y);
    const uint32_t cb6 = cvt_e2m1x2(sb6v.x, sb6v.y);
    const uint32_t ca4 = cvt_e2m1x2(sa4v.x, sa4v.y);
    const uint32_t cb4 = cvt_e2m1x2(sb4v.x, sb4v.y);
    const float2 qa6 = e2m1x2_to_float2(ca6), qb6 = e2m1x2_to_float2(cb6);
    const float2 qa4 = e2m1x2_to_float2(ca4), qb4 = e2m1x2_to_float2(cb4);
    // dequantized candidates minus x, two elements per packed instruction (every lane rounds as the scalar op does)
    const F2 da6 = f2_sub(div_const2<1536>(f2_mul(F2{qa6.x, qa6.y}, f2_splat(sa6))), xa);
    const F2 db6 = f2_sub(div_const2<1536>(f2_mul(F2{qb6.x, qb6.y}, f2_splat(sa6))), xb);
    const F2 da4 = f2_sub(div_const2<1536>(f2_mul(F2{qa4.x, qa4.y}, f2_splat(sa4))), xa);
    const F2 db4 = f2_sub(div_const2<1536>(f2_mul(F2{qb4.x, qb4.y}, f2_splat(sa4))), xb);
    if (RULE == LLNV_RULE_MSE) {
      // lanes 2j and 2j+1 of the 8-lane partial sums: element i plus element i+8
      const F2 l6 = f2_add(f2_mul(da6, da6), f2_mul(db6, db6));
      const F2 l4 = f2_add(f2_mul(da4, da4), f2_mul(db4, db4));
      // running sums of both candidates side by side: (e6, e4) + lane 2j, then + lane 2j+1
      if (j == 0) {
        const F2 e = f2_add(F2{l6.x, l4.x}, F2{l6.y, l4.y});
        e6 = e.x; e4 = e.y;
      } else {
        const F2 e = f2_add(f2_add(F2{e6, e4}, F2{l6.x, l4.x}), F2{l6.y, l4.y});
        e6 = e.x; e4 = e.y;
      }
    } else {
      const float t6a0 = fabsf(da6.x), t6a1 = fabsf(da6.y), t6b0 = fabsf(db6.x), t6b1 = fabsf(db6.y);
      const float t4a0 = fabsf(da4.x), t4a1 = fabsf(da4.y), t4b0 = fabsf(db4.x), t4b1 = fabsf(db4.y);
      if (RULE == LLNV_RULE_ABS_MAX) {
        e6 = fmaxf(fmaxf(e6, fmaxf(t6a0, t6b0)), fmaxf(t6a1, t6b1));
        e4 = fmaxf(fmaxf(e4, fmaxf(t4a0, t4b0)), fmaxf(t4a1, t4b1));
      } else {
        const float l6a = __fadd_rn(t6a0, t6b0), l6b = __fadd_rn(t6a1, t6b1);   // lanes 2j and 2j+1
        const float l4a = __fadd_rn(t4a0, t4b0), l4b = __fadd_rn(t4a1, t4b1);
        e6 = j == 0 ? __fadd_rn(l6a, l6b) : __fadd_rn(__fadd_rn(e6, l6a), l6b);
        e4 = j == 0 ? __fadd_rn(l4a, l4b) : __fadd_rn(__fadd_rn(e4, l4a), l4b);
      }
    }
  }
  return e4 < e6;
}

// The same out of line, for the few blocks that need it.
template <int RULE>
__device__ __noinline__ bool four_is_better_call(uint4 w0, uint4 w1, float inv6, float inv4, float sa6, float sa4) {
  const uint32_t w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
  return four_is_better<RULE>(w, inv6, inv4, sa6, sa4);
}

// Whether candidate 4's codes stand for candidate 6's values at a scale 1.5 times as large: (6, 4), (3, 2), (1.5, 1) or (0, 0) in
// every element, in codes (7, 6), (5, 4), (3, 2), (0, 0) and the same sign.  p0 .. p3: code bytes of candidate 6 (even) and 4 (odd).
__device__ __forceinline__ bool same_values(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3) {
  uint32_t bad = 0;
  const uint32_t p[4] = {p0, p1, p2, p3};
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const uint32_t c6 = __byte_perm(p[i], p[i + 1], 0x6420), c4 = __byte_perm(p[i], p[i + 1], 0x7531);
    const uint32_t odd = c6 & 0x11111111u;
    bad |= (c4 ^ c6 ^ odd) | (c6 & 0x77777777u & ~(odd * 7u));
  }
  return bad == 0;
}

// One 16-element block.  w: 8 words of packed bf16 (element 2j in the low half of w[j]).
// Output: c_lo = codes of elements 0..7 (nibble j), c_hi = codes of elements 8..15, sf byte.
template <int RULE>
__device__ __forceinline__ void quant_block(const uint32_t (&w)[8], const QuantConsts& qc, uint32_t& c_lo, uint32_t& c_hi,
                                            uint32_t& sf_out) {
  constexpr bool kStatic = (RULE == LLNV_RULE_STATIC_6 || RULE == LLNV_RULE_STATIC_4);
  // block maximum on the packed 15-bit magnitudes
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < 8; j += 2) m = __vimax3_u16x2(m, w[j] & 0x7FFF7FFFu, w[j + 1] & 0x7FFF7FFFu);
  const float bmax = __uint_as_float(max(m & 0xFFFFu, m >> 16) << 16);
  float hp;
  if (qc.amax == 0.f) hp = 0.f;
  else if (RULE == LLNV_RULE_STATIC_4) hp = __fmul_rn(__fmul_rn(bmax, 0.25f), qc.enc);
  else hp = __fmul_rn(qc.fast ? div_const<6>(bmax) : __fdiv_rn(bmax, 6.f), qc.enc);

  const uint32_t sc = cvt_e4m3x2(hp, kStatic ? 0.f : __fmul_rn(hp, 1.5f));       // byte 0: 6-scale, byte 1: 4-scale
  const float2 sv = e4m3x2_to_float2(sc);
  const float s6 = sv.x, s4 = sv.y;
  const float inv6 = __frcp_rn(__fmul_rn(qc.dec, s6));

  // Slow path: the corner cases listed in the file header.  2^-100 keeps every quotient, product
  // and error term of the fast path far from the denormal range.
  const float xs_max = __fmul_rn(bmax, inv6);                                    // infinite or NaN where s6 == 0
  if (!qc.fast || !(xs_max < 6.75f) || bmax < 1.0e-28f) {
    if (bmax == 0.f) { c_lo = c_hi = 0u; sf_out = 0u; return; }
    quant_block_slow<RULE>(w, qc, hp, c_lo, c_hi, sf_out);
    return;
  }

  if (kStatic) {
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo |= cvt_e2m1x2(__fmaf_rn(bf16_lo(w[j]), inv6, 0.f), __fmaf_rn(bf16_hi(w[j]), inv6, 0.f)) << (8 * j);
      hi |= cvt_e2m1x2(__fmaf_rn(bf16_lo(w[j + 4]), inv6, 0.f), __fmaf_rn(bf16_hi(w[j + 4]), inv6, 0.f)) << (8 * j);
    }
    c_lo = lo; c_hi = hi; sf_out = sc & 0xFFu;
    return;
  }
  const float inv4 = __frcp_rn(__fmul_rn(qc.dec, s4));
  // Codes of both candidates, and an estimate of both errors in units of the candidate's step: with d = q - x * inv the error of
  // a candidate is s^2 * sum d^2 (s * sum |d|) times a power of dec that both share.
  constexpr bool kEstimate = RULE != LLNV_RULE_ABS_MAX;
  uint32_t pa[8];
  F2 n6 = f2_splat(0.f), n4 = f2_splat(0.f);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const F2 x = {bf16_lo(w[j]), bf16_hi(w[j])};
    // the +0 addend turns a -0 product (input -0.0) into +0, as the reference's sign(x)*|.| does
    const F2 t6 = f2_fma(x, f2_splat(inv6), f2_splat(0.f)), t4 = f2_fma(x, f2_splat(inv4), f2_splat(0.f));
    const uint32_t k6 = cvt_e2m1x2(t6.x, t6.y), k4 = cvt_e2m1x2(t4.x, t4.y);
    // candidate-6 and candidate-4 code bytes of this pair side by side; the selected ones are gathered at the end
    pa[j] = __byte_perm(k6, k4, 0x0040);
    if (!kEstimate) continue;
    const F2 d6 = e2m1x2_minus(k6, t6), d4 = e2m1x2_minus(k4, t4);
    if (RULE == LLNV_RULE_MSE) {
      n6 = f2_fma(d6, d6, n6);
      n4 = f2_fma(d4, d4, n4);
    } else {
      n6.x += fabsf(d6.x), n6.y += fabsf(d6.y);
      n4.x += fabsf(d4.x), n4.y += fabsf(d4.y);
    }
  }
  const float sa6 = __fmul_rn(s6, qc.amax), sa4 = __fmul_rn(s4, qc.amax);        // exact (4 + 8 significant bits)
  // bytes (c6_0, c4_0, c6_1, c4_1) and so on: the even ones are candidate 6's, the odd ones candidate 4's
  const uint32_t p0 = __byte_perm(pa[0], pa[1], 0x5410), p1 = __byte_perm(pa[2], pa[3], 0x5410);
  const uint32_t p2 = __byte_perm(pa[4], pa[5], 0x5410), p3 = __byte_perm(pa[6], pa[7], 0x5410);
  bool sel4;
  if (kEstimate) {
    // The choice is the estimate's where its margin exceeds what rounding can move.  In units of a step |x * inv| < 6.75 and
    // |q| <= 6, so the reference's d (three roundings of at most 2^-24 * 6.75) and the one here (x * inv with five roundings
    // behind it, and one subtraction) are each within 2.5e-6 of the exact difference: D = 5e-6 between them.  With n = sum d^2
    // of 16 terms that moves n by at most 2 D * 4 sqrt(n) + 16 D^2 < 2.1e-5 (n + 1), and the roundings of the sums by less than
    // 3e-6 n; a sum of magnitudes moves by 16 D = 8e-5 plus 3e-6 n.  The margin is almost twice that.  Of Gaussian data
    // about one block in 2000 falls inside it and is decided by the reference's own arithmetic; of blocks with one or a few values up to a
    // third do, nearly all because both candidates stand for the same values.
    // us for 2640 x 14336 bf16, amax given, exact arithmetic for every block / for those inside the margin / and for those of them whose
    // values differ: Gaussian 39.2 / 28.2 / 28.4, 90 % zeros 51 / 58 / 44, one value a block 48 / 56 / 40, all equal 39 / 48 / 29, after a
    // ReLU 39 / 30 / 28.5.  (With the largest |d| as the criterion both candidates often share the block maximum's error exactly, and
    // estimating first cost 20 %.)
    constexpr bool kMse = RULE == LLNV_RULE_MSE;
    const float u6 = kMse ? __fmul_rn(s6, s6) : s6, u4 = kMse ? __fmul_rn(s4, s4) : s4;
    const float e6 = __fmul_rn(u6, n6.x + n6.y), e4 = __fmul_rn(u4, n4.x + n4.y);
    constexpr float kTolRel = kMse ? 4.2e-5f : 6.0e-6f, kTolAbs = kMse ? 4.2e-5f : 1.6e-4f;
    sel4 = e4 < e6;
    if (!(fabsf(e4 - e6) > kTolRel * (e4 + e6) + kTolAbs * (u4 + u6))) {
      // equal values have equal errors, whatever the rounding: 6 stays
      if (s4 == 1.5f * s6 && same_values(p0, p1, p2, p3)) sel4 = false;
      else sel4 = four_is_better_call<RULE>(make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]), inv6, inv4, sa6, sa4);
    }
  } else {
    sel4 = four_is_better<RULE>(w, inv6, inv4, sa6, sa4);
  }
  const uint32_t pick = sel4 ? 0x7531u : 0x6420u;
  c_lo = __byte_perm(p0, p1, pick);
  c_hi = __byte_perm(p2, p3, pick);
  sf_out = sel4 ? (sc >> 8) : (sc & 0xFFu);
}

// Constants of a tensor with the given amax (reference.py:142-166).
template <int RULE>
__device__ __forceinline__ QuantConsts make_consts(float amax) {
  constexpr float kE2 = RULE == LLNV_RULE_STATIC_4 ? 4.f : 6.f;
  constexpr float kE4 = (RULE == LLNV_RULE_STATIC_6 || RULE == LLNV_RULE_STATIC_4) ? 448.f : 256.f;
  QuantConsts qc;
  qc.amax = amax;
  qc.enc = __fdiv_rn(kE2 * kE4, qc.amax);     // reference.py:142-151
  qc.dec = __fdiv_rn(1.f, qc.enc);            // reference.py:159-166
  qc.fast = (__float_as_uint(qc.amax) & 0xFFFFu) == 0u && qc.amax > 1.0e-20f && qc.amax < 1.0e30f;
  return qc;
}

}  // namespace quant
}  // namespace llnv
