// Packed quantizer arithmetic shared by the append step (append_fast.cu) and the functional quantizers
// (quantize_fast.cu): two 16-bit elements per register, rounded per operation in the data dtype like the reference
// (src/dart/quantization.py:178-186, src/dart/mixed.py:200-209).
#pragma once

#include "common.cuh"

namespace {

// range / qmax rounded to the data dtype.  For bf16 the quotient of two 8-bit significands is never within
// 2^-17 of a rounding boundary (see below), so a multiply by the fp32 reciprocal rounds to the same bf16.
template <int DT>
__device__ __forceinline__ float scale_of(float mn, float mx, float qmax) {
  float range = rnd<DT>(__fsub_rn(mx, mn));
  range = fmaxf(range, rnd<DT>(1e-4f));
  // qmax is one of 3, 15, 255: correctly rounded fp32 reciprocals as constants
  const float inv_qmax = qmax == 3.0f ? 0.3333333432674408f : (qmax == 15.0f ? 0.06666667014360428f : 0.003921568859368563f);
  if (DT == DARTKV_BF16) return rnd<DT>(__fmul_rn(range, inv_qmax));
  return rnd<DT>(__fdiv_rn(range, qmax));
}
// 1 / scale for the quotients below: the approximate reciprocal is within 2^-22 (0 for an infinite scale)
__device__ __forceinline__ float inverse_scale(float scale) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(scale));
  return r;
}

// ---- packed code computation -------------------------------------------------------------------
// Two elements that share (min, scale) travel as one 16-bit pair.  The reference computes
//   code = clamp(rint(r16(r16(x - min) / scale)), 0, qmax)        (r16 = round to the data dtype)
// which is evaluated here as
//   a2   = x2 - min2                      packed subtract, one rounding (exact for the 16-bit formats)
//   q    = a * (1/scale)         bf16: the quotient of two 8-bit significands is never within 2^-17 of a bf16
//                                rounding boundary and never on one, so a reciprocal multiply rounds to the
//                                same bf16 as the IEEE quotient
//          q + (a - q*scale)/scale   fp16: a boundary b between two fp16 numbers has a 12-bit odd significand N, so
//                                a = b * scale would need 11 bits to hold N * (odd part of scale) >= 2^11 + 1:
//                                never on a boundary, and |a - b*scale| is at least one unit of a product below
//                                2^23, i.e. the quotient stays 2^-23 (relative) away from every boundary, while
//                                one exact-residual step leaves q within 2^-24.  An infinite scale (the range of
//                                the group overflows fp16) enters as scale = 1/scale = 0.
//   r2   = r16(q) packed
//   m2   = r2 + magic                     magic = 128 (bf16) / 1024 (fp16): the sum has unit ulp, so the
//                                         packed add rounds half-to-even to an integer = rint
// leaving the codes in the low mantissa bits of each half.  bf16 cannot hold 128 + code for 8-bit
// codes; that combination uses scalar rint.
template <int DT> struct Pack16;
template <> struct Pack16<DARTKV_BF16> {
  static constexpr uint32_t kMagic = 0x43004300u;   // 128.0 | 128.0
  static constexpr uint32_t kInfinity = 0x7F807F80u;
  static __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
    uint32_t d; asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
    uint32_t d; asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) {
    uint32_t d; asm("min.NaN.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t cap2(uint32_t a, uint32_t b) {   // a NaN becomes the cap
    uint32_t d; asm("min.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t floor2(uint32_t a, uint32_t b) {
    uint32_t d; asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    uint32_t d; asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ float lo(uint32_t v) { return __uint_as_float(v << 16); }
  static __device__ __forceinline__ float hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
  static __device__ __forceinline__ uint32_t pack(float hi_v, float lo_v) {
    uint32_t d; asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi_v), "f"(lo_v)); return d;
  }
  // the quotients of a pair, rounded to bf16: both products in one packed fp32 multiply
  static __device__ __forceinline__ uint32_t quotients(uint32_t a2, float, float, float inv_lo, float inv_hi) {
    uint32_t d;
    asm("{\n.reg .b64 a, b, q;\n.reg .f32 ql, qh;\n"
        "mov.b64 a, {%1, %2};\nmov.b64 b, {%3, %4};\nmul.rn.f32x2 q, a, b;\nmov.b64 {ql, qh}, q;\n"
        "cvt.rn.bf16x2.f32 %0, qh, ql;\n}"
        : "=r"(d) : "f"(lo(a2)), "f"(hi(a2)), "f"(inv_lo), "f"(inv_hi));
    return d;
  }
  static __device__ __forceinline__ uint16_t bits(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }
};
template <> struct Pack16<DARTKV_F16> {
  static constexpr uint32_t kMagic = 0x64006400u;   // 1024.0 | 1024.0
  static constexpr uint32_t kInfinity = 0x7C007C00u;
  static __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
    uint32_t d; asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
    uint32_t d; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) {
    uint32_t d; asm("min.NaN.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t cap2(uint32_t a, uint32_t b) {
    uint32_t d; asm("min.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t floor2(uint32_t a, uint32_t b) {
    uint32_t d; asm("max.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    uint32_t d; asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
  }
  static __device__ __forceinline__ float lo(uint32_t v) { return __half2float(__ushort_as_half((uint16_t)(v & 0xFFFFu))); }
  static __device__ __forceinline__ float hi(uint32_t v) { return __half2float(__ushort_as_half((uint16_t)(v >> 16))); }
  static __device__ __forceinline__ uint32_t pack(float hi_v, float lo_v) {
    uint32_t d; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi_v), "f"(lo_v)); return d;
  }
  static __device__ __forceinline__ float quotient(float a, float s, float inv) {
    const float q = __fmul_rn(a, inv);
    return __fmaf_rn(__fmaf_rn(-q, s, a), inv, q);
  }
  static __device__ __forceinline__ uint32_t quotients(uint32_t a2, float s_lo, float s_hi, float inv_lo, float inv_hi) {
    return pack(quotient(hi(a2), s_hi, inv_hi), quotient(lo(a2), s_lo, inv_lo));
  }
  static __device__ __forceinline__ uint16_t bits(float v) { return __half_as_ushort(__float2half_rn(v)); }
};


// whether an element of the pair is Inf or NaN
template <int DT>
__device__ __forceinline__ bool pair_nonfinite(uint32_t v) {
  constexpr uint32_t kUnit = DT == DARTKV_BF16 ? 0x00800080u : 0x04000400u;   // one step of the exponent
  return ((v & 0x7FFF7FFFu) + kUnit) & 0x80008000u;
}

// magic exponents in the codes of a pair (none where scalar rint produced them)
template <int DT, int BITS>
__host__ __device__ constexpr uint32_t pair_magic() {
  return DT == DARTKV_BF16 && BITS == 8 ? 0u : (DT == DARTKV_BF16 ? 0x43004300u : 0x64006400u);
}
// largest code of a pair, as pair_codes() compares it
template <int DT>
__device__ __forceinline__ uint32_t cap_pair(float qmax_lo, float qmax_hi) {
  constexpr float kBase = DT == DARTKV_BF16 ? 128.0f : 1024.0f;
  return (uint32_t)Pack16<DT>::bits(kBase + qmax_lo) | ((uint32_t)Pack16<DT>::bits(kBase + qmax_hi) << 16);
}
// codes of a pair, plus pair_magic(): low element in bits [15:0], high element in bits [31:16]
template <int DT, int BITS>
__device__ __forceinline__ uint32_t pair_codes(uint32_t x2, uint32_t mn2, float s_lo, float s_hi, float inv_lo, float inv_hi,
                                               uint32_t cap2) {
  using P = Pack16<DT>;
  const uint32_t r2 = P::quotients(P::sub(x2, mn2), s_lo, s_hi, inv_lo, inv_hi);
  if (DT == DARTKV_BF16 && BITS == 8)
    return (uint32_t)fminf(rintf(P::lo(r2)), 255.0f) | ((uint32_t)fminf(rintf(P::hi(r2)), 255.0f) << 16);
  return P::cap2(P::add(r2, P::kMagic), cap2);
}

// sum of 4^... shifted magic exponents of a gather register: `count` pairs, `step` bits apart (modulo 2^32)
__host__ __device__ constexpr uint32_t magic_sum(uint32_t magic, int count, int step) {
  uint32_t sum = 0;
  for (int i = 0; i < count; ++i) sum += magic << (step * i);
  return sum;
}

// acc + (codes << shift) as one multiply-add
__device__ __forceinline__ uint32_t gather(uint32_t acc, uint32_t codes, int shift) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(codes), "r"(1u << shift), "r"(acc));
  return d;
}

// two neighbouring metadata values (scale or zero point), rounded to the metadata dtype
__device__ __forceinline__ void store_pair(void* p, int md, int64_t pair, float a, float b) {
  if (md == DARTKV_F32) reinterpret_cast<float2*>(p)[pair] = make_float2(a, b);
  else if (md == DARTKV_F16) reinterpret_cast<uint32_t*>(p)[pair] = Pack16<DARTKV_F16>::pack(b, a);
  else reinterpret_cast<uint32_t*>(p)[pair] = Pack16<DARTKV_BF16>::pack(b, a);
}

}  // namespace
