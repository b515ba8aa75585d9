// Packed codes of any width to 16-bit numbers, two codes with scales of their own per register: MMA operands (decode_rows.cu,
// decode_many.cuh) and restored keys and values (materialize.cu, quantize_fast.cu).
#pragma once

#include "mma_utils.cuh"

namespace {

// scale and zero point of the two elements of a register, made ready for codes at any of the in-mantissa positions.
// MD: metadata dtype (the arithmetic), OUT: cache dtype (the MMA operand), FP32: the fp32 flavour.  WIDE: any scale, at one
// operation more (the magic number is subtracted first); without it magic * scale must not overflow.
template <int MD, int OUT, bool FP32, bool WIDE = false>
struct PairAffine {
  using H = Half2Ops<MD>;
  static constexpr bool kFp32 = FP32;
  uint32_t ss, zz, ms[3];
  float s0, s1, z0, z1;
  template <int POSITIONS>
  __device__ __forceinline__ void init(uint32_t scales, uint32_t zeros) {
    if (FP32) {
      unpack16<MD>(scales, s0, s1);
      unpack16<MD>(zeros, z0, z1);
    } else {
      ss = scales; zz = zeros;
      if (!WIDE)
#pragma unroll
        for (int j = 0; j < POSITIONS; ++j) ms[j] = H::mul(ss, H::neg_magic(j));
    }
  }
  // m = magic(J) + code in both halves
  template <int J>
  __device__ __forceinline__ uint32_t restore(uint32_t m) const {
    if (!FP32) return cast16<MD, OUT>(H::add(WIDE ? H::mul(H::add(m, H::neg_magic(J)), ss) : H::fma(m, ss, ms[J]), zz));
    float c0, c1;
    unpack16<MD>(H::add(m, H::neg_magic(J)), c0, c1);
    return pack16<OUT>(__fmaf_rn(c0, s0, z0), __fmaf_rn(c1, s1, z1));
  }
};

// eight 2-bit codes per half of x -> eight registers
template <int MD, int OUT, bool FP32, bool WIDE>
__device__ __forceinline__ void restore_codes2(const CodeConsts<MD>& k, uint32_t x, const PairAffine<MD, OUT, FP32, WIDE>& a, uint32_t (&r)[8]) {
  constexpr int P0 = Half2Ops<MD>::kFirstPos;
  const uint32_t x0 = align_codes(x, 0, P0), x1 = align_codes(x, 3, P0), x2 = align_codes(x, 6, P0);
  r[0] = a.template restore<0>(and_or(x0, k.mask[0], k.magic[0]));
  r[1] = a.template restore<1>(and_or(x0, k.mask[1], k.magic[1]));
  r[2] = a.template restore<2>(and_or(x0, k.mask[2], k.magic[2]));
  r[3] = a.template restore<0>(and_or(x1, k.mask[0], k.magic[0]));
  r[4] = a.template restore<1>(and_or(x1, k.mask[1], k.magic[1]));
  r[5] = a.template restore<2>(and_or(x1, k.mask[2], k.magic[2]));
  r[6] = a.template restore<0>(and_or(x2, k.mask[0], k.magic[0]));
  r[7] = a.template restore<1>(and_or(x2, k.mask[1], k.magic[1]));
}

// eight codes per half split over a low and a high plane (code = low | high << 2) -> eight registers
template <int MD, int OUT, bool FP32, bool WIDE>
__device__ __forceinline__ void restore_codes22(const CodeConsts<MD>& k, uint32_t xl, uint32_t xh, const PairAffine<MD, OUT, FP32, WIDE>& a,
                                                uint32_t (&r)[8]) {
  constexpr int P0 = Half2Ops<MD>::kFirstPos;
#pragma unroll
  for (int grp = 0; grp < 4; ++grp) {
    const uint32_t l = align_codes(xl, 2 * grp, P0), h = align_codes(xh, 2 * grp, P0, 2);
    r[2 * grp] = a.template restore<0>(and_or(h, k.mask[1], and_or(l, k.mask[0], k.magic[0])));
    r[2 * grp + 1] = a.template restore<1>(and_or(h, k.mask[2], and_or(l, k.mask[1], k.magic[1])));
  }
}

// four 4-bit codes per half of x -> four registers (bits 4..7 of an fp16 mantissa, 0..3 of a bf16 mantissa: magic(0))
template <int MD, int OUT, bool FP32, bool WIDE>
__device__ __forceinline__ void restore_codes4(const CodeConsts<MD>& k, uint32_t mask4, uint32_t x, const PairAffine<MD, OUT, FP32, WIDE>& a,
                                               uint32_t* r) {
  constexpr int P0 = Half2Ops<MD>::kFirstPos;
#pragma unroll
  for (int u = 0; u < 4; ++u) r[u] = a.template restore<0>(and_or(align_codes(x, 2 * u, P0), mask4, k.magic[0]));
}

// the four 8-bit codes of a word for each half -> four registers.  Eight bits fit an fp16 mantissa (1024 + code; the magic
// is subtracted first, 1024 * scale could overflow) but not a bf16 one: there through fp32 (8388608 + code, exact).
template <int MD, int OUT, bool FP32, bool WIDE>
__device__ __forceinline__ void restore_codes8(uint32_t w0, uint32_t w1, const PairAffine<MD, OUT, FP32, WIDE>& a, uint32_t* r) {
  using H = Half2Ops<MD>;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (FP32 || MD == DARTKV_BF16) {
      const float c0 = __uint_as_float(prmt(w0, 0x4B000000u, j | 0x7540u)) - 8388608.0f;
      const float c1 = __uint_as_float(prmt(w1, 0x4B000000u, j | 0x7540u)) - 8388608.0f;
      r[j] = FP32 ? pack16<OUT>(__fmaf_rn(c0, a.s0, a.z0), __fmaf_rn(c1, a.s1, a.z1))
                  : cast16<MD, OUT>(H::add(H::mul(pack16<MD>(c0, c1), a.ss), a.zz));
    } else {
      const uint32_t m = and_or(prmt(w0, w1, j * 0x0011u | (4 + j) * 0x1100u), 0x00FF00FFu, 0x64006400u);
      r[j] = cast16<MD, OUT>(H::add(H::mul(H::add(m, 0xE400E400u), a.ss), a.zz));
    }
  }
}

// The codes of one word of each of two neighbouring columns, BITS wide (0: 2-bit codes with a second plane for promoted columns), in
// kColumnParts<BITS> parts of N elements: element part * N + u of both columns is r[u].
template <int BITS> constexpr int kColumnParts = BITS == 8 ? 1 : 2;
template <int MD, int OUT, bool FP32, int BITS, int N>
__device__ __forceinline__ void restore_columns(const CodeConsts<MD>& k, const uint32_t (&w)[2], const uint32_t (&high)[2],
                                                const PairAffine<MD, OUT, FP32, true>& affine, int part, uint32_t (&r)[N]) {
  static_assert(N * kColumnParts<BITS> == 32 / (BITS == 0 ? 2 : BITS), "a word's elements");
  if constexpr (BITS == 8) {
    restore_codes8<MD, OUT>(w[0], w[1], affine, r);
  } else {
    const uint32_t sel = part ? 0x7632u : 0x5410u, x = prmt(w[0], w[1], sel);
    if constexpr (BITS == 0) restore_codes22<MD, OUT>(k, x, prmt(high[0], high[1], sel), affine, r);
    else if constexpr (BITS == 2) restore_codes2<MD, OUT>(k, x, affine, r);
    else restore_codes4<MD, OUT>(k, 0x000F000Fu << (2 * Half2Ops<MD>::kFirstPos), x, affine, r);
  }
}

// Eight neighbouring codes of a row, BITS wide, of one group.
template <int MD, int OUT, bool FP32, int BITS>
__device__ __forceinline__ void restore_row(const CodeConsts<MD>& k, uint64_t codes, uint32_t scale, uint32_t zero, uint32_t (&r)[4]) {
  constexpr int P0 = Half2Ops<MD>::kFirstPos;
  PairAffine<MD, OUT, FP32, true> affine;
  affine.template init<0>(low_twice(scale), low_twice(zero));
  const uint32_t lo = (uint32_t)codes, hi = (uint32_t)(codes >> 32);
  if constexpr (BITS == 8) {
    restore_codes8<MD, OUT>(prmt(lo, hi, 0x6420u), prmt(lo, hi, 0x7531u), affine, r);
  } else if constexpr (BITS == 4) {
    // the odd codes move up to the half-word above the even ones: two pairs a word, eight bits apart
    constexpr uint32_t mask = 0x000F000Fu << (2 * P0);
    const uint32_t x[2] = {(lo & 0xFFFFu) | ((lo << 12) & 0xFFFF0000u), (lo >> 16) | ((lo >> 4) & 0xFFFF0000u)};
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = affine.template restore<0>(and_or(align_codes(x[i >> 1], 4 * (i & 1), P0), mask, k.magic[0]));
  } else {
    const uint32_t x = lo | (lo << 14);   // pair i four bits on from pair i - 1: positions 0 and 2 of two alignments
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t y = align_codes(x, 4 * i, P0);
      r[2 * i] = affine.template restore<0>(and_or(y, k.mask[0], k.magic[0]));
      r[2 * i + 1] = affine.template restore<2>(and_or(y, k.mask[2], k.magic[2]));
    }
  }
}

__device__ __forceinline__ uint32_t lds_u16(const uint8_t* p) { return *reinterpret_cast<const uint16_t*>(p); }
__device__ __forceinline__ uint32_t lds_u32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t d;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(x));
  return d;
}

}  // namespace
