// Packed codes of any width to 16-bit numbers, two codes with scales of their own per register (decode_rows.cu, decode_many.cu).
#pragma once

#include "mma_utils.cuh"

namespace {

// scale and zero point of the two elements of a register, made ready for codes at any of the in-mantissa positions.
// MD: metadata dtype (the arithmetic), OUT: cache dtype (the MMA operand), FP32: the fp32 flavour.
template <int MD, int OUT, bool FP32>
struct PairAffine {
  using H = Half2Ops<MD>;
  uint32_t ss, zz, ms[3];
  float s0, s1, z0, z1;
  template <int POSITIONS>
  __device__ __forceinline__ void init(uint32_t scales, uint32_t zeros) {
    if (FP32) {
      unpack16<MD>(scales, s0, s1);
      unpack16<MD>(zeros, z0, z1);
    } else {
      ss = scales; zz = zeros;
#pragma unroll
        for (int j = 0; j < POSITIONS; ++j) ms[j] = H::mul(ss, H::neg_magic(j));
    }
  }
  // m = magic(J) + code in both halves
  template <int J>
  __device__ __forceinline__ uint32_t restore(uint32_t m) const {
    if (!FP32) return cast16<MD, OUT>(H::add(H::fma(m, ss, ms[J]), zz));
    float c0, c1;
    unpack16<MD>(H::add(m, H::neg_magic(J)), c0, c1);
    return pack16<OUT>(__fmaf_rn(c0, s0, z0), __fmaf_rn(c1, s1, z1));
  }
};

// eight 2-bit codes per half of x -> eight registers
template <int MD, int OUT, bool FP32>
__device__ __forceinline__ void restore_codes2(const CodeConsts<MD>& k, uint32_t x, const PairAffine<MD, OUT, FP32>& a, uint32_t (&r)[8]) {
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
template <int MD, int OUT, bool FP32>
__device__ __forceinline__ void restore_codes22(const CodeConsts<MD>& k, uint32_t xl, uint32_t xh, const PairAffine<MD, OUT, FP32>& a,
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
template <int MD, int OUT, bool FP32>
__device__ __forceinline__ void restore_codes4(const CodeConsts<MD>& k, uint32_t mask4, uint32_t x, const PairAffine<MD, OUT, FP32>& a,
                                               uint32_t* r) {
  constexpr int P0 = Half2Ops<MD>::kFirstPos;
#pragma unroll
  for (int u = 0; u < 4; ++u) r[u] = a.template restore<0>(and_or(align_codes(x, 2 * u, P0), mask4, k.magic[0]));
}

// the four 8-bit codes of a word for each half -> four registers.  Eight bits fit an fp16 mantissa (1024 + code; the magic
// is subtracted first, 1024 * scale could overflow) but not a bf16 one: there through fp32 (8388608 + code, exact).
template <int MD, int OUT, bool FP32>
__device__ __forceinline__ void restore_codes8(uint32_t w0, uint32_t w1, const PairAffine<MD, OUT, FP32>& a, uint32_t* r) {
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

__device__ __forceinline__ uint32_t lds_u16(const uint8_t* p) { return *reinterpret_cast<const uint16_t*>(p); }
__device__ __forceinline__ uint32_t lds_u32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t d;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(x));
  return d;
}

}  // namespace
