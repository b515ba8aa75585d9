// One page of the per-op rounded decode on tensor cores, as one warp works on it, or one of two warps on half of its tokens:
// contraction table, logits, online softmax, P.V.
//
// Packed 2-bit codes are turned into exactly rounded 16-bit operands with one logic op and two packed fma/add per pair
// (mma_utils.cuh) and fed straight into m16n8k16 MMAs; K and V are never materialized.  Keys: a register of the operand
// pairs two tokens of one channel (they share the channel's scale and zero point), which is the MMA's non-contraction
// direction, so the contraction index is doubled, k = (channel, j), against a block-diagonal query operand whose columns
// are (query head, j).  Values: the code words of two tokens are byte-interleaved so that a register pairs two TOKENS of
// one channel, the contraction direction itself; each half of the packed arithmetic carries its own token's scale and
// zero point, the probability operand is plain (p[a], p[b]), and its eight columns hold the high and the low 16-bit parts
// of the four heads' probabilities, so one MMA accumulates both.
//
// Lane (g, c) = (lane >> 2, lane & 3).  A thread reads the whole 32-bit word g of a channel's code row, tokens 16g .. 16g+15;
// register u pairs tokens 16g + u and 16g + u + 8, and registers 2mt, 2mt + 1 are the row halves of m-tile mt.
#pragma once

#include "decode_fast_common.cuh"

namespace {

constexpr int kProbStride = 136;   // 16-bit elements per (part, head) row of the probabilities: 128 tokens, 8 pad

// what a warp needs beside a staged page; the probabilities take the table's place after the logits
union PageScratch {
  // by contraction position: (s, s), (z, z), (-magic0*s, -magic1*s), (-magic2*s, byte offset of the channel's row)
  uint4 table[128];
  uint16_t prob[2 * 4 * kProbStride];   // [hi/lo][head][local token]
};

// the dequantized registers of a code word, from the metadata dtype to the cache dtype (nothing when they agree)
template <int DT, int OUT, int N>
__device__ __forceinline__ void cast_registers(uint32_t (&r)[N]) {
  if (DT != OUT) {
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = cast16<DT, OUT>(r[i]);
  }
}


// DT = metadata dtype (the arithmetic of the dequantization), OUT = cache dtype (the MMA operands): when they differ
// every dequantized register is cast, as the reference casts its dequantized pages (src/dart/quantization.py:103-106).
// GN: value groups per token (1 or 2).  KP: promoted channels per page when that is a multiple of eight known to
// the host (0, 8, 16, 24, 32), else -1 (read from the descriptor): with the count fixed the logits loops have
// constant trip counts and no per-position "is this slot promoted" test.
template <int DT, int OUT, int GN, int KP>
struct PageWork {
  using H = Half2Ops<DT>;
  using HO = Half2Ops<OUT>;
  // Unrolling, for whole pages: longer bodies cost instruction fetch on the first pages of a call, shorter ones expose
  // shared-memory latency.  Batch 128, 32,768 tokens: 1,026 us; with two promoted steps 1,042, with two or six of the other
  // logits' 1,035 and 1,037, with two of P.V 1,027.  fp16 scales beside bf16, 32 x 8,192 tokens: two of the other logits' steps
  // 112.3 us, four 114.5.
  static constexpr int kPromUnroll = 4, kQkUnroll = DT == OUT ? 4 : 2, kPvUnroll = 1;
  CodeConsts<DT> cc;
  const dartkv_cache_desc& d;
  const uint8_t* q_thread;   // this thread's column of the query: + 32 * channel
  float scale2;
  int lane, g, c, K, prom_steps;
  bool gv;                   // this thread's sixteen channels are of value group 1
  float o_acc[8][4];         // [m-tile][c-reg]: channel 16g + mt + 8(i>>1), head 2(c&1) + (i&1), high (c<2) or low part of P
  float m_run, l_run;        // head c, log2 domain

  __device__ __forceinline__ PageWork(const dartkv_cache_desc& desc, const void* query_table, float scale, int lane_)
      : d(desc), scale2(scale * kLog2e), lane(lane_), g(lane_ >> 2), c(lane_ & 3) {
    cc.init();
    K = KP >= 0 ? KP : (d.key_mode == DARTKV_MIXED_PAGE ? d.promoted : 0);
    prom_steps = (K + 7) >> 3;
    gv = (16 * g) / d.value_group;
    q_thread = reinterpret_cast<const uint8_t*>(query_table) + 4 * g;
  }

  // column n = g of the query operand: head g >> 1 in half j' = g & 1, zero in the other; row32 = 32 * channel
  __device__ __forceinline__ uint32_t query(uint32_t row32) const {
    return *reinterpret_cast<const uint32_t*>(q_thread + row32);
  }

  __device__ __forceinline__ void start_row() {
#pragma unroll
    for (int mt = 0; mt < 8; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) o_acc[mt][i] = 0.0f;
    m_run = -INFINITY;
    l_run = 0.0f;
  }

  // contraction table: the promoted slots first, then the other channels in order
  __device__ __forceinline__ void fill_table(const uint8_t* keys, PageScratch& scratch) const {
    const uint16_t* kscale = reinterpret_cast<const uint16_t*>(keys + d.key_off_scale);
    const uint16_t* kzero = reinterpret_cast<const uint16_t*>(keys + d.key_off_zero);
    auto fill = [&](int pos, int ch) {
      const uint32_t ss = (uint32_t)kscale[ch] * 0x00010001u, zz = (uint32_t)kzero[ch] * 0x00010001u;
      const uint32_t m01 = H::mul(ss, (H::neg_magic(0) & 0xFFFFu) | (H::neg_magic(1) & 0xFFFF0000u));
      const uint32_t m2 = H::mul(ss, H::neg_magic(2));
      scratch.table[pos] = make_uint4(ss, zz, m01, prmt(m2, 32u * ch, 0x5410u));
    };
    int slot_channel = -1;
    if (K > 0 && lane < K) slot_channel = reinterpret_cast<const int32_t*>(keys + d.key_off_index)[lane] & 127;
    if (slot_channel >= 0) fill(lane, slot_channel);
    int position = K;   // of the first channel of the next 32
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t promoted = 0;
      if (K > 0) promoted = __reduce_or_sync(0xffffffffu, (slot_channel >> 5) == i ? 1u << (slot_channel & 31) : 0u);
      const uint32_t below = promoted & ((1u << lane) - 1u);
      if (!((promoted >> lane) & 1u)) fill(min(position + lane - __popc(below), 127), 32 * i + lane);
      position += 32 - __popc(promoted);
    }
  }

  // logits S[token pair][(head, j')] over the doubled contraction (channel, j), eight positions per step.  MT: m-tiles, 4 for
  // the whole page or 2 for the half `hf` of it (codes u = 4hf .. 4hf + 3 of each half of a word)
  template <int MT>
  __device__ __forceinline__ void logits(const uint8_t* keys, const PageScratch& scratch, int hf, float (&s_acc)[MT][4]) const {
    const uint8_t* const low_thread = keys + 4 * g;                                                     // + 32 * channel
    const uint32_t* const high_thread = reinterpret_cast<const uint32_t*>(keys + d.key_off_high) + g;   // + 8 * slot
    const int shift = MT == 4 ? 0 : 8 * hf;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s_acc[mt][i] = 0.0f;
#pragma unroll kPromUnroll
    for (int i = 0; i < prom_steps; ++i) {
      const int s0 = 8 * i + c, s1 = s0 + 4;
      const uint4 e0 = scratch.table[s0], e1 = scratch.table[s1];
      const uint32_t o0 = e0.w >> 16, o1 = e1.w >> 16;
      const uint32_t w0 = *reinterpret_cast<const uint32_t*>(low_thread + o0) >> shift;
      const uint32_t w1 = *reinterpret_cast<const uint32_t*>(low_thread + o1) >> shift;
      // with a promoted count that is a multiple of eight every position of a promoted step is a promoted slot
      const uint32_t h0 = (KP >= 0 || s0 < K) ? high_thread[s0 * 8] >> shift : 0u;
      const uint32_t h1 = (KP >= 0 || s1 < K) ? high_thread[s1 * 8] >> shift : 0u;
      uint32_t r0[2 * MT], r1[2 * MT];
      dequant_word4<DT>(cc, w0, h0, e0.x, e0.y, low_twice(e0.z), high_twice(e0.z), r0);
      dequant_word4<DT>(cc, w1, h1, e1.x, e1.y, low_twice(e1.z), high_twice(e1.z), r1);
      cast_registers<DT, OUT>(r0);
      cast_registers<DT, OUT>(r1);
      const uint32_t b0 = query(o0), b1 = query(o1);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) HO::mma(s_acc[mt], r0[2 * mt], r0[2 * mt + 1], r1[2 * mt], r1[2 * mt + 1], b0, b1);
    }
#pragma unroll kQkUnroll
    for (int i = prom_steps; i < 16; ++i) {
      const int s0 = 8 * i + c, s1 = s0 + 4;
      const uint4 e0 = scratch.table[s0], e1 = scratch.table[s1];
      const uint32_t o0 = e0.w >> 16, o1 = e1.w >> 16;
      const uint32_t w0 = *reinterpret_cast<const uint32_t*>(low_thread + o0) >> shift;
      const uint32_t w1 = *reinterpret_cast<const uint32_t*>(low_thread + o1) >> shift;
      uint32_t r0[2 * MT], r1[2 * MT];
      dequant_word2<DT>(cc, w0, e0.x, e0.y, low_twice(e0.z), high_twice(e0.z), low_twice(e0.w), r0);
      dequant_word2<DT>(cc, w1, e1.x, e1.y, low_twice(e1.z), high_twice(e1.z), low_twice(e1.w), r1);
      cast_registers<DT, OUT>(r0);
      cast_registers<DT, OUT>(r1);
      const uint32_t b0 = query(o0), b1 = query(o1);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) HO::mma(s_acc[mt], r0[2 * mt], r0[2 * mt + 1], r1[2 * mt], r1[2 * mt + 1], b0, b1);
    }
  }

  // online softmax for head c (this thread's tokens are 16g + u + 8j, u = 2mt + (i >> 1), j = i & 1, in a half + 4hf); the
  // probabilities go to the table with the pairs (u, u + 8) side by side.  mask_below: tokens before it drop out.
  template <int MT>
  __device__ __forceinline__ void softmax(float (&s_acc)[MT][4], int hf, int mask_below, PageScratch& scratch) {
    const int first = 16 * g + (MT == 4 ? 0 : 4 * hf);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s_acc[mt][i] *= scale2;
    if (mask_below > 0) {   // the page that holds the row's first live token
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (first + 2 * mt + (i >> 1) + 8 * (i & 1) < mask_below) s_acc[mt][i] = -INFINITY;
    }
    float mx = -INFINITY;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) mx = fmaxf(mx, s_acc[mt][i]);
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    const float m_new = fmaxf(m_run, mx);
    const float m_ref = m_new == -INFINITY ? 0.0f : m_new;   // nothing live yet: every weight below comes out zero
    const float alpha = fast_exp2(m_run - m_ref);
    m_run = m_new;
    float psum = 0.0f;
    uint32_t hi[2 * MT], lo[2 * MT];
#pragma unroll
    for (int u = 0; u < 2 * MT; ++u) {
      const float p0 = fast_exp2(s_acc[u >> 1][2 * (u & 1)] - m_ref), p1 = fast_exp2(s_acc[u >> 1][2 * (u & 1) + 1] - m_ref);
      psum += p0 + p1;
      hi[u] = pack16<OUT>(p0, p1);
      float h0, h1;
      unpack16<OUT>(hi[u], h0, h1);
      lo[u] = pack16<OUT>(p0 - h0, p1 - h1);
    }
    uint4* const row_hi = reinterpret_cast<uint4*>(&scratch.prob[c * kProbStride + 16 * g]) + (MT == 4 ? 0 : hf);
    uint4* const row_lo = reinterpret_cast<uint4*>(&scratch.prob[(4 + c) * kProbStride + 16 * g]) + (MT == 4 ? 0 : hf);
#pragma unroll
    for (int k = 0; k < MT / 2; ++k) {
      row_hi[k] = make_uint4(hi[4 * k], hi[4 * k + 1], hi[4 * k + 2], hi[4 * k + 3]);
      row_lo[k] = make_uint4(lo[4 * k], lo[4 * k + 1], lo[4 * k + 2], lo[4 * k + 3]);
    }
    l_run = l_run * alpha + psum;
    // the running maximum rarely moves after the first pages: skip the rescale when no lane needs it.  This thread's
    // accumulator columns belong to heads 2(c&1) and 2(c&1)+1, whose factors live in the lanes c' = head of its quad.
    if (__any_sync(0xffffffffu, alpha != 1.0f)) {
      const float alpha_even = __shfl_sync(0xffffffffu, alpha, (lane & ~3) | (2 * (c & 1)));
      const float alpha_odd = __shfl_sync(0xffffffffu, alpha, (lane & ~3) | (2 * (c & 1) + 1));
#pragma unroll
      for (int mt = 0; mt < 8; ++mt) {
        o_acc[mt][0] *= alpha_even; o_acc[mt][1] *= alpha_odd;
        o_acc[mt][2] *= alpha_even; o_acc[mt][3] *= alpha_odd;
      }
    }
  }

  // O[channel][(part, head)] += V^T P, 16 tokens per step; in a half, whose tokens are 16s + 4hf .. + 3 and 8 more, of two
  // s a step.  The code words of two tokens are byte-interleaved (low halves
  // together: channels 0..7 of both tokens; high halves: channels 8..15), so that the packed dequantization sees token a in
  // the low half and token b in the high half.  m-tile mt, row g is channel 16g + mt, row g+8 channel 16g + 8 + mt.
  template <int MT>
  __device__ __forceinline__ void weigh_values(const uint8_t* values, const PageScratch& scratch, int hf) {
    constexpr int kStep = MT == 4 ? 16 : 32, kSecond = MT == 4 ? 4 : 16;   // tokens from step to step, to the second pair
    const int base = c + (MT == 4 ? 0 : 4 * hf);
    const uint32_t* vcodes = reinterpret_cast<const uint32_t*>(values) + g;   // word g of a token row: + 8 * token
    const uint8_t* vmeta = values + kValueCodes;
    const uint32_t* pb = reinterpret_cast<const uint32_t*>(&scratch.prob[g * kProbStride]) + base;   // column n = g
    // byte selectors that bring the scale (zero point) of this thread's value group of tokens a and b together
    const uint32_t sel_s = GN == 2 ? (gv ? 0x7632u : 0x5410u) : 0x5410u;
    const uint32_t sel_z = GN == 2 ? (gv ? 0x7632u : 0x5410u) : 0x7632u;
    auto token_pair = [&](int ta, uint32_t (&r_lo)[8], uint32_t (&r_hi)[8]) {   // tokens ta and ta + 8
      const uint32_t wa = vcodes[ta * 8], wb = vcodes[ta * 8 + 64];
      uint32_t ss, zz;
      if (GN == 2) {
        const uint2 ma = *reinterpret_cast<const uint2*>(vmeta + ta * 8);        // {s0,s1} {z0,z1}
        const uint2 mb = *reinterpret_cast<const uint2*>(vmeta + ta * 8 + 64);
        ss = prmt(ma.x, mb.x, sel_s);
        zz = prmt(ma.y, mb.y, sel_z);
      } else {
        const uint32_t ma = *reinterpret_cast<const uint32_t*>(vmeta + ta * 4);   // {s0, z0}
        const uint32_t mb = *reinterpret_cast<const uint32_t*>(vmeta + ta * 4 + 32);
        ss = prmt(ma, mb, sel_s);
        zz = prmt(ma, mb, sel_z);
      }
      const uint32_t ms0 = H::mul(ss, H::neg_magic(0)), ms1 = H::mul(ss, H::neg_magic(1)), ms2 = H::mul(ss, H::neg_magic(2));
      dequant_word2<DT>(cc, prmt(wa, wb, 0x5410u), ss, zz, ms0, ms1, ms2, r_lo);
      dequant_word2<DT>(cc, prmt(wa, wb, 0x7632u), ss, zz, ms0, ms1, ms2, r_hi);
      cast_registers<DT, OUT>(r_lo);
      cast_registers<DT, OUT>(r_hi);
    };
#pragma unroll kPvUnroll
    for (int s = 0; s < 2 * MT; ++s) {
      uint32_t r0_lo[8], r0_hi[8], r1_lo[8], r1_hi[8];
      token_pair(kStep * s + base, r0_lo, r0_hi);             // contraction index 2c, 2c + 1
      token_pair(kStep * s + base + kSecond, r1_lo, r1_hi);   // contraction index 2c + 8, 2c + 9
      // the pairs (t, t + 8) of sixteen tokens are eight words
      const uint32_t b0 = pb[kStep / 2 * s], b1 = pb[kStep / 2 * s + (MT == 4 ? 4 : 8)];
#pragma unroll
      for (int mt = 0; mt < 8; ++mt) HO::mma(o_acc[mt], r0_lo[mt], r0_hi[mt], r1_lo[mt], r1_hi[mt], b0, b1);
    }
  }

  // this warp's state for the merge: m_run and l_run of head c, accumulators [head][channel]
  __device__ __forceinline__ void hand_over(float* acc) {
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 4);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 8);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 16);
#pragma unroll
    for (int mt = 0; mt < 8; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // lanes c and c ^ 2 hold what the high and the low parts of the probabilities contributed
        const float v = o_acc[mt][i] + __shfl_xor_sync(0xffffffffu, o_acc[mt][i], 2);
        if (c < 2) acc[(2 * c + (i & 1)) * 128 + 16 * g + mt + 8 * (i >> 1)] = v;
      }
  }
};

// the query of a KV head's group, pre-shifted for the block-diagonal operand: [channel][2 * head + j'].  A thread has a channel of
// heads r and r + 2 (zero for absent heads).
struct QueryPair { uint32_t value[2]; };
__device__ __forceinline__ QueryPair load_query(const void* q, int64_t first_row, int rep, int tid) {
  QueryPair v;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = (tid >> 7) + 2 * i;
    v.value[i] = r < rep ? reinterpret_cast<const uint16_t*>(q)[(first_row + r) * 128 + (tid & 127)] : 0u;
  }
  return v;
}
__device__ __forceinline__ void store_query(uint32_t (*q32)[8], const QueryPair& v, int tid) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
    *reinterpret_cast<uint2*>(&q32[tid & 127][2 * ((tid >> 7) + 2 * i)]) = make_uint2(v.value[i], v.value[i] << 16);
}

}  // namespace
