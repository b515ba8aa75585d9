// Tensor-core fused decode attention with the arithmetic of the reference's Triton attention kernels
// (src/dart/fused_attention.py:149-262): key = code * scale + zero and value = code * scale + zero in
// fp32 with no rounding to the cache dtype, fp32 logits, fp32 online softmax.  Same page geometry, work
// split and staging as decode_fast.cu (which reproduces the per-op rounded dequantization instead).
//
// Because nothing is rounded per element, the affine map leaves the inner loop:
//   logit[t,h]  = sum_ch (q[h,ch] * s[ch]) * code[t,ch]  +  sum_ch q[h,ch] * z[ch]
//   out[h,ch]   = sum_t  (p[t,h] * s[t,grp]) * code[t,ch] +  sum_t  p[t,h] * z[t,grp]
// The packed 2-bit codes become MMA operands with ONE logic op per register: `word & mask` leaves a
// code in mantissa bits 2p..2p+1 of each 16-bit half with a zero exponent, which read as fp16 is the
// subnormal code * 4^p * 2^-24 -- exact, and the tensor cores take subnormal fp16 operands at full
// accuracy.  The power of two is constant per accumulator row (a row always reads the same code
// position), so it is folded into the fp32 scaling that follows the MMA.  The other operand carries
// the weights q*s (per page) and p*s (per token) as fp16 after an exact power-of-two normalisation
// chosen from the largest scale in sight, so no input magnitude overflows or underflows the format.
// The zero-point terms are plain fp32 dot products.  A promoted channel's code is low + 4 * high: its
// high plane is just more contraction steps with weight 4 * q * s.
//
// As in decode_fast.cu a 32-bit register of codes pairs two elements along the MMA's non-contraction
// direction, so the contraction index is doubled, (channel, j) for K and (token, j) for V, against a
// block-diagonal weight operand whose columns are (query head, j').  For V the pair is arranged as
// (channel of value group 0, channel of value group 1), which lets one operand carry both groups'
// scales.  Algorithmic HBM bytes per page and (batch, kv head): 10880.

#include <atomic>

#include "decode_fast_common.cuh"

namespace {

constexpr int kUStride = 132;   // 32-bit words per head of a warp's weight table: 128 tokens, 4 pad

// what a warp needs beside a staged page
union FusedScratch {
  struct {
    uint2 w_low[128];      // per channel: fp16 q*s*f of heads (0,1) and (2,3)
    uint2 w_high[32];      // per promoted slot: fp16 4*q*s*f of its channel, zero past the last slot
    uint2 w_high_lo[32];   // what the fp16 rounding of w_high dropped, as fp16: the high plane carries most of a
                           // promoted (outlier) channel's magnitude, so its weights get a second term
  };
  // takes their place after the logits: [head][token] = fp16 p*s*fv of (value group 0 | group 1 << 16)
  uint32_t u[4 * kUStride];
};

struct FusedWarpSmem {
  uint8_t keys[kPageBytesK];
  uint8_t values[kStageBytes - kPageBytesK];   // codes, then scales and zero points
  FusedScratch scratch;
};

static_assert(sizeof(FusedScratch) >= 512 * sizeof(float), "the scratch of a warp takes its state at the end of a row");

struct FusedBlockSmem {
  uint2 query[128];              // [channel]: the 16-bit query values of the four heads (zero for absent heads)
  float merge_m[kWarps][4];
  float merge_l[kWarps][4];
  int slot_map[128];
  uint64_t k_bar[kWarps], v_bar[kWarps];
};

template <int DT>
__device__ __forceinline__ float md_to_float(uint32_t bits16) {
  if (DT == DARTKV_BF16) return __uint_as_float(bits16 << 16);
  return __half2float(__ushort_as_half((uint16_t)bits16));
}
// both halves of a packed pair of 16-bit floats
template <int DT>
__device__ __forceinline__ void md_pair_to_float(uint32_t pair, float& lo, float& hi) {
  if (DT == DARTKV_BF16) {
    lo = __uint_as_float(pair << 16);
    hi = __uint_as_float(pair & 0xFFFF0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&pair));
    lo = f.x;
    hi = f.y;
  }
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
// Power of two f with bound * f < 2^15 (so bound * f fits fp16), and 1/f; bound >= 0 finite.
__device__ __forceinline__ void pow2_normaliser(float bound, float& f, float& f_inv) {
  int eb = (int)(__float_as_uint(bound) >> 23);   // bound < 2^(eb - 126)
  eb = min(max(eb, 15), 253);
  f = __uint_as_float((uint32_t)(268 - eb) << 23);       // 2^(141 - eb)
  f_inv = __uint_as_float((uint32_t)(eb - 14) << 23);    // 2^(eb - 141)
}

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One page, as one warp works on it.  DT: dtype of the cache and the query; MD: dtype of the scales and zero points.
// GN: value groups per token (1 or 2).  KP: promoted channels per page when that is a multiple of eight known to
// the host (0, 8, 16, 24, 32), else -1 (read from the descriptor).
template <int DT, int MD, int GN, int KP>
struct FusedWork {
  // 64 x 32,768 tokens: 382 us; with 4 and 4 386, with 2 and 2 396 (on one GPU; others give this version 392 to 414)
  static constexpr int kQkUnroll = 16, kPvUnroll = 4;
  const dartkv_cache_desc& d;
  const uint2* query;
  float scale2;
  int lane, g, c, K, prom_steps;
  uint32_t sel_w, mask_u;
  float q_absmax;
  float o_acc[4][4];           // [m-tile][c-reg], in units of 4^p * 2^-24 / fv_run
  float m_run, l_run;          // head c, log2 domain
  float zs[2];                 // this thread's share of sum_t p * z for (head c, value group j)
  float fv_run, fv_inv_run;
  float bias, f_inv;           // of the page in work

  __device__ __forceinline__ FusedWork(const dartkv_cache_desc& desc, const uint2* query_table, float scale, int lane_)
      : d(desc), query(query_table), scale2(scale * kLog2e), lane(lane_), g(lane_ >> 2), c(lane_ & 3) {
    K = KP >= 0 ? KP : (d.key_mode == DARTKV_MIXED_PAGE ? d.promoted : 0);
    prom_steps = (K + 7) >> 3;
    // weight operand: column n = g is (head g >> 1, j' = g & 1); the 32-bit word read holds the fp16 weights of the
    // head pair g >> 2.  Take the head's half into half j' and zeros (from the second source) into the other.
    const uint32_t head_bytes = ((g >> 1) & 1) ? 0x32u : 0x10u;
    sel_w = (g & 1) ? (0x0054u | (head_bytes << 8)) : (head_bytes | 0x5400u);
    mask_u = (g & 1) ? 0xFFFF0000u : 0x0000FFFFu;
  }

  __device__ __forceinline__ float4 query_of(int ch) const {
    const uint2 x = query[ch];
    float4 q;
    md_pair_to_float<DT>(x.x, q.x, q.y);
    md_pair_to_float<DT>(x.y, q.z, q.w);
    return q;
  }

  // the query table is complete: its largest magnitude bounds the weights q*s
  __device__ __forceinline__ void start_row() {
    q_absmax = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 q = query_of(32 * i + lane);
      q_absmax = fmaxf(q_absmax, fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) q_absmax = fmaxf(q_absmax, __shfl_xor_sync(0xffffffffu, q_absmax, off));
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) o_acc[mt][i] = 0.0f;
    m_run = -INFINITY; l_run = 0.0f; zs[0] = zs[1] = 0.0f;
    fv_run = __uint_as_float(253u << 23); fv_inv_run = __uint_as_float(1u << 23);
  }

  // weights of the page's channels and promoted slots
  __device__ __forceinline__ void fill_table(const uint8_t* keys, FusedScratch& ws) {
    const uint32_t* kscale2 = reinterpret_cast<const uint32_t*>(keys + d.key_off_scale);
    const uint32_t* kzero2 = reinterpret_cast<const uint32_t*>(keys + d.key_off_zero);
    const uint32_t sc[2] = {kscale2[lane], kscale2[32 + lane]}, zp[2] = {kzero2[lane], kzero2[32 + lane]};
    // scales are positive finite 16-bit floats: their bit patterns order like the values
    const uint32_t smax = __reduce_max_sync(0xffffffffu, max(max(sc[0] & 0xFFFFu, sc[0] >> 16), max(sc[1] & 0xFFFFu, sc[1] >> 16)));
    float f;
    pow2_normaliser(4.0f * q_absmax * md_to_float<MD>(smax), f, f_inv);
    float bz[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < 2; ++i) {   // channels 2 * tp and 2 * tp + 1
      const int tp = 32 * i + lane;
      float s0, s1, z0, z1;
      md_pair_to_float<MD>(sc[i], s0, s1);
      md_pair_to_float<MD>(zp[i], z0, z1);
      const float4 qa = query_of(2 * tp), qb = query_of(2 * tp + 1);
      const float sa = s0 * f, sb = s1 * f;
      *reinterpret_cast<uint4*>(&ws.w_low[2 * tp]) = make_uint4(pack_f16x2(qa.x * sa, qa.y * sa), pack_f16x2(qa.z * sa, qa.w * sa),
                                                                pack_f16x2(qb.x * sb, qb.y * sb), pack_f16x2(qb.z * sb, qb.w * sb));
      bz[0] += fmaf(qa.x, z0, qb.x * z1); bz[1] += fmaf(qa.y, z0, qb.y * z1);
      bz[2] += fmaf(qa.z, z0, qb.z * z1); bz[3] += fmaf(qa.w, z0, qb.w * z1);
    }
    if (prom_steps > 0) {   // lane = slot
      uint2 wh = make_uint2(0u, 0u), wl = make_uint2(0u, 0u);
      if (lane < K) {
        const int ch = reinterpret_cast<const int32_t*>(keys + d.key_off_index)[lane] & 127;
        const float s4 = 4.0f * f * md_to_float<MD>(reinterpret_cast<const uint16_t*>(keys + d.key_off_scale)[ch]);
        const float4 qh = query_of(ch);
        const float e0 = qh.x * s4, e1 = qh.y * s4, e2 = qh.z * s4, e3 = qh.w * s4;
        wh = make_uint2(pack_f16x2(e0, e1), pack_f16x2(e2, e3));
        const float2 h01 = __half22float2(*reinterpret_cast<const __half2*>(&wh.x));
        const float2 h23 = __half22float2(*reinterpret_cast<const __half2*>(&wh.y));
        wl = make_uint2(pack_f16x2(e0 - h01.x, e1 - h01.y), pack_f16x2(e2 - h23.x, e3 - h23.y));
      }
      ws.w_high[lane] = wh;
      ws.w_high_lo[lane] = wl;
    }
    // sum_ch q*z per head: four sums over 32 lanes in 6 shuffles, halving the number of sums a lane carries at the
    // first two levels; head 2*up16 + up8 ends up in the lanes of that eighth
    const bool up16 = lane & 16, up8 = lane & 8;
    const float k0 = (up16 ? bz[2] : bz[0]) + __shfl_xor_sync(0xffffffffu, up16 ? bz[0] : bz[2], 16);
    const float k1 = (up16 ? bz[3] : bz[1]) + __shfl_xor_sync(0xffffffffu, up16 ? bz[1] : bz[3], 16);
    float k = (up8 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, up8 ? k0 : k1, 8);
    k += __shfl_xor_sync(0xffffffffu, k, 4);
    k += __shfl_xor_sync(0xffffffffu, k, 2);
    k += __shfl_xor_sync(0xffffffffu, k, 1);
    bias = __shfl_sync(0xffffffffu, k, 8 * c) * scale2;
  }

  // logits S[token pair][(head, j')] over the doubled contraction (channel, j).  A thread reads the whole word g of a
  // channel's code row (tokens 16g .. 16g+15); row g of m-tile mt is code u = 2mt of both halves, row g+8 u = 2mt + 1:
  // u = 0..4 at positions 0..4 of the mantissa, 5..7 at positions 0..2 after a shift.  MT: m-tiles, 4 for the whole page or 2
  // for the half `hf` of it (u = 4hf .. 4hf + 3, at positions 0..3).
  template <int MT>
  __device__ __forceinline__ void logits(const uint8_t* keys, const FusedScratch& ws, int hf, float (&s_acc)[MT][4]) const {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s_acc[mt][i] = 0.0f;
    const int shift = MT == 4 ? 0 : 8 * hf;
    // the A operands of two code words, m-tile by m-tile
    auto tiles = [&](uint32_t w0, uint32_t w1, auto multiply) {
      w0 >>= shift; w1 >>= shift;
      multiply(s_acc[0], w0 & 0x00030003u, w0 & 0x000C000Cu, w1 & 0x00030003u, w1 & 0x000C000Cu);
      multiply(s_acc[1], w0 & 0x00300030u, w0 & 0x00C000C0u, w1 & 0x00300030u, w1 & 0x00C000C0u);
      if constexpr (MT == 4) {
        const uint32_t y0 = w0 >> 10, y1 = w1 >> 10;
        multiply(s_acc[2], w0 & 0x03000300u, y0 & 0x00030003u, w1 & 0x03000300u, y1 & 0x00030003u);
        multiply(s_acc[3], y0 & 0x000C000Cu, y0 & 0x00300030u, y1 & 0x000C000Cu, y1 & 0x00300030u);
      }
    };
    const uint8_t* const low = keys + 4 * g + 32 * c;                          // + 256 * step (+128)
    const int w_thread = 8 * c + 4 * (g >> 2);                                 // + 64 * step (+32)
    const uint8_t* const w_low = reinterpret_cast<const uint8_t*>(ws.w_low) + w_thread;
#pragma unroll kQkUnroll
    for (int ks = 0; ks < 16; ++ks) {
      const uint32_t w0 = *reinterpret_cast<const uint32_t*>(low + 256 * ks);
      const uint32_t w1 = *reinterpret_cast<const uint32_t*>(low + 256 * ks + 128);
      const uint32_t b0 = prmt(*reinterpret_cast<const uint32_t*>(w_low + 64 * ks), 0u, sel_w);
      const uint32_t b1 = prmt(*reinterpret_cast<const uint32_t*>(w_low + 64 * ks + 32), 0u, sel_w);
      tiles(w0, w1, [&](float (&s)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) { mma_f16(s, a0, a1, a2, a3, b0, b1); });
    }
    // high plane of the promoted slots: the same codes against both terms of the weights
    const uint8_t* const high = keys + d.key_off_high + 4 * g + 32 * c;
    const uint8_t* const w_high = reinterpret_cast<const uint8_t*>(ws.w_high) + w_thread;
    const uint8_t* const w_high_lo = reinterpret_cast<const uint8_t*>(ws.w_high_lo) + w_thread;
    for (int ks = 0; ks < prom_steps; ++ks) {
      const uint32_t w0 = *reinterpret_cast<const uint32_t*>(high + 256 * ks);
      const uint32_t w1 = *reinterpret_cast<const uint32_t*>(high + 256 * ks + 128);
      const uint32_t b0 = prmt(*reinterpret_cast<const uint32_t*>(w_high + 64 * ks), 0u, sel_w);
      const uint32_t b1 = prmt(*reinterpret_cast<const uint32_t*>(w_high + 64 * ks + 32), 0u, sel_w);
      const uint32_t l0 = prmt(*reinterpret_cast<const uint32_t*>(w_high_lo + 64 * ks), 0u, sel_w);
      const uint32_t l1 = prmt(*reinterpret_cast<const uint32_t*>(w_high_lo + 64 * ks + 32), 0u, sel_w);
      tiles(w0, w1, [&](float (&s)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
        mma_f16(s, a0, a1, a2, a3, b0, b1);
        mma_f16(s, a0, a1, a2, a3, l0, l1);
      });
    }
  }

  // online softmax for head c over the page or half of it (this thread: tokens 16g + u + 8j, u = 2mt + (i >> 1), j = i & 1, in
  // a half + 4hf); the probabilities leave as weights p*s*fv.  wait_for_values() returns when the page's values have landed.
  template <int MT, class Wait>
  __device__ __forceinline__ void softmax(float (&s_acc)[MT][4], int hf, int mask_below, FusedScratch& ws, Wait wait_for_values,
                                          const uint8_t* values) {
    const int first = 16 * g + (MT == 4 ? 0 : 4 * hf);
    {
      const float base = scale2 * f_inv * 16777216.0f;
      const float cm[5] = {base, base * 0.25f, base * 0.0625f, base * 0.015625f, base * 0.00390625f};
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int u = 2 * mt + (i >> 1);
          s_acc[mt][i] = fmaf(s_acc[mt][i], cm[u < 5 ? u : u - 5], bias);
        }
    }
    if (mask_below > 0) {   // the page that holds the row's first live token: the tokens before it drop out
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

    // largest value scale of the page; the normaliser only ever shrinks, so accumulators are rescaled at most a handful
    // of times per run
    wait_for_values();
    const uint8_t* const vmeta = values + kValueCodes;
    uint32_t smax;
    {
      const uint4 m0 = reinterpret_cast<const uint4*>(vmeta)[lane];
      if (GN == 2) {
        const uint4 m1 = reinterpret_cast<const uint4*>(vmeta)[32 + lane];
        smax = max(max(max(m0.x & 0xFFFFu, m0.x >> 16), max(m0.z & 0xFFFFu, m0.z >> 16)),
                   max(max(m1.x & 0xFFFFu, m1.x >> 16), max(m1.z & 0xFFFFu, m1.z >> 16)));
      } else {
        smax = max(max(m0.x & 0xFFFFu, m0.y & 0xFFFFu), max(m0.z & 0xFFFFu, m0.w & 0xFFFFu));
      }
    }
    smax = __reduce_max_sync(0xffffffffu, smax);
    float fv_page, fv_inv_page;
    pow2_normaliser(md_to_float<MD>(smax), fv_page, fv_inv_page);
    const bool shrink = fv_page < fv_run;
    const float factor = shrink ? alpha * (fv_page * fv_inv_run) : alpha;
    if (shrink) { fv_run = fv_page; fv_inv_run = fv_inv_page; }
    const float fv = fv_run;

    float psum = 0.0f, zs0 = 0.0f, zs1 = 0.0f;
    constexpr int kQuads = MT / 2;   // fours of tokens on each side of j, eight tokens apart
    uint32_t* const row = &ws.u[c * kUStride + first];
#pragma unroll
    for (int k4 = 0; k4 < MT; ++k4) {   // tokens `first` + from .. + 3
      const int from = kQuads == 2 ? 4 * k4 : 8 * k4;
      uint32_t packed[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int u = kQuads == 2 ? 4 * (k4 & 1) + k : k, j = k4 / kQuads;
        const float p = fast_exp2(s_acc[u >> 1][2 * (u & 1) + j] - m_ref);
        psum += p;
        const float pf = p * fv;
        const int tok = first + from + k;
        if (GN == 2) {
          const uint2 m = *reinterpret_cast<const uint2*>(vmeta + tok * 8);   // (s0 | s1 << 16), (z0 | z1 << 16)
          float s0, s1, z0, z1;
          md_pair_to_float<MD>(m.x, s0, s1);
          md_pair_to_float<MD>(m.y, z0, z1);
          zs0 = fmaf(p, z0, zs0);
          zs1 = fmaf(p, z1, zs1);
          packed[k] = pack_f16x2(pf * s0, pf * s1);
        } else {
          float s0, z0;
          md_pair_to_float<MD>(*reinterpret_cast<const uint32_t*>(vmeta + tok * 4), s0, z0);
          zs0 = fmaf(p, z0, zs0);
          const float w = pf * s0;
          packed[k] = pack_f16x2(w, w);
        }
      }
      *reinterpret_cast<uint4*>(row + from) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
    l_run = l_run * alpha + psum;
    zs[0] = zs[0] * alpha + zs0;
    zs[1] = zs[1] * alpha + (GN == 2 ? zs1 : zs0);
    // the running maximum and the normaliser rarely move after the first pages
    if (__any_sync(0xffffffffu, factor != 1.0f)) {
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) o_acc[mt][i] *= factor;
    }
  }

  // O[channel pair][(head, j')] += V^T U over the doubled contraction (token, j): lane row g reads the
  // code words wi = g & 3 and wi + 4 of a token row and pairs their low (g < 4) or high (g >= 4) halves, so a
  // register holds (channel 16wi + 8xy + u of group 0, the same channel + 64 of group 1).  Step ks covers the
  // eight tokens from 8ks on, in a half the tokens 16ks + 4hf .. + 3 and 16ks + 4hf + 8 .. + 11.
  template <int MT>
  __device__ __forceinline__ void weigh_values(const uint8_t* values, const FusedScratch& ws, int hf) {
    constexpr int kStep = MT == 4 ? 8 : 16, kSecond = MT == 4 ? 4 : 8;   // tokens from step to step, to the second four
    const int base = c + (MT == 4 ? 0 : 4 * hf);
    const int wi = g & 3;
    const uint32_t sel_v = (g >> 2) ? 0x7632u : 0x5410u;
    const uint8_t* const vthread = values + 32 * base + 4 * wi;            // + 32 * tokens
    const uint32_t* const uthread = &ws.u[(g >> 1) * kUStride + base];     // + tokens
#pragma unroll kPvUnroll
    for (int ks = 0; ks < 4 * MT; ++ks) {
      const uint8_t* const va = vthread + 32 * kStep * ks;
      const uint8_t* const vb = va + 32 * kSecond;
      const uint32_t x0 = prmt(*reinterpret_cast<const uint32_t*>(va), *reinterpret_cast<const uint32_t*>(va + 16), sel_v);
      const uint32_t x1 = prmt(*reinterpret_cast<const uint32_t*>(vb), *reinterpret_cast<const uint32_t*>(vb + 16), sel_v);
      const uint32_t y0 = x0 >> 10, y1 = x1 >> 10;   // codes 5, 6, 7 at positions 0, 1, 2
      const uint32_t b0 = uthread[kStep * ks] & mask_u;
      const uint32_t b1 = uthread[kStep * ks + kSecond] & mask_u;
      mma_f16(o_acc[0], x0 & 0x00030003u, x0 & 0x000C000Cu, x1 & 0x00030003u, x1 & 0x000C000Cu, b0, b1);
      mma_f16(o_acc[1], x0 & 0x00300030u, x0 & 0x00C000C0u, x1 & 0x00300030u, x1 & 0x00C000C0u, b0, b1);
      mma_f16(o_acc[2], x0 & 0x03000300u, y0 & 0x00030003u, x1 & 0x03000300u, y1 & 0x00030003u, b0, b1);
      mma_f16(o_acc[3], y0 & 0x000C000Cu, y0 & 0x00300030u, y1 & 0x000C000Cu, y1 & 0x00300030u, b0, b1);
    }
  }

  // this warp's state for the merge: m_run and l_run of head c, accumulators [head][channel]
  __device__ __forceinline__ void hand_over(float* acc) {
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
      l_run += __shfl_xor_sync(0xffffffffu, l_run, off);
      zs[0] += __shfl_xor_sync(0xffffffffu, zs[0], off);
      zs[1] += __shfl_xor_sync(0xffffffffu, zs[1], off);
    }
    const int wi = g & 3, xy = g >> 2;
    const float unit = fv_inv_run * 16777216.0f;   // accumulators hold codes * 4^p * 2^-24 * fv
    const float pos_scale[5] = {unit, unit * 0.25f, unit * 0.0625f, unit * 0.015625f, unit * 0.00390625f};
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int u = 2 * mt + (i >> 1), jp = i & 1;
        acc[c * 128 + 64 * jp + 16 * wi + 8 * xy + u] = fmaf(o_acc[mt][i], pos_scale[u < 5 ? u : u - 5], zs[jp]);
      }
  }
};

// the work split of decode_fast_kernel, FEW included
template <int DT, int MD, int GN, int KP, bool FEW>
__global__ void __launch_bounds__(kThreads, 2) decode_fused32_kernel(dartkv_cache_desc d, FastArgs a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous();
  FusedBlockSmem& bs = *reinterpret_cast<FusedBlockSmem*>(smem_raw + sizeof(FusedWarpSmem) * kWarps);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rep = a.query_heads / d.kv_heads;

  if ((int)blockIdx.x >= a.stream_blocks) {
    const int bh = blockIdx.x - a.stream_blocks;
    float* const warp_out = reinterpret_cast<float*>(smem_raw);   // [warp][head][128]
    dense_block<DT, MD>(d, a, bs, warp_out, bh);
    __syncthreads();
    block_merge(a, bs, warp_out, bh / d.kv_heads, bh % d.kv_heads, rep, 0);
    return;
  }

  const int sb = blockIdx.x;
  int unit = (int)((int64_t)sb * a.units / a.stream_blocks);   // the host keeps the unit count below 2^31
  const int unit_end = (int)((int64_t)(sb + 1) * a.units / a.stream_blocks);
  FusedWarpSmem& ws = reinterpret_cast<FusedWarpSmem*>(smem_raw)[warp];
  int bh = unit / a.quads, quad = unit - bh * a.quads;
  // the row's first live token, its query and the state are requested together
  const int first_live = first_live_token(d, a, bh);
  const QueryWords first_query = load_query_compact(a.q, (int64_t)(bh / d.kv_heads) * a.query_heads + bh % d.kv_heads * rep, warp == 0 ? rep : 0, lane);
  const int k_end = d.state[2], v_end = d.state[3], sink_filled = d.state[4];
  const int fast_end = fast_range_end(d.sink_tokens, d.page_size, k_end, v_end, sink_filled);
  const int total_pages = fast_end > d.sink_tokens ? (fast_end - d.sink_tokens) / 128 : 0;
  constexpr int kMetaBytes = 128 * 2 * GN * 2;
  auto issue_keys = [&](int bh, int pg) {
    mbar_expect_tx(&bs.k_bar[warp], d.key_page_bytes);
    bulk_copy_g2s(ws.keys, d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes, d.key_page_bytes, &bs.k_bar[warp]);
  };
  auto issue_values = [&](int bh, int pg) {
    mbar_expect_tx(&bs.v_bar[warp], kValueCodes + kMetaBytes);
    const int64_t vrow = (int64_t)bh * d.max_value_tokens + (int64_t)pg * 128;
    bulk_copy_g2s(ws.values, d.v_codes + vrow * 32, kValueCodes, &bs.v_bar[warp]);
    bulk_copy_g2s(ws.values + kValueCodes, reinterpret_cast<const uint8_t*>(d.v_meta) + vrow * (4 * GN), kMetaBytes, &bs.v_bar[warp]);
  };
  if (lane == 0) {
    mbar_init(&bs.k_bar[warp], 1);
    mbar_init(&bs.v_bar[warp], 1);
    mbar_fence_init();
  }
  __syncwarp();
  FusedWork<DT, MD, GN, KP> work(d, bs.query, a.scale, lane);
  bool ok = true;
  uint32_t parity = 0;   // of the pages this warp has consumed so far

  RowPiece now = row_piece(d, a, first_live, quad, min(a.quads - quad, unit_end - unit), total_pages);
  // this warp's first page is requested before anything else, so its latency overlaps the query load below
  if (lane == 0 && now.begin + warp < now.end) { issue_keys(bh, now.begin + warp); issue_values(bh, now.begin + warp); }
  if (warp == 0) store_query_compact(bs.query, first_query, lane);
  __syncthreads();

  while (unit < unit_end) {
    unit += min(a.quads - quad, unit_end - unit);
    quad = 0;
    // this warp's first page of the next row: requested as soon as its buffers are free, before the rows are merged
    auto next_row = [&](auto issue) {
      if (lane != 0 || unit >= unit_end) return;
      const RowPiece next = row_piece(d, a, first_live_token(d, a, bh + 1), 0, min(a.quads, unit_end - unit), total_pages);
      if (next.begin + warp < next.end) issue(bh + 1, next.begin + warp);
    };

    work.start_row();
    if constexpr (FEW) {
      // the block's only unit: warps w and w + 4 share page w, half of its tokens each
      const int hf = warp >> 2, shared = warp & 3;
      const FusedWarpSmem& page = reinterpret_cast<const FusedWarpSmem*>(smem_raw)[shared];
      if (now.begin + shared < now.end) {
        ok = mbar_wait(&bs.k_bar[shared], 0) && ok;
        work.fill_table(page.keys, ws.scratch);
        __syncwarp();
        float s_acc[2][4];
        work.template logits<2>(page.keys, ws.scratch, hf, s_acc);
        __syncwarp();
        work.template softmax<2>(s_acc, hf, now.first_live - (d.sink_tokens + 128 * (now.begin + shared)), ws.scratch,
                                 [&] { ok = mbar_wait(&bs.v_bar[shared], 0) && ok; }, page.values);
        __syncwarp();
        work.template weigh_values<2>(page.values, ws.scratch, hf);
      }
    } else {
      for (int pg = now.begin + warp; pg < now.end; pg += kWarps, parity ^= 1) {
        const bool last = pg + kWarps >= now.end;
        ok = mbar_wait(&bs.k_bar[warp], parity) && ok;
        work.fill_table(ws.keys, ws.scratch);
        __syncwarp();
        float s_acc[4][4];
        work.template logits<4>(ws.keys, ws.scratch, 0, s_acc);
        __syncwarp();
        // the keys are consumed: their buffer takes the next page's while the values are worked on
        if (last) next_row(issue_keys);
        else if (lane == 0) issue_keys(bh, pg + kWarps);
        work.template softmax<4>(s_acc, 0, now.first_live - (d.sink_tokens + 128 * pg), ws.scratch,
                                 [&] { ok = mbar_wait(&bs.v_bar[warp], parity) && ok; }, ws.values);
        __syncwarp();
        work.template weigh_values<4>(ws.values, ws.scratch, 0);
        __syncwarp();
        if (last) next_row(issue_values);
        else if (lane == 0) issue_values(bh, pg + kWarps);
      }
    }

    if (now.begin + warp >= now.end) {   // no page of this row for this warp
      next_row(issue_keys);
      next_row(issue_values);
    }
    // the states meet in the warps' scratch: nothing there is in use between the rows
    __syncwarp();
    work.hand_over(reinterpret_cast<float*>(&ws.scratch));
    if (lane < 4) { bs.merge_m[warp][lane] = merge_maximum(work.m_run, work.l_run); bs.merge_l[warp][lane] = work.l_run; }
    __syncthreads();
    block_merge<false, sizeof(FusedWarpSmem) / sizeof(float)>(a, bs, reinterpret_cast<const float*>(&reinterpret_cast<FusedWarpSmem*>(smem_raw)->scratch),
                                                     bh / d.kv_heads, bh % d.kv_heads, rep,
                                                     1 + sb - dartkv_block_of_unit((int64_t)bh * a.quads, a.stream_blocks, a.units));
    if (unit >= unit_end) break;
    ++bh;
    now = row_piece(d, a, first_live_token(d, a, bh), 0, min(a.quads, unit_end - unit), total_pages);
    if (warp == 0) store_query_compact(bs.query, load_query_compact(a.q, (int64_t)(bh / d.kv_heads) * a.query_heads + bh % d.kv_heads * rep, rep, lane), lane);
    __syncthreads();
  }
  if (!ok && lane == 0) atomicExch(a.status, 1);
}

constexpr size_t kFusedSmemBytes = sizeof(FusedWarpSmem) * kWarps + sizeof(FusedBlockSmem);

}  // namespace

int dartkv_decode_fused32_supported(const dartkv_cache_desc* d, int q_dtype, int query_heads) {
  if (d->head_dim != 128 || d->page_size != 128 || d->key_group != 128 || !d->regular_pages) return 0;
  if (d->dtype != DARTKV_F16 && d->dtype != DARTKV_BF16) return 0;
  if ((d->md_dtype != DARTKV_F16 && d->md_dtype != DARTKV_BF16) || q_dtype != d->dtype) return 0;
  if (d->value_bits != 2 || (d->value_group != 64 && d->value_group != 128)) return 0;
  if (d->key_mode == DARTKV_QUANTIZED_PAGE && d->key_bits != 2) return 0;
  if (d->key_page_bytes % 16 || d->key_page_bytes > kPageBytesK) return 0;   // at most 32 promoted channels
  if (query_heads % d->kv_heads || query_heads / d->kv_heads > 4) return 0;
  if (d->max_value_tokens % 8) return 0;   // keeps every page of value metadata 16-byte aligned
  if ((uintptr_t)d->k_pages % 16 || (uintptr_t)d->v_codes % 16 || (uintptr_t)d->v_meta % 16) return 0;
  return 1;
}

// every (cache dtype, metadata dtype, value groups, promoted count) variant of the kernel; a cache whose metadata
// dtype differs from its dtype gets the promoted counts 0 and 32 specialized, the others read the count at run time
using FusedKernel = void (*)(dartkv_cache_desc, FastArgs);
template <bool FEW, int DT, int GN>
static FusedKernel fused_variant_kp(int kp) {
  switch (kp) {
    case 0: return decode_fused32_kernel<DT, DT, GN, 0, FEW>;
    case 8: return decode_fused32_kernel<DT, DT, GN, 8, FEW>;
    case 16: return decode_fused32_kernel<DT, DT, GN, 16, FEW>;
    case 24: return decode_fused32_kernel<DT, DT, GN, 24, FEW>;
    case 32: return decode_fused32_kernel<DT, DT, GN, 32, FEW>;
    default: return decode_fused32_kernel<DT, DT, GN, -1, FEW>;
  }
}
template <bool FEW, int DT, int MD, int GN>
static FusedKernel fused_mixed_kp(int kp) {
  switch (kp) {
    case 0: return decode_fused32_kernel<DT, MD, GN, 0, FEW>;
    case 32: return decode_fused32_kernel<DT, MD, GN, 32, FEW>;
    default: return decode_fused32_kernel<DT, MD, GN, -1, FEW>;
  }
}
template <bool FEW>
static FusedKernel fused_variant_of(int dtype, int md, int value_groups, int kp) {
  if (md == dtype) {
    if (dtype == DARTKV_BF16) return value_groups == 2 ? fused_variant_kp<FEW, DARTKV_BF16, 2>(kp) : fused_variant_kp<FEW, DARTKV_BF16, 1>(kp);
    return value_groups == 2 ? fused_variant_kp<FEW, DARTKV_F16, 2>(kp) : fused_variant_kp<FEW, DARTKV_F16, 1>(kp);
  }
  if (dtype == DARTKV_BF16)
    return value_groups == 2 ? fused_mixed_kp<FEW, DARTKV_BF16, DARTKV_F16, 2>(kp) : fused_mixed_kp<FEW, DARTKV_BF16, DARTKV_F16, 1>(kp);
  return value_groups == 2 ? fused_mixed_kp<FEW, DARTKV_F16, DARTKV_BF16, 2>(kp) : fused_mixed_kp<FEW, DARTKV_F16, DARTKV_BF16, 1>(kp);
}

static FusedKernel fused_variant(bool few, int dtype, int md, int value_groups, int kp) {
  return few ? fused_variant_of<true>(dtype, md, value_groups, kp) : fused_variant_of<false>(dtype, md, value_groups, kp);
}

int dartkv_decode_fused32_launch(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads, float scale,
                                 int flavour, int unit_pages, int quads, int stream_blocks, long long units, int total_splits,
                                 float* part_m, float* part_l, float* part_acc, int* status, const int32_t* row_start,
                                 cudaStream_t stream) {
  (void)q_dtype;
  FastArgs a{query, query_heads, scale, flavour, quads, stream_blocks, units, total_splits, part_m, part_l, part_acc, status,
             row_start, unit_pages};
  dim3 grid(stream_blocks + d->batch * d->kv_heads);
  const bool few = dartkv_few_pages(unit_pages, units, stream_blocks);
  {
    // the shared-memory opt-in is per device and per kernel: ask once per device (the flags are atomic; two threads
    // that race on a device's first call both set the attribute, which is harmless)
    static std::atomic<bool> ready[64];
    int device = 0;
    DARTKV_CUDA_OK(cudaGetDevice(&device));
    if (device < 0 || device >= 64 || !ready[device].load(std::memory_order_acquire)) {
      for (int dt : {DARTKV_BF16, DARTKV_F16})
        for (int md : {DARTKV_BF16, DARTKV_F16})
          for (int gn : {1, 2})
            for (int kp : {-1, 0, 8, 16, 24, 32})
              for (bool each : {false, true})   // the next call, of another length, may be under graph capture
                DARTKV_CUDA_OK(cudaFuncSetAttribute(fused_variant(each, dt, md, gn, kp), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)kFusedSmemBytes));
      if (device >= 0 && device < 64) ready[device].store(true, std::memory_order_release);
    }
  }
  const int promoted = d->key_mode == DARTKV_MIXED_PAGE ? d->promoted : 0;
  const int kp = (promoted % 8 == 0 && promoted <= 32) ? promoted : -1;
  DARTKV_CUDA_OK(launch_following(fused_variant(few, d->dtype, d->md_dtype, d->value_groups, kp), grid, kThreads, kFusedSmemBytes,
                                  stream, *d, a));
  DARTKV_LAUNCH_OK("decode_fused32_kernel");
  return DARTKV_OK;
}
