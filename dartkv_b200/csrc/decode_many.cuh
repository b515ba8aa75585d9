// Tensor-core decode attention for many query rows per KV head: 9 to 32 of them in one pass over the pages (several query
// tokens at once, wide GQA groups; more rows go in groups of up to 32).  The geometries of decode_rows.cu, per-op rounded
// flavour.
//
// What bounds it: instructions.  With every row of a KV head in one block a page is restored once, whatever the number of
// rows, where groups of eight rows (decode_rows.cu) restore it for every group.  So that the MMAs of all rows can share the
// restored numbers without the accumulators of a warp growing with the rows, a block of eight warps restores a page of keys and
// one of values into two shared tiles and splits both contractions over its warps by their M rows: tokens for the logits,
// channels for P.V.  A warp then holds four accumulators per eight rows (a warp that kept all channels would need 32).
//   * tiles: [channel][token] for keys and [token][channel] for values, the order of the packed words, so that a word's sixteen
//     numbers are two 16-byte stores; MMA operands come out of both with ldmatrix.trans.  The places of sixteen tokens (channels)
//     in a tile follow the registers that hold them: tile_element() is the element at a place.  Rows of 272 bytes keep the stores and
//     ldmatrix free of bank conflicts.
//   * the rows' maxima meet in shared memory (atomic maximum of ordered integers) while the values are restored, the
//     probabilities, as a high and a low 16-bit part, go to shared memory as the B operands that P.V reads.
//   * a page's packed bytes are staged by bulk copies; the next page's are requested as soon as the tile is made.
//   * dense tokens (sinks and tail) are copied into the same tiles, 128 at a time, as if they were pages.
// Work split: `pieces` blocks per KV head and row group, an even share of its chunks of dense tokens and pages each.
//
// B200, five query tokens on batch 8, 4,096 tokens, 32 heads on 8, 2-bit: 41.8 us, as three groups of seven rows in
// decode_rows.cu 62.9 us.  On the way: 48.7 us with the code widths read at run time, a block per KV head for the dense tokens and
// every warp reading all probabilities; 45.8 with the promoted channels found by reductions in every warp.  8,900 warp
// instructions per page and dense chunk, issue 48 % of the active cycles.

#pragma once

#include "decode_fast_common.cuh"
#include "code_pairs.cuh"

struct DecodeManyCall {
  const dartkv_cache_desc* d;
  const void* query;
  int query_heads;
  float scale;
  int pieces, total_splits;
  float *part_m, *part_l, *part_acc;
  int* status;
  const int32_t* row_start;
  cudaStream_t stream;
};

namespace {

constexpr int kTileRow = 272;                  // bytes of a tile row: 128 numbers and 16 bytes of padding
constexpr int kTileBytes = 128 * kTileRow;
constexpr uint32_t kKeyOfMinusInf = 0x807FFFFFu;

struct ManyGeom {
  int promoted;                // promoted channels of a page, 0 for uniform keys
  int k_stage, v_codes;        // bytes of the staged keys and of the value codes beside them (the metadata follow)
  int pieces;                  // stream blocks per (batch, KV head, row group)
  int groups, group_rows;      // row groups per KV head, query rows of a group (the last one may have fewer)
};

template <int NT>
struct ManySmem {
  uint64_t k_bar, v_bar;
  int row_max[2][8 * NT];            // ordered integers, by parity of the page
  float row_sum[kWarps][8 * NT];
  int slot[2][128];                  // dense tokens: promoted slots of the channels of up to two key pages
  int promoted_at[128];              // last step in whose page the channel was a promoted one
  uint4 q_frag[NT][4][32];           // B operands of the logits: two k-steps per entry
  uint4 p_frag[8][NT][32];           // B operands of P.V by k-step: high part, low part
  __align__(16) uint8_t keys[kTileBytes];
  __align__(16) uint8_t values[kTileBytes];
};

// sixteen codes
template <int BITS> struct CodeWord { using type = uint32_t; };
template <> struct CodeWord<4> { using type = uint2; };
template <> struct CodeWord<8> { using type = uint4; };

// Floats as integers that order like them (no NaN here).
__device__ __forceinline__ int ordered_key(float x) {
  const int b = __float_as_int(x);
  return b >= 0 ? b : b ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float ordered_value(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7FFFFFFF); }

// The token (channel) whose number stands at a place of a tile row: 2-bit words hold eight elements in each half, a register
// (u, u + 8); 4-bit words and pairs of 8-bit words (u, u + 4).
__device__ __forceinline__ int tile_element(int place, bool two_bits) {
  return two_bits ? (place & ~15) + ((place & 15) >> 1) + 8 * (place & 1) : (place & ~7) + ((place & 7) >> 1) + 4 * (place & 1);
}

__device__ __forceinline__ void store_tile(uint8_t* at, const uint32_t (&r)[8]) {
  reinterpret_cast<uint4*>(at)[0] = make_uint4(r[0], r[1], r[2], r[3]);
  reinterpret_cast<uint4*>(at)[1] = make_uint4(r[4], r[5], r[6], r[7]);
}

template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// NT: eights of query rows of a group.  KB: width of a key code, 2 (with or without promoted channels) or 4; VB: of a value code.  20 rows, batch
// 16, 8,192 tokens: 134 us, with both widths read at run time 155 (144 with the query's operands in shared memory, where registers
// no longer spill), with that of the values alone 151 (144) (B200).
template <int DT, int MD, int NT, int KB, int VB>
__global__ void __launch_bounds__(kThreads, 2) decode_many_kernel(const __grid_constant__ dartkv_cache_desc d, const __grid_constant__ FastArgs a,
                                                                  const __grid_constant__ ManyGeom w) {
  using HO = Half2Ops<DT>;
  using Affine = PairAffine<MD, DT, false>;
  constexpr bool key2 = KB == 2, value2 = VB == 2;
  constexpr bool kHoldQuery = NT <= 3;   // the query's operands in registers: with 32 rows they would spill
  constexpr int vrb = 16 * VB;           // bytes of a row of value codes
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous();
  ManySmem<NT>& sm = *reinterpret_cast<ManySmem<NT>*>(smem_raw);
  uint8_t* const k_stage = smem_raw + (sizeof(ManySmem<NT>) + 127) / 128 * 128;
  uint8_t* const v_stage = k_stage + w.k_stage;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, c = lane & 3;
  // the part of a warp's four tile rows that this lane makes: row `sub`, sixteen numbers from 16 * word on.  Eight neighbouring lanes
  // take four words of two rows: 272 bytes apart, their 16-byte stores fall into different banks.
  const int word = (lane & 3) | ((lane >> 1) & 4), sub = ((lane >> 2) & 1) | ((lane >> 4) << 1);
  const int rep = a.query_heads / d.kv_heads;
  const int seen = d.state[0], k_end = d.state[2], v_end = d.state[3], sink_filled = d.state[4];
  const int fast_end = fast_range_end(d.sink_tokens, d.page_size, k_end, v_end, sink_filled);
  const int total_pages = fast_end > d.sink_tokens ? (fast_end - d.sink_tokens) / 128 : 0;

  const int work_row = blockIdx.x / w.pieces, piece = blockIdx.x - work_row * w.pieces;   // (batch, KV head, row group)
  const int bh = work_row / w.groups, b = bh / d.kv_heads;
  const int head0 = (work_row - bh * w.groups) * w.group_rows, rows = min(rep - head0, w.group_rows);
  const int64_t first_row = (int64_t)b * a.query_heads + (bh - b * d.kv_heads) * rep + head0;   // of the query and the partials
  // A row's work: chunks of 128 live dense tokens (the sinks and the tokens from fast_end on, counted through), then the pages from
  // the first one with a live token on; steps [step, step_end) of them are this block's.
  const int row_first = a.row_start ? max(a.row_start[b], 0) : 0;
  const int sinks = sink_filled - min(row_first, sink_filled), tail = max(fast_end, row_first);
  const int dense_tokens = sinks + max(seen - tail, 0), chunks = (dense_tokens + 127) / 128;
  const int first_page = row_first > d.sink_tokens ? min((row_first - d.sink_tokens) >> 7, total_pages) : 0;
  const int64_t steps = chunks + total_pages - first_page;
  int step = (int)(steps * piece / w.pieces);
  const int step_end = (int)(steps * (piece + 1) / w.pieces);
  auto dense_token = [&](int i) { return i < sinks ? sink_filled - sinks + i : tail + (i - sinks); };   // the i-th live one
  const int meta_row = 4 * d.value_groups;
  auto issue_keys = [&](int pg) {
    mbar_expect_tx(&sm.k_bar, d.key_page_bytes);
    bulk_copy_g2s(k_stage, d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes, d.key_page_bytes, &sm.k_bar);
  };
  auto issue_values = [&](int pg) {
    const int64_t vrow = (int64_t)bh * d.max_value_tokens + (int64_t)pg * 128;
    mbar_expect_tx(&sm.v_bar, 128 * (vrb + meta_row));
    bulk_copy_g2s(v_stage, d.v_codes + vrow * vrb, 128 * vrb, &sm.v_bar);
    bulk_copy_g2s(v_stage + w.v_codes, reinterpret_cast<const uint8_t*>(d.v_meta) + vrow * meta_row, 128 * meta_row, &sm.v_bar);
  };
  if (tid == 0) {
    mbar_init(&sm.k_bar, 1);
    mbar_init(&sm.v_bar, 1);
    mbar_fence_init();
    if (step < step_end && step >= chunks) { issue_keys(first_page + step - chunks); issue_values(first_page + step - chunks); }
  }
  for (int i = tid; i < NT * 128; i += kThreads) {
    const int l = i & 31, ks = 2 * ((i >> 5) & 3), n = 8 * (i >> 7) + (l >> 2);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (n < rows) {   // the query is 4-byte aligned, no more
      const uint32_t* q = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint16_t*>(a.q) + (first_row + n) * 128 + 16 * ks) + (l & 3);
      v = make_uint4(q[0], q[4], q[8], q[12]);
    }
    sm.q_frag[i >> 7][(i >> 5) & 3][l] = v;
  }
  for (int i = tid; i < 16 * NT; i += kThreads) reinterpret_cast<int*>(sm.row_max)[i] = (int)kKeyOfMinusInf;
  if (tid < 128) sm.promoted_at[tid] = -1;
  __syncthreads();   // the barriers are ready, too

  CodeConsts<MD> cc;
  cc.init();
  const uint32_t mask4 = reg_const(0x000F000Fu << (2 * Half2Ops<MD>::kFirstPos));
  const float scale2 = a.scale * kLog2e;
  const int K = key2 ? w.promoted : 0;
  bool ok = true;

  // sixteen codes of a row, in one word, two or four
  auto restore = [&](auto codes, const Affine& affine, uint32_t (&r)[8]) {
    if constexpr (sizeof(codes) == 4) {
      restore_codes2<MD, DT, false>(cc, codes, affine, r);
    } else if constexpr (sizeof(codes) == 8) {
      restore_codes4<MD, DT, false>(cc, mask4, codes.x, affine, r);
      restore_codes4<MD, DT, false>(cc, mask4, codes.y, affine, r + 4);
    } else {
      restore_codes8<MD, DT, false>(codes.x, codes.y, affine, r);
      restore_codes8<MD, DT, false>(codes.z, codes.w, affine, r + 4);
    }
  };
  using KeyWord = typename CodeWord<KB>::type;
  using ValueWord = typename CodeWord<VB>::type;
  constexpr int kKeyPositions = KB == 2 ? 3 : 1, kValuePositions = VB == 2 ? 3 : VB == 4 ? 1 : 0;
  // the promoted channels of the page of that step, once its keys have landed
  auto mark_promoted = [&](int of_step) {
    for (int k = tid; k < K; k += kThreads) sm.promoted_at[reinterpret_cast<const int32_t*>(k_stage + d.key_off_index)[k] & 127] = of_step;
  };
  // the staged page's keys to the tile
  auto make_keys = [&]() {
    const uint16_t* scale = reinterpret_cast<const uint16_t*>(k_stage + d.key_off_scale) + 4 * warp + sub;
    const uint16_t* zero = reinterpret_cast<const uint16_t*>(k_stage + d.key_off_zero) + 4 * warp + sub;
    const uint8_t* codes = k_stage + (4 * warp + sub) * (16 * KB) + word * (2 * KB);
    uint8_t* to = sm.keys + (4 * warp + sub) * kTileRow + 32 * word;
    KeyWord x[4];
    uint32_t ss[4], zz[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // channel 32 * i + 4 * warp + sub
      x[i] = *reinterpret_cast<const KeyWord*>(codes + 32 * i * (16 * KB));
      ss[i] = scale[32 * i];
      zz[i] = zero[32 * i];
    }
    int promoted[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) promoted[i] = K > 0 ? sm.promoted_at[32 * i + 4 * warp + sub] : -1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      Affine affine;
      affine.template init<kKeyPositions>(low_twice(ss[i]), low_twice(zz[i]));
      uint32_t r[8];
      restore(x[i], affine, r);
      if (promoted[i] != step) store_tile(to + 32 * i * kTileRow, r);   // else made below
    }
    if constexpr (key2) {
      for (int s = 4 * warp + sub; s < K; s += 32) {
        const int ch = reinterpret_cast<const int32_t*>(k_stage + d.key_off_index)[s] & 127;
        Affine affine;
        affine.template init<2>(low_twice(lds_u16(k_stage + d.key_off_scale + 2 * ch)), low_twice(lds_u16(k_stage + d.key_off_zero + 2 * ch)));
        uint32_t r[8];
        restore_codes22<MD, DT, false>(cc, lds_u32(k_stage + 32 * ch + 4 * word), lds_u32(k_stage + d.key_off_high + 32 * s + 4 * word), affine, r);
        store_tile(sm.keys + ch * kTileRow + 32 * word, r);
      }
    }
  };
  const int vgroup2 = 2 * (16 * word / d.value_group);
  auto make_values = [&]() {
    const int t0 = tile_element(4 * warp + sub, key2);   // place 32 * i further holds token 32 * i further
    const uint8_t* meta = v_stage + w.v_codes + t0 * meta_row + vgroup2;
    const uint8_t* codes = v_stage + t0 * vrb + word * (2 * VB);
    uint8_t* to = sm.values + (4 * warp + sub) * kTileRow + 32 * word;
    ValueWord x[4];
    uint32_t ss[4], zz[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = *reinterpret_cast<const ValueWord*>(codes + 32 * i * vrb);
      ss[i] = lds_u16(meta + 32 * i * meta_row);
      zz[i] = lds_u16(meta + 32 * i * meta_row + 2 * d.value_groups);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      Affine affine;
      affine.template init<kValuePositions>(low_twice(ss[i]), low_twice(zz[i]));
      uint32_t r[8];
      restore(x[i], affine, r);
      store_tile(to + 32 * i * kTileRow, r);
    }
  };
  // dense tokens from the i0-th on to the tiles: keys as [token][channel].  A token that is packed on this side (the other side's
  // value or key is dense) is restored element by element.
  auto make_dense = [&](int i0, int side) {
    const int page0 = (dense_token(max(i0, min(sinks, dense_tokens - 1))) - d.sink_tokens) / 128;   // the first one of a chunk's packed tokens
    if (side == 0 && d.key_mode == DARTKV_MIXED_PAGE && k_end > fast_end) {
      for (int i = tid; i < 256; i += kThreads) sm.slot[i >> 7][i & 127] = -1;
      __syncthreads();
      for (int i = tid; i < 2 * K; i += kThreads) {
        const int pg = page0 + i / K;
        if (d.sink_tokens + 128 * pg < k_end) {
          const int ch = reinterpret_cast<const int32_t*>(d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes + d.key_off_index)[i % K];
          if (ch >= 0 && ch < 128) sm.slot[i / K][ch] = i % K;
        }
      }
      __syncthreads();
    }
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      const int place = 32 * i + 4 * warp + sub;
      uint32_t x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = 0u;
      if (i0 + place < dense_tokens) {
        const int t = dense_token(i0 + place);
        if (t < sink_filled || t >= (side == 0 ? k_end : v_end)) {
          const uint16_t* row = t < sink_filled
              ? reinterpret_cast<const uint16_t*>(side == 0 ? d.k_sink : d.v_sink) + ((int64_t)bh * d.sink_tokens + t) * 128
              : reinterpret_cast<const uint16_t*>(side == 0 ? d.k_ring : d.v_ring) + ((int64_t)bh * d.ring_tokens + t % d.ring_tokens) * 128;
          const uint4 lo = reinterpret_cast<const uint4*>(row)[2 * word], hi = reinterpret_cast<const uint4*>(row)[2 * word + 1];
          x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
          x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
        } else {
          const int pg = (t - d.sink_tokens) / 128, j = (t - d.sink_tokens) & 127;
          const uint8_t* keys = d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes;
          const int64_t vrow = (int64_t)bh * d.max_value_tokens + (t - d.sink_tokens);
          const int bits = side == 1 ? VB : KB;
          const uint32_t mask = (1u << bits) - 1u;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int ch = 16 * word + e;
            uint32_t code;
            uint16_t s, z;
            if (side == 0) {
              code = (keys[ch * 16 * bits + j * bits / 8] >> (j * bits & 7)) & mask;
              const int slot = K > 0 ? sm.slot[(pg - page0) & 1][ch] : -1;
              if (slot >= 0) code |= ((keys[d.key_off_high + 32 * slot + j / 4] >> (2 * j & 7)) & 3u) << 2;
              s = reinterpret_cast<const uint16_t*>(keys + d.key_off_scale)[ch];
              z = reinterpret_cast<const uint16_t*>(keys + d.key_off_zero)[ch];
            } else {
              code = (d.v_codes[vrow * vrb + ch * bits / 8] >> (ch * bits & 7)) & mask;
              s = reinterpret_cast<const uint16_t*>(d.v_meta)[vrow * 2 * d.value_groups + ch / d.value_group];
              z = reinterpret_cast<const uint16_t*>(d.v_meta)[vrow * 2 * d.value_groups + d.value_groups + ch / d.value_group];
            }
            const float v = restore16<DT, MD>((float)code, Half2Ops<MD>::to_float(s), Half2Ops<MD>::to_float(z), DARTKV_DEQUANT_PER_OP);
            x[e >> 1] |= (uint32_t)HO::from_float(v) << (16 * (e & 1));
          }
        }
      }
      if (side == 0) {
        store_tile(sm.keys + place * kTileRow + 32 * word, x);
      } else {   // channel pairs (2k, 2k + 1) to the places that restored values have
        uint32_t r[8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t sel = u & 1 ? 0x7632u : 0x5410u;
          if (value2) {
            r[u] = prmt(x[u >> 1], x[4 + (u >> 1)], sel);
            r[4 + u] = prmt(x[2 + (u >> 1)], x[6 + (u >> 1)], sel);
          } else {
            r[u] = prmt(x[u >> 1], x[2 + (u >> 1)], sel);
            r[4 + u] = prmt(x[4 + (u >> 1)], x[6 + (u >> 1)], sel);
          }
        }
        store_tile(sm.values + place * kTileRow + 32 * word, r);
      }
    }
  };

  // A operands: matrix lane >> 3 of a fragment, row lane & 7 of it.  Logits: this warp's sixteen tokens, all channels.  P.V: 32 channels
  // and half of the tokens, so that the warps read the probabilities four times and not eight.
  const int fr = lane & 7, fi = lane >> 3, quarter = warp & 3, half = warp >> 2;
  const uint32_t trans_row = ((fi >> 1) * 8 + fr) * kTileRow + (fi & 1) * 16;
  const uint32_t keys_trans = smem_u32(sm.keys) + trans_row + 32 * warp;                                                       // + 16 tile rows per k-step
  const uint32_t keys_plain = smem_u32(sm.keys) + (16 * warp + (fi & 1) * 8 + fr) * kTileRow + (fi >> 1) * 16;                 // + 32 bytes per k-step
  const uint32_t values_at = smem_u32(sm.values) + trans_row + 64 * quarter + 64 * half * kTileRow;                            // + 16 tile rows per k-step
  uint4 held[kHoldQuery ? NT : 1][4];
  if constexpr (kHoldQuery) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int k = 0; k < 4; ++k) held[nt][k] = sm.q_frag[nt][k][lane];
  }

  float o_acc[2][NT][4];                // channel place 32 * quarter + 16 * mt + g + 8 * (i >> 1), row 8 * nt + 2c + (i & 1); half of the tokens
  float m_run[NT][2], l_run[NT][2];     // row 8 * nt + 2c + e, log2 domain; l_run: this lane's tokens only
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int i = 0; i < 8; ++i) o_acc[i >> 2][nt][i & 3] = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; ++e) { m_run[nt][e] = -INFINITY; l_run[nt][e] = 0.0f; }
  }

  uint32_t copies = 0, buffer = 0;   // parities: of the staged pages consumed, of the steps
  if (step < step_end && step >= chunks && K > 0) {
    ok = mbar_wait(&sm.k_bar, 0) && ok;
    mark_promoted(step);
    __syncthreads();
  }
  for (; step < step_end; ++step, buffer ^= 1) {
    const bool dense = step < chunks, fetch = step + 1 < step_end && step + 1 >= chunks;
    const int page = first_page + step - chunks;
    if (dense) {
      make_dense(128 * step, 0);
    } else {
      ok = mbar_wait(&sm.k_bar, copies) && ok;
      make_keys();
    }
    __syncthreads();   // the keys' tile is made; the values' tile, the maxima of the step before and its probabilities have been read
    if (tid == 0 && fetch) issue_keys(page + 1);
    int* const row_max = sm.row_max[buffer];

    // ---- logits of this warp's sixteen tokens
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[nt][i] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < 8; ks += 2) {
      uint32_t a0[4], a1[4];
      if (dense) {
        ldmatrix4<false>(a0, keys_plain + 32 * ks);
        ldmatrix4<false>(a1, keys_plain + 32 * ks + 32);
      } else {
        ldmatrix4<true>(a0, keys_trans + 16 * kTileRow * ks);
        ldmatrix4<true>(a1, keys_trans + 16 * kTileRow * (ks + 1));
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint4 q = kHoldQuery ? held[kHoldQuery ? nt : 0][ks >> 1] : sm.q_frag[nt][ks >> 1][lane];
        HO::mma(s[nt], a0[0], a0[1], a0[2], a0[3], q.x, q.y);
        HO::mma(s[nt], a1[0], a1[1], a1[2], a1[3], q.z, q.w);
      }
    }
    // ---- their maxima
    int live_from, live_to, t0, t1;   // in tokens of the page
    if (dense) {
      t0 = 16 * warp + g; t1 = t0 + 8; live_from = 0; live_to = dense_tokens - 128 * step;
    } else {
      t0 = tile_element(16 * warp + g, key2); t1 = tile_element(16 * warp + g + 8, key2);
      live_from = row_first - (d.sink_tokens + 128 * page); live_to = 128;
    }
    const bool live0 = t0 >= live_from && t0 < live_to, live1 = t1 >= live_from && t1 < live_to;
    float mine = -INFINITY;   // the maximum that this lane reports
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[nt][e] = live0 ? s[nt][e] * scale2 : -INFINITY;
        s[nt][2 + e] = live1 ? s[nt][2 + e] * scale2 : -INFINITY;
        float mx = fmaxf(s[nt][e], s[nt][2 + e]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        if (g == 2 * nt + e) mine = mx;
      }
    if (g < 2 * NT) atomicMax(&row_max[8 * (g >> 1) + 2 * c + (g & 1)], ordered_key(fmaxf(mine, -INFINITY)));
    if (tid < 8 * NT) sm.row_max[buffer ^ 1][tid] = (int)kKeyOfMinusInf;   // for the next step

    if (dense) {
      make_dense(128 * step, 1);
    } else {
      ok = mbar_wait(&sm.v_bar, copies) && ok;
      make_values();
      copies ^= 1;
    }
    __syncthreads();   // the maxima and the values' tile are complete
    if (tid == 0 && fetch) issue_values(page + 1);

    // ---- probabilities of this warp's tokens: k-step `warp` of P.V
    float alpha[NT][2];
    bool moved = false;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int2 mx = *reinterpret_cast<const int2*>(&row_max[8 * nt + 2 * c]);
      float m_ref[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float m_new = fmaxf(m_run[nt][e], ordered_value(e ? mx.y : mx.x));
        m_ref[e] = m_new == -INFINITY ? 0.0f : m_new;   // nothing live yet: every weight below comes out zero
        alpha[nt][e] = fast_exp2(m_run[nt][e] - m_ref[e]);
        m_run[nt][e] = m_new;
        moved = moved || alpha[nt][e] != 1.0f;
      }
      uint32_t hi[2], lo[2];
      l_run[nt][0] *= alpha[nt][0];
      l_run[nt][1] *= alpha[nt][1];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float p0 = fast_exp2(s[nt][2 * i] - m_ref[0]), p1 = fast_exp2(s[nt][2 * i + 1] - m_ref[1]);
        l_run[nt][0] += p0;
        l_run[nt][1] += p1;
        hi[i] = pack16<DT>(p0, p1);
        float h0, h1;
        unpack16<DT>(hi[i], h0, h1);
        lo[i] = pack16<DT>(p0 - h0, p1 - h1);
      }
      sm.p_frag[warp][nt][lane] = make_uint4(transpose8x8(hi[0]), transpose8x8(hi[1]), transpose8x8(lo[0]), transpose8x8(lo[1]));
    }
    if (__any_sync(0xffffffffu, moved)) {   // the running maximum rarely moves after the first pages
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 8; ++i) o_acc[i >> 2][nt][i & 3] *= alpha[nt][i & 1];
    }
    if (K > 0 && fetch) {   // the next page's keys were requested at the beginning of the step
      ok = mbar_wait(&sm.k_bar, copies) && ok;
      mark_promoted(step + 1);
    }
    __syncthreads();   // the probabilities and the next page's marks are complete

    // ---- O[channel][row] += V^T P
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t v0[4], v1[4];
      ldmatrix4<true>(v0, values_at + 16 * kTileRow * ks);
      ldmatrix4<true>(v1, values_at + 16 * kTileRow * ks + 32);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint4 p = sm.p_frag[4 * half + ks][nt][lane];
        HO::mma(o_acc[0][nt], v0[0], v0[1], v0[2], v0[3], p.x, p.y);
        HO::mma(o_acc[1][nt], v1[0], v1[1], v1[2], v1[3], p.x, p.y);
        HO::mma(o_acc[0][nt], v0[0], v0[1], v0[2], v0[3], p.z, p.w);
        HO::mma(o_acc[1][nt], v1[0], v1[1], v1[2], v1[3], p.z, p.w);
      }
    }
  }

  // ---- the block's partial: one maximum for all warps, so the halves of the tokens and the sums just add up
  __syncthreads();   // the tiles are no longer read
  float* const other = reinterpret_cast<float*>(sm.keys) + (quarter * 32 + lane) * (8 * NT + 4);   // 16-byte rows, a lane each
  if (half == 1) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        reinterpret_cast<float4*>(other)[mt * NT + nt] = make_float4(o_acc[mt][nt][0], o_acc[mt][nt][1], o_acc[mt][nt][2], o_acc[mt][nt][3]);
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float l = l_run[nt][e];
      l += __shfl_xor_sync(0xffffffffu, l, 4);
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      if (g == 0) sm.row_sum[warp][8 * nt + 2 * c + e] = l;
    }
  __syncthreads();
  if (half == 0) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const float4 x = reinterpret_cast<const float4*>(other)[mt * NT + nt];
        const float add[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = 8 * nt + 2 * c + (i & 1);
          if (n < rows)
            a.part_acc[((first_row + n) * a.total_splits + 1 + piece) * 128 + tile_element(32 * quarter + 16 * mt + g + 8 * (i >> 1), value2)] =
                o_acc[mt][nt][i] + add[i];
        }
      }
  } else if (warp == 4 && g == 0) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = 8 * nt + 2 * c + e;
        if (n >= rows) continue;
        float l = 0.0f;
#pragma unroll
        for (int v = 0; v < kWarps; ++v) l += sm.row_sum[v][n];
        const int64_t row = (first_row + n) * a.total_splits;
        a.part_m[row + 1 + piece] = merge_maximum(m_run[nt][e] == -INFINITY ? -INFINITY : m_run[nt][e] * 0.6931471805599453f, l);
        a.part_l[row + 1 + piece] = l;
        if (piece == 0) {   // the slot that the other kernels have a dense block for
          a.part_m[row] = -INFINITY;
          a.part_l[row] = 0.0f;
        }
      }
  }
  if (!ok && lane == 0) atomicExch(a.status, 1);
}

ManyGeom many_geometry(const dartkv_cache_desc* d, int rep) {
  ManyGeom w{};
  w.promoted = d->key_mode == DARTKV_MIXED_PAGE ? d->promoted : 0;
  w.k_stage = (d->key_page_bytes + 127) / 128 * 128;
  w.v_codes = 128 * d->value_row_bytes;
  w.groups = (rep + 31) / 32;
  w.group_rows = (rep + w.groups - 1) / w.groups;
  return w;
}

template <int NT>
size_t many_smem_of(const dartkv_cache_desc* d, const ManyGeom& w) {
  return (sizeof(ManySmem<NT>) + 127) / 128 * 128 + w.k_stage + w.v_codes + 128 * 4 * d->value_groups;
}
size_t many_smem(const dartkv_cache_desc* d, const ManyGeom& w) {
  const int nt = (w.group_rows + 7) / 8;
  return nt <= 2 ? many_smem_of<2>(d, w) : nt == 3 ? many_smem_of<3>(d, w) : many_smem_of<4>(d, w);
}

// Not for 8-bit values beside 4-bit keys: such pages leave no room for two blocks of decode_rows.cu, whose geometries these are.
using ManyKernel = void (*)(dartkv_cache_desc, FastArgs, ManyGeom);
template <int DT, int MD, int NT>
ManyKernel many_variant_of(int kb, int vb) {
  if (kb == 2) return vb == 2 ? decode_many_kernel<DT, MD, NT, 2, 2> : vb == 4 ? decode_many_kernel<DT, MD, NT, 2, 4> : decode_many_kernel<DT, MD, NT, 2, 8>;
  return vb == 2 ? decode_many_kernel<DT, MD, NT, 4, 2> : decode_many_kernel<DT, MD, NT, 4, 4>;
}
template <int DT, int MD>
ManyKernel many_variant(int nt, int kb, int vb) {
  return nt <= 2 ? many_variant_of<DT, MD, 2>(kb, vb) : nt == 3 ? many_variant_of<DT, MD, 3>(kb, vb) : many_variant_of<DT, MD, 4>(kb, vb);
}

// Launches the kernel of these types.  The 15 kernels of a pair of types are a translation unit (decode_many_*.cu): a module is loaded as a
// whole by the first call that reaches it, which took 37 ms with all of them in one and every one's attribute set, 27 ms with
// the attribute of one and 4 ms so.
template <int DT, int MD>
int many_launch(const DecodeManyCall& c) {
  const dartkv_cache_desc* d = c.d;
  const int rep = c.query_heads / d->kv_heads;
  ManyGeom w = many_geometry(d, rep);
  w.pieces = c.pieces;
  const int work_rows = d->batch * d->kv_heads * w.groups;
  const FastArgs a{c.query, c.query_heads, c.scale, DARTKV_DEQUANT_PER_OP, 0, work_rows * c.pieces, 0, c.total_splits, c.part_m, c.part_l, c.part_acc,
                   c.status, c.row_start};
  const int kb = w.promoted ? 2 : d->key_bits, vb = d->value_bits, nt = max(2, (w.group_rows + 7) / 8);
  const ManyKernel kernel = many_variant<DT, MD>(nt, kb, vb);
  static SharedMemoryOptIn<3 * 5> opt_in;
  DARTKV_CUDA_OK(opt_in((nt - 2) * 5 + (kb == 4 ? 3 : 0) + (vb == 2 ? 0 : vb == 4 ? 1 : 2), kernel, 160 * 1024));
  DARTKV_CUDA_OK(launch_following(kernel, dim3(work_rows * c.pieces), dim3(kThreads), many_smem(d, w), c.stream, *d, a, w));
  DARTKV_LAUNCH_OK("decode_many_kernel");
  return DARTKV_OK;
}

}  // namespace
