// Tensor-core decode attention with packed codes turned into MMA operands in registers, for groups of up to 4 or 8
// query rows of a KV head: pages of 128 tokens with one key group, 2/4-bit keys or 2+2-bit promoted channels,
// 2/4/8-bit values in groups of 16..128 channels, the rounded flavours of the dequantization.  It serves the
// geometries of decode_wide.cu that fit this description, and calls with more than four query rows per KV head
// (several query tokens at once, wide GQA groups), which otherwise take one call per four rows.  More than eight rows
// are split into groups of equal size; a group is a row of work like a (batch, KV head) pair, so all of them run in
// one launch and find each other's pages in L2.  decode_many.cuh takes such calls where they are large.
//
// What bounds it: as in decode_fast.cu, the dependent phases of a page (order, table, logits, softmax, P.V) at four warps
// per scheduler, here with instruction fetch as the largest stall; time moves with the number of instructions (three
// packed operations per operand register).  What the layout is for:
//   * keys: a register pairs two CHANNELS of one token (the contraction direction).  The half-words of two channel
//     rows are put side by side with one prmt, after which every register is one logic op plus the packed arithmetic
//     with the two channels' scales side by side.  Register u of a thread is token 16g + 8*HF + u, the same for 2-bit
//     and 4-bit codes; two registers (u, u + 1) are the two row halves of an m16n8k16 A operand, the query rows are its
//     N columns, so one dequantization serves 8 rows per MMA.
//   * values: a register pairs two TOKENS of one channel.  The contraction order of P.V is free, so it follows the
//     logits' accumulators: packed to 16 bits and transposed by movmatrix they are the B operand, without shared
//     memory.  That makes the four lanes of a quad read rows 32 tokens apart; the staged page is cut into four
//     32-token pieces with 32 bytes between them, which keeps these reads free of bank conflicts.
//   * the probabilities travel as a high and a low 16-bit part: side by side in the eight columns with up to four
//     query rows (columns 4..7 repeat rows 0..3, so the same lane sees both), in MMAs of their own with more.
//   * the two warps of a pair share a staged page and split its tokens; nothing is exchanged between them.
//   * uniform pages take the channels in their order: the query rows wait as MMA operands, code addresses are constants, and a
//     table entry holds the parameters of both channel pairs of a k-step (64.9 us, with the promoted pages' row offsets in the
//     table, to 61.3 at the size below; two steps unrolled, four 63.5).  Value parameters of groups of 64 in one wide load and a
//     select instead of four narrow ones: 62.3, the registers run out.
// Staging is by bulk copies on mbarriers, keys and values separately: with one buffer each (4-bit pages) the next
// page's keys arrive during P.V and its values during the logits, two blocks per SM stay resident.
//
// B200: 4-bit fp16 pages, batch 24, 6,001 tokens, 32 heads on 8: 115 us through decode_wide.cu, 60 us here (the query
// rows in M instead of N needed 64 + 32 accumulators and spilled).  Two query tokens on batch 8, 4,096 tokens,
// 2-bit: 69 us as two passes of decode_fast.cu, 44 us here in one launch.  One
// query token on the 2-bit pages of decode_fast.cu stays there: 1,026 us against 1,462 us at batch 128, 32,768 tokens.

#include "decode_fast_common.cuh"
#include "code_pairs.cuh"

namespace {

struct RowsGeom {
  int key_kind;      // 2, 4: uniform code width; 22: 2-bit codes plus a 2-bit plane for the promoted channels
  int key_row;       // bytes of a channel row of key codes, and of a channel's row in the query table
  int v_piece;       // shared bytes from one 32-token piece of value codes to the next
  int v_meta, v_meta_piece;   // offset of the value metadata in a value stage, bytes from piece to piece
  int k_stage, v_stage;       // bytes per stage
  int stages;        // 1 or 2
  int pair_bytes;
  int groups, group_rows;    // row groups per KV head, query rows of a group (the last one may have fewer)
};

constexpr int kTableBytes = 64 * 16 + 256;   // per warp: channel-pair entries, contraction order, promoted flags

template <int R>
struct RowsSmem {
  uint64_t k_bar[kPairs][2], v_bar[kPairs][2];
  float merge_m[kWarps][R];
  float merge_l[kWarps][R];
  int slot_map[128];
};

// Block merge of the eight warp states of R rows each (block_merge of decode_fast_common.cuh takes four rows).
template <int R>
__device__ __forceinline__ void rows_merge(const FastArgs& a, const RowsSmem<R>& bs, const float* warp_out, int64_t first_row, int rows, int slot) {
  const int ch = threadIdx.x & 127;
  for (int r = threadIdx.x >> 7; r < rows; r += kThreads / 128) {
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, bs.merge_m[w][r]);
    float l = 0.0f, acc = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float mw = bs.merge_m[w][r];
      if (mw != -INFINITY) {
        const float wgt = fast_exp2(mw - m);
        l += bs.merge_l[w][r] * wgt;
        acc += warp_out[(w * R + r) * 128 + ch] * wgt;
      }
    }
    const int64_t row = (first_row + r) * a.total_splits + slot;
    if (ch == 0) {
      a.part_m[row] = merge_maximum(m == -INFINITY ? -INFINITY : m * 0.6931471805599453f, l);
      a.part_l[row] = l;
    }
    a.part_acc[row * 128 + ch] = acc;
  }
}

// R: most query rows of a group, 4 or 8.  UNIFORM: no promoted channels; in one kernel with them the two forms take each other's registers and
// instruction fetch: promoted 2-bit pages with fp16 metadata beside bf16, eight rows, 16 x 16,384 tokens 166 us, apart 156; 4-bit, four
// rows, 94.7 and 93.5 (B200).
template <int DT, int MD, bool FP32, int R, bool UNIFORM>
__global__ void __launch_bounds__(kThreads, 2) decode_rows_kernel(dartkv_cache_desc d, FastArgs a, RowsGeom w) {
  using H = Half2Ops<MD>;
  using HO = Half2Ops<DT>;
  using Affine = PairAffine<MD, DT, FP32>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous();
  RowsSmem<R>& bs = *reinterpret_cast<RowsSmem<R>*>(smem_raw);
  uint8_t* q_table = smem_raw + (sizeof(RowsSmem<R>) + 127) / 128 * 128;   // [channel] rows of w.key_row bytes: 8 columns; uniform pages: [k-step][lane] operands
  uint8_t* pair_base = q_table + 128 * w.key_row;
  float* warp_out = reinterpret_cast<float*>(pair_base);   // merge buffer: aliases the staging memory

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, c = lane & 3;
  const int rep = a.query_heads / d.kv_heads;

  if ((int)blockIdx.x >= a.stream_blocks) {
    // dense tokens of one (batch, kv head), four query rows: partial slot 0
    const int heads = d.batch * d.kv_heads, idx = blockIdx.x - a.stream_blocks;
    const int bh = idx % heads, head0 = 4 * (idx / heads);
    dense_block<DT, MD, true>(d, a, bs, warp_out, bh, head0);
    __syncthreads();
    block_merge<true>(a, bs, warp_out, bh / d.kv_heads, bh % d.kv_heads, rep, 0, head0);
    return;
  }

  const int sb = blockIdx.x;
  int unit = (int)((int64_t)sb * a.units / a.stream_blocks);
  const int unit_end = (int)((int64_t)(sb + 1) * a.units / a.stream_blocks);
  const int pair = warp >> 1, hf = warp & 1;
  uint8_t* const pair_mem = pair_base + pair * w.pair_bytes;
  uint8_t* const k_mem = pair_mem;
  uint8_t* const v_mem = pair_mem + w.stages * w.k_stage;
  uint8_t* const my_table = v_mem + w.stages * w.v_stage + hf * kTableBytes;
  uint4* const table = reinterpret_cast<uint4*>(my_table);   // [64] channel pairs: scales, zero points, row offsets
  uint8_t* const order = my_table + 1024;
  uint8_t* const flag = my_table + 1024 + 128;
  const int k_end = d.state[2], v_end = d.state[3], sink_filled = d.state[4];
  const int fast_end = fast_range_end(d.sink_tokens, d.page_size, k_end, v_end, sink_filled);
  const int total_pages = fast_end > d.sink_tokens ? (fast_end - d.sink_tokens) / 128 : 0;
  const int vrb = d.value_row_bytes, meta_row = 4 * d.value_groups;
  int bh = 0;
  // the first warp of a pair fetches: one lane announces the bytes, then one lane per copy
  auto issue_keys = [&](int pg, int stage) {
    if (lane == 0) {
      mbar_expect_tx(&bs.k_bar[pair][stage], d.key_page_bytes);
      bulk_copy_g2s(k_mem + stage * w.k_stage, d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes, d.key_page_bytes,
                    &bs.k_bar[pair][stage]);
    }
  };
  auto issue_values = [&](int pg, int stage) {
    if (lane == 0) mbar_expect_tx(&bs.v_bar[pair][stage], 128 * (vrb + meta_row));
    __syncwarp();
    if (lane < 4) {
      const int64_t vrow = (int64_t)bh * d.max_value_tokens + (int64_t)pg * 128 + 32 * lane;
      uint8_t* dst = v_mem + stage * w.v_stage;
      bulk_copy_g2s(dst + lane * w.v_piece, d.v_codes + vrow * vrb, 32 * vrb, &bs.v_bar[pair][stage]);
      bulk_copy_g2s(dst + w.v_meta + lane * w.v_meta_piece, reinterpret_cast<const uint8_t*>(d.v_meta) + vrow * meta_row, 32 * meta_row,
                    &bs.v_bar[pair][stage]);
    }
  };
  if (hf == 0 && lane == 0) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bs.k_bar[pair][s], 1);
      mbar_init(&bs.v_bar[pair][s], 1);
    }
    mbar_fence_init();
  }
  __syncthreads();
  const int K = UNIFORM ? 0 : d.promoted;
  const int prom_steps = (K + 15) >> 4;
  const float scale2 = a.scale * kLog2e;
  const int vgroup = (16 * g) / d.value_group;
  const uint8_t* const q_thread = q_table + 2 * g;
  bool ok = true;
  CodeConsts<MD> cc;
  cc.init();
  const uint32_t mask4 = reg_const(0x000F000Fu << (2 * H::kFirstPos));
  const int ahead = w.stages * kPairs;   // a page's buffers are refilled with the page that many pages on
  int iter = 0;   // pages this pair has consumed so far: stage and barrier parity carry over from row to row

  while (unit < unit_end) {
    const int work_row = unit / a.quads;   // (batch, KV head, row group)
    bh = work_row / w.groups;
    const int head0 = (work_row - bh * w.groups) * w.group_rows, rows = min(rep - head0, w.group_rows);
    const int quad_begin = unit - work_row * a.quads;
    const int quad_count = min(a.quads - quad_begin, unit_end - unit);
    unit += quad_count;
    const int b = bh / d.kv_heads;
    const int64_t first_row = (int64_t)b * a.query_heads + (bh - b * d.kv_heads) * rep + head0;   // of the query and the partials
    // tokens before the row's first live one get no weight: whole pages of them are not even fetched
    const int row_first = a.row_start ? max(a.row_start[b], 0) : 0;
    const int p_begin = max(4 * quad_begin, row_first > d.sink_tokens ? (row_first - d.sink_tokens) >> 7 : 0);
    const int p_end = min(4 * (quad_begin + quad_count), total_pages);
    const int pg0 = p_begin + pair;
    if (hf == 0) {
      for (int s = 0; s < w.stages; ++s)
        if (pg0 + s * kPairs < p_end) {
          const int stage = w.stages == 2 ? (iter + s) & 1 : 0;
          issue_keys(pg0 + s * kPairs, stage);
          issue_values(pg0 + s * kPairs, stage);
        }
    }
    for (int i = tid; i < 8 * 128; i += kThreads) {
      const int col = i >> 7, ch = i & 127, r = R == 4 ? col & 3 : col;
      uint16_t v = 0;
      if (r < rows) v = reinterpret_cast<const uint16_t*>(a.q)[(first_row + r) * 128 + ch];
      // uniform pages: a lane's operand of a k-step as it goes into the MMA
      const int at = UNIFORM ? 8 * (32 * (ch >> 4) + 4 * col + (ch & 3)) + 2 * ((ch >> 2) & 3) : ch * w.key_row + 2 * col;
      *reinterpret_cast<uint16_t*>(q_table + at) = v;
    }
    __syncthreads();

    // [m-tile mt][i]: channel 16g + 2mt + (i >> 1), column 2c + (i & 1)
    float o_acc[8][4];
    float m_run[2], l_run[2];   // this lane's columns, log2 domain; l_run: this lane's tokens only
#pragma unroll
    for (int mt = 0; mt < 8; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) o_acc[mt][i] = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; ++e) { m_run[e] = -INFINITY; l_run[e] = 0.0f; }

    for (int pg = pg0; pg < p_end; pg += kPairs, ++iter) {
      const int stage = w.stages == 2 ? iter & 1 : 0;
      const uint32_t parity = (w.stages == 2 ? iter >> 1 : iter) & 1;
      ok = mbar_wait(&bs.k_bar[pair][stage], parity) && ok;
      const uint8_t* blob = k_mem + stage * w.k_stage;

      // ---- contraction order of the channels (promoted slots first), then one entry per channel pair: a k-step is
      // sixteen positions, lane c of a quad takes positions (c, c + 4) and (c + 8, c + 12) of it
      if constexpr (!UNIFORM) {
        reinterpret_cast<uint32_t*>(flag)[lane] = 0;
        __syncwarp();
        const int32_t* idx = reinterpret_cast<const int32_t*>(blob + d.key_off_index);
        for (int k = lane; k < K; k += 32) {
          const int ch = idx[k] & 127;
          flag[ch] = 1;
          order[k] = (uint8_t)ch;
        }
        __syncwarp();
        const uint32_t flags = reinterpret_cast<const uint32_t*>(flag)[lane];   // channels 4*lane .. +3
        const int mine = 4 - __popc(flags & 0x01010101u);
        int before = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, before, off);
          if (lane >= off) before += up;
        }
        int pos = K + before - mine;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (!((flags >> (8 * i)) & 1u)) order[min(pos++, 127)] = (uint8_t)(4 * lane + i);
        __syncwarp();
      }
      auto param = [&](int off, int c0, int c1) { return prmt(lds_u16(blob + off + 2 * c0), lds_u16(blob + off + 2 * c1), 0x5410u); };
      if constexpr (UNIFORM) {
        // channels in their order: one entry holds both pairs of a k-step and lane of a quad
        const int ch = 16 * (lane >> 2) + c;
        table[lane] = make_uint4(param(d.key_off_scale, ch, ch + 4), param(d.key_off_zero, ch, ch + 4),
                                 param(d.key_off_scale, ch + 8, ch + 12), param(d.key_off_zero, ch + 8, ch + 12));
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int f = lane + 32 * i;
          const int p0 = 16 * (f >> 3) + 8 * ((f >> 2) & 1) + (f & 3);
          const int ch0 = order[p0], ch1 = order[p0 + 4];
          table[f] = make_uint4(param(d.key_off_scale, ch0, ch1), param(d.key_off_zero, ch0, ch1), (uint32_t)(ch0 * w.key_row),
                                (uint32_t)(ch1 * w.key_row));
        }
      }
      __syncwarp();

      // ---- logits over eight k-steps: [m-tile][i] = token 16g + 8*HF + 2mt + (i >> 1), column 2c + (i & 1)
      float s_acc[4][4];
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) s_acc[mt][i] = 0.0f;
      auto products = [&](const uint32_t (&ra)[8], const uint32_t (&rb)[8], uint32_t b0, uint32_t b1) {
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) HO::mma(s_acc[mt], ra[2 * mt], ra[2 * mt + 1], rb[2 * mt], rb[2 * mt + 1], b0, b1);
      };
      auto multiply = [&](const uint4& ea, const uint4& eb, const uint32_t (&ra)[8], const uint32_t (&rb)[8]) {
        products(ra, rb, prmt(lds_u16(q_thread + ea.z), lds_u16(q_thread + ea.w), 0x5410u),
                 prmt(lds_u16(q_thread + eb.z), lds_u16(q_thread + eb.w), 0x5410u));
      };
      if (UNIFORM && w.key_kind == 4) {
        const uint2* const q_ready = reinterpret_cast<const uint2*>(q_table) + lane;
        const uint8_t* codes = blob + 64 * c + 8 * g + 4 * hf;
#pragma unroll 2
        for (int i = 0; i < 8; ++i, codes += 16 * 64) {
          const uint4 e = table[4 * i + c];
          const uint2 q = q_ready[32 * i];
          uint32_t ra[8], rb[8];
          Affine aff;
          aff.template init<1>(e.x, e.y);
          uint32_t w0 = lds_u32(codes), w1 = lds_u32(codes + 4 * 64);
          restore_codes4<MD, DT, FP32>(cc, mask4, prmt(w0, w1, 0x5410u), aff, ra);
          restore_codes4<MD, DT, FP32>(cc, mask4, prmt(w0, w1, 0x7632u), aff, ra + 4);
          aff.template init<1>(e.z, e.w);
          w0 = lds_u32(codes + 8 * 64); w1 = lds_u32(codes + 12 * 64);
          restore_codes4<MD, DT, FP32>(cc, mask4, prmt(w0, w1, 0x5410u), aff, rb);
          restore_codes4<MD, DT, FP32>(cc, mask4, prmt(w0, w1, 0x7632u), aff, rb + 4);
          products(ra, rb, q.x, q.y);
        }
      } else if (UNIFORM) {
        const uint2* const q_ready = reinterpret_cast<const uint2*>(q_table) + lane;
        const uint8_t* codes = blob + 32 * c + 4 * g + 2 * hf;
#pragma unroll 2
        for (int i = 0; i < 8; ++i, codes += 16 * 32) {
          const uint4 e = table[4 * i + c];
          const uint2 q = q_ready[32 * i];
          uint32_t ra[8], rb[8];
          Affine aff;
          aff.template init<3>(e.x, e.y);
          restore_codes2<MD, DT, FP32>(cc, prmt(lds_u16(codes), lds_u16(codes + 4 * 32), 0x5410u), aff, ra);
          aff.template init<3>(e.z, e.w);
          restore_codes2<MD, DT, FP32>(cc, prmt(lds_u16(codes + 8 * 32), lds_u16(codes + 12 * 32), 0x5410u), aff, rb);
          products(ra, rb, q.x, q.y);
        }
      } else {
        const uint8_t* codes = blob + 4 * g + 2 * hf;
        const uint8_t* high = blob + d.key_off_high + 4 * g + 2 * hf;
#pragma unroll 1
        for (int i = 0; i < prom_steps; ++i) {
          const uint4 ea = table[8 * i + c], eb = table[8 * i + 4 + c];
          auto plane = [&](int p) { return p < K ? lds_u16(high + 32 * p) : 0u; };
          uint32_t ra[8], rb[8];
          Affine aff;
          aff.template init<2>(ea.x, ea.y);
          restore_codes22<MD, DT, FP32>(cc, prmt(lds_u16(codes + ea.z), lds_u16(codes + ea.w), 0x5410u),
                                        prmt(plane(16 * i + c), plane(16 * i + c + 4), 0x5410u), aff, ra);
          aff.template init<2>(eb.x, eb.y);
          restore_codes22<MD, DT, FP32>(cc, prmt(lds_u16(codes + eb.z), lds_u16(codes + eb.w), 0x5410u),
                                        prmt(plane(16 * i + c + 8), plane(16 * i + c + 12), 0x5410u), aff, rb);
          multiply(ea, eb, ra, rb);
        }
#pragma unroll 2
        for (int i = prom_steps; i < 8; ++i) {
          const uint4 ea = table[8 * i + c], eb = table[8 * i + 4 + c];
          uint32_t ra[8], rb[8];
          Affine aff;
          aff.template init<3>(ea.x, ea.y);
          restore_codes2<MD, DT, FP32>(cc, prmt(lds_u16(codes + ea.z), lds_u16(codes + ea.w), 0x5410u), aff, ra);
          aff.template init<3>(eb.x, eb.y);
          restore_codes2<MD, DT, FP32>(cc, prmt(lds_u16(codes + eb.z), lds_u16(codes + eb.w), 0x5410u), aff, rb);
          multiply(ea, eb, ra, rb);
        }
      }
      if (w.stages == 1) {
        pair_barrier(pair);   // both warps have read the keys: their buffer takes the next page's
        if (hf == 0 && pg + ahead < p_end) issue_keys(pg + ahead, 0);
      }

      // ---- online softmax of this lane's columns over the warp's 64 tokens
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) s_acc[mt][i] *= scale2;
      const int mask_below = row_first - (d.sink_tokens + 128 * pg);
      if (mask_below > 0) {   // the page that holds the row's first live token: the tokens before it drop out
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (16 * g + 8 * hf + 2 * mt + (i >> 1) < mask_below) s_acc[mt][i] = -INFINITY;
      }
      uint32_t p_hi[8], p_lo[8];   // B operands of P.V; with R = 4 p_hi holds both parts
      float alpha[2], m_ref[2];
      bool moved = false;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float mx = -INFINITY;
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) mx = fmaxf(mx, fmaxf(s_acc[mt][e], s_acc[mt][2 + e]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float m_new = fmaxf(m_run[e], mx);
        m_ref[e] = m_new == -INFINITY ? 0.0f : m_new;   // nothing live yet: every weight below comes out zero
        alpha[e] = fast_exp2(m_run[e] - m_ref[e]);
        m_run[e] = m_new;
        l_run[e] *= alpha[e];
        moved = moved || alpha[e] != 1.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float p0 = fast_exp2(s_acc[u >> 1][2 * (u & 1)] - m_ref[0]), p1 = fast_exp2(s_acc[u >> 1][2 * (u & 1) + 1] - m_ref[1]);
        l_run[0] += p0;
        l_run[1] += p1;
        const uint32_t hi = pack16<DT>(p0, p1);
        float h0, h1;
        unpack16<DT>(hi, h0, h1);
        const uint32_t lo = pack16<DT>(p0 - h0, p1 - h1);
        p_hi[u] = transpose8x8(R == 4 && c >= 2 ? lo : hi);
        if (R > 4) p_lo[u] = transpose8x8(lo);
      }
      if (__any_sync(0xffffffffu, moved)) {   // the running maximum rarely moves after the first pages
#pragma unroll
        for (int mt = 0; mt < 8; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) o_acc[mt][i] *= alpha[i & 1];
      }

      // ---- O[channel][column] += V^T P, sixteen tokens per step: contraction index 2c, 2c + 1 = tokens T, T + 16 with
      // T = 32c + 8*HF + 2s, and 2c + 8, 2c + 9 = tokens T + 1, T + 17
      ok = mbar_wait(&bs.v_bar[pair][stage], parity) && ok;
      {
        const uint8_t* vs = v_mem + stage * w.v_stage;
        const uint8_t* vm = vs + w.v_meta + c * w.v_meta_piece + 8 * hf * meta_row + 2 * vgroup;
        const uint8_t* vc = vs + c * w.v_piece + 8 * hf * vrb + g * (vrb >> 3);
        auto params = [&](int tok) {
          const uint8_t* m0 = vm + tok * meta_row;
          const uint8_t* m1 = m0 + 16 * meta_row;
          const int zero = 2 * d.value_groups;
          return make_uint2(prmt(lds_u16(m0), lds_u16(m1), 0x5410u), prmt(lds_u16(m0 + zero), lds_u16(m1 + zero), 0x5410u));
        };
        auto accumulate = [&](int s, int mt0, const uint32_t (&ra)[8], const uint32_t (&rb)[8]) {
#pragma unroll
          for (int mt = 0; mt < 4; ++mt) {
            HO::mma(o_acc[mt0 + mt], ra[2 * mt], ra[2 * mt + 1], rb[2 * mt], rb[2 * mt + 1], p_hi[2 * s], p_hi[2 * s + 1]);
            if (R > 4) HO::mma(o_acc[mt0 + mt], ra[2 * mt], ra[2 * mt + 1], rb[2 * mt], rb[2 * mt + 1], p_lo[2 * s], p_lo[2 * s + 1]);
          }
        };
        if (d.value_bits == 4) {
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const uint2 wa0 = *reinterpret_cast<const uint2*>(vc + 2 * s * 64), wa1 = *reinterpret_cast<const uint2*>(vc + (2 * s + 16) * 64);
            const uint2 wb0 = *reinterpret_cast<const uint2*>(vc + (2 * s + 1) * 64), wb1 = *reinterpret_cast<const uint2*>(vc + (2 * s + 17) * 64);
            Affine fa, fb;
            const uint2 pa = params(2 * s), pb = params(2 * s + 1);
            fa.template init<1>(pa.x, pa.y);
            fb.template init<1>(pb.x, pb.y);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const uint32_t a0 = half ? wa0.y : wa0.x, a1 = half ? wa1.y : wa1.x, b0 = half ? wb0.y : wb0.x, b1 = half ? wb1.y : wb1.x;
              uint32_t ra[8], rb[8];
              restore_codes4<MD, DT, FP32>(cc, mask4, prmt(a0, a1, 0x5410u), fa, ra);
              restore_codes4<MD, DT, FP32>(cc, mask4, prmt(a0, a1, 0x7632u), fa, ra + 4);
              restore_codes4<MD, DT, FP32>(cc, mask4, prmt(b0, b1, 0x5410u), fb, rb);
              restore_codes4<MD, DT, FP32>(cc, mask4, prmt(b0, b1, 0x7632u), fb, rb + 4);
              accumulate(s, 4 * half, ra, rb);
            }
          }
        } else if (d.value_bits == 8) {
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            Affine fa, fb;
            const uint2 pa = params(2 * s), pb = params(2 * s + 1);
            fa.template init<0>(pa.x, pa.y);
            fb.template init<0>(pb.x, pb.y);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              auto words = [&](int tok) { return *reinterpret_cast<const uint2*>(vc + tok * 128 + 8 * half); };
              const uint2 a0 = words(2 * s), a1 = words(2 * s + 16), b0 = words(2 * s + 1), b1 = words(2 * s + 17);
              uint32_t ra[8], rb[8];
              restore_codes8<MD, DT, FP32>(a0.x, a1.x, fa, ra);
              restore_codes8<MD, DT, FP32>(a0.y, a1.y, fa, ra + 4);
              restore_codes8<MD, DT, FP32>(b0.x, b1.x, fb, rb);
              restore_codes8<MD, DT, FP32>(b0.y, b1.y, fb, rb + 4);
              accumulate(s, 4 * half, ra, rb);
            }
          }
        } else {
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const uint32_t wa0 = lds_u32(vc + 2 * s * 32), wa1 = lds_u32(vc + (2 * s + 16) * 32);
            const uint32_t wb0 = lds_u32(vc + (2 * s + 1) * 32), wb1 = lds_u32(vc + (2 * s + 17) * 32);
            Affine fa, fb;
            const uint2 pa = params(2 * s), pb = params(2 * s + 1);
            fa.template init<3>(pa.x, pa.y);
            fb.template init<3>(pb.x, pb.y);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              uint32_t ra[8], rb[8];
              restore_codes2<MD, DT, FP32>(cc, prmt(wa0, wa1, half ? 0x7632u : 0x5410u), fa, ra);
              restore_codes2<MD, DT, FP32>(cc, prmt(wb0, wb1, half ? 0x7632u : 0x5410u), fb, rb);
              accumulate(s, 4 * half, ra, rb);
            }
          }
        }
      }
      pair_barrier(pair);   // both warps have read the page
      if (hf == 0 && pg + ahead < p_end) {
        if (w.stages == 2) issue_keys(pg + ahead, stage);
        issue_values(pg + ahead, stage);
      }
    }

    // ---- hand the warp state to the block merge
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 4);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 8);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 16);
    }
    __syncthreads();   // every warp is done with its stages: the staging memory becomes the merge buffer
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = 2 * c + e;
      if (g == 0 && row < R) { bs.merge_m[warp][row] = merge_maximum(m_run[e], l_run[e]); bs.merge_l[warp][row] = l_run[e]; }
#pragma unroll
      for (int mt = 0; mt < 8; ++mt)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float v = o_acc[mt][2 * i + e];
          if (R == 4) v += __shfl_xor_sync(0xffffffffu, v, 2);   // lanes c and c ^ 2: the high and the low parts
          if (row < R) warp_out[(warp * R + row) * 128 + 16 * g + 2 * mt + i] = v;
        }
    }
    __syncthreads();
    rows_merge<R>(a, bs, warp_out, first_row, rows, 1 + sb - dartkv_block_of_unit((int64_t)work_row * a.quads, a.stream_blocks, a.units));
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();   // the merge buffer is staging memory again, the query table may be overwritten
  }
  if (!ok && lane == 0) atomicExch(a.status, 1);
}

RowsGeom rows_geometry(const dartkv_cache_desc* d, int stages) {
  RowsGeom w{};
  const bool mixed = d->key_mode == DARTKV_MIXED_PAGE;
  w.key_kind = mixed ? 22 : d->key_bits;
  w.key_row = mixed ? 32 : 16 * d->key_bits;
  w.v_piece = 32 * d->value_row_bytes + 32;
  w.v_meta = 4 * w.v_piece;
  w.v_meta_piece = 128 * d->value_groups + 16;
  w.k_stage = (d->key_page_bytes + 127) / 128 * 128;
  w.v_stage = (w.v_meta + 4 * w.v_meta_piece + 127) / 128 * 128;
  w.stages = stages;
  w.pair_bytes = stages * (w.k_stage + w.v_stage) + 2 * kTableBytes;
  return w;
}

template <int R>
size_t rows_smem_bytes(const RowsGeom& w) {
  const size_t streaming = (size_t)kPairs * w.pair_bytes;
  const size_t merge = (size_t)kWarps * R * 128 * sizeof(float);
  const size_t dense = (size_t)(kWarps * 4 * 128 + kWarps * 64) * sizeof(float);   // warp states + probability tables
  const size_t body = streaming > merge ? streaming : merge;
  return (sizeof(RowsSmem<R>) + 127) / 128 * 128 + 128 * w.key_row + (body > dense ? body : dense);
}
int rows_for(int rep) { return rep <= 4 ? 4 : 8; }
size_t rows_smem(const RowsGeom& w, int rows) { return rows == 8 ? rows_smem_bytes<8>(w) : rows_smem_bytes<4>(w); }
bool two_blocks(size_t smem) { return 2 * (smem + 1024) <= 228 * 1024; }
// two stages where two blocks still fit an SM
RowsGeom rows_geometry_for(const dartkv_cache_desc* d, int rows) {
  const RowsGeom w = rows_geometry(d, 2);
  return two_blocks(rows_smem(w, rows)) ? w : rows_geometry(d, 1);
}

using RowsKernel = void (*)(dartkv_cache_desc, FastArgs, RowsGeom);
template <int DT, int MD, bool UNIFORM>
RowsKernel rows_variant_of(bool fp32, int rows) {
  if (rows == 8) return decode_rows_kernel<DT, MD, false, 8, UNIFORM>;
  return fp32 ? decode_rows_kernel<DT, MD, true, 4, UNIFORM> : decode_rows_kernel<DT, MD, false, 4, UNIFORM>;
}
template <bool UNIFORM>
RowsKernel rows_variant(int dtype, int md, bool fp32, int rows) {
  if (dtype == DARTKV_BF16)
    return md == DARTKV_BF16 ? rows_variant_of<DARTKV_BF16, DARTKV_BF16, UNIFORM>(fp32, rows) : rows_variant_of<DARTKV_BF16, DARTKV_F16, UNIFORM>(fp32, rows);
  return md == DARTKV_BF16 ? rows_variant_of<DARTKV_F16, DARTKV_BF16, UNIFORM>(fp32, rows) : rows_variant_of<DARTKV_F16, DARTKV_F16, UNIFORM>(fp32, rows);
}

}  // namespace

// `rep` query rows per KV head run as this many groups of equal size (the last one may be smaller)
int dartkv_decode_rows_groups(int rep) { return (rep + 7) / 8; }

// up to 4 query rows per KV head, or up to 64 with the per-op flavour; pages that leave room for two blocks per SM
int dartkv_decode_rows_supported(const dartkv_cache_desc* d, int q_dtype, int rep, int flavour) {
  if (d->head_dim != 128 || d->page_size != 128 || d->key_group != 128 || !d->regular_pages) return 0;
  if (d->dtype != DARTKV_F16 && d->dtype != DARTKV_BF16) return 0;
  if ((d->md_dtype != DARTKV_F16 && d->md_dtype != DARTKV_BF16) || q_dtype != d->dtype) return 0;
  if (flavour == DARTKV_DEQUANT_FUSED || rep < 1 || rep > (flavour == DARTKV_DEQUANT_PER_OP ? 64 : 4)) return 0;
  if (d->value_group < 16 || d->value_group > 128 || (d->value_group & (d->value_group - 1))) return 0;
  if (d->value_bits != 2 && d->value_bits != 4 && d->value_bits != 8) return 0;
  if (d->key_mode == DARTKV_QUANTIZED_PAGE && d->key_bits != 2 && d->key_bits != 4) return 0;
  if (d->key_mode == DARTKV_MIXED_PAGE && (d->promoted < 1 || d->promoted > 128)) return 0;
  if (d->key_page_bytes % 16 || d->max_value_tokens % 8) return 0;
  if ((uintptr_t)d->k_pages % 16 || (uintptr_t)d->v_codes % 16 || (uintptr_t)d->v_meta % 16) return 0;
  const int rows = rows_for(rep);
  return two_blocks(rows_smem(rows_geometry_for(d, rows), rows)) ? 1 : 0;
}

int dartkv_decode_rows_launch(const dartkv_cache_desc* d, const void* query, int query_heads, float scale, int flavour, int quads,
                              int stream_blocks, long long units, int total_splits, float* part_m, float* part_l, float* part_acc,
                              int* status, const int32_t* row_start, cudaStream_t stream) {
  FastArgs a{query, query_heads, scale, flavour, quads, stream_blocks, units, total_splits, part_m, part_l, part_acc, status, row_start};
  const int rep = query_heads / d->kv_heads, rows = rows_for(rep);
  RowsGeom w = rows_geometry_for(d, rows);
  w.groups = dartkv_decode_rows_groups(rep);
  w.group_rows = (rep + w.groups - 1) / w.groups;
  const bool uniform = w.key_kind != 22, fp32 = flavour == DARTKV_DEQUANT_FP32;
  const RowsKernel kernel = (uniform ? rows_variant<true> : rows_variant<false>)(d->dtype, d->md_dtype, fp32, rows);
  static SharedMemoryOptIn<4 * 3 * 2> opt_in;
  DARTKV_CUDA_OK(opt_in((2 * (d->dtype == DARTKV_BF16) + (d->md_dtype == DARTKV_BF16)) * 6 + (rows == 8 ? 2 : fp32 ? 1 : 0) * 2 + uniform, kernel,
                        113 * 1024));
  dim3 grid(stream_blocks + d->batch * d->kv_heads * ((rep + 3) / 4));
  DARTKV_CUDA_OK(launch_following(kernel, grid, kThreads, rows_smem(w, rows), stream, *d, a, w));
  DARTKV_LAUNCH_OK("decode_rows_kernel");
  return DARTKV_OK;
}
