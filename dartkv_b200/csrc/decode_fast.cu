// Tensor-core fused decode attention for the common page geometry: head_dim 128, 128-token pages,
// one 128-token key group, 2-bit values with 64/128-channel groups, 2-bit keys (uniform or with up to
// 32 promoted 2+2-bit channels), 16-bit data whose metadata has the same dtype, up to 4 query heads
// per KV head.  Everything else takes the generic kernel in decode_attention.cu.
//
// Work split: one unit = four or eight consecutive pages of a (batch, kv head) row.  The units of all rows are dealt out
// evenly to the stream blocks (aligned to rows, or one block per resident slot whose share may run from one
// row into the next; the host chooses).  A warp of a block's eight takes every eighth page of the block's run by itself
// (decode_page.cuh), from buffers of its own that bulk async copies fill, completion on an mbarrier: the keys' buffer is
// refilled as soon as the logits are done, the values' after P.V, with the first page of the next row after a row's last one.
// Where blocks have one unit and an SM each, two warps share a page, half of its tokens each.  The block merges the eight
// states when it leaves a row, in the warps' scratch and not in their buffers, so that the next row's pages arrive meanwhile
// (batch 128, 32,768 tokens: 1,087 us with the states in the buffers, 1,061 to 1,068 so; 32 x 8,192: 89.7 and 87.7), and
// writes one partial per row it touched.  One more short block per row, launched after the stream blocks, handles the
// dense tokens: the sink prefix and everything after the last page that is packed on both the key and the value side.
//
// What bounds it: two pipes that take a warp instruction every other cycle, each busy half of the time (logic: one LOP3 per
// operand register, address arithmetic, shifts; packed 16-bit arithmetic: two per register), and four warps per scheduler to
// keep them so.  Batch 128, 32,768 tokens: 1,144 us with two warps per page that split the logits by channels, the rest by
// tokens, and met twice per page; 1,089 us with a warp per page, which fills one table instead of two and exchanges nothing
// (B200; the instructions of a launch went from 3,340 to 3,287 per page); 1,026 us now (states merged beside the next row's
// pages, shorter dense blocks, half-register operands).
// Algorithmic HBM bytes per page and (batch, kv head): 10880.

#include <atomic>

#include "decode_page.cuh"

namespace {

struct WarpSmem {
  uint8_t keys[kPageBytesK];
  uint8_t values[kStageBytes - kPageBytesK];   // codes, then scales and zero points
  PageScratch scratch;
};

static_assert(sizeof(PageScratch) >= 512 * sizeof(float), "the scratch of a warp takes its state at the end of a row");

struct BlockSmem {
  uint32_t q32[128][8];      // [channel][2*head + j']: query pre-shifted into the low (j'=0) or high (j'=1) half
  float merge_m[kWarps][4];
  float merge_l[kWarps][4];
  int slot_map[128];
  uint64_t k_bar[kWarps], v_bar[kWarps];
};

// GN: value groups per token (1 or 2).  KP: promoted channels per page when that is a multiple of eight known to
// the host (0, 8, 16, 24, 32), else -1 (read from the descriptor): with the count fixed the logits loops have
// constant trip counts and no per-position "is this slot promoted" test.  FEW: one unit per block (see dartkv_few_pages).
template <int DT, int OUT, int GN, int KP, bool FEW>
__global__ void __launch_bounds__(kThreads, 2) decode_fast_kernel(dartkv_cache_desc d, FastArgs a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous();
  BlockSmem& bs = *reinterpret_cast<BlockSmem*>(smem_raw + sizeof(WarpSmem) * kWarps);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rep = a.query_heads / d.kv_heads;

  if ((int)blockIdx.x >= a.stream_blocks) {
    // dense tokens of one (batch, kv head): partial slot 0.  These short blocks come last in launch order and fill
    // the slots the stream blocks leave.
    const int bh = blockIdx.x - a.stream_blocks;
    float* const warp_out = reinterpret_cast<float*>(smem_raw);   // [warp][head][128]
    dense_block<OUT, DT>(d, a, bs, warp_out, bh);
    __syncthreads();
    block_merge(a, bs, warp_out, bh / d.kv_heads, bh % d.kv_heads, rep, 0);
    return;
  }

  // ---- stream block: an even share of all (row, unit) work, possibly spanning several rows
  const int sb = blockIdx.x;
  int unit = (int)((int64_t)sb * a.units / a.stream_blocks);   // the host keeps the unit count below 2^31
  const int unit_end = (int)((int64_t)(sb + 1) * a.units / a.stream_blocks);
  WarpSmem& ws = reinterpret_cast<WarpSmem*>(smem_raw)[warp];
  int bh = unit / a.quads, quad = unit - bh * a.quads;
  // the row's first live token, its query and the state are requested together
  const int first_live = first_live_token(d, a, bh);
  const QueryPair first_query = load_query(a.q, (int64_t)(bh / d.kv_heads) * a.query_heads + bh % d.kv_heads * rep, rep, tid);
  const int k_end = d.state[2], v_end = d.state[3], sink_filled = d.state[4];
  const int fast_end = fast_range_end(d.sink_tokens, d.page_size, k_end, v_end, sink_filled);
  const int total_pages = fast_end > d.sink_tokens ? (fast_end - d.sink_tokens) / 128 : 0;
  constexpr int kMetaBytes = 128 * 2 * GN * 2;
  // one lane starts the copies of a page; the barriers complete when all bytes landed
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
  PageWork<DT, OUT, GN, KP> work(d, bs.q32, a.scale, lane);
  bool ok = true;
  uint32_t parity = 0;   // of the pages this warp has consumed so far

  RowPiece now = row_piece(d, a, first_live, quad, min(a.quads - quad, unit_end - unit), total_pages);
  // this warp's first page is requested before anything else, so its latency overlaps the query load below
  if (lane == 0 && now.begin + warp < now.end) { issue_keys(bh, now.begin + warp); issue_values(bh, now.begin + warp); }
  store_query(bs.q32, first_query, tid);
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
      const WarpSmem& page = reinterpret_cast<const WarpSmem*>(smem_raw)[shared];
      if (now.begin + shared < now.end) {
        ok = mbar_wait(&bs.k_bar[shared], 0) && ok;
        work.fill_table(page.keys, ws.scratch);
        __syncwarp();
        float s_acc[2][4];
        work.template logits<2>(page.keys, ws.scratch, hf, s_acc);
        __syncwarp();
        work.template softmax<2>(s_acc, hf, now.first_live - (d.sink_tokens + 128 * (now.begin + shared)), ws.scratch);
        __syncwarp();
        ok = mbar_wait(&bs.v_bar[shared], 0) && ok;
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
        work.template softmax<4>(s_acc, 0, now.first_live - (d.sink_tokens + 128 * pg), ws.scratch);
        __syncwarp();
        ok = mbar_wait(&bs.v_bar[warp], parity) && ok;
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
    block_merge<false, sizeof(WarpSmem) / sizeof(float)>(a, bs, reinterpret_cast<const float*>(&reinterpret_cast<WarpSmem*>(smem_raw)->scratch),
                                                     bh / d.kv_heads, bh % d.kv_heads, rep,
                                                     1 + sb - dartkv_block_of_unit((int64_t)bh * a.quads, a.stream_blocks, a.units));
    if (unit >= unit_end) break;
    ++bh;
    now = row_piece(d, a, first_live_token(d, a, bh), 0, min(a.quads, unit_end - unit), total_pages);
    store_query(bs.q32, load_query(a.q, (int64_t)(bh / d.kv_heads) * a.query_heads + bh % d.kv_heads * rep, rep, tid), tid);
    __syncthreads();
  }
  if (!ok && lane == 0) atomicExch(a.status, 1);
}

constexpr size_t kSmemBytes = sizeof(WarpSmem) * kWarps + sizeof(BlockSmem);

}  // namespace

int dartkv_decode_fast_supported(const dartkv_cache_desc* d, int q_dtype, int query_heads) {
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

// every (metadata dtype, cache dtype, value groups, promoted count) variant of the kernel; a cache whose metadata
// dtype differs from its dtype gets the promoted counts 0 and 32 specialized, the others read the count at run time
using FastKernel = void (*)(dartkv_cache_desc, FastArgs);
template <bool FEW, int DT, int GN>
static FastKernel fast_variant_kp(int kp) {
  switch (kp) {
    case 0: return decode_fast_kernel<DT, DT, GN, 0, FEW>;
    case 8: return decode_fast_kernel<DT, DT, GN, 8, FEW>;
    case 16: return decode_fast_kernel<DT, DT, GN, 16, FEW>;
    case 24: return decode_fast_kernel<DT, DT, GN, 24, FEW>;
    case 32: return decode_fast_kernel<DT, DT, GN, 32, FEW>;
    default: return decode_fast_kernel<DT, DT, GN, -1, FEW>;
  }
}
template <bool FEW, int DT, int OUT, int GN>
static FastKernel mixed_variant_kp(int kp) {
  switch (kp) {
    case 0: return decode_fast_kernel<DT, OUT, GN, 0, FEW>;
    case 32: return decode_fast_kernel<DT, OUT, GN, 32, FEW>;
    default: return decode_fast_kernel<DT, OUT, GN, -1, FEW>;
  }
}
template <bool FEW>
static FastKernel fast_variant_of(int md, int dtype, int value_groups, int kp) {
  if (md == dtype) {
    if (dtype == DARTKV_BF16) return value_groups == 2 ? fast_variant_kp<FEW, DARTKV_BF16, 2>(kp) : fast_variant_kp<FEW, DARTKV_BF16, 1>(kp);
    return value_groups == 2 ? fast_variant_kp<FEW, DARTKV_F16, 2>(kp) : fast_variant_kp<FEW, DARTKV_F16, 1>(kp);
  }
  if (md == DARTKV_F16)
    return value_groups == 2 ? mixed_variant_kp<FEW, DARTKV_F16, DARTKV_BF16, 2>(kp) : mixed_variant_kp<FEW, DARTKV_F16, DARTKV_BF16, 1>(kp);
  return value_groups == 2 ? mixed_variant_kp<FEW, DARTKV_BF16, DARTKV_F16, 2>(kp) : mixed_variant_kp<FEW, DARTKV_BF16, DARTKV_F16, 1>(kp);
}
static FastKernel fast_variant(bool few, int md, int dtype, int value_groups, int kp) {
  return few ? fast_variant_of<true>(md, dtype, value_groups, kp) : fast_variant_of<false>(md, dtype, value_groups, kp);
}

int dartkv_decode_fast_launch(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads, float scale,
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
      for (int md : {DARTKV_BF16, DARTKV_F16})
        for (int dt : {DARTKV_BF16, DARTKV_F16})
          for (int gn : {1, 2})
            for (int kp : {-1, 0, 8, 16, 24, 32})
              for (bool each : {false, true})   // the next call, of another length, may be under graph capture
                DARTKV_CUDA_OK(cudaFuncSetAttribute(fast_variant(each, md, dt, gn, kp), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)kSmemBytes));
      if (device >= 0 && device < 64) ready[device].store(true, std::memory_order_release);
    }
  }
  const int promoted = d->key_mode == DARTKV_MIXED_PAGE ? d->promoted : 0;
  const int kp = (promoted % 8 == 0 && promoted <= 32) ? promoted : -1;
  DARTKV_CUDA_OK(launch_following(fast_variant(few, d->md_dtype, d->dtype, d->value_groups, kp), grid, kThreads, kSmemBytes, stream, *d,
                                  a));
  DARTKV_LAUNCH_OK("decode_fast_kernel");
  return DARTKV_OK;
}
