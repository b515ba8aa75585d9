// Fused single-token decode attention over the device-resident paged cache.
//
// Split-K over the token range: every (batch, KV head, split) block keeps an fp32 online-softmax
// state (m, l, acc) for the query heads of its KV head (GQA group) and writes one partial; a merge
// kernel combines the partials, normalizes and casts.  Numerics follow the reference's
// page-streaming attention (src/dart/attention.py:60-87): dequantize to the cache dtype, fp32
// logits q.k * scale, fp32 online softmax, acc / max(l, 1e-20), cast to the query dtype.
//
// This file holds the generic kernel (any page geometry, bit width, dtype; CUDA-core fp32 math)
// and the merge; the tensor-core kernel for the headline geometry is in decode_fast.cu.

#include <atomic>
#include <cstdlib>
#include <cstring>

#include <cooperative_groups.h>

#include "common.cuh"
#include "mma_utils.cuh"

#define GEN_THREADS 256
#define GEN_WARPS (GEN_THREADS / 32)
#define GEN_TILE 32
#define GEN_MAX_REP 16
#define GEN_MAX_D 256

__device__ __forceinline__ int gen_find_page(const dartkv_cache_desc& d, int pages, int t) {
  int lo = 0, hi = pages - 1;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (d.page_start[mid] + d.page_tokens[mid] > t) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// Tokens [sink_tokens, fast_range_end) are whole pages packed on both the key and the value side.
__host__ __device__ __forceinline__ int dartkv_fast_range_end(int sink_tokens, int page_size, int k_end, int v_end,
                                                              int sink_filled) {
  int packed = min(k_end, v_end);
  if (packed <= sink_tokens) return sink_filled;
  return sink_tokens + (packed - sink_tokens) / page_size * page_size;
}

struct GenericArgs {
  const void* q;
  int q_dt, query_heads, flavour;
  float scale;
  int tok_begin, tok_end;   // tok_end < 0: up to the number of tokens seen
  int chunk, split_base, total_splits;
  float* part_m;
  float* part_l;
  float* part_acc;
  const int32_t* row_start;   // optional [batch] first live token of every batch row
  int cluster;                // decode_tiles_kernel: blocks of a (batch, kv head)
  void* out;                  // and where their results go; null: to the partials, one per row
};

// One block per (batch, kv head) and run of tokens, in tiles of 32 tokens.  Keys: lane = token, the channels are dealt
// out to the warps, so the codes of a channel are one short coalesced read, its scale and the query are broadcasts and
// a dot product needs no shuffles; the warps' partial logits meet in shared memory.  Values: thread = channel, the
// tile's tokens split over the remaining threads.  Nothing dequantized is staged.  Latency is what counts here (small
// fp32 caches): loads of several channels / tokens are in flight together, and a call is cut into tiles until every SM
// has a block.  [1,8,256,128] fp32, 2-bit: 98 us per call with one serial dot product per thread and staged tiles, 31 us so
// (B200; decode_tiles_kernel, which takes such small calls of uniform pages, 16).
template <int REP>
__global__ void __launch_bounds__(GEN_THREADS) decode_generic_kernel(const __grid_constant__ dartkv_cache_desc d,
                                                                     const __grid_constant__ GenericArgs a) {
  extern __shared__ float smem[];
  wait_previous();
  const int D = d.head_dim;
  const int rep = a.query_heads / d.kv_heads;            // at most REP
  float* s_q = smem;                                     // [D][REP]: a channel's heads together
  float* s_part = s_q + D * REP;                         // [warp][REP][32] partial logits, then [split][REP][D] sums
  float* s_p = s_part + GEN_WARPS * REP * GEN_TILE;      // [32][REP] probabilities of the tile
  float* s_alpha = s_p + GEN_TILE * REP;                 // [REP]
  float* s_m = s_alpha + REP;
  float* s_l = s_m + REP;
  int* s_slot = reinterpret_cast<int*>(s_l + REP);       // [D]

  const int bh = blockIdx.x, split = blockIdx.y;
  const int b = bh / d.kv_heads, h = bh % d.kv_heads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int seen = d.state[0], pages = d.state[1], k_end = d.state[2], v_end = d.state[3], sink_filled = d.state[4];
  const int end = a.tok_end < 0 ? seen : min(a.tok_end, seen);
  // tok_begin < 0: start where the tensor-core kernel stops (last full page packed on both sides)
  int begin = a.tok_begin;
  if (begin < 0) begin = dartkv_fast_range_end(d.sink_tokens, d.page_size, k_end, v_end, sink_filled);
  const int first = begin + split * a.chunk;
  const int hi = (int)min((int64_t)first + a.chunk, (int64_t)end);
  // left padding: the tokens before the row's first live one get no weight (a split wholly before it stays empty)
  const int lo = a.row_start ? max(first, a.row_start[b]) : first;

  for (int i = tid; i < D * REP; i += GEN_THREADS) {
    const int r = i % REP, c = i / REP;
    s_q[i] = r < rep ? load_f(a.q, a.q_dt, ((int64_t)b * a.query_heads + h * rep + r) * D + c) : 0.0f;
  }
  if (tid < REP) { s_m[tid] = -INFINITY; s_l[tid] = 0.0f; }
  // values: this thread's channel and share of the tile's tokens (D is at most the block)
  const int vsplits = GEN_THREADS / D, vsplit = tid / D, vc = tid % D;
  float acc[REP];
#pragma unroll
  for (int r = 0; r < REP; ++r) acc[r] = 0.0f;
  __syncthreads();

  // A packed value segment [vs, ve) (page_size tokens from sink_tokens on, the last one ending at the packed end)
  // that a key-segment boundary cuts is materialized by the reference with its per-op dequantization: the key
  // boundaries are the page edges and the end of the packed keys.
  auto value_flavour = [&](int tok) -> int {
    if (a.flavour == DARTKV_DEQUANT_PER_OP || d.regular_pages) return a.flavour;   // regular pages share the value edges
    const int vs = d.sink_tokens + (tok - d.sink_tokens) / d.page_size * d.page_size;
    const int ve = min(v_end, vs + d.page_size);
    if (vs >= k_end) return a.flavour;
    const int pg = gen_find_page(d, pages, vs);
    return d.page_start[pg] + d.page_tokens[pg] < ve ? DARTKV_DEQUANT_PER_OP : a.flavour;
  };
  int t = lo;
  while (t < hi) {
    // ---- locate the key segment that holds token t
    int seg_end, kind, page_first = 0, page_n = 1;
    int key_flavour = a.flavour;
    const uint8_t* page = nullptr;
    if (t < sink_filled) {
      kind = 0; seg_end = min(hi, sink_filled);
    } else if (t < k_end) {
      kind = 1;
      const int pg = d.regular_pages ? (t - d.sink_tokens) / d.page_size : gen_find_page(d, pages, t);
      page_first = d.page_start[pg];
      page_n = d.page_tokens[pg];
      seg_end = min(hi, page_first + page_n);
      page = d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes;
      // A key page that a value-segment boundary cuts is materialized by the reference with its per-op
      // dequantization whatever the device (src/dart/cache.py:557-560); only whole pages reach its fp32 kernels.
      // Value boundaries: sink_tokens + i * page_size below the packed end of the values, and that end itself.
      if (a.flavour != DARTKV_DEQUANT_PER_OP && page_first < v_end) {
        const int next_value_edge = d.sink_tokens + ((page_first - d.sink_tokens) / d.page_size + 1) * d.page_size;
        if (min(next_value_edge, v_end) < page_first + page_n) key_flavour = DARTKV_DEQUANT_PER_OP;
      }
      if (d.key_mode == DARTKV_MIXED_PAGE) {
        __syncthreads();
        for (int c = tid; c < D; c += GEN_THREADS) s_slot[c] = -1;
        __syncthreads();
        const int32_t* idx = reinterpret_cast<const int32_t*>(page + d.key_off_index);
        for (int k = tid; k < d.promoted; k += GEN_THREADS) {
          const int c = idx[k];
          if (c >= 0 && c < D) s_slot[c] = k;
        }
        __syncthreads();
      }
    } else {
      kind = 2; seg_end = hi;
    }
    const bool mixed = d.key_mode == DARTKV_MIXED_PAGE;
    const int Gk = d.key_group, G = ceil_div(page_n, Gk), bits = mixed ? 2 : d.key_bits, vpb = 8 / bits;
    const int plane = ceil_div(Gk, 4);                                    // mixed: bytes of one group's plane
    const int row_bytes = mixed ? G * plane : ceil_div(G * Gk, vpb);
    for (int tile0 = t; tile0 < seg_end; tile0 += GEN_TILE) {
      const int nt = min(GEN_TILE, seg_end - tile0);
      // ---- partial logits of this warp's channels (lanes past the tile repeat its last token)
      float dot[REP];
#pragma unroll
      for (int r = 0; r < REP; ++r) dot[r] = 0.0f;
      const int tok = tile0 + min(lane, nt - 1);
      auto add = [&](int c, float k) {
#pragma unroll
        for (int r = 0; r < REP; ++r) dot[r] = fmaf(s_q[c * REP + r], k, dot[r]);
      };
      if (kind == 1) {
        const int j = tok - page_first, g = j / Gk;
        const int at = mixed ? g * plane + (j - g * Gk) / 4 : j / vpb;
        const int shift = mixed ? ((j - g * Gk) % 4) * 2 : (j % vpb) * bits;
        const uint32_t mask = (1u << bits) - 1u;
        const uint8_t *scale = page + d.key_off_scale, *zero = page + d.key_off_zero;
#pragma unroll 8
        for (int c = warp; c < D; c += GEN_WARPS) {
          uint32_t code = (page[c * row_bytes + at] >> shift) & mask;
          const float s = load_f(scale, d.md_dtype, c * G + g), z = load_f(zero, d.md_dtype, c * G + g);
          if (mixed && s_slot[c] >= 0) code |= ((page[d.key_off_high + s_slot[c] * row_bytes + at] >> shift) & 3u) << 2;
          add(c, affine_restore((float)code, s, z, d.md_dtype, d.dtype, key_flavour));
        }
      } else {
        const void* rows = kind == 0 ? d.k_sink : d.k_ring;
        const int64_t row = kind == 0 ? (int64_t)bh * d.sink_tokens + tok : (int64_t)bh * d.ring_tokens + tok % d.ring_tokens;
#pragma unroll 8
        for (int c = warp; c < D; c += GEN_WARPS) add(c, load_f(rows, d.dtype, row * D + c));
      }
#pragma unroll
      for (int r = 0; r < REP; ++r) s_part[(warp * REP + r) * GEN_TILE + lane] = dot[r];
      __syncthreads();
      // ---- online softmax state, a warp per query head
      for (int r = warp; r < rep; r += GEN_WARPS) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < GEN_WARPS; ++w) v += s_part[(w * REP + r) * GEN_TILE + lane];
        v = lane < nt ? v * a.scale : -INFINITY;
        float mx = v;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float m_old = s_m[r], m_new = fmaxf(m_old, mx);
        const float m_ref = m_new == -INFINITY ? 0.0f : m_new;   // every logit so far -Inf or NaN: the former weigh nothing
        const float e = expf(v - m_ref);
        float sum = e;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        s_p[lane * REP + r] = e;
        __syncwarp();
        if (lane == 0) {
          const float alpha = expf(m_old - m_ref);
          s_alpha[r] = alpha;
          s_m[r] = m_new;
          s_l[r] = s_l[r] * alpha + sum;
        }
      }
      __syncthreads();
      // ---- values
      if (vsplit < vsplits) {
#pragma unroll
        for (int r = 0; r < REP; ++r) acc[r] *= r < rep ? s_alpha[r] : 0.0f;
        const int vbits = d.value_bits, per = 8 / vbits, vg = vc / d.value_group;
        const uint32_t vmask = (1u << vbits) - 1u;
        auto weigh = [&](int tt, float v) {
#pragma unroll
          for (int r = 0; r < REP; ++r) acc[r] = fmaf(r < rep ? s_p[tt * REP + r] : 0.0f, v, acc[r]);
        };
        if (tile0 >= sink_filled && tile0 + nt <= v_end) {
#pragma unroll 8
          for (int tt = vsplit; tt < nt; tt += vsplits) {
            const int64_t row = (int64_t)bh * d.max_value_tokens + (tile0 + tt - d.sink_tokens);
            const uint32_t code = (d.v_codes[row * d.value_row_bytes + vc / per] >> ((vc % per) * vbits)) & vmask;
            const float s = load_f(d.v_meta, d.md_dtype, (row * 2 + 0) * d.value_groups + vg);
            const float z = load_f(d.v_meta, d.md_dtype, (row * 2 + 1) * d.value_groups + vg);
            weigh(tt, affine_restore((float)code, s, z, d.md_dtype, d.dtype, value_flavour(tile0 + tt)));
          }
        } else {
#pragma unroll 4
          for (int tt = vsplit; tt < nt; tt += vsplits) {
            const int vt = tile0 + tt;
            float v;
            if (vt < sink_filled) v = load_f(d.v_sink, d.dtype, ((int64_t)bh * d.sink_tokens + vt) * D + vc);
            else if (vt >= v_end) v = load_f(d.v_ring, d.dtype, ((int64_t)bh * d.ring_tokens + (vt % d.ring_tokens)) * D + vc);
            else {
              const int64_t row = (int64_t)bh * d.max_value_tokens + (vt - d.sink_tokens);
              const uint32_t code = (d.v_codes[row * d.value_row_bytes + vc / per] >> ((vc % per) * vbits)) & vmask;
              const float s = load_f(d.v_meta, d.md_dtype, (row * 2 + 0) * d.value_groups + vg);
              const float z = load_f(d.v_meta, d.md_dtype, (row * 2 + 1) * d.value_groups + vg);
              v = affine_restore((float)code, s, z, d.md_dtype, d.dtype, value_flavour(vt));
            }
            weigh(tt, v);
          }
        }
      }
      __syncthreads();
    }
    t = seg_end;
  }

  // the token shares of a channel meet in shared memory
  if (vsplits > 1) {
    if (vsplit < vsplits)
#pragma unroll
      for (int r = 0; r < REP; ++r) s_part[(vsplit * REP + r) * D + vc] = acc[r];
    __syncthreads();
    if (vsplit == 0)
#pragma unroll
      for (int r = 0; r < REP; ++r) {
        acc[r] = 0.0f;
        for (int s = 0; s < vsplits; ++s) acc[r] += s_part[(s * REP + r) * D + vc];
      }
  }
  const int slot = a.split_base + split;
#pragma unroll
  for (int r = 0; r < REP; ++r) {
    if (r < rep) {
      const int64_t row = ((int64_t)b * a.query_heads + h * rep + r) * a.total_splits + slot;
      // a NaN logit does not show in the maximum: the merge must not take a split of nothing else for an empty one
      if (tid == 0) { a.part_m[row] = s_l[r] == s_l[r] ? s_m[r] : s_l[r]; a.part_l[row] = s_l[r]; }
      if (vsplit == 0) a.part_acc[row * D + vc] = acc[r];
    }
  }
}

template <int MD> __device__ __forceinline__ float load_md(const void* p, int64_t i) {
  if (MD == DARTKV_F16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  if (MD == DARTKV_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return reinterpret_cast<const float*>(p)[i];
}

// Uniform key pages of few tokens: what decode_generic_kernel does, one tile of 32 tokens per block, with the chain of memory
// latencies cut to two.  Every lane finds the place of its own token (sink, page, dense tail), so a tile is not cut at segment
// edges; pages are found without a search where there are at most 32; the tile's values, packed or dense, are requested with
// its keys.  The blocks of a (batch, KV head), a.cluster of them, are a cluster that merges its results through distributed
// shared memory.  What such a call waits for longest is its own instructions, each of which runs once: so the metadata dtype and
// whether the cache is fp32 are template arguments (F32), what concerns a token (packed or dense, flavour, ring row) is found
// once by its lane and kept as bits, and addresses of a thread's tokens and channels are a first one plus steps.  [1,8,256,128]
// fp32, 2-bit: 12.5 us, with all of that found again for every element 15.0 us (of which requesting the values took 4.7).
template <int REP, int MD, bool F32>
__global__ void __launch_bounds__(GEN_THREADS, 2) decode_tiles_kernel(const __grid_constant__ dartkv_cache_desc d,
                                                                      const __grid_constant__ GenericArgs a) {
  extern __shared__ float smem[];
  wait_previous();
  const int D = d.head_dim;
  const int rep = a.query_heads / d.kv_heads;            // at most REP
  float* s_q = smem;                                     // [D][REP]
  float* s_part = s_q + D * REP;                         // [warp][REP][32] partial logits, then [split][REP][D] sums
  float* s_p = s_part + GEN_THREADS * REP;               // [32][REP] probabilities of the tile
  float* s_m = s_p + GEN_TILE * REP;                     // [REP]
  float* s_l = s_m + REP;
  static_assert(GEN_WARPS * GEN_TILE <= GEN_THREADS, "partial logits and sums share memory");

  const int tiles = a.cluster ? a.cluster : a.total_splits, split = blockIdx.x % tiles, bh = blockIdx.x / tiles;
  const int b = bh / d.kv_heads, h = bh % d.kv_heads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int seen = d.state[0], pages = d.state[1], k_end = d.state[2], v_end = d.state[3], sink_filled = d.state[4];
  const int first = split * GEN_TILE;
  const int lo = a.row_start ? max(first, a.row_start[b]) : first;
  const int nt = min(first + GEN_TILE, seen) - lo;       // tokens of this block, none or less where the row starts behind them
  // irregular pages, a page per lane where there are few; regular ones are computed
  int my_first = 0, my_tokens = 0;
  const bool by_lane = !d.regular_pages && pages <= 32;
  if (by_lane && lane < pages) { my_first = d.page_start[lane]; my_tokens = d.page_tokens[lane]; }
  for (int i = tid; i < D * REP; i += GEN_THREADS) {
    const int r = i % REP, c = i / REP;
    s_q[i] = r < rep ? load_f(a.q, a.q_dt, ((int64_t)b * a.query_heads + h * rep + r) * D + c) : 0.0f;
  }
  if (tid < REP) { s_m[tid] = -INFINITY; s_l[tid] = 0.0f; }
  const int vsplits = GEN_THREADS / D, vsplit = tid / D, vc = tid % D;
  float acc[REP];
#pragma unroll
  for (int r = 0; r < REP; ++r) acc[r] = 0.0f;
  const int bits = d.key_bits, vbits = d.value_bits, vg = vc / d.value_group;   // 2, 4 or 8 bits: no code lies across bytes
  const uint32_t mask = (1u << bits) - 1u, vmask = (1u << vbits) - 1u;
  auto value_flavour = [&](int tok) -> int {             // see decode_generic_kernel
    if (a.flavour == DARTKV_DEQUANT_PER_OP || d.regular_pages) return a.flavour;
    const int vs = d.sink_tokens + (tok - d.sink_tokens) / d.page_size * d.page_size;
    const int ve = min(v_end, vs + d.page_size);
    if (vs >= k_end) return a.flavour;
    const int pg = gen_find_page(d, pages, vs);
    return d.page_start[pg] + d.page_tokens[pg] < ve ? DARTKV_DEQUANT_PER_OP : a.flavour;
  };
  __syncthreads();

  if (nt > 0) {
    const int tok = lo + min(lane, nt - 1);              // lanes past the tile repeat its last token
    // ---- the place of this lane's key
    const bool packed = tok >= sink_filled && tok < k_end;
    int page_first = 0, page_n = 1, pg = 0;
    bool key_per_op = a.flavour == DARTKV_DEQUANT_PER_OP;
    if (by_lane) {
      for (int i = 0; i < pages; ++i) {
        const int f = __shfl_sync(0xffffffffu, my_first, i), n = __shfl_sync(0xffffffffu, my_tokens, i);
        if (f <= tok && tok < f + n) { page_first = f; page_n = n; pg = i; }
      }
    } else if (packed && d.regular_pages) {
      pg = (tok - d.sink_tokens) / d.page_size;
      page_first = d.sink_tokens + pg * d.page_size;
      page_n = d.page_size;
    } else if (packed) {
      pg = gen_find_page(d, pages, tok);
      page_first = d.page_start[pg];
      page_n = d.page_tokens[pg];
    }
    const uint8_t* page = d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes;
    if (!key_per_op && packed && page_first < v_end) {   // see decode_generic_kernel
      const int next_value_edge = d.sink_tokens + ((page_first - d.sink_tokens) / d.page_size + 1) * d.page_size;
      key_per_op = min(next_value_edge, v_end) < page_first + page_n;
    }
    // ---- bits of the tile's tokens: values packed, and restored with per-op rounding
    const uint32_t value_packed = __ballot_sync(0xffffffffu, tok >= sink_filled && tok < v_end);
    const uint32_t value_per_op = __ballot_sync(0xffffffffu, a.flavour == DARTKV_DEQUANT_PER_OP || value_flavour(tok) == DARTKV_DEQUANT_PER_OP);
    // ---- the tile's values are requested, kAhead of this thread's tokens at a time, the first ones before the keys are
    // waited for.  A dense value takes the scale's register.  One copy of this code serves all of a tile's tokens.  Dense
    // [1,8,20,256] fp32, one query row per KV head: 20.5 us with dense values loaded one by one behind the softmax, 21.2 with a
    // second copy of the code for the first tokens, 16.4 so.  Sixteen ahead with more query rows: 16 rows of that shape 37.2 us
    // instead of 33.1.
    constexpr int kAhead = REP <= 4 ? 16 : 8;
    uint32_t v_code[kAhead];
    float v_scale[kAhead], v_zero[kAhead];
    const int64_t row0 = (int64_t)bh * d.max_value_tokens + (lo - d.sink_tokens);   // of the tile's first token, whether packed or not
    const uint8_t* const codes0 = d.v_codes + row0 * d.value_row_bytes + (vc * vbits >> 3);
    const int meta_step = 2 * d.value_groups, ring_row = lo % d.ring_tokens;
    const int64_t meta0 = row0 * meta_step + vg;
    const int64_t sink0 = ((int64_t)bh * d.sink_tokens + lo) * D + vc, ring0 = (int64_t)bh * d.ring_tokens * D + vc;
    auto dense = [&](const void* p, int64_t i) { return F32 ? reinterpret_cast<const float*>(p)[i] : load_f(p, d.dtype, i); };
    auto request_values = [&](int base) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int tt = vsplit + (base + i) * vsplits;
        v_code[i] = 0; v_scale[i] = v_zero[i] = 0.0f;
        if (tt < nt) {
          if ((value_packed >> tt) & 1u) {
            v_code[i] = codes0[tt * d.value_row_bytes];
            v_scale[i] = load_md<MD>(d.v_meta, meta0 + tt * meta_step);
            v_zero[i] = load_md<MD>(d.v_meta, meta0 + tt * meta_step + d.value_groups);
          } else if (lo + tt < sink_filled) {
            v_scale[i] = dense(d.v_sink, sink0 + tt * D);
          } else {
            int row = ring_row + tt;
            while (row >= d.ring_tokens) row -= d.ring_tokens;
            v_scale[i] = dense(d.v_ring, ring0 + row * D);
          }
        }
      }
    };
    if (vsplit < vsplits) request_values(0);
    auto restore = [&](uint32_t code, float s, float z, bool per_op) {
      if (!F32) return affine_restore((float)code, s, z, MD, d.dtype, per_op ? DARTKV_DEQUANT_PER_OP : a.flavour);
      const float rounded = rnd<MD>(__fadd_rn(rnd<MD>(__fmul_rn((float)code, s)), z)), fused = __fmaf_rn((float)code, s, z);
      return per_op ? rounded : fused;   // fp32 caches round neither result again
    };
    // ---- partial logits of this warp's channels
    float dot[REP];
#pragma unroll
    for (int r = 0; r < REP; ++r) dot[r] = 0.0f;
    auto add = [&](int c, float k) {
#pragma unroll
      for (int r = 0; r < REP; ++r) dot[r] = fmaf(s_q[c * REP + r], k, dot[r]);
    };
    if (packed) {
      const int j = tok - page_first, g = j / d.key_group, G = ceil_div(page_n, d.key_group);
      const int row_bytes = (G * d.key_group * bits + 7) >> 3;
      const uint8_t* codes = page + (j * bits >> 3) + warp * row_bytes;
      const int shift = j * bits & 7;
      const uint8_t *scale = page + d.key_off_scale, *zero = page + d.key_off_zero;
#pragma unroll 1
      for (int c0 = warp; c0 < D; c0 += 8 * GEN_WARPS) {
        uint32_t code[8];
        float s[8], z[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {   // channels past the last one repeat it
          const int c = min(c0 + i * GEN_WARPS, D - 1);
          code[i] = codes[(c - warp) * row_bytes];
          s[i] = load_md<MD>(scale, c * G + g);
          z[i] = load_md<MD>(zero, c * G + g);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (c0 + i * GEN_WARPS < D) add(c0 + i * GEN_WARPS, restore((code[i] >> shift) & mask, s[i], z[i], key_per_op));
      }
    } else {
      const void* rows = tok < sink_filled ? d.k_sink : d.k_ring;
      const int64_t row = tok < sink_filled ? (int64_t)bh * d.sink_tokens + tok : (int64_t)bh * d.ring_tokens + tok % d.ring_tokens;
#pragma unroll 8
      for (int c = warp; c < D; c += GEN_WARPS) add(c, dense(rows, row * D + c));
    }
#pragma unroll
    for (int r = 0; r < REP; ++r) s_part[(warp * REP + r) * GEN_TILE + lane] = dot[r];
    __syncthreads();
    // ---- softmax over the tile, a warp per query head
    for (int r = warp; r < rep; r += GEN_WARPS) {
      float v = 0.0f;
#pragma unroll
      for (int w = 0; w < GEN_WARPS; ++w) v += s_part[(w * REP + r) * GEN_TILE + lane];
      v = lane < nt ? v * a.scale : -INFINITY;
      float m = v;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
      const float e = expf(v - (m == -INFINITY ? 0.0f : m));   // every logit -Inf or NaN: the former weigh nothing
      float sum = e;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      s_p[lane * REP + r] = e;
      if (lane == 0) { s_m[r] = m; s_l[r] = sum; }
    }
    __syncthreads();
    // ---- values
    if (vsplit < vsplits) {
      const int vshift = vc * vbits & 7;
#pragma unroll 1
      for (int base = 0; vsplit + base * vsplits < nt; base += kAhead) {
        if (base > 0) request_values(base);
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int tt = vsplit + (base + i) * vsplits;
          if (tt >= nt) break;
          const float v = (value_packed >> tt) & 1u ? restore((v_code[i] >> vshift) & vmask, v_scale[i], v_zero[i], (value_per_op >> tt) & 1u)
                                                    : v_scale[i];
#pragma unroll
          for (int r = 0; r < REP; ++r) acc[r] = fmaf(r < rep ? s_p[tt * REP + r] : 0.0f, v, acc[r]);
        }
      }
    }
    __syncthreads();
  }

  // the token shares of a channel meet in shared memory
  if (vsplit < vsplits)
#pragma unroll
    for (int r = 0; r < REP; ++r) s_part[(vsplit * REP + r) * D + vc] = acc[r];
  __syncthreads();
  if (vsplit == 0)
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      acc[r] = 0.0f;
      for (int s = 0; s < vsplits; ++s) acc[r] += s_part[(s * REP + r) * D + vc];
      s_part[r * D + vc] = acc[r];   // nobody else reads these entries before the cluster meets
    }
  if (a.cluster == 0) {   // more tiles than a cluster has blocks: a partial each, for the merge kernel
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      if (r < rep) {
        const int64_t row = ((int64_t)b * a.query_heads + h * rep + r) * a.total_splits + split;
        if (tid == 0) { a.part_m[row] = s_l[r] == s_l[r] ? s_m[r] : s_l[r]; a.part_l[row] = s_l[r]; }   // see decode_generic_kernel
        if (vsplit == 0) a.part_acc[row * D + vc] = acc[r];
      }
    }
    return;
  }
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int i = split * GEN_THREADS + tid; i < rep * D; i += a.cluster * GEN_THREADS) {
    const int r = i / D, c = i - r * D;
    float m = -INFINITY, l = 0.0f, sum = 0.0f;
    for (int k = 0; k < a.cluster; ++k) m = fmaxf(m, *cluster.map_shared_rank(&s_m[r], k));
    for (int k = 0; k < a.cluster; ++k) {
      const float mk = *cluster.map_shared_rank(&s_m[r], k), lk = *cluster.map_shared_rank(&s_l[r], k);
      if (mk != -INFINITY || lk != lk) {   // a NaN logit does not show in the maximum
        const float w = lk == lk ? expf(mk - m) : lk;
        l = fmaf(lk, w, l);
        sum = fmaf(*cluster.map_shared_rank(&s_part[r * D + c], k), w, sum);   // Inf and NaN count even where the weight is zero
      }
    }
    const float v = sum * (1.0f / fmaxf(l, 1e-20f));
    const int64_t row = (int64_t)b * a.query_heads + h * rep + r;
    if (a.out != nullptr) {
      store_f(a.out, a.q_dt, row * D + c, v);
    } else {   // the row's only partial: the merge kernel delivers the same numbers to the peers
      a.part_acc[row * D + c] = v;
      if (c == 0) { a.part_m[row] = 0.0f; a.part_l[row] = 1.0f; }
    }
  }
  cluster.sync();   // no block leaves while another one reads its results
}

static size_t tiles_smem(int D, int rep) {
  return ((size_t)D * rep + (size_t)GEN_THREADS * rep + (size_t)GEN_TILE * rep + 2 * rep) * sizeof(float);
}

using GenericKernel = void (*)(const dartkv_cache_desc, const GenericArgs);
template <int MD, bool F32>
static GenericKernel tiles_variant_of(int rep) {
  switch (rep) {
    case 1: return decode_tiles_kernel<1, MD, F32>;
    case 2: return decode_tiles_kernel<2, MD, F32>;
    case 4: return decode_tiles_kernel<4, MD, F32>;
    case 8: return decode_tiles_kernel<8, MD, F32>;
    default: return decode_tiles_kernel<16, MD, F32>;
  }
}
template <bool F32>
static GenericKernel tiles_variant(int md, int rep) {
  return md == DARTKV_F32 ? tiles_variant_of<DARTKV_F32, F32>(rep) : md == DARTKV_F16 ? tiles_variant_of<DARTKV_F16, F32>(rep) : tiles_variant_of<DARTKV_BF16, F32>(rep);
}

// shared memory of decode_generic_kernel<REP>; the sums of up to GEN_THREADS channels reuse the partial logits
static size_t generic_smem(int D, int rep) {
  return ((size_t)D * rep + (size_t)GEN_WARPS * rep * GEN_TILE + (size_t)GEN_TILE * rep + 3 * rep) * sizeof(float) + (size_t)D * sizeof(int);
}

// one block per (batch, query head): combine split partials, normalize, cast
// With stream_blocks > 0 (tensor-core layouts) a row's valid slots are its dense slot 0 plus one per stream block
// that touched its (batch, kv head); the remaining slots of the row hold stale data and are skipped.
// With peers.world_size > 1 the normalized rows are also stored into every rank's gathered output tensor (plain
// stores through peer-mapped pointers over NVLink), and the block that finishes last publishes this rank's arrival
// flag on every peer and then waits, with a bound, for every peer's flag on this rank: when the kernel ends, the
// gathered tensor of this rank is complete.  Nothing here waits on another kernel of the same GPU.
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

constexpr int kFewSplits = 17;          // slots of a row on the tensor-core layouts
constexpr int kManyThreads = 512;       // block of the merge where a row has more slots than kFewSplits

__global__ void decode_merge_kernel(const float* __restrict__ part_m, const float* __restrict__ part_l,
                                    const float* __restrict__ part_acc, int total_splits, int D, void* out, int out_dt,
                                    int stream_blocks, int64_t units, int quads, int query_heads, int kv_heads, int row_groups,
                                    dartkv_peer_scatter peers, int* status, unsigned int* done_counter) {
  wait_previous();
  int64_t row = blockIdx.x;
  int splits = total_splits;
  if (stream_blocks > 0) {
    // the work rows of the split are (batch, KV head, group of the head's query rows)
    const int rep = query_heads / kv_heads, group_rows = (rep + row_groups - 1) / row_groups, head = (int)(row % query_heads);
    const int64_t bh = ((row / query_heads) * kv_heads + head / rep) * row_groups + head % rep / group_rows;
    splits = 2 + dartkv_block_of_unit(bh * quads + quads - 1, stream_blocks, units) -
             dartkv_block_of_unit(bh * quads, stream_blocks, units);
  }
  part_m += row * total_splits;
  part_l += row * total_splits;
  part_acc += row * total_splits * D;
  const int64_t out_row = blockIdx.x;
  const int64_t peer_row = (int64_t)(peers.dst_row_begin + out_row / query_heads) * peers.dst_heads_total +
                           peers.dst_head_begin + out_row % query_heads;
  auto deliver = [&](int c, float v) {
    store_f(out, out_dt, out_row * D + c, v);
    for (int p = 0; p < peers.world_size; ++p) store_f(peers.out[p], out_dt, peer_row * D + c, v);
  };
  const int lane = threadIdx.x & 31;
  if (splits <= kFewSplits) {
    // the partials of a channel are requested before the weights are known: one memory latency instead of three
    for (int c0 = 0; c0 < D; c0 += blockDim.x) {   // every thread takes part in the shuffles
      const int c = c0 + threadIdx.x;
      float v[kFewSplits];
#pragma unroll
      for (int s = 0; s < kFewSplits; ++s) v[s] = s < splits && c < D ? part_acc[s * D + c] : 0.0f;
      const float ms = lane < splits ? part_m[lane] : -INFINITY, ls = lane < splits ? part_l[lane] : 0.0f;
      float m = ms;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
      const bool live = ms != -INFINITY;   // the sums of an empty split may be anything
      const float w = live ? expf(ms - m) : 0.0f;
      float l = live ? ls * w : 0.0f;
      const uint32_t lives = __ballot_sync(0xffffffffu, live);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
      float acc = 0.0f;
#pragma unroll
      for (int s = 0; s < kFewSplits; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, s);
        if ((lives >> s) & 1u) acc = fmaf(v[s], ws, acc);   // Inf and NaN count even where the weight is zero
      }
      if (c < D) deliver(c, acc * (1.0f / fmaxf(l, 1e-20f)));
    }
  } else {
    // many splits: warps of equal channels take every `groups`-th split
    extern __shared__ float s_sum[];   // [groups][D]
    const int groups = blockDim.x / D, group = threadIdx.x / D, c = threadIdx.x % D;
    float m = -INFINITY;
    for (int s = lane; s < splits; s += 32) m = fmaxf(m, part_m[s]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    float l = 0.0f;
    for (int s = lane; s < splits; s += 32) {
      const float ms = part_m[s];
      if (ms != -INFINITY) l += part_l[s] * expf(ms - m);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
    float acc = 0.0f;
    if (group < groups) {
#pragma unroll 8
      for (int s = group; s < splits; s += groups) {
        const float ms = part_m[s], v = part_acc[s * D + c];
        if (ms != -INFINITY) acc = fmaf(v, expf(ms - m), acc);
      }
      s_sum[group * D + c] = acc;
    }
    __syncthreads();
    if (group == 0) {
      for (int g = 1; g < groups; ++g) acc += s_sum[g * D + c];
      deliver(c, acc * (1.0f / fmaxf(l, 1e-20f)));
    }
  }
  if (peers.world_size > 1) {
    // the block's peer stores are ordered before the barrier; one cumulative system-scope fence after it makes
    // them all visible system-wide before the block reports in (a fence per thread costs microseconds per wave)
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();
      const unsigned int ticket = atomicAdd(done_counter, 1u);
      if (ticket == gridDim.x - 1) {
        *done_counter = 0;      // ready for the next call on this stream
        __threadfence_system();
        for (int p = 0; p < peers.world_size; ++p) st_release_sys(peers.flags[p] + peers.rank, peers.epoch);
        // every peer's rows have landed here once its flag shows this step (or a later one)
        bool ok = true;
        for (int p = 0; p < peers.world_size && ok; ++p) {
          ok = false;
          for (int spin = 0; spin < (1 << 21); ++spin) {   // about half a second with the sleep below
            if ((int)(ld_acquire_sys(peers.flags[peers.rank] + p) - peers.epoch) >= 0) { ok = true; break; }
            __nanosleep(200);
          }
        }
        if (!ok) atomicExch(status, 2);
      }
    }
  }
}

// The merge of rows of few slots without peers: a warp per row, four channels a lane, eight rows a block.  Bound by latency;
// a block per row with a channel per thread takes the larger calls two waves of blocks and every thread seventeen predicated
// loads: whole decode call of batch 128, 32,768 tokens 1,097 -> 1,089 us, batch 32, 8,192 tokens 94.3 -> 91.5, batch 24 of
// 6,001 tokens in 4 bits 73.4 -> 69.4.  Eight slots: with room for five only, calls of six to eight slots (batch 1, 2,700 and
// 3,300 tokens) take 14.3 us instead of 12.3; with room for seventeen, calls of two and three slots take 13.3 to 14.3 us
// instead of 12.3 and calls of nine to seventeen gain nothing (B200).
constexpr int kRowSlots = 8;   // the lanes of the reductions below
constexpr int kRowDim = 128;   // channels of the tensor-core layouts
__global__ void __launch_bounds__(256) decode_merge_rows_kernel(const float* __restrict__ part_m, const float* __restrict__ part_l,
                                                                const float* __restrict__ part_acc, int total_splits, void* out,
                                                                int out_dt, int stream_blocks, int64_t units, int quads, int query_heads,
                                                                int kv_heads, int row_groups, int rows) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int rep = query_heads / kv_heads, group_rows = (rep + row_groups - 1) / row_groups, head = row % query_heads;
  const int64_t bh = ((int64_t)(row / query_heads) * kv_heads + head / rep) * row_groups + head % rep / group_rows;
  const int splits = 2 + dartkv_block_of_unit(bh * quads + quads - 1, stream_blocks, units) -
                     dartkv_block_of_unit(bh * quads, stream_blocks, units);
  const int64_t base = (int64_t)row * total_splits;
  wait_previous();
  const int c = 4 * lane;
  float4 v[kRowSlots];   // requested before the weights are known
#pragma unroll
  for (int s = 0; s < kRowSlots; ++s) {
    v[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (s < splits) {
      const float2* at = reinterpret_cast<const float2*>(part_acc + (base + s) * kRowDim + c);   // 8-byte aligned
      const float2 a = at[0], b = at[1];
      v[s] = make_float4(a.x, a.y, b.x, b.y);
    }
  }
  const float ms = lane < splits ? part_m[base + lane] : -INFINITY, ls = lane < splits ? part_l[base + lane] : 0.0f;
  float m = ms;
#pragma unroll
  for (int off = kRowSlots / 2; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  const bool live = ms != -INFINITY;   // the sums of an empty split may be anything
  const float w = live ? expf(ms - m) : 0.0f;
  float l = live ? ls * w : 0.0f;
#pragma unroll
  for (int off = kRowSlots / 2; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
  const float norm = 1.0f / fmaxf(__shfl_sync(0xffffffffu, l, 0), 1e-20f);
  const uint32_t lives = __ballot_sync(0xffffffffu, live);
  float r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int s = 0; s < kRowSlots; ++s) {
    const float ws = __shfl_sync(0xffffffffu, w, s);
    if ((lives >> s) & 1u) {   // Inf and NaN count even where the weight is zero
      r[0] = fmaf(v[s].x, ws, r[0]); r[1] = fmaf(v[s].y, ws, r[1]);
      r[2] = fmaf(v[s].z, ws, r[2]); r[3] = fmaf(v[s].w, ws, r[3]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] *= norm;
  const uint2 x = out_dt == DARTKV_BF16 ? make_uint2(pack16<DARTKV_BF16>(r[0], r[1]), pack16<DARTKV_BF16>(r[2], r[3]))
                                        : make_uint2(pack16<DARTKV_F16>(r[0], r[1]), pack16<DARTKV_F16>(r[2], r[3]));
  *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(out) + (int64_t)row * kRowDim + c) = x;
}

// ---------------------------------------------------------------------------- host side
struct DecodeLayout {
  int generic_splits, generic_chunk;   // generic kernel over the whole range (fallback)
  int fast;                            // tensor-core kernel for the packed pages: 1 per-op rounded, 2 unrounded fp32
  int quads, stream_blocks;            // tensor-core layouts: units per work row, stream blocks
  long long units;                     // of all work rows: (batch, kv head, group of the head's query rows)
  int unit_pages;                      // pages of a unit, four or eight
  int total_splits;
  int row_groups;                      // layout 4: groups of the query rows of a KV head, else 1
  int pieces;                          // large calls of more than eight rows (decode_many.cuh): blocks per work row, else 0
};

int dartkv_decode_fast_supported(const dartkv_cache_desc* d, int q_dtype, int query_heads);
int dartkv_decode_fast_launch(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads, float scale,
                              int flavour, int unit_pages, int quads, int stream_blocks, long long units, int total_splits,
                              float* part_m, float* part_l, float* part_acc, int* status, const int32_t* row_start,
                              cudaStream_t stream);
int dartkv_decode_fused32_supported(const dartkv_cache_desc* d, int q_dtype, int query_heads);
int dartkv_decode_fused32_launch(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads, float scale,
                                 int flavour, int unit_pages, int quads, int stream_blocks, long long units, int total_splits,
                                 float* part_m, float* part_l, float* part_acc, int* status, const int32_t* row_start,
                              cudaStream_t stream);

int dartkv_decode_wide_supported(const dartkv_cache_desc* d, int q_dtype, int query_heads);
int dartkv_decode_wide_blocks_per_sm(const dartkv_cache_desc* d, int q_dtype, int rep, int flavour);
int dartkv_decode_rows_supported(const dartkv_cache_desc* d, int q_dtype, int rep, int flavour);
int dartkv_decode_rows_groups(int rep);
int dartkv_decode_rows_launch(const dartkv_cache_desc* d, const void* query, int query_heads, float scale, int flavour, int quads,
                              int stream_blocks, long long units, int total_splits, float* part_m, float* part_l, float* part_acc,
                              int* status, const int32_t* row_start, cudaStream_t stream);
int dartkv_decode_many_groups(int rep);
int dartkv_decode_many_pieces(const dartkv_cache_desc* d, int rep, int pages);
int dartkv_decode_many_launch(const dartkv_cache_desc* d, const void* query, int query_heads, float scale, int pieces, int total_splits,
                              float* part_m, float* part_l, float* part_acc, int* status, const int32_t* row_start, cudaStream_t stream);
int dartkv_decode_wide_launch(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads, float scale,
                              int flavour, int quads, int stream_blocks, long long units, int total_splits,
                              float* part_m, float* part_l, float* part_acc, int* status, const int32_t* row_start,
                              cudaStream_t stream);

int dartkv_sm_count() {
  // per device: a process may drive GPUs of different sizes
  static std::atomic<int> cached[64];
  int device = 0, count = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 148;
  count = cached[device].load(std::memory_order_relaxed);
  if (count == 0) {
    if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0) count = 148;   // B200
    cached[device].store(count, std::memory_order_relaxed);
  }
  return count;
}

// work-split override: a debugging / testing knob, kept off the per-call path (the environment is read once)
static char g_split_override[64] = "";
static bool g_split_override_ready = false;
static const char* split_override() {
  if (!g_split_override_ready) {
    const char* env = getenv("DARTKV_DECODE_SPLIT");
    if (env) { strncpy(g_split_override, env, sizeof(g_split_override) - 1); g_split_override[sizeof(g_split_override) - 1] = 0; }
    g_split_override_ready = true;
  }
  return g_split_override[0] ? g_split_override : nullptr;
}
extern "C" int dartkv_decode_split_override(const char* spec) {
  g_split_override_ready = true;
  g_split_override[0] = 0;
  if (spec) { strncpy(g_split_override, spec, sizeof(g_split_override) - 1); g_split_override[sizeof(g_split_override) - 1] = 0; }
  return DARTKV_OK;
}

// Splits of the generic kernel: four blocks per SM where the tokens allow tiles for them, however many slots that gives
// the merge.  One (batch, KV head) of 131,072 fp32 tokens, 2-bit: 592 splits 210 us, 296 splits 316 us, 128 splits 609 us;
// of 8,192 tokens (256 tiles): 256 splits 60 us, 128 splits 69 us (B200).
static int generic_splits_for(int bh, int tokens) {
  return min(max(1, (148 * 4 + bh - 1) / bh), max(1, (tokens + GEN_TILE - 1) / GEN_TILE));
}

// Work split of the 2-bit kernels.  Two families are compared with a cost model in rounds of eight pages, one per warp:
//   aligned    rows * s blocks, s = 1..16 pieces per row, in units of four pages;
//   unaligned  one block per resident slot, in units of eight pages: a block may finish one row and start the next (at most 15
//              blocks touch a row), and what it does of a row is whole rounds but for the row's last one.
// Of a round beside another block on the SM, a round alone takes 0.6, one of four pages whose warps have a page each 0.7 (shared by two
// warps, alone, 0.3), a row that a block touches 0.3 more, the dense block of a row 0.7 of a slot's time, and up to 0.45 where
// dense blocks are left over for a second turn; the unaligned family counts 1 % more.  Fitted to 88 shapes (8 to 1,024 rows, 4 to
// 255 pages, both kernels), of which the model's choice takes 0.2 % more than the best of both families on average and 4 % at most;
// in units of four pages and with the constants of kernels of four pages a round 8 x 2,200 tokens took 17.2 us and not 14.5, unrounded
// 16 x 2,200 19.2 and not 15.6, 32 x 8,192 86.2 and not 82.9, 24 x 6,001 55.6 and not 52.6.  Aligned and unaligned: batch 128, 32,768
// tokens 1,054 and 1,075, 112 x 10,000 364 and 321 (B200).
static void two_bit_split(DecodeLayout& L, int bh, int pages, int resident, const char* force) {
  constexpr double kRow = 0.3, kDense = 0.7, kAlone = 0.6, kShared = 0.3, kHalf = 0.7, kTail = 0.45, kAcross = 1.01;
  const bool force_unaligned = force && force[0] == 'u', force_aligned = force && force[0] == 'a';
  const int sms = dartkv_sm_count();
  int best_pieces = 1;
  double best_cost = 1e30;
  for (int q = max(1, (L.quads + 15) / 16); q <= L.quads; ++q) {
    const int pieces = (L.quads + q - 1) / q;
    const long long blocks = (long long)bh * pieces;
    const bool alone = blocks <= sms;
    const double rounds = (q == 1 ? (alone ? kShared : kHalf) : (q + 1) / 2 * (alone ? kAlone : 1.0)) + kRow;
    const double left_over = blocks + bh > resident ? (double)(blocks + bh - resident) / sms : 0.0;
    const double by_waves = (double)((blocks + resident - 1) / resident) * rounds + kTail * (left_over < 1.0 ? left_over : 1.0);
    const double by_work = (double)bh * (pieces * rounds + kDense) / resident;
    const double cost = by_waves > by_work ? by_waves : by_work;
    if (cost < best_cost - 1e-9) { best_cost = cost; best_pieces = pieces; }
  }
  L.stream_blocks = bh * best_pieces;
  L.total_splits = best_pieces + 1;
  const int octs = (pages + 7) / 8;
  const long long units = (long long)bh * octs, min_share = (octs + 14) / 15;
  long long blocks = min((long long)resident, units / min_share);
  if (force_unaligned && strchr(force, ':')) {
    const long long wanted = atoll(strchr(force, ':') + 1);
    if (wanted >= 1 && wanted < blocks) blocks = wanted;
  }
  if (blocks < 1 || force_aligned) return;
  const double share = (double)((units + blocks - 1) / blocks);
  const double cost = kAcross * (share * (blocks <= sms ? kAlone : 1.0) + kRow * (share / octs + 1.0) + (double)bh * kDense / resident);
  if (cost >= best_cost && !force_unaligned) return;
  L.unit_pages = 8;
  L.quads = octs;
  L.units = units;
  L.stream_blocks = (int)blocks;
  const long long w = units / blocks;   // smallest share of a block
  L.total_splits = (int)((octs + w - 2) / w + 1) + 1;
}

// rows_call: the call came through dartkv_decode_attention_rows, the only one that runs more than four query rows per
// KV head on the tensor cores
static DecodeLayout decode_layout(const dartkv_cache_desc* d, int q_dtype, int query_heads, int flavour, int tokens,
                                  bool rows_call = false) {
  DecodeLayout L{};
  const int rep = query_heads / d->kv_heads;
  int bh = d->batch * d->kv_heads;
  L.row_groups = 1;
  L.unit_pages = 4;
  L.fast = rows_call && rep > 4 && dartkv_decode_rows_supported(d, q_dtype, rep, flavour) ? 4 : 0;
  if (L.fast == 4) {
    L.row_groups = dartkv_decode_rows_groups(rep);
    bh *= L.row_groups;   // at most eight
  }
  if (flavour == DARTKV_DEQUANT_PER_OP && dartkv_decode_fast_supported(d, q_dtype, query_heads)) L.fast = 1;
  if (flavour == DARTKV_DEQUANT_FUSED && dartkv_decode_fused32_supported(d, q_dtype, query_heads)) L.fast = 2;
  // every other packed geometry with 128-token pages and head_dim 128, and the fp32 flavour of all of them
  if (!L.fast && flavour != DARTKV_DEQUANT_FUSED && dartkv_decode_wide_supported(d, q_dtype, query_heads)) L.fast = 3;
  // the tensor-core kernels index (row, four-page unit) pairs with 32 bits
  if (L.fast && (long long)bh * ((max(1, (tokens - d->sink_tokens) / d->page_size) + 3) / 4) >= (1ll << 31)) {
    L.fast = 0;
    L.row_groups = 1;
    bh = d->batch * d->kv_heads;
  }
  if (L.fast) {
    // One unit = four consecutive pages of a (batch, kv head).  The units of all rows are dealt out evenly to `stream_blocks`
    // blocks (two_bit_split() for the 2-bit kernels).  Two families of splits are compared with a cost model in units of a round of four pages
    // (a block costs its rounds plus 1.75 per row it touches: query load, first-page latency, merge of its eight warps;
    // the dense block of a row about 2; blocks run in waves of two per SM):
    //   aligned    rows * s blocks, s = 1..16 pieces per row;
    //   unaligned  one block per resident slot, a block may finish one row and start the next (at most 16 blocks
    //              touch a row); measured ~3 % slower per unit than aligned blocks, but it fills every slot when
    //              the rows do not (e.g. 256 rows on 296 slots: 9 % faster at context 32768).
    // The constants were fitted to B200 timings.
    const int pages = max(1, (tokens - d->sink_tokens) / d->page_size);
    L.quads = (pages + 3) / 4;
    L.units = (long long)bh * L.quads;
    // (sinks and rings from any multiple of 8 bytes on serve decode_rows.cu, decode_many.cuh reads them 16 bytes at a time)
    if (L.fast == 4 && rep > 8 && ((uintptr_t)d->k_sink | (uintptr_t)d->v_sink | (uintptr_t)d->k_ring | (uintptr_t)d->v_ring) % 16 == 0) {
      // Every block of decode_many.cuh works for all rows of a KV head (of a group of up to 32), one page after another: less work,
      // but a longer chain than that of decode_rows.cu's blocks, which take four pages at a time for eight rows.  It pays where its
      // blocks, counted once for every eight rows, come near two per SM.  2-bit, 8 KV heads, before and after (B200): 20 rows,
      // 1 x 4,096 tokens (64 blocks, counted 192) 17.0 and 20.8 us, 1 x 8,192 (384) 23.2 and 21.3, 4 x 2,100 (384) 22.8 and 20.1,
      // 8 x 4,096 (768) 62.9 and 41.1; 9 rows, 2 x 4,096 (256) 20.8 and 18.5, 8 x 1,100 (256) 22.5 and 17.5.  With two eights of
      // rows and as many blocks per KV head as a row has slots for, 1 x 16,384 tokens take 23.5 and 27.9.  Nor does it pay where
      // decode_rows.cu has room for all of its units and dense blocks at once: 64 rows, 1 x 1,100 tokens (128 units and 128 dense
      // blocks, 32 blocks here) 14.4 and 21.6, 48 rows, 1 x 2,100 (288 together) 18.4 and 19.2; 2 x 1,100 (384) 22.6 and 19.2.
      const long long at_once = (long long)bh * min(L.quads, 16) + (long long)d->batch * d->kv_heads * ((rep + 3) / 4);
      const int groups = dartkv_decode_many_groups(rep), pieces = dartkv_decode_many_pieces(d, rep, pages);
      const long long work_rows = (long long)d->batch * d->kv_heads * groups, blocks = work_rows * pieces;
      if (10 * blocks * L.row_groups >= 17 * dartkv_sm_count() && (L.row_groups > 2 || pieces < 15) && at_once > 2 * dartkv_sm_count()) {
        L.pieces = pieces;
        L.row_groups = groups;
        L.units = work_rows * L.quads;
        L.stream_blocks = (int)blocks;
        L.total_splits = pieces + 1;
        return L;
      }
    }
    const int resident = (L.fast == 3 ? dartkv_decode_wide_blocks_per_sm(d, q_dtype, rep, flavour) : 2) * dartkv_sm_count();
    // "aligned" | "unaligned" | "unaligned:<blocks>" overrides the model (tests exercise both families, and
    // blocks that span several rows, with it): set through dartkv_decode_split_override(), or once per process
    // from the environment variable DARTKV_DECODE_SPLIT
    const char* force = split_override();
    if (L.fast == 1 || L.fast == 2) {
      two_bit_split(L, bh, pages, resident, force);
      return L;
    }
    // dense blocks of the many-row layout (one per four rows): with 2.0 instead of 4.0 8 x 1,177 tokens, 12 rows, take 39.9
    // instead of 33.8 us; with 8.0 16 x 2,125 tokens, 8 rows, 48 instead of 44
    const double block_fixed = 1.75, dense_cost = L.fast == 4 ? 4.0 : 2.0;
    int best_pieces = 1;
    double best_cost = 1e30;
    for (int q = max(1, (L.quads + 15) / 16); q <= L.quads; ++q) {
      const int pieces = (L.quads + q - 1) / q;
      const long long blocks = (long long)bh * pieces;
      const long long waves = (blocks + resident - 1) / resident;
      const double by_waves = (double)waves * (q + block_fixed);
      const double by_work = (double)bh * (pieces * (q + block_fixed) + dense_cost) / resident;
      const double cost = by_waves > by_work ? by_waves : by_work;
      if (cost < best_cost - 1e-9) { best_cost = cost; best_pieces = pieces; }
    }
    L.stream_blocks = bh * best_pieces;
    L.total_splits = best_pieces + 1;
    {
      const long long min_share = (L.quads + 14) / 15;
      long long blocks = resident;
      if (blocks > L.units / min_share) blocks = L.units / min_share;
      const bool force_unaligned = force && force[0] == 'u', force_aligned = force && force[0] == 'a';
      if (force_unaligned && strchr(force, ':')) {
        const long long wanted = atoll(strchr(force, ':') + 1);
        if (wanted >= 1 && wanted < blocks) blocks = wanted;
      }
      if (blocks >= 1 && !force_aligned) {
        const double share = (double)L.units / blocks;
        const double cost = 1.03 * (share + block_fixed * (share / L.quads + 1.0)) + (double)bh * dense_cost / resident;
        if (cost < best_cost || force_unaligned) {
          const long long w = L.units / blocks;   // smallest share of a block
          L.stream_blocks = (int)blocks;
          L.total_splits = (int)((L.quads + w - 2) / w + 1) + 1;
        }
      }
    }
  } else {
    L.generic_splits = generic_splits_for(bh, tokens);
    int chunk = (tokens + L.generic_splits - 1) / L.generic_splits;
    L.generic_chunk = max(GEN_TILE, (chunk + GEN_TILE - 1) / GEN_TILE * GEN_TILE);
    L.generic_splits = max(1, (tokens + L.generic_chunk - 1) / L.generic_chunk);
    L.total_splits = L.generic_splits;
  }
  return L;
}

static int64_t layout_bytes(const dartkv_cache_desc* d, int query_heads, const DecodeLayout& L) {
  int64_t rows = (int64_t)d->batch * query_heads * L.total_splits;
  return 16 + rows * (2 + d->head_dim) * (int64_t)sizeof(float);
}

extern "C" int64_t dartkv_decode_workspace_bytes(const dartkv_cache_desc* d, int query_heads, int max_tokens) {
  if (!d || query_heads <= 0 || max_tokens <= 0) return 0;
  // upper bound over query dtypes, dequant flavours and every token count up to max_tokens
  int64_t best = 0;
  for (int dt = 0; dt < 3; ++dt)
    for (int flavour = 0; flavour < 3; ++flavour) {
      DecodeLayout L = decode_layout(d, dt, query_heads, flavour, max_tokens);
      // the tensor-core layouts use at most 16 stream slots + 1 dense slot per row whatever the token count
      if (L.fast || dartkv_decode_rows_supported(d, dt, query_heads / d->kv_heads, flavour)) L.total_splits = max(L.total_splits, 17);
      best = max(best, layout_bytes(d, query_heads, L));
    }
  // The generic layout may serve any smaller token count (and is what a tensor-core cache falls back to for other
  // query dtypes).  Its split count is not monotonic in the token count, because the chunk is rounded up to whole
  // tiles, but it never exceeds generic_splits_for(): rounding the chunk up only lowers it.
  {
    const int bh = d->batch * d->kv_heads;
    DecodeLayout L{};
    L.total_splits = generic_splits_for(bh, max_tokens);
    best = max(best, layout_bytes(d, query_heads, L));
  }
  return best;
}

static int decode_plan_impl(const dartkv_cache_desc* d, int q_dtype, int query_heads, int flavour, int tokens, bool rows_call,
                            dartkv_decode_plan_info* out) {
  DARTKV_REQUIRE(d != nullptr && out != nullptr, "decode_plan received a null pointer");
  DARTKV_REQUIRE(dartkv_valid_dtype(q_dtype), "query must be f32, f16 or bf16");
  DARTKV_REQUIRE(query_heads > 0 && query_heads % d->kv_heads == 0, "query heads must be divisible by cache KV heads");
  DARTKV_REQUIRE(tokens > 0, "cache is empty");
  DARTKV_REQUIRE(flavour >= DARTKV_DEQUANT_PER_OP && flavour <= DARTKV_DEQUANT_FUSED, "unknown dequant flavour %d", flavour);
  const DecodeLayout L = decode_layout(d, q_dtype, query_heads, flavour, tokens, rows_call);
  out->kernel = L.fast;
  out->quads = L.fast ? L.quads : 0;
  out->stream_blocks = L.fast ? L.stream_blocks : 0;
  out->total_splits = L.total_splits;
  out->units = L.fast ? L.units : 0;
  out->generic_splits = L.fast ? 0 : L.generic_splits;
  out->generic_chunk = L.fast ? 0 : L.generic_chunk;
  out->unit_pages = L.fast && !L.pieces ? L.unit_pages : 0;
  out->row_groups = L.fast ? L.row_groups : 0;
  return DARTKV_OK;
}

extern "C" int dartkv_decode_plan(const dartkv_cache_desc* d, int q_dtype, int query_heads, int flavour, int tokens,
                                  dartkv_decode_plan_info* out) {
  return decode_plan_impl(d, q_dtype, query_heads, flavour, tokens, false, out);
}

extern "C" int dartkv_decode_plan_rows(const dartkv_cache_desc* d, int q_dtype, int query_heads, int flavour, int tokens,
                                       dartkv_decode_plan_info* out) {
  return decode_plan_impl(d, q_dtype, query_heads, flavour, tokens, true, out);
}

extern "C" int dartkv_decode_status(const void* workspace, int* status_out, void* stream) {
  DARTKV_REQUIRE(workspace && status_out, "decode_status received a null pointer");
  DARTKV_CUDA_OK(cudaMemcpyAsync(status_out, workspace, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  DARTKV_CUDA_OK(cudaStreamSynchronize((cudaStream_t)stream));
  return DARTKV_OK;
}

static int decode_attention_impl(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads,
                                 float scale, int flavour, int tokens, void* workspace, int64_t workspace_bytes,
                                 void* out, const dartkv_peer_scatter* peers, const int32_t* row_start,
                                 void* stream_, bool rows_call = false) {
  DARTKV_REQUIRE(d != nullptr, "null descriptor");
  DARTKV_REQUIRE(query && out && workspace, "decode_attention received a null pointer");
  DARTKV_REQUIRE(dartkv_valid_dtype(q_dtype), "query must be f32, f16 or bf16");
  DARTKV_REQUIRE(query_heads > 0 && query_heads % d->kv_heads == 0, "query heads must be divisible by cache KV heads");
  DARTKV_REQUIRE(tokens > 0, "cache is empty");
  DARTKV_REQUIRE(flavour >= DARTKV_DEQUANT_PER_OP && flavour <= DARTKV_DEQUANT_FUSED, "unknown dequant flavour %d", flavour);
  const int rep = query_heads / d->kv_heads;
  DecodeLayout L = decode_layout(d, q_dtype, query_heads, flavour, tokens, rows_call);
  DARTKV_REQUIRE(rep <= GEN_MAX_REP || L.fast == 4, "at most %d query heads per KV head are supported", GEN_MAX_REP);
  DARTKV_REQUIRE(d->head_dim <= GEN_MAX_D, "decode attention supports head_dim up to %d", GEN_MAX_D);
  // the dense-token blocks of the tensor-core kernels read the query two channels at a time
  DARTKV_REQUIRE(!L.fast || (uintptr_t)query % 4 == 0, "the query must be 4-byte aligned");
  cudaStream_t stream = (cudaStream_t)stream_;
  const int64_t rows = (int64_t)d->batch * query_heads * L.total_splits;
  DARTKV_REQUIRE(workspace_bytes >= layout_bytes(d, query_heads, L), "decode workspace too small: need %lld bytes",
                 (long long)layout_bytes(d, query_heads, L));
  DARTKV_REQUIRE((uintptr_t)workspace % 4 == 0, "the decode workspace must be 4-byte aligned");
  // The status word and the counter of finished blocks, then the partials, which move two floats at a time: from a multiple of eight
  // bytes on, wherever the workspace begins.
  int* status = reinterpret_cast<int*>(workspace);
  float* part_m = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 16 - (uintptr_t)workspace % 8);
  float* part_l = part_m + rows;
  float* part_acc = part_l + rows;
  const int bh = d->batch * d->kv_heads;
  const int D = d->head_dim;
  if (L.pieces) {
    int rc = dartkv_decode_many_launch(d, query, query_heads, scale, L.pieces, L.total_splits, part_m, part_l, part_acc, status, row_start,
                                       stream);
    if (rc) return rc;
  } else if (L.fast == 4) {
    int rc = dartkv_decode_rows_launch(d, query, query_heads, scale, flavour, L.quads, L.stream_blocks, L.units, L.total_splits, part_m,
                                       part_l, part_acc, status, row_start, stream);
    if (rc) return rc;
  } else if (L.fast) {
    int rc = L.fast == 3 ? dartkv_decode_wide_launch(d, query, q_dtype, query_heads, scale, flavour, L.quads, L.stream_blocks, L.units,
                                                     L.total_splits, part_m, part_l, part_acc, status, row_start, stream)
                         : (L.fast == 2 ? dartkv_decode_fused32_launch : dartkv_decode_fast_launch)(
                               d, query, q_dtype, query_heads, scale, flavour, L.unit_pages, L.quads, L.stream_blocks, L.units, L.total_splits,
                               part_m, part_l, part_acc, status, row_start, stream);
    if (rc) return rc;
  } else {
    GenericArgs a;
    a.q = query; a.q_dt = q_dtype; a.query_heads = query_heads; a.flavour = flavour; a.scale = scale;
    a.total_splits = L.total_splits; a.part_m = part_m; a.part_l = part_l; a.part_acc = part_acc;
    a.tok_begin = 0; a.tok_end = -1; a.chunk = L.generic_chunk; a.split_base = 0;
    a.row_start = row_start;
    DARTKV_REQUIRE(L.generic_splits <= 65535, "too many splits");
    const int padded_rep = rep <= 1 ? 1 : rep <= 2 ? 2 : rep <= 4 ? 4 : rep <= 8 ? 8 : 16;
    // Uniform pages where a block has one tile at most go to decode_tiles_kernel.  Its blocks of a KV head are a cluster (of the
    // portable size) and finish the row where there are up to eight of them and all are resident; clusters that wait for room cost
    // more than partials and a merge.  Calls of 16-bit caches with more blocks than that stay with decode_generic_kernel.  fp32, 128
    // channels: [1,8,256] 12.5 us (31.2 in decode_generic_kernel), [1,8,1000] 25.1 -> 16.7, [4,8,300] (320 blocks) 31.8 -> 18.8, [24,8,96] (576
    // blocks) 24.4 there, 32.7 in clusters of three and 22.4 as partials; 16 bits, 64 channels, [128,8,20] 27.9 and 30.9 (B200).
    const long long blocks = (long long)bh * L.generic_splits;
    const bool resident = blocks <= 2 * dartkv_sm_count();
    const bool tiles = d->key_mode == DARTKV_QUANTIZED_PAGE && L.generic_chunk == GEN_TILE && (resident || d->dtype == DARTKV_F32);
    a.cluster = tiles && L.generic_splits <= 8 && (resident || L.generic_splits == 1) ? L.generic_splits : 0;
    a.out = peers ? nullptr : out;
    const size_t smem = tiles ? tiles_smem(D, padded_rep) : generic_smem(D, padded_rep);
    const GenericKernel kernel = tiles ? (d->dtype == DARTKV_F32 ? tiles_variant<true>(d->md_dtype, padded_rep) : tiles_variant<false>(d->md_dtype, padded_rep)) : padded_rep == 1 ? decode_generic_kernel<1> : padded_rep == 2 ? decode_generic_kernel<2>
                      : padded_rep == 4 ? decode_generic_kernel<4> : padded_rep == 8 ? decode_generic_kernel<8> : decode_generic_kernel<16>;
    if (smem > 48 * 1024) DARTKV_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (a.cluster) {
      DARTKV_CUDA_OK(launch_clusters(a.cluster, kernel, dim3((unsigned)(bh * a.cluster)), dim3(GEN_THREADS), smem, stream, *d, a));
      DARTKV_LAUNCH_OK("decode_tiles_kernel");
      if (!peers) return DARTKV_OK;
      L.total_splits = 1;
    } else if (tiles) {
      DARTKV_CUDA_OK(launch_following(kernel, dim3((unsigned)(bh * L.generic_splits)), dim3(GEN_THREADS), smem, stream, *d, a));
      DARTKV_LAUNCH_OK("decode_tiles_kernel");
    } else {
      DARTKV_CUDA_OK(launch_following(kernel, dim3(bh, L.generic_splits), GEN_THREADS, smem, stream, *d, a));
      DARTKV_LAUNCH_OK("decode_generic_kernel");
    }
  }
  {
    const bool few = L.total_splits <= kFewSplits;
    // few slots a row of a tensor-core layout (128 channels, 16 bits): a warp per row, which moves four channels at a time
    if (L.fast && L.total_splits <= kRowSlots && !peers && (uintptr_t)out % 8 == 0 &&
        rows / L.total_splits < (1ll << 31)) {
      const int out_rows = (int)(rows / L.total_splits);
      DARTKV_CUDA_OK(launch_following(decode_merge_rows_kernel, dim3((out_rows + 7) / 8), dim3(256), 0, stream, part_m, part_l, part_acc,
                                      L.total_splits, out, q_dtype, L.stream_blocks, L.units, L.quads, query_heads, d->kv_heads,
                                      L.row_groups, out_rows));
      DARTKV_LAUNCH_OK("decode_merge_rows_kernel");
      return DARTKV_OK;
    }
    dartkv_peer_scatter none{};
    unsigned int* done_counter = reinterpret_cast<unsigned int*>(reinterpret_cast<char*>(workspace) + 4);
    DARTKV_CUDA_OK(launch_following(decode_merge_kernel, dim3((unsigned)((int64_t)d->batch * query_heads)),
                                    dim3(few ? min(256, (D + 31) / 32 * 32) : kManyThreads),
                                    few ? 0 : (size_t)(kManyThreads / D) * D * sizeof(float), stream, part_m, part_l, part_acc,
                                    L.total_splits, D, out, q_dtype, L.fast ? L.stream_blocks : 0, L.units, L.quads, query_heads,
                                    d->kv_heads, L.row_groups, peers ? *peers : none, status, done_counter));
  }
  DARTKV_LAUNCH_OK("decode_merge_kernel");
  return DARTKV_OK;
}

extern "C" int dartkv_decode_attention(const dartkv_cache_desc* d, const void* query, int q_dtype, int query_heads,
                                       float scale, int flavour, int tokens, void* workspace,
                                       int64_t workspace_bytes, void* out, void* stream) {
  return decode_attention_impl(d, query, q_dtype, query_heads, scale, flavour, tokens, workspace, workspace_bytes, out,
                               nullptr, nullptr, stream);
}

extern "C" int dartkv_decode_attention_padded(const dartkv_cache_desc* d, const void* query, int q_dtype,
                                              int query_heads, float scale, int flavour, int tokens,
                                              const int32_t* row_start, void* workspace, int64_t workspace_bytes,
                                              void* out, void* stream) {
  return decode_attention_impl(d, query, q_dtype, query_heads, scale, flavour, tokens, workspace, workspace_bytes, out,
                               nullptr, row_start, stream);
}

// Below this many tokens passes of four rows stay, not for speed but for their results: a token's is bit for bit that of a
// call with this token alone, which many-row blocks with their own order of sums do not give.  Batch 8, 32 heads on 8,
// 2-bit pages, device time of a call: 600 tokens 2 queries 48 us in passes, 26 us at once, 5 queries 110 / 38; 1,100
// tokens 50 / 26 and 118 / 40; 4,096 tokens 69 / 44 and 161 / 42 (B200).
constexpr int kRowsMinTokens = 1024;

extern "C" int dartkv_decode_rows_limit(const dartkv_cache_desc* d, int q_dtype, int flavour, int tokens) {
  if (!d || tokens < kRowsMinTokens || !dartkv_decode_rows_supported(d, q_dtype, 64, flavour)) return 0;
  // as many as keep the partials of a call (17 slots per row) within 64 MiB, in steps of a row group
  const int64_t row_bytes = 17 * (2 + (int64_t)d->head_dim) * sizeof(float) * d->batch * d->kv_heads;
  const int64_t fit = ((int64_t)64 << 20) / row_bytes / 8 * 8;
  return fit < 8 ? 8 : fit > 64 ? 64 : (int)fit;
}

extern "C" int dartkv_decode_attention_rows(const dartkv_cache_desc* d, const void* query, int q_dtype,
                                            int query_heads, float scale, int flavour, int tokens,
                                            const int32_t* row_start, void* workspace, int64_t workspace_bytes,
                                            void* out, void* stream) {
  return decode_attention_impl(d, query, q_dtype, query_heads, scale, flavour, tokens, workspace, workspace_bytes, out,
                               nullptr, row_start, stream, true);
}

extern "C" int dartkv_decode_attention_scatter(const dartkv_cache_desc* d, const void* query, int q_dtype,
                                               int query_heads, float scale, int flavour, int tokens, void* workspace,
                                               int64_t workspace_bytes, void* out, const dartkv_peer_scatter* peers,
                                               void* stream) {
  DARTKV_REQUIRE(peers != nullptr, "decode_attention_scatter received a null pointer");
  DARTKV_REQUIRE(peers->world_size >= 1 && peers->world_size <= DARTKV_MAX_PEERS, "world_size must be in [1, %d]",
                 DARTKV_MAX_PEERS);
  DARTKV_REQUIRE(peers->rank >= 0 && peers->rank < peers->world_size, "rank must be in [0, world_size)");
  DARTKV_REQUIRE(peers->dst_row_begin >= 0 && peers->dst_head_begin >= 0 &&
                     peers->dst_head_begin + query_heads <= peers->dst_heads_total,
                 "the rows of this rank do not fit the gathered tensor");
  for (int p = 0; p < peers->world_size; ++p)
    DARTKV_REQUIRE(peers->out[p] != nullptr && peers->flags[p] != nullptr, "peer %d has a null pointer", p);
  return decode_attention_impl(d, query, q_dtype, query_heads, scale, flavour, tokens, workspace, workspace_bytes, out,
                               peers, nullptr, stream);
}

// ---------------------------------------------------------------------------- built-in scratch variant
// Split-K scratch that lives in the library image instead of caller memory.  Every device that
// loads the library carries these 32 MiB until the process exits.
#define DARTKV_BUILTIN_SCRATCH_BYTES (32ll << 20)
static __device__ __align__(256) unsigned char g_builtin_scratch[DARTKV_BUILTIN_SCRATCH_BYTES];

#include <mutex>

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
void* g_scratch_address[kMaxDevices] = {};   // device address of g_builtin_scratch, per device ordinal
}  // namespace

// In host code `g_builtin_scratch` is only a handle for the symbol, not memory a kernel can use:
// the device address has to be asked for, with the target device current, once per device.
static int builtin_scratch_address(void** out) {
  int device = -1;
  DARTKV_CUDA_OK(cudaGetDevice(&device));
  DARTKV_REQUIRE(device >= 0 && device < kMaxDevices, "device ordinal %d is outside the supported range", device);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_address[device] == nullptr) {
    void* address = nullptr;
    DARTKV_CUDA_OK(cudaGetSymbolAddress(&address, g_builtin_scratch));
    DARTKV_REQUIRE(address != nullptr, "cudaGetSymbolAddress returned a null address for the built-in scratch");
    g_scratch_address[device] = address;
  }
  *out = g_scratch_address[device];
  return DARTKV_OK;
}

extern "C" int64_t dartkv_builtin_scratch_bytes(void) { return DARTKV_BUILTIN_SCRATCH_BYTES; }

extern "C" int dartkv_decode_attention_builtin_scratch(const dartkv_cache_desc* d, const void* query, int q_dtype,
                                                       int query_heads, float scale, int flavour, int tokens,
                                                       void* out, void* stream) {
  DARTKV_REQUIRE(d != nullptr, "null descriptor");
  DARTKV_REQUIRE(dartkv_valid_dtype(q_dtype), "query must be f32, f16 or bf16");
  DARTKV_REQUIRE(query_heads > 0 && query_heads % d->kv_heads == 0, "query heads must be divisible by cache KV heads");
  DARTKV_REQUIRE(tokens > 0, "cache is empty");
  DARTKV_REQUIRE(flavour >= DARTKV_DEQUANT_PER_OP && flavour <= DARTKV_DEQUANT_FUSED, "unknown dequant flavour %d", flavour);
  const DecodeLayout L = decode_layout(d, q_dtype, query_heads, flavour, tokens);
  const int64_t need = layout_bytes(d, query_heads, L);
  if (need > DARTKV_BUILTIN_SCRATCH_BYTES) {
    dartkv_set_error("this call needs %lld bytes of split scratch but the built-in scratch holds %lld; "
                     "use dartkv_decode_attention with a caller-provided workspace",
                     (long long)need, (long long)DARTKV_BUILTIN_SCRATCH_BYTES);
    return DARTKV_ELIMIT;
  }
  void* scratch = nullptr;
  int rc = builtin_scratch_address(&scratch);
  if (rc) return rc;
  // the array keeps whatever the previous call left; only the status word has to start at zero
  DARTKV_CUDA_OK(cudaMemsetAsync(scratch, 0, 16, (cudaStream_t)stream));
  return dartkv_decode_attention(d, query, q_dtype, query_heads, scale, flavour, tokens, scratch,
                                 DARTKV_BUILTIN_SCRATCH_BYTES, out, stream);
}
