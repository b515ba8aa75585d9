// Dense rows and device-side metadata of an append step, shared by the general path (cache_append.cu) and the
// page-shaped kernel (append_fast.cu).
#pragma once

#include "common.cuh"

__device__ __forceinline__ void publish_append(const dartkv_cache_desc& d, const dartkv_append_plan& p) {
  for (int pg = threadIdx.x; pg < p.num_pages; pg += blockDim.x) {
    d.page_start[p.first_page + pg] = p.page_token_start + pg * d.page_size;
    d.page_tokens[p.first_page + pg] = (pg == p.num_pages - 1) ? p.last_page_tokens : d.page_size;
  }
  if (threadIdx.x == 0) {
    d.state[0] = p.seen_after;
    d.state[1] = p.key_pages_after;
    d.state[2] = p.k_packed_end_after;
    d.state[3] = p.v_packed_end_after;
    d.state[4] = min(p.seen_after, d.sink_tokens);
  }
}

// true when a 16-byte piece of `dt` elements holds an Inf or NaN
__device__ __forceinline__ bool piece_nonfinite(uint4 v, int dt) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t flag = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (dt == DARTKV_F32) flag |= ((w[i] & 0x7FFFFFFFu) + 0x00800000u) & 0x80000000u;
    else flag |= ((w[i] & 0x7FFF7FFFu) + (dt == DARTKV_BF16 ? 0x00800080u : 0x04000400u)) & 0x80008000u;
  }
  return flag != 0;
}

// The chunk tokens of a step that stay dense, as copy rows 0..rows-1: row r is chunk token r while r < sink_copy
// (sink rows), then chunk token ring_first + (r - sink_copy) (ring rows, where the side's own range begins later the
// row is skipped).
struct DenseRows {
  int ring_first, rows;
};
__host__ __device__ __forceinline__ DenseRows dense_rows(const dartkv_append_plan& p) {
  const int chunk_end = p.chunk_start + p.chunk_tokens;
  DenseRows r{p.chunk_tokens, 0};
  if (p.sink_copy > 0 || p.ring_begin < chunk_end || p.value_end < chunk_end) {
    const int first_dense = p.ring_begin < (p.value_end > p.chunk_start ? p.value_end : p.chunk_start)
                                ? p.ring_begin : (p.value_end > p.chunk_start ? p.value_end : p.chunk_start);
    r.ring_first = first_dense - p.chunk_start > p.sink_copy ? first_dense - p.chunk_start : p.sink_copy;
    r.rows = p.sink_copy + (p.chunk_tokens - r.ring_first);
  }
  return r;
}

// Copy rows [r_begin, r_end) of one (batch, head) and side, the block's threads over the row pieces: 16-byte pieces
// where `vector_ok`, else elements.  Returns whether a copied element is Inf or NaN.
__device__ __forceinline__ bool copy_dense_rows(const dartkv_cache_desc& d, const dartkv_append_plan& p, const void* src,
                                                int64_t src_base, int64_t st, int ring_first, int r_begin, int r_end,
                                                int vector_ok, int bh, int side) {
  const int ring_begin = side == 0 ? p.ring_begin : p.value_end;  // values not packed by this step stay dense
  const int esize = dartkv_dtype_size(d.dtype);
  const int pieces = vector_ok ? d.head_dim * esize / 16 : d.head_dim;   // units per row
  bool bad = false;
  for (int i = threadIdx.x; i < (r_end - r_begin) * pieces; i += blockDim.x) {
    const int r = r_begin + i / pieces, c = i % pieces;
    const int j = r < p.sink_copy ? r : ring_first + (r - p.sink_copy);
    const int t = p.chunk_start + j;
    const bool to_sink = j < p.sink_copy;
    if (!to_sink && t < ring_begin) continue;
    void* dst = to_sink ? (side == 0 ? d.k_sink : d.v_sink) : (side == 0 ? d.k_ring : d.v_ring);
    const int64_t drow = to_sink ? ((int64_t)bh * d.sink_tokens + t) : ((int64_t)bh * d.ring_tokens + (t % d.ring_tokens));
    const int64_t srow = src_base + (int64_t)j * st;
    if (vector_ok) {
      const uint4 v = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(src) + srow * esize)[c];
      bad |= piece_nonfinite(v, d.dtype);
      reinterpret_cast<uint4*>(reinterpret_cast<char*>(dst) + drow * d.head_dim * esize)[c] = v;
    } else {
      const float v = load_f(src, d.dtype, srow + c);
      bad |= !isfinite(v);
      store_f(dst, d.dtype, drow * d.head_dim + c, v);
    }
  }
  return bad;
}

static inline int validate_desc(const dartkv_cache_desc* d) {
  DARTKV_REQUIRE(d != nullptr, "null descriptor");
  DARTKV_REQUIRE(d->key_page_bytes > 0 && d->value_row_bytes > 0, "descriptor geometry not filled (call dartkv_cache_geometry)");
  DARTKV_REQUIRE(d->k_ring && d->v_ring && d->k_pages && d->v_codes && d->v_meta && d->page_start && d->page_tokens && d->state,
                 "descriptor has a null pool pointer");
  DARTKV_REQUIRE(d->sink_tokens == 0 || (d->k_sink && d->v_sink), "descriptor has a null sink pointer");
  return DARTKV_OK;
}
