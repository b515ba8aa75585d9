// Materialization of the paged cache (DartKVCache.get, src/dart/cache.py:192-199): packed pages and dense rows back to
// [B,H,T,D] tensors.
//
// 16-bit caches whose groups fill whole code words take materialize_spans_kernel: a block restores one 128-token span
// (the span of a key page) of one (batch, head) and side with whole-word reads of the codes and whole-line stores; a
// thread owns the tokens of one key code word for two neighbouring channels, or eight channels of a value row.
// Everything else takes materialize_kernel, which walks a tile of tokens element pair by element pair.
// Bound by instructions and the latency of the codes, the stores stay in L2: 2 x 20 MB out of 8 MB packed (fp16 [4,8,2500,128],
// 2-bit + promoted keys) take 24.7 us element by element and 16.1 with two codes per register (code_pairs.cuh), some 2 us of
// the difference from the form of the launch; 222 us for the pass that appends them too with one block per token, which built
// the page's slot map 128 times over (B200).

#include "code_pairs.cuh"
#include "common.cuh"
#include "append_common.cuh"

namespace {

// first page whose range ends after token t (pages are contiguous from sink_tokens)
__device__ __forceinline__ int find_page(const dartkv_cache_desc& d, int pages, int t) {
  int lo = 0, hi = pages - 1;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (d.page_start[mid] + d.page_tokens[mid] > t) hi = mid; else lo = mid + 1;
  }
  return lo;
}


// One restored element from its code, with the cache's rounding.
__device__ __forceinline__ float restore_code(uint32_t code, float s, float z, const dartkv_cache_desc& d, int flavour) {
  return affine_restore((float)code, s, z, d.md_dtype, d.dtype, flavour);
}

// Tokens [first, end) of one (batch, head) and side, by the whole block (any geometry).  The range is walked segment
// by segment (dense rows, or one key page with its slot map), a thread owning two neighbouring channels of every
// few tokens.  row0 + token = output row; s_slot: [D].
__device__ void materialize_tokens(const dartkv_cache_desc& d, int bh, int side, int first, int end, int64_t row0, int flavour,
                                   void* out, int out_dt, int* s_slot) {
  const int D = d.head_dim, pairs = (D + 1) / 2, threads = blockDim.x;
  const int sink_filled = d.state[4], packed_end = side == 0 ? d.state[2] : d.state[3];
  // two channels are one store where the rows and the output (any element-aligned pointer) allow it
  const bool wide = D % 2 == 0 && (uintptr_t)out % (out_dt == DARTKV_F32 ? 8 : 4) == 0;
  auto put = [&](int t, int c, float a, float b) {
    const int64_t at = (row0 + t) * D + c;
    if (wide && out_dt == DARTKV_F32) reinterpret_cast<float2*>(out)[at / 2] = make_float2(a, b);
    else if (wide && out_dt == DARTKV_F16) reinterpret_cast<__half2*>(out)[at / 2] = __floats2half2_rn(a, b);
    else if (wide) reinterpret_cast<__nv_bfloat162*>(out)[at / 2] = __floats2bfloat162_rn(a, b);
    else {
      store_f(out, out_dt, at, a);
      if (c + 1 < D) store_f(out, out_dt, at + 1, b);
    }
  };
  // the block's threads as (token offset, channel pair); `step` tokens at a time
  const int step = max(1, threads / pairs);
  const int mine = threadIdx.x / pairs;   // threads past step * pairs idle where pairs does not divide the block
  for (int t = first; t < end;) {
    if (t < sink_filled || t >= packed_end) {
      const int stop = t < sink_filled ? min(end, sink_filled) : end;
      const void* src = t < sink_filled ? (side == 0 ? d.k_sink : d.v_sink) : (side == 0 ? d.k_ring : d.v_ring);
      if (mine < step)
        for (int tok = t + mine; tok < stop; tok += step)
          for (int p = threadIdx.x % pairs; p < pairs; p += threads) {
            const int64_t row = t < sink_filled ? (int64_t)bh * d.sink_tokens + tok : (int64_t)bh * d.ring_tokens + tok % d.ring_tokens;
            const int c = 2 * p;
            put(tok, c, load_f(src, d.dtype, row * D + c), c + 1 < D ? load_f(src, d.dtype, row * D + c + 1) : 0.0f);
          }
      t = stop;
      continue;
    }
    if (side == 1) {
      const int stop = min(end, packed_end), bits = d.value_bits, vpb = 8 / bits;
      const uint32_t mask = (1u << bits) - 1u;
      if (mine < step)
        for (int tok = t + mine; tok < stop; tok += step)
          for (int p = threadIdx.x % pairs; p < pairs; p += threads) {
            const int64_t row = (int64_t)bh * d.max_value_tokens + (tok - d.sink_tokens);
            const uint8_t* codes = d.v_codes + row * d.value_row_bytes;
            float v[2] = {0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int c = 2 * p + i;
              if (c < D) {
                const int g = c / d.value_group;
                v[i] = restore_code((codes[c / vpb] >> ((c % vpb) * bits)) & mask,
                                    load_f(d.v_meta, d.md_dtype, (row * 2 + 0) * d.value_groups + g),
                                    load_f(d.v_meta, d.md_dtype, (row * 2 + 1) * d.value_groups + g), d, flavour);
              }
            }
            put(tok, 2 * p, v[0], v[1]);
          }
      t = stop;
      continue;
    }
    const int pg = d.regular_pages ? (t - d.sink_tokens) / d.page_size : find_page(d, d.state[1], t);
    const int page_first = d.page_start[pg], n = d.page_tokens[pg], stop = min(end, page_first + n);
    const uint8_t* page = d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes;
    const bool mixed = d.key_mode == DARTKV_MIXED_PAGE;
    if (mixed) {
      __syncthreads();
      for (int c = threadIdx.x; c < D; c += blockDim.x) s_slot[c] = -1;
      __syncthreads();
      const int32_t* idx = reinterpret_cast<const int32_t*>(page + d.key_off_index);
      for (int k = threadIdx.x; k < d.promoted; k += blockDim.x) {
        const int c = idx[k];
        if (c >= 0 && c < D) s_slot[c] = k;
      }
      __syncthreads();
    }
    const int Gk = d.key_group, G = ceil_div(n, Gk), bits = mixed ? 2 : d.key_bits, vpb = 8 / bits;
    const int pb = ceil_div(Gk, 4);                            // mixed: bytes of a group's plane
    const int row_bytes = mixed ? G * pb : ceil_div(G * Gk, vpb);
    const uint32_t mask = (1u << bits) - 1u;
    if (mine < step)
      for (int p = threadIdx.x % pairs; p < pairs; p += threads) {
        // the scale and zero point of a channel change only with the group
        int held = -1;
        float s[2] = {0.0f, 0.0f}, z[2] = {0.0f, 0.0f};
        for (int tok = t + mine; tok < stop; tok += step) {
          const int j = tok - page_first, g = j / Gk;
          const int at = mixed ? g * pb + (j - g * Gk) / 4 : j / vpb;
          const int shift = mixed ? ((j - g * Gk) % 4) * 2 : (j % vpb) * bits;
          float v[2] = {0.0f, 0.0f};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int c = 2 * p + i;
            if (c < D) {
              if (g != held) {
                s[i] = load_f(page + d.key_off_scale, d.md_dtype, c * G + g);
                z[i] = load_f(page + d.key_off_zero, d.md_dtype, c * G + g);
              }
              uint32_t code = (page[c * row_bytes + at] >> shift) & mask;
              if (mixed && s_slot[c] >= 0) code |= ((page[d.key_off_high + s_slot[c] * row_bytes + at] >> shift) & 3u) << 2;
              v[i] = restore_code(code, s[i], z[i], d, flavour);
            }
          }
          held = g;
          put(tok, 2 * p, v[0], v[1]);
        }
      }
    t = stop;
  }
}

constexpr int kTileTokens = 32, kTileThreads = 128, kSpan = 128, kSpanThreads = 256;

struct MaterializeArgs {
  int side0, t0, t1, flavour, out_dt;   // t0, t1: the tokens of the launch
  int out_first, out_tokens;            // first token and row count of the output per (batch, head)
  void *out_k, *out_v;
};

// grid (bh, tile, side)
__global__ void __launch_bounds__(kTileThreads) materialize_kernel(const __grid_constant__ dartkv_cache_desc d,
                                                                   const __grid_constant__ MaterializeArgs a) {
  extern __shared__ int s_slot[];
  wait_previous();
  const int bh = blockIdx.x, side = a.side0 + blockIdx.z, first = a.t0 + blockIdx.y * kTileTokens;
  materialize_tokens(d, bh, side, first, min(a.t1, first + kTileTokens), (int64_t)bh * a.out_tokens - a.out_first, a.flavour,
                     side == 0 ? a.out_k : a.out_v, a.out_dt, s_slot);
}

// A page of n tokens, the tokens [lo, hi) of it wanted; out: row of the page's first token.  BITS 0: mixed keys.
template <int MD, int DT, int BITS>
__device__ __forceinline__ void restore_page(const dartkv_cache_desc& d, const uint8_t* page, int n, int lo, int hi, int flavour,
                                             uint16_t* out, const int* s_slot) {
  constexpr int PB = BITS == 0 ? 2 : BITS, TOK = 32 / PB;
  CodeConsts<MD> consts;
  consts.init();
  const int groups = ceil_div(n, d.key_group), row_words = groups * d.key_group * PB / 32;
  const uint32_t* codes = reinterpret_cast<const uint32_t*>(page);
  const uint32_t* high = reinterpret_cast<const uint32_t*>(page + d.key_off_high);
  const int pairs = d.head_dim / 2, items = pairs * ceil_div(n, TOK);
  for (int item = threadIdx.x; item < items; item += kSpanThreads) {
    const int p = item % pairs, w = item / pairs, t = w * TOK, g = t / d.key_group;
    if (t + TOK <= lo || t >= hi) continue;
    uint32_t code[2], more[2] = {0, 0}, s[2], z[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = 2 * p + i;
      code[i] = codes[c * row_words + w];
      if (BITS == 0 && s_slot[c] >= 0) more[i] = high[s_slot[c] * row_words + w];
      s[i] = reinterpret_cast<const uint16_t*>(page + d.key_off_scale)[c * groups + g];
      z[i] = reinterpret_cast<const uint16_t*>(page + d.key_off_zero)[c * groups + g];
    }
    constexpr int PARTS = kColumnParts<BITS>, N = TOK / PARTS;
    uint32_t* to = reinterpret_cast<uint32_t*>(out + (int64_t)t * d.head_dim) + p;
    auto restore = [&](auto affine) {
      affine.template init<0>(s[0] | (s[1] << 16), z[0] | (z[1] << 16));
#pragma unroll
      for (int part = 0; part < PARTS; ++part) {
        uint32_t v[N];
        restore_columns<MD, DT, decltype(affine)::kFp32, BITS>(consts, code, more, affine, part, v);
#pragma unroll
        for (int u = 0; u < N; ++u, to += pairs)
          if (t + part * N + u >= lo && t + part * N + u < hi) *to = v[u];
      }
    };
    if (flavour == DARTKV_DEQUANT_PER_OP) restore(PairAffine<MD, DT, false, true>());
    else restore(PairAffine<MD, DT, true, true>());
  }
}

// Packed value rows [lo, hi) (absolute tokens); out + token * D: the token's output row.
template <int MD, int DT, int BITS>
__device__ __forceinline__ void restore_values(const dartkv_cache_desc& d, int bh, int lo, int hi, int flavour, uint16_t* out) {
  CodeConsts<MD> consts;
  consts.init();
  const int per_row = d.head_dim / 8, items = (hi - lo) * per_row;
  for (int item = threadIdx.x; item < items; item += kSpanThreads) {
    const int t = lo + item / per_row, k = item % per_row, g = 8 * k / d.value_group;
    const int64_t row = (int64_t)bh * d.max_value_tokens + (t - d.sink_tokens);
    const uint8_t* codes = d.v_codes + row * d.value_row_bytes;
    uint64_t q;
    if (BITS == 2) q = reinterpret_cast<const uint16_t*>(codes)[k];
    else if (BITS == 4) q = reinterpret_cast<const uint32_t*>(codes)[k];
    else q = reinterpret_cast<const uint64_t*>(codes)[k];
    const uint16_t* meta = reinterpret_cast<const uint16_t*>(d.v_meta) + row * 2 * d.value_groups + g;
    const uint32_t s = meta[0], z = meta[d.value_groups];
    uint32_t v[4];
    if (flavour == DARTKV_DEQUANT_PER_OP) restore_row<MD, DT, false, BITS>(consts, q, s, z, v);
    else restore_row<MD, DT, true, BITS>(consts, q, s, z, v);
    reinterpret_cast<uint4*>(out + (int64_t)t * d.head_dim)[k] = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

// grid (bh, span, side): span 0 holds the sink tokens, span i the 128 tokens from sink_tokens + 128 * (i - 1) on
template <int MD, int DT>
__global__ void __launch_bounds__(kSpanThreads) materialize_spans_kernel(const __grid_constant__ dartkv_cache_desc d,
                                                                         const __grid_constant__ MaterializeArgs a, int first_span) {
  extern __shared__ int s_slot[];
  wait_previous();
  const int bh = blockIdx.x, side = a.side0 + blockIdx.z, span = first_span + blockIdx.y, D = d.head_dim;
  const int span_lo = span == 0 ? 0 : d.sink_tokens + kSpan * (span - 1);
  const int span_hi = span == 0 ? d.sink_tokens : span_lo + kSpan;
  const int lo = max(a.t0, span_lo), hi = min(a.t1, span_hi);
  if (lo >= hi) return;
  const int packed_hi = span == 0 ? lo : min(hi, max(lo, side == 0 ? d.state[2] : d.state[3]));
  const int64_t row0 = (int64_t)bh * a.out_tokens - a.out_first;
  uint16_t* out = reinterpret_cast<uint16_t*>(side == 0 ? a.out_k : a.out_v);
  if (lo < packed_hi && side == 1) {
    uint16_t* rows = out + row0 * D;
    if (d.value_bits == 2) restore_values<MD, DT, 2>(d, bh, lo, packed_hi, a.flavour, rows);
    else if (d.value_bits == 4) restore_values<MD, DT, 4>(d, bh, lo, packed_hi, a.flavour, rows);
    else restore_values<MD, DT, 8>(d, bh, lo, packed_hi, a.flavour, rows);
  } else if (lo < packed_hi) {
    // pages that were flushed partially filled shift the later ones off the spans: those ranges are walked instead
    const int pg = span - 1;
    const bool aligned = pg < d.state[1] && d.page_start[pg] == span_lo && span_lo + d.page_tokens[pg] >= packed_hi;
    if (!aligned) {
      materialize_tokens(d, bh, 0, lo, packed_hi, row0, a.flavour, out, a.out_dt, s_slot);
    } else {
      const uint8_t* page = d.k_pages + ((int64_t)bh * d.max_key_pages + pg) * d.key_page_bytes;
      uint16_t* rows = out + (row0 + span_lo) * D;
      const int n = d.page_tokens[pg], from = lo - span_lo, to = packed_hi - span_lo;
      if (d.key_mode == DARTKV_MIXED_PAGE) {
        for (int c = threadIdx.x; c < D; c += kSpanThreads) s_slot[c] = -1;
        __syncthreads();
        const int32_t* idx = reinterpret_cast<const int32_t*>(page + d.key_off_index);
        for (int k = threadIdx.x; k < d.promoted; k += kSpanThreads) {
          const int c = idx[k];
          if (c >= 0 && c < D) s_slot[c] = k;
        }
        __syncthreads();
        restore_page<MD, DT, 0>(d, page, n, from, to, a.flavour, rows, s_slot);
      } else if (d.key_bits == 2) restore_page<MD, DT, 2>(d, page, n, from, to, a.flavour, rows, s_slot);
      else if (d.key_bits == 4) restore_page<MD, DT, 4>(d, page, n, from, to, a.flavour, rows, s_slot);
      else restore_page<MD, DT, 8>(d, page, n, from, to, a.flavour, rows, s_slot);
    }
  }
  // dense rows: sinks, or what is not packed yet
  const int pieces = D / 8, dense_lo = max(lo, packed_hi);
  const uint4* src = reinterpret_cast<const uint4*>(span == 0 ? (side == 0 ? d.k_sink : d.v_sink) : (side == 0 ? d.k_ring : d.v_ring));
  for (int i = threadIdx.x; i < (hi - dense_lo) * pieces; i += kSpanThreads) {
    const int t = dense_lo + i / pieces, k = i % pieces;
    const int64_t row = span == 0 ? (int64_t)bh * d.sink_tokens + t : (int64_t)bh * d.ring_tokens + t % d.ring_tokens;
    reinterpret_cast<uint4*>(out + (row0 + t) * D)[k] = src[row * pieces + k];
  }
}

// whole code words per group, 16-byte rows, one dtype on both ends
bool span_shapes(const dartkv_cache_desc* d, const void* out_k, const void* out_v, int out_dtype) {
  const int key_bits = d->key_mode == DARTKV_MIXED_PAGE ? 2 : d->key_bits;
  return (d->dtype == DARTKV_F16 || d->dtype == DARTKV_BF16) && out_dtype == d->dtype &&
         (d->md_dtype == DARTKV_F16 || d->md_dtype == DARTKV_BF16) && d->page_size == kSpan && d->head_dim % 8 == 0 &&
         d->key_group * key_bits % 32 == 0 && d->key_page_bytes % 4 == 0 && d->value_group % 8 == 0 &&
         d->value_row_bytes % 8 == 0 && ((uintptr_t)out_k | (uintptr_t)out_v) % 16 == 0 && (uintptr_t)d->k_pages % 4 == 0 &&
         (uintptr_t)d->v_codes % 8 == 0;
}

constexpr int kMaxGridY = 65535;   // spans or tiles of one launch; longer ranges go in pieces

int launch_materialize(const dartkv_cache_desc* d, int side, int sides, int t0, int t1, int flavour, void* out_k, void* out_v,
                       int out_dtype, cudaStream_t stream) {
  MaterializeArgs a{side, t0, t1, flavour, out_dtype, t0, t1 - t0, out_k, out_v};
  const unsigned bh = d->batch * d->kv_heads;
  const size_t smem = d->head_dim * sizeof(int);
  if (span_shapes(d, out_k, out_v, out_dtype)) {
    auto span_of = [&](int t) { return t < d->sink_tokens ? 0 : 1 + (t - d->sink_tokens) / kSpan; };
    const int end = span_of(t1 - 1) + 1;
    for (int first = span_of(t0); first < end; first += kMaxGridY) {
      const dim3 grid(bh, min(end - first, kMaxGridY), sides);
      const bool half_md = d->md_dtype == DARTKV_F16, half = d->dtype == DARTKV_F16;
      DARTKV_CUDA_OK(launch_following(half_md ? (half ? materialize_spans_kernel<DARTKV_F16,
                                      DARTKV_F16> : materialize_spans_kernel<DARTKV_F16, DARTKV_BF16>)
                                              : (half ? materialize_spans_kernel<DARTKV_BF16, DARTKV_F16> : materialize_spans_kernel<DARTKV_BF16, DARTKV_BF16>),
                                      grid, dim3(kSpanThreads), smem, stream, *d, a, first));
      DARTKV_LAUNCH_OK("materialize_spans_kernel");
    }
    return DARTKV_OK;
  }
  for (int64_t first = t0; first < t1; first += (int64_t)kMaxGridY * kTileTokens) {
    a.t0 = (int)first;
    a.t1 = (int)min((int64_t)t1, first + (int64_t)kMaxGridY * kTileTokens);
    DARTKV_CUDA_OK(launch_following(materialize_kernel, dim3(bh, ceil_div(a.t1 - a.t0, kTileTokens), sides), dim3(kTileThreads), smem,
                                    stream, *d, a));
    DARTKV_LAUNCH_OK("materialize_kernel");
  }
  return DARTKV_OK;
}

}  // namespace

extern "C" int dartkv_cache_materialize(const dartkv_cache_desc* desc, int side, int32_t t0, int32_t t1, int flavour,
                                        void* out, int out_dtype, void* stream) {
  int rc = validate_desc(desc);
  if (rc) return rc;
  DARTKV_REQUIRE(side == 0 || side == 1, "side must be 0 (keys) or 1 (values)");
  DARTKV_REQUIRE(t0 >= 0 && t1 >= t0, "bad token range");
  DARTKV_REQUIRE(dartkv_valid_dtype(out_dtype), "unsupported output dtype");
  DARTKV_REQUIRE(flavour == DARTKV_DEQUANT_PER_OP || flavour == DARTKV_DEQUANT_FP32, "unknown dequant flavour %d", flavour);
  if (t1 == t0) return DARTKV_OK;
  DARTKV_REQUIRE(out != nullptr, "materialize received a null output");
  return launch_materialize(desc, side, 1, t0, t1, flavour, out, out, out_dtype, (cudaStream_t)stream);
}

// Both sides at once (DartKVCache.get, src/dart/cache.py:192-199), one launch.
extern "C" int dartkv_cache_materialize_both(const dartkv_cache_desc* desc, int32_t t0, int32_t t1, int flavour, void* out_k,
                                             void* out_v, int out_dtype, void* stream) {
  int rc = validate_desc(desc);
  if (rc) return rc;
  DARTKV_REQUIRE(t0 >= 0 && t1 >= t0, "bad token range");
  DARTKV_REQUIRE(dartkv_valid_dtype(out_dtype), "unsupported output dtype");
  DARTKV_REQUIRE(flavour == DARTKV_DEQUANT_PER_OP || flavour == DARTKV_DEQUANT_FP32, "unknown dequant flavour %d", flavour);
  if (t1 == t0) return DARTKV_OK;
  DARTKV_REQUIRE(out_k != nullptr && out_v != nullptr, "materialize received a null output");
  return launch_materialize(desc, 0, 2, t0, t1, flavour, out_k, out_v, out_dtype, (cudaStream_t)stream);
}
