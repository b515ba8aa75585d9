// Append step for the common geometry: head_dim 128, 16-bit data, 128-token key pages with one 128-token key group,
// value groups of 16/32/64/128 channels.  One kernel does a whole step: quantize + pack the key pages, quantize +
// pack the value rows, copy the dense sink / ring rows and publish the page table and the state words.
//
// Grid (head, batch row, page of the step and role): a block of 256 threads takes the 128 key tokens of a page or the 128
// value rows beside it.  The ring rows a step reads are those of its first page only, so the block of that page also
// writes the step's dense rows of its side, after a block barrier: no ordering between blocks is needed, and a
// generation-time append is one launch instead of three.
//
// Keys: thread (tq, p) owns the channel pair (2p, 2p+1) of 32 tokens (quarter tq of the page) and keeps them in
// registers as packed 16-bit pairs: one pass for min / max / sum|k|, the splits' statistics combined in shared
// memory, the rank of the 128 channels by one integer key, then the codes.  Values: four lanes per token row
// (32 channels per lane), group min/max by xor-shuffles.
//
// What bounds it: the instruction stream.  Per pair of elements the quantizer needs a subtract, two unpacks, two
// multiplies, a pack, the rounding add and a cap; gathering the codes is one shift-add per pair (the magic exponents
// are subtracted once per register, and 4-bit codes split into their low and high plane once per eight tokens).
// HBM traffic per page: 64 KiB read (K and V rows), 10.6 KiB written (2-bit, 32 promoted).
// The arithmetic is the reference's per-op rounding in the data dtype
// (src/dart/quantization.py:178-186, src/dart/mixed.py:200-209).

#include "common.cuh"
#include "append_common.cuh"
#include "quant_math.cuh"

namespace {

constexpr int kD = 128;
constexpr int kP = 128;
constexpr int kThreads = 256;
constexpr int kSplits = 4;              // token splits of a key page
constexpr int kTok = kP / kSplits;      // tokens per thread

struct RowSource {
  const void* chunk;
  const void* ring;
  int64_t sb, sh, st;
  int chunk_start, ring_tokens;
  // base pointers of this block's (batch, head): chunk rows then ring rows
  __device__ __forceinline__ void bases(int bh, const uint16_t*& chunk_base, const uint16_t*& ring_base) const {
    chunk_base = reinterpret_cast<const uint16_t*>(chunk) + (int64_t)blockIdx.y * sb + (int64_t)blockIdx.x * sh;
    ring_base = reinterpret_cast<const uint16_t*>(ring) + (int64_t)bh * ring_tokens * kD;
  }
  __device__ __forceinline__ const uint16_t* row_from(const uint16_t* chunk_base, const uint16_t* ring_base, int t) const {
    if (t >= chunk_start) return chunk_base + (int64_t)(t - chunk_start) * st;
    return ring_base + (t % ring_tokens) * kD;
  }
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The dense rows of a step for one (batch, head) and side, 64 rows at a time with 16 lanes per row: load() brings
// a batch into registers (beside the loads of the page, so that a small step waits for memory once), store() puts
// it into the sink and ring rows once the block has read the ring.
template <int DT>
struct DenseBatch {
  static constexpr int ROWS = 4;   // rows per thread
  uint4 v[ROWS];
  const uint16_t* chunk;
  uint4 *sink, *ring;
  int sink_copy, ring_first, rows, ring_begin, chunk_start, ring_tokens;
  int64_t st;

  __device__ __forceinline__ void init(const dartkv_cache_desc& d, const RowSource& src, const dartkv_append_plan& plan,
                                       int bh, int role) {
    const DenseRows r = dense_rows(plan);
    const uint16_t* ring_base;
    src.bases(bh, chunk, ring_base);
    sink = reinterpret_cast<uint4*>(role == 0 ? d.k_sink : d.v_sink) + (int64_t)bh * d.sink_tokens * 16;
    ring = reinterpret_cast<uint4*>(role == 0 ? d.k_ring : d.v_ring) + (int64_t)bh * d.ring_tokens * 16;
    sink_copy = plan.sink_copy; ring_first = r.ring_first; rows = r.rows;
    ring_begin = role == 0 ? plan.ring_begin : plan.value_end;
    chunk_start = src.chunk_start; ring_tokens = src.ring_tokens; st = src.st;
  }
  __device__ __forceinline__ int chunk_row(int r) const { return r < sink_copy ? r : ring_first + (r - sink_copy); }
  __device__ __forceinline__ void load(int first) {
    const int piece = threadIdx.x & 15;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const int r = first + (threadIdx.x >> 4) + 16 * k;
      if (r < rows) v[k] = reinterpret_cast<const uint4*>(chunk + (int64_t)chunk_row(r) * st)[piece];
    }
  }
  __device__ __forceinline__ bool store(int first) {   // whether a stored element is Inf or NaN
    const int piece = threadIdx.x & 15;
    bool bad = false;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const int r = first + (threadIdx.x >> 4) + 16 * k;
      if (r >= rows) continue;
      const int t = chunk_start + chunk_row(r);
      if (r >= sink_copy && t < ring_begin) continue;
      bad |= piece_nonfinite(v[k], DT);
      if (r < sink_copy) sink[t * 16 + piece] = v[k];
      else ring[(t % ring_tokens) * 16 + piece] = v[k];
    }
    return bad;
  }
  // the batch in registers, then whatever rows are left
  __device__ __forceinline__ bool store_all() {
    bool bad = store(0);
    for (int first = 16 * ROWS; first < rows; first += 16 * ROWS) {
      load(first);
      bad |= store(first);
    }
    return bad;
  }
};

struct KeySmem {
  __align__(16) uint32_t page[kP * 64];   // [token][channel pair]
  uint32_t mn[kSplits][64], mx[kSplits][64];
  float sum[2][kSplits][64];        // [low | high channel]
  double exact[2][kSplits][64];
  __align__(16) uint32_t score[64];
  int rank[kSplits][kD];            // [block of 32 others][channel]
};

// One key page.  KBITS: 0 = mixed 2+2-bit keys, else uniform keys with KBITS bits.
template <int DT, int KBITS>
__device__ __forceinline__ bool key_page(const dartkv_cache_desc& d, const RowSource& src, KeySmem& sm, int bh, int pg,
                                         int first_slot, int num_pages, int page_token_start,
                                         const int32_t* __restrict__ indices, DenseBatch<DT>& dense) {
  using P = Pack16<DT>;
  const int p = threadIdx.x & 63, tq = threadIdx.x >> 6;
  const uint16_t *chunk_base, *ring_base;
  src.bases(bh, chunk_base, ring_base);
  // stage the page: piece threadIdx % 16 of rows threadIdx / 16, + 16, ...
  {
    const int piece = threadIdx.x & 15, r0 = threadIdx.x >> 4, first = page_token_start + pg * kP;
    uint32_t* to = sm.page + r0 * 64 + piece * 4;
    if (first >= src.chunk_start) {
      const uint16_t* from = chunk_base + (int64_t)(first - src.chunk_start + r0) * src.st + piece * 8;
      if (src.st == kD) {   // rows of one head lie together: every address is the first one plus a constant
#pragma unroll
        for (int k = 0; k < kP / 16; ++k) cp_async16(to + k * 1024, from + k * 16 * kD);
      } else {
#pragma unroll
        for (int k = 0; k < kP / 16; ++k, from += 16 * src.st) cp_async16(to + k * 1024, from);
      }
    } else {                // the first tokens of the page wait in the ring
#pragma unroll
      for (int k = 0; k < kP / 16; ++k)
        cp_async16(to + k * 1024, src.row_from(chunk_base, ring_base, first + r0 + 16 * k) + piece * 8);
    }
  }
  if (dense.rows > 0) dense.load(0);
  cp_async_wait_all();
  __syncthreads();
  bool bad = false;
  if (dense.rows > 0) bad = dense.store_all();   // every ring row of the page has been read
  const uint32_t* x = sm.page + (tq * kTok) * 64 + p;   // + 64 * token
  uint8_t* page = d.k_pages + ((int64_t)bh * d.max_key_pages + first_slot + pg) * d.key_page_bytes;
  // the scores are only needed when the kernel ranks the channels itself
  const bool ranked = KBITS == 0 && indices == nullptr && d.promoted > 0 && d.promoted < kD;

  // pass 1: packed min / max (NaN-propagating, so Inf/NaN inputs surface in them) and sum |k| per channel.  The score
  // is the exact sum rounded to fp32, divided and rounded to the data dtype.  bf16: an fp32 sum decides it unless the
  // rounding boundary lies within the sum's error (about 1 page in 16 has such a channel), then the block sums again in
  // double; fp16 scores have 11 bits and almost
  // every page would, so they are summed in double at once.
  uint32_t mn2 = x[0], mx2 = mn2;
  float part_lo[2] = {0.0f, 0.0f}, part_hi[2] = {0.0f, 0.0f};
  double e_lo = 0.0, e_hi = 0.0;
#pragma unroll
  for (int j = 0; j < kTok; ++j) {
    const uint32_t v = x[64 * j];
    mn2 = P::min2(mn2, v);
    mx2 = P::max2(mx2, v);
    if (KBITS == 0 && DT == DARTKV_BF16) { part_lo[j & 1] += fabsf(P::lo(v)); part_hi[j & 1] += fabsf(P::hi(v)); }
    if (KBITS == 0 && DT == DARTKV_F16) { e_lo += (double)fabsf(P::lo(v)); e_hi += (double)fabsf(P::hi(v)); }
  }
  float sum_lo = part_lo[0] + part_lo[1], sum_hi = part_hi[0] + part_hi[1];
  sm.mn[tq][p] = mn2;
  sm.mx[tq][p] = mx2;
  if (KBITS == 0 && DT == DARTKV_BF16) { sm.sum[0][tq][p] = sum_lo; sm.sum[1][tq][p] = sum_hi; }
  if (KBITS == 0 && DT == DARTKV_F16) { sm.exact[0][tq][p] = e_lo; sm.exact[1][tq][p] = e_hi; }
  __syncthreads();
  mn2 = sm.mn[0][p];
  mx2 = sm.mx[0][p];
#pragma unroll
  for (int o = 1; o < kSplits; ++o) { mn2 = P::min2(mn2, sm.mn[o][p]); mx2 = P::max2(mx2, sm.mx[o][p]); }
  const float mn_lo = P::lo(mn2), mn_hi = P::hi(mn2), mx_lo = P::lo(mx2), mx_hi = P::hi(mx2);
  bad |= !(isfinite(mn_lo) && isfinite(mn_hi) && isfinite(mx_lo) && isfinite(mx_hi));

  int slot_lo = -1, slot_hi = -1;
  float qmax_lo, qmax_hi;
  if (KBITS == 0) {
    const int K = d.promoted;
    int32_t* idx_field = reinterpret_cast<int32_t*>(page + d.key_off_index);
    const int c_lo = 2 * p, c_hi = 2 * p + 1;
    if (indices != nullptr) {
      const int32_t* mine = indices + ((int64_t)bh * num_pages + pg) * K;
      for (int k = 0; k < K; ++k) {
        const int ch = mine[k];
        if (ch == c_lo) slot_lo = k;
        if (ch == c_hi) slot_hi = k;
      }
      for (int k = threadIdx.x; k < K; k += kThreads) idx_field[k] = mine[k];
    } else if (K == kD) {
      slot_lo = c_lo; slot_hi = c_hi;
      if (tq == 0) { idx_field[c_lo] = c_lo; idx_field[c_hi] = c_hi; }
    } else if (ranked) {
      // score bits of a channel from its sum
      auto score = [](float sum) -> uint32_t { return P::bits(__fmul_rn(sum, 1.0f / kP)); };   // a power of two: exact like the division
      uint32_t score_lo = 0, score_hi = 0;
      bool unsure = true;
      if (DT == DARTKV_BF16) {
        sum_lo = (sm.sum[0][0][p] + sm.sum[0][1][p]) + (sm.sum[0][2][p] + sm.sum[0][3][p]);
        sum_hi = (sm.sum[1][0][p] + sm.sum[1][1][p]) + (sm.sum[1][2][p] + sm.sum[1][3][p]);
        // 15 additions per partial sum and three more: at most 18 rounding errors of 2^-24 each, and one of the product
        constexpr float kError = 20.0f / 16777216.0f, kBelow = 1.0f - kError, kAbove = 1.0f + kError;
        score_lo = score(sum_lo * kBelow);
        score_hi = score(sum_hi * kBelow);
        unsure = score_lo != score(sum_lo * kAbove) || score_hi != score(sum_hi * kAbove) ||
                 !(sum_lo < 1e37f) || !(sum_hi < 1e37f);
      }
      const bool exact = DT == DARTKV_F16 || __syncthreads_or(unsure);
      if (exact) {
        if (DT == DARTKV_BF16) {
#pragma unroll 8
          for (int j = 0; j < kTok; ++j) {
            const uint32_t again = x[64 * j];
            e_lo += (double)fabsf(P::lo(again));
            e_hi += (double)fabsf(P::hi(again));
          }
          sm.exact[0][tq][p] = e_lo;
          sm.exact[1][tq][p] = e_hi;
          __syncthreads();
        }
        e_lo = (sm.exact[0][0][p] + sm.exact[0][1][p]) + (sm.exact[0][2][p] + sm.exact[0][3][p]);
        e_hi = (sm.exact[1][0][p] + sm.exact[1][1][p]) + (sm.exact[1][2][p] + sm.exact[1][3][p]);
        score_lo = score((float)e_lo);
        score_hi = score((float)e_hi);
      }
      // Rank by (score descending, channel ascending).  Scores are non-negative 16-bit floats, so their bit patterns
      // order like integers with NaN above everything: each channel has a rank of its own whatever the keys hold.  The
      // 128 x 128 comparisons go as 16 squares of 32 channels against 32 others, two squares per warp, lane = channel,
      // two others per subtraction: bit 15 of (other | 0x8000) - than is set where other >= than (than is at most
      // 0x8000, so the halves do not borrow from each other), and the 2 x 16 bits of a square are counted at once.  A
      // channel with the same score counts if it comes first, i.e. against the score itself instead of the next number.
      if (tq == 0) sm.score[p] = score_lo | (score_hi << 16) | 0x80008000u;
      __syncthreads();
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int mine = warp >> 1, others = 2 * (warp & 1) + i;     // blocks of 32 channels
        const uint32_t bits = reinterpret_cast<const uint16_t*>(sm.score)[32 * mine + lane] & 0x7FFFu;
        const uint32_t from = bits * 0x00010001u, above = from + 0x00010001u;
        uint32_t flags = 0;
        auto compare = [&](uint32_t other, uint32_t than) { flags = (flags >> 1) | ((other - than) & 0x80008000u); };
        const uint4* o4 = reinterpret_cast<const uint4*>(sm.score) + 4 * others;
        if (others != mine) {
          const uint32_t than = others < mine ? from : above;
#pragma unroll
          for (int r4 = 0; r4 < 4; ++r4) {
            const uint4 o = o4[r4];
            compare(o.x, than); compare(o.y, than); compare(o.z, than); compare(o.w, than);
          }
        } else {   // others 2r and 2r + 1 of the channel's own block come before it, after it, or on both sides
          const uint32_t both = lane & 1 ? (from & 0xFFFFu) | (above & 0xFFFF0000u) : above;
#pragma unroll
          for (int r = 0; r < 16; ++r) compare(sm.score[16 * others + r], r < lane >> 1 ? from : (r == lane >> 1 ? both : above));
        }
        sm.rank[others][32 * mine + lane] = __popc(flags);
      }
      __syncthreads();
      int rank_lo, rank_hi;
      rank_lo = 0; rank_hi = 0;
#pragma unroll
      for (int o = 0; o < kSplits; ++o) {
        const int2 r = *reinterpret_cast<const int2*>(&sm.rank[o][c_lo]);
        rank_lo += r.x; rank_hi += r.y;
      }
      if (rank_lo < K) { slot_lo = rank_lo; if (tq == 0) idx_field[rank_lo] = c_lo; }
      if (rank_hi < K) { slot_hi = rank_hi; if (tq == 0) idx_field[rank_hi] = c_hi; }
    }
    qmax_lo = slot_lo >= 0 ? 15.0f : 3.0f;
    qmax_hi = slot_hi >= 0 ? 15.0f : 3.0f;
  } else {
    qmax_lo = qmax_hi = (float)((1 << KBITS) - 1);
  }
  float scale_lo = scale_of<DT>(mn_lo, mx_lo, qmax_lo), scale_hi = scale_of<DT>(mn_hi, mx_hi, qmax_hi);
  if (tq == 0) {
    store_pair(page + d.key_off_scale, d.md_dtype, p, scale_lo, scale_hi);
    store_pair(page + d.key_off_zero, d.md_dtype, p, mn_lo, mn_hi);
  }
  const float inv_lo = inverse_scale(scale_lo), inv_hi = inverse_scale(scale_hi);
  if (DT == DARTKV_F16) {   // an infinite scale enters the quotient as zero
    scale_lo = isinf(scale_lo) ? 0.0f : scale_lo;
    scale_hi = isinf(scale_hi) ? 0.0f : scale_hi;
  }
  const uint32_t cap2 = cap_pair<DT>(qmax_lo, qmax_hi);

  // pass 2: the codes of a channel pair gather in registers, channel 2p in the low half and 2p+1 in the high half,
  // 16 / BITS tokens each; two such registers split into one 32-bit word per channel.
  constexpr int BITS = KBITS == 0 ? 2 : KBITS;      // bits per stored plane
  constexpr int PER_HALF = 16 / BITS;               // tokens per 16-bit half of a plane word
  constexpr int WORDS = kP / (2 * PER_HALF);        // 32-bit words per channel and plane
  constexpr int MY_WORDS = WORDS / kSplits;         // words of this split: 2, 4 or 8
  constexpr uint32_t MAGIC = pair_magic<DT, KBITS == 0 ? 4 : KBITS>();
  constexpr int CHUNK = MY_WORDS < 4 ? 2 : 4;       // words per store
#pragma unroll
  for (int w0 = 0; w0 < MY_WORDS; w0 += CHUNK) {
    uint32_t a_lo[CHUNK], a_hi[CHUNK], b_lo[CHUNK], b_hi[CHUNK];   // a: low plane, b: high plane
#pragma unroll
    for (int w = 0; w < CHUNK; ++w) {
      uint32_t acc_a[2], acc_b[2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int base = (2 * (w0 + w) + half) * PER_HALF;
        auto codes = [&](int j) {
          return pair_codes<DT, KBITS == 0 ? 4 : KBITS>(x[64 * j], mn2, scale_lo, scale_hi, inv_lo, inv_hi, cap2);
        };
        if (KBITS == 0) {
          // 4-bit codes of the even and of the odd tokens as nibbles, then the planes of all eight tokens at once
          uint32_t even = 0u - magic_sum(MAGIC, 4, 4), odd = even;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            even = gather(even, codes(base + 2 * u), 4 * u);
            odd = gather(odd, codes(base + 2 * u + 1), 4 * u);
          }
          acc_a[half] = (even & 0x33333333u) | ((odd << 2) & 0xCCCCCCCCu);
          acc_b[half] = ((even >> 2) & 0x33333333u) | (odd & 0xCCCCCCCCu);
        } else {
          uint32_t acc = 0u - magic_sum(MAGIC, PER_HALF, BITS);
#pragma unroll
          for (int u = 0; u < PER_HALF; ++u) acc = gather(acc, codes(base + u), BITS * u);
          acc_a[half] = acc;
          acc_b[half] = 0;
        }
      }
      a_lo[w] = __byte_perm(acc_a[0], acc_a[1], 0x5410);
      a_hi[w] = __byte_perm(acc_a[0], acc_a[1], 0x7632);
      b_lo[w] = __byte_perm(acc_b[0], acc_b[1], 0x5410);
      b_hi[w] = __byte_perm(acc_b[0], acc_b[1], 0x7632);
    }
    auto store_words = [&](uint8_t* row, const uint32_t (&v)[CHUNK]) {
      uint32_t* to = reinterpret_cast<uint32_t*>(row) + tq * MY_WORDS + w0;
      if (CHUNK == 2) *reinterpret_cast<uint2*>(to) = make_uint2(v[0], v[1]);
      else *reinterpret_cast<uint4*>(to) = make_uint4(v[0], v[1], v[CHUNK - 2], v[CHUNK - 1]);
    };
    store_words(page + (2 * p) * (WORDS * 4), a_lo);
    store_words(page + (2 * p + 1) * (WORDS * 4), a_hi);
    if (KBITS == 0) {
      if (slot_lo >= 0) store_words(page + d.key_off_high + slot_lo * (WORDS * 4), b_lo);
      if (slot_hi >= 0) store_words(page + d.key_off_high + slot_hi * (WORDS * 4), b_hi);
    }
  }
  return bad;
}

// 128 value rows from `first` (relative to value_begin; rows past `count` are skipped): four lanes per token row,
// 32 channels per lane, so a warp holds eight rows and a block goes twice over 64.  A group is half a lane
// (value_group 16), one lane (32), or 2 / 4 neighbouring lanes.
template <int DT, int VBITS>
__device__ __forceinline__ bool value_rows(const dartkv_cache_desc& d, const RowSource& src, int bh, int first,
                                           int value_begin, int count) {
  using P = Pack16<DT>;
  constexpr int ROWS = 2;               // rows per thread, all loads in flight together
  const int lane = threadIdx.x & 31, part = lane & 3;
  const int row0 = first + (threadIdx.x >> 2);
  const uint16_t *chunk_base, *ring_base;
  src.bases(bh, chunk_base, ring_base);
  bool bad = false;
  if (first + (threadIdx.x & ~31) / 4 >= count) return bad;   // the whole warp is past the end
  const bool from_ring = value_begin + first < src.chunk_start;   // only blocks of the step's first rows
  uint4 raw[ROWS][4];
#pragma unroll
  for (int s = 0; s < ROWS; ++s) {
    const int t = value_begin + min(row0 + 64 * s, count - 1);
    const uint16_t* row = chunk_base + (int64_t)(t - src.chunk_start) * src.st;
    if (from_ring && t < src.chunk_start) row = ring_base + (t % src.ring_tokens) * kD;
    const uint4* ptr = reinterpret_cast<const uint4*>(row + part * 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) raw[s][i] = ptr[i];
  }
  constexpr float qmax = (float)((1 << VBITS) - 1);
  const uint32_t cap2 = cap_pair<DT>(qmax, qmax);
  const bool half_lane = d.value_group == 16;
  const int lanes = d.value_group >> 5;   // lanes per group
#pragma unroll
  for (int s = 0; s < ROWS; ++s) {
    uint32_t x[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) { x[4 * i] = raw[s][i].x; x[4 * i + 1] = raw[s][i].y; x[4 * i + 2] = raw[s][i].z; x[4 * i + 3] = raw[s][i].w; }
    uint32_t mn2[2], mx2[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mn2[h] = mx2[h] = x[8 * h];
#pragma unroll
      for (int i = 1; i < 8; ++i) { mn2[h] = P::min2(mn2[h], x[8 * h + i]); mx2[h] = P::max2(mx2[h], x[8 * h + i]); }
    }
    if (!half_lane) {
      mn2[0] = P::min2(mn2[0], mn2[1]);
      mx2[0] = P::max2(mx2[0], mx2[1]);
      for (int off = 1; off < lanes; off <<= 1) {
        mn2[0] = P::min2(mn2[0], __shfl_xor_sync(0xffffffffu, mn2[0], off));
        mx2[0] = P::max2(mx2[0], __shfl_xor_sync(0xffffffffu, mx2[0], off));
      }
      mn2[1] = mn2[0];
      mx2[1] = mx2[0];
    }
    float mn[2], scale[2], inv[2], s_q[2];
    uint32_t mnp[2];
    const bool live = row0 + 64 * s < count;
    auto group = [&](int h) {
      // NaN-propagating min / max: any Inf or NaN of the group ends up in mn or mx
      const uint32_t mn1 = P::min2(mn2[h], mn2[h] >> 16), mx1 = P::max2(mx2[h], mx2[h] >> 16);
      mn[h] = P::lo(mn1);
      const float mx = P::lo(mx1);
      bad |= live && !(isfinite(mn[h]) && isfinite(mx));
      scale[h] = scale_of<DT>(mn[h], mx, qmax);
      inv[h] = inverse_scale(scale[h]);
      s_q[h] = DT == DARTKV_F16 && isinf(scale[h]) ? 0.0f : scale[h];
      mnp[h] = (mn1 & 0xFFFFu) * 0x00010001u;
    };
    group(0);
    if (half_lane) {
      group(1);
    } else {
      mn[1] = mn[0]; scale[1] = scale[0]; inv[1] = inv[0]; s_q[1] = s_q[0]; mnp[1] = mnp[0];
    }
    // codes of 8 / VBITS pairs gather in one register (even channels in the low half, odd ones in the high half)
    constexpr int PAIRS = 8 / VBITS;                      // pairs per gather register
    constexpr int GATHERS = 16 / PAIRS;
    constexpr uint32_t MAGIC = pair_magic<DT, VBITS>();
    constexpr uint32_t LOMASK = VBITS == 2 ? 0x3333u : VBITS == 4 ? 0x0F0Fu : 0x00FFu;
    uint32_t half_word[GATHERS];
#pragma unroll
    for (int g = 0; g < GATHERS; ++g) {
      uint32_t acc = 0u - magic_sum(MAGIC, PAIRS, 2 * VBITS);
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) {
        const int k = g * PAIRS + i, h = k / 8;
        acc = gather(acc, pair_codes<DT, VBITS>(x[k], mnp[h], s_q[h], s_q[h], inv[h], inv[h], cap2), 2 * VBITS * i);
      }
      half_word[g] = (acc & LOMASK) | ((acc >> (16 - VBITS)) & (LOMASK << VBITS));
    }
    if (!live) continue;
    const int64_t out_row = (int64_t)bh * d.max_value_tokens + (value_begin + row0 + 64 * s - d.sink_tokens);
    uint32_t* codes = reinterpret_cast<uint32_t*>(d.v_codes + out_row * d.value_row_bytes) + part * (GATHERS / 2);
    if (VBITS == 2) {
      *reinterpret_cast<uint2*>(codes) = make_uint2(half_word[0] | (half_word[1] << 16), half_word[2] | (half_word[3] << 16));
    } else {
#pragma unroll
      for (int g = 0; g + 7 < GATHERS; g += 8)
        reinterpret_cast<uint4*>(codes)[g / 8] = make_uint4(half_word[g] | (half_word[g + 1] << 16), half_word[g + 2] | (half_word[g + 3] << 16),
                                                            half_word[g + 4] | (half_word[g + 5] << 16), half_word[g + 6] | (half_word[g + 7] << 16));
    }
    if (half_lane) {
      const int64_t pair = out_row * d.value_groups + part;       // groups 2*part, 2*part + 1 of the scale row
      store_pair(d.v_meta, d.md_dtype, pair, scale[0], scale[1]);
      store_pair(d.v_meta, d.md_dtype, pair + d.value_groups / 2, mn[0], mn[1]);
    } else if ((part & (lanes - 1)) == 0) {
      const int g = part >> (lanes >> 1);   // lanes per group: 1, 2 or 4
      store_f(d.v_meta, d.md_dtype, (out_row * 2 + 0) * d.value_groups + g, scale[0]);
      store_f(d.v_meta, d.md_dtype, (out_row * 2 + 1) * d.value_groups + g, mn[0]);
    }
  }
  return bad;
}

struct StepArgs {
  RowSource source;                        // strides of the chunk; pointers and first token are set per block
  const void *keys, *values;
  dartkv_append_plan plan;
  const dartkv_append_plan* device_plan;   // where the plan was made on the device: *plan then only sizes the grid
  const int32_t* indices;
  int32_t* nonfinite;
  int roles, role_begin;                   // 2: keys and values; 1: role_begin only (0 keys, 1 values)
  int copies;                              // the step's dense rows and metadata are written here
};

// KBITS as in key_page().  Four blocks per SM (64 registers, 42 KB of shared memory each): 32 warps, every block's page
// in flight as asynchronous copies.
template <int DT, int KBITS, int VBITS>
__global__ void __launch_bounds__(kThreads, 4) append_step_kernel(const __grid_constant__ dartkv_cache_desc d,
                                                                  const __grid_constant__ StepArgs a) {
  __shared__ KeySmem sm;
  wait_previous();
  // read through the pointer where it is needed: the plan's numbers are not kept in registers across the page code
  const dartkv_append_plan& plan = a.device_plan ? *a.device_plan : a.plan;
  // grid: (kv head, batch row, page and role): no division to find any of them
  const int bh = blockIdx.y * gridDim.x + blockIdx.x;
  const int pg = a.roles == 2 ? blockIdx.z >> 1 : blockIdx.z, role = a.roles == 2 ? (int)(blockIdx.z & 1) : a.role_begin;
  RowSource src = a.source;
  src.chunk = role == 0 ? a.keys : a.values;
  src.ring = role == 0 ? d.k_ring : d.v_ring;
  src.chunk_start = plan.chunk_start;
  const bool writes_dense = a.copies && pg == 0;
  if (writes_dense && bh == 0 && role == 0) publish_append(d, plan);
  bool bad = false;
  DenseBatch<DT> dense;
  dense.rows = 0;
  if (role == 0 && pg < plan.num_pages) {
    if (writes_dense) dense.init(d, src, plan, bh, role);
    bad = key_page<DT, KBITS>(d, src, sm, bh, pg, plan.first_page, plan.num_pages, plan.page_token_start, a.indices, dense);
  } else {
    if (role == 1 && pg * kP < plan.value_end - plan.value_begin)
      bad = value_rows<DT, VBITS>(d, src, bh, pg * kP, plan.value_begin, plan.value_end - plan.value_begin);
    if (writes_dense) {
      // value blocks are done well before the key blocks: their dense rows come last
      dense.init(d, src, plan, bh, role);
      __syncthreads();   // every ring row of these values has been read
      dense.load(0);
      bad |= dense.store_all();
    }
  }
  if (bad && a.nonfinite) *a.nonfinite = 1;
}

using StepKernel = void (*)(dartkv_cache_desc, StepArgs);
template <int DT, int KBITS>
StepKernel step_variant_v(int value_bits) {
  return value_bits == 2 ? append_step_kernel<DT, KBITS, 2> : value_bits == 4 ? append_step_kernel<DT, KBITS, 4>
                                                                              : append_step_kernel<DT, KBITS, 8>;
}
template <int DT>
StepKernel step_variant_k(int key_bits, int value_bits) {
  switch (key_bits) {
    case 0: return step_variant_v<DT, 0>(value_bits);
    case 2: return step_variant_v<DT, 2>(value_bits);
    case 4: return step_variant_v<DT, 4>(value_bits);
    default: return step_variant_v<DT, 8>(value_bits);
  }
}

int launch_step(const dartkv_cache_desc& d, StepArgs a, int blocks, int roles, cudaStream_t stream) {
  DARTKV_REQUIRE(blocks * roles <= 65535, "too many pages in one append (limit 65535)");
  DARTKV_REQUIRE(d.batch <= 65535, "batch above 65535");
  a.roles = roles;
  const int key_bits = d.key_mode == DARTKV_MIXED_PAGE ? 0 : d.key_bits;
  const StepKernel kernel = d.dtype == DARTKV_F16 ? step_variant_k<DARTKV_F16>(key_bits, d.value_bits)
                                                  : step_variant_k<DARTKV_BF16>(key_bits, d.value_bits);
  DARTKV_CUDA_OK(launch_following(kernel, dim3(d.kv_heads, d.batch, blocks * roles), dim3(kThreads), 0, stream, d, a));
  DARTKV_LAUNCH_OK("append_step_kernel");
  return DARTKV_OK;
}

}  // namespace

// bit 0: the keys of the step have the geometry of this file; bit 1: its values have
int dartkv_append_fast_supported(const dartkv_cache_desc* d, const dartkv_append_plan* p, int64_t st) {
  if ((d->dtype != DARTKV_F16 && d->dtype != DARTKV_BF16) || d->head_dim != kD || st % 8) return 0;
  int ok = 0;
  if (d->page_size == kP && d->key_group == kP && (p->num_pages == 0 || p->last_page_tokens == kP) &&
      (d->key_mode == DARTKV_QUANTIZED_PAGE || d->promoted <= kD))
    ok |= 1;
  if (d->value_group == 16 || d->value_group == 32 || d->value_group == 64 || d->value_group == 128) ok |= 2;
  return ok;
}

// device_plan (optional): the step's plan in device memory, written by a kernel earlier on the stream; *p then
// only sizes the grid (the most pages / rows the step can bring)
static StepArgs step_args(const dartkv_cache_desc* d, const dartkv_append_plan* p, const void* keys, const void* values,
                          int64_t sb, int64_t sh, int64_t st, const int32_t* indices, int32_t* nonfinite,
                          const dartkv_append_plan* device_plan) {
  StepArgs a{};
  a.source = RowSource{nullptr, nullptr, sb, sh, st, p->chunk_start, d->ring_tokens};
  a.keys = keys;
  a.values = values;
  a.plan = *p;
  a.device_plan = device_plan;
  a.indices = indices;
  a.nonfinite = nonfinite;
  return a;
}

// Whether one launch can do the whole step: the value rows are those of the key pages, no page but the first
// reads the ring (a local window longer than a page leaves more than a page waiting there), and keys and values of all
// pages fit the grid's 65,535 layers together.
int dartkv_append_fast_whole_step(const dartkv_append_plan* p) {
  const bool same_rows = p->num_pages == 0 ? p->value_end <= p->value_begin
                                           : p->value_begin == p->page_token_start &&
                                                 p->value_end == p->page_token_start + p->num_pages * kP;
  return same_rows && p->num_pages <= 65535 / 2 && (p->num_pages <= 1 || p->page_token_start + kP >= p->chunk_start);
}

int dartkv_append_fast_step(const dartkv_cache_desc* d, const dartkv_append_plan* p, const void* keys, const void* values,
                            int64_t sb, int64_t sh, int64_t st, const int32_t* indices, int32_t* nonfinite,
                            cudaStream_t stream, const dartkv_append_plan* device_plan) {
  StepArgs a = step_args(d, p, keys, values, sb, sh, st, indices, nonfinite, device_plan);
  a.copies = 1;
  return launch_step(*d, a, max(1, p->num_pages), 2, stream);
}

int dartkv_append_fast_keys(const dartkv_cache_desc* d, const dartkv_append_plan* p, const void* keys, int64_t sb,
                            int64_t sh, int64_t st, const int32_t* indices, int32_t* nonfinite, cudaStream_t stream,
                            const dartkv_append_plan* device_plan) {
  if (p->num_pages == 0) return DARTKV_OK;
  return launch_step(*d, step_args(d, p, keys, nullptr, sb, sh, st, indices, nonfinite, device_plan), p->num_pages, 1, stream);
}

int dartkv_append_fast_values(const dartkv_cache_desc* d, const dartkv_append_plan* p, const void* values, int64_t sb,
                              int64_t sh, int64_t st, int32_t* nonfinite, cudaStream_t stream,
                              const dartkv_append_plan* device_plan) {
  if (p->value_end <= p->value_begin) return DARTKV_OK;
  StepArgs a = step_args(d, p, nullptr, values, sb, sh, st, nullptr, nonfinite, device_plan);
  a.role_begin = 1;
  return launch_step(*d, a, ceil_div(p->value_end - p->value_begin, kP), 1, stream);
}
