// Functional quantizers and dequantizers for 16-bit data whose groups fill whole 32-bit words: the shapes a model's
// keys (groups along the tokens, channels contiguous) and values (groups along the channels) have.  Any other shape
// keeps the kernels of quantize.cu, which handle one group (or element) per thread.
//
// All of these are bound by memory latency and by the few instructions per element, not by capacity: a group's tokens
// are split over up to four threads per channel pair, and requested at once where they fit registers, codes gather in
// registers (quant_math.cuh) and leave as whole words.  fp16 [8,8,1024,128], 2-bit + promoted keys in groups of 128 / 2-bit
// values, a call of the Python API among others, with its allocations and the check of its input: keys with the selection
// 33.7 us (36.7 with the tokens of a column group read twice), values 24.3; all four calls with their waits 92.5 us, 503 with one
// group or element per thread.  The GPU's share of restoring keys is 10.3 us element by element and 6.5 with two codes per
// register (code_pairs.cuh), of values 8.3 and 4.9, some 2 us of each from the form of the launch (B200).

#include <cooperative_groups.h>

#include "code_pairs.cuh"
#include "common.cuh"
#include "quant_math.cuh"

namespace {

constexpr int kSlab = 128;   // columns per block: 64 threads, two neighbouring columns each

// ---------------------------------------------------------------------------- groups along a strided axis
struct ColumnArgs {
  const uint16_t* x;
  int64_t so, sn;                      // element strides of the outer index and of the quantized axis
  int n, inner, group, groups;
  int64_t packed_bytes;                // per (outer, column) row, all groups
  uint8_t *values, *high;              // mixed keys: low plane and promoted high plane
  const int32_t* indices;              // mixed keys: [outer][promoted]
  int promoted, md;
  void *scale, *zero;
  int32_t* nonfinite;
};

// grid (group, slab of columns, outer); 64 threads per token split.  KB: 0 = mixed 2+2-bit keys, else the code width.
// TOK: tokens of a thread, which is the group over the token splits, where that is 8, 16 or 32: all are requested at once and
// kept in registers between the search for minimum and maximum and the codes; 0 for other groups, which read them twice, eight at a time.
template <int DT, int KB, int TOK>
__global__ void __launch_bounds__(256, TOK == 32 ? 2 : 4) quantize_columns_kernel(const __grid_constant__ ColumnArgs a) {
  using P = Pack16<DT>;
  constexpr int PB = KB == 0 ? 2 : KB, CODE_BITS = KB == 0 ? 4 : KB;
  constexpr int PER_HALF = 16 / PB;
  constexpr uint32_t MAGIC = pair_magic<DT, CODE_BITS>();
  wait_previous();
  __shared__ int s_slot[KB == 0 ? kSlab : 1];
  __shared__ uint32_t s_mn[4][64], s_mx[4][64];
  const int p = threadIdx.x & 63, split = threadIdx.x >> 6, splits = blockDim.x >> 6;
  const int g = blockIdx.x, c0 = blockIdx.y * kSlab + 2 * p;
  const int64_t o = blockIdx.z;
  const bool live = c0 < a.inner;      // the column count is even
  if (KB == 0) {
    for (int i = threadIdx.x; i < kSlab; i += blockDim.x) s_slot[i] = -1;
    __syncthreads();
    for (int k = threadIdx.x; k < a.promoted; k += blockDim.x) {
      const int c = a.indices[o * a.promoted + k] - (int)blockIdx.y * kSlab;
      if (c >= 0 && c < kSlab) s_slot[c] = k;
    }
  }
  const int words = a.group * PB / 32, mine = words / splits;           // words per group and plane, of this thread
  const int tok = mine * 2 * PER_HALF, t_begin = g * a.group + split * tok;
  const uint16_t* col = a.x + o * a.so + (live ? c0 : 0);
  // the last group is padded by repeating the final element
  auto at = [&](int t) { return __ldg(reinterpret_cast<const uint32_t*>(col + (int64_t)min(t, a.n - 1) * a.sn)); };
  uint32_t held[TOK > 0 ? TOK : 1];
  uint32_t mn2, mx2;
  if constexpr (TOK > 0) {
#pragma unroll
    for (int j = 0; j < TOK; ++j) held[j] = at(t_begin + j);
    mn2 = mx2 = held[0];
#pragma unroll
    for (int j = 1; j < TOK; ++j) {
      mn2 = P::min2(mn2, held[j]);
      mx2 = P::max2(mx2, held[j]);
    }
  } else {
    mn2 = mx2 = at(t_begin);
#pragma unroll 8
    for (int j = 1; j < tok; ++j) {
      const uint32_t v = at(t_begin + j);
      mn2 = P::min2(mn2, v);
      mx2 = P::max2(mx2, v);
    }
  }
  s_mn[split][p] = mn2;
  s_mx[split][p] = mx2;
  const bool odd = pair_nonfinite<DT>(mn2) || pair_nonfinite<DT>(mx2);
  if (odd && live && a.nonfinite) *a.nonfinite = 1;
  const bool odd_block = __syncthreads_or(odd);
  if (odd_block) {   // Inf or NaN in the block's groups: minimum and maximum leave the NaNs out, like quantize.cu
    mn2 = P::kInfinity; mx2 = P::kInfinity | 0x80008000u;
    for (int j = 0; j < tok; ++j) {
      const uint32_t v = at(t_begin + j);
      mn2 = P::cap2(mn2, v);
      mx2 = P::floor2(mx2, v);
    }
    __syncthreads();
    s_mn[split][p] = mn2;
    s_mx[split][p] = mx2;
    __syncthreads();
  }
  for (int s = 0; s < splits; ++s) { mn2 = P::cap2(mn2, s_mn[s][p]); mx2 = P::floor2(mx2, s_mx[s][p]); }
  if (!live) return;
  const float mn_lo = P::lo(mn2), mn_hi = P::hi(mn2), mx_lo = P::lo(mx2), mx_hi = P::hi(mx2);
  const int slot_lo = KB == 0 ? s_slot[2 * p] : -1, slot_hi = KB == 0 ? s_slot[2 * p + 1] : -1;
  const float qmax_lo = KB == 0 ? (slot_lo >= 0 ? 15.0f : 3.0f) : (float)((1 << CODE_BITS) - 1);
  const float qmax_hi = KB == 0 ? (slot_hi >= 0 ? 15.0f : 3.0f) : (float)((1 << CODE_BITS) - 1);
  float scale_lo = scale_of<DT>(mn_lo, mx_lo, qmax_lo), scale_hi = scale_of<DT>(mn_hi, mx_hi, qmax_hi);
  const int64_t row = o * a.inner + c0;
  if (split == 0) {
    store_f(a.scale, a.md, row * a.groups + g, scale_lo);
    store_f(a.scale, a.md, (row + 1) * a.groups + g, scale_hi);
    store_f(a.zero, a.md, row * a.groups + g, mn_lo);
    store_f(a.zero, a.md, (row + 1) * a.groups + g, mn_hi);
  }
  auto word_at = [&](uint8_t* plane, int64_t r, int w) -> uint32_t& {
    return reinterpret_cast<uint32_t*>(plane + r * a.packed_bytes + (int64_t)g * words * 4)[split * mine + w];
  };
  if (odd_block || isinf(scale_lo) || isinf(scale_hi)) {
    // element by element: the packed arithmetic would give a NaN quotient (Inf / Inf too) the largest code, not code 0
    constexpr uint32_t MASK = (1u << PB) - 1u;
#pragma unroll 1
    for (int w = 0; w < mine; ++w) {
      uint32_t low[2] = {0, 0}, high[2] = {0, 0};
#pragma unroll 1
      for (int u = 0; u < 2 * PER_HALF; ++u) {
        const uint32_t v = at(t_begin + w * 2 * PER_HALF + u);
        const uint32_t code[2] = {group_code(P::lo(v), mn_lo, scale_lo, qmax_lo, DT), group_code(P::hi(v), mn_hi, scale_hi, qmax_hi, DT)};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          low[i] |= (code[i] & MASK) << (PB * u);
          if (KB == 0) high[i] |= (code[i] >> 2) << (PB * u);
        }
      }
      word_at(a.values, row, w) = low[0];
      word_at(a.values, row + 1, w) = low[1];
      if (KB == 0) {
        if (slot_lo >= 0) word_at(a.high, o * a.promoted + slot_lo, w) = high[0];
        if (slot_hi >= 0) word_at(a.high, o * a.promoted + slot_hi, w) = high[1];
      }
    }
    return;
  }
  const float inv_lo = inverse_scale(scale_lo), inv_hi = inverse_scale(scale_hi);
  const uint32_t cap2 = cap_pair<DT>(qmax_lo, qmax_hi);
#pragma unroll (TOK > 0 ? TOK / (2 * PER_HALF) : 1)
  for (int w = 0; w < (TOK > 0 ? TOK / (2 * PER_HALF) : mine); ++w) {
    uint32_t acc_a[2], acc_b[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int base = t_begin + (2 * w + half) * PER_HALF;
      uint32_t x[PER_HALF];
#pragma unroll
      for (int u = 0; u < PER_HALF; ++u) x[u] = TOK > 0 ? held[(2 * w + half) * PER_HALF + u] : at(base + u);
      auto codes = [&](int u) { return pair_codes<DT, CODE_BITS>(x[u], mn2, scale_lo, scale_hi, inv_lo, inv_hi, cap2); };
      if (KB == 0) {
        uint32_t even = 0u - magic_sum(MAGIC, 4, 4), odd = even;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          even = gather(even, codes(2 * u), 4 * u);
          odd = gather(odd, codes(2 * u + 1), 4 * u);
        }
        acc_a[half] = (even & 0x33333333u) | ((odd << 2) & 0xCCCCCCCCu);
        acc_b[half] = ((even >> 2) & 0x33333333u) | (odd & 0xCCCCCCCCu);
      } else {
        uint32_t acc = 0u - magic_sum(MAGIC, PER_HALF, PB);
#pragma unroll
        for (int u = 0; u < PER_HALF; ++u) acc = gather(acc, codes(u), PB * u);
        acc_a[half] = acc;
        acc_b[half] = 0;
      }
    }
    word_at(a.values, row, w) = __byte_perm(acc_a[0], acc_a[1], 0x5410);
    word_at(a.values, row + 1, w) = __byte_perm(acc_a[0], acc_a[1], 0x7632);
    if (KB == 0) {
      if (slot_lo >= 0) word_at(a.high, o * a.promoted + slot_lo, w) = __byte_perm(acc_b[0], acc_b[1], 0x5410);
      if (slot_hi >= 0) word_at(a.high, o * a.promoted + slot_hi, w) = __byte_perm(acc_b[0], acc_b[1], 0x7632);
    }
  }
}

using ColumnsKernel = void (*)(ColumnArgs);
template <int DT, int KB>
ColumnsKernel columns_variant_of(int tok) {
  if (tok == 32) return quantize_columns_kernel<DT, KB, 32>;
  if (tok == 16) return quantize_columns_kernel<DT, KB, 16>;
  return tok == 8 && KB >= 4 ? quantize_columns_kernel<DT, KB, (KB >= 4 ? 8 : 0)> : quantize_columns_kernel<DT, KB, 0>;
}
template <int DT>
ColumnsKernel columns_variant(int kb, int tok) {
  return kb == 0 ? columns_variant_of<DT, 0>(tok) : kb == 2 ? columns_variant_of<DT, 2>(tok)
       : kb == 4 ? columns_variant_of<DT, 4>(tok) : columns_variant_of<DT, 8>(tok);
}

bool is16(int dt) { return dt == DARTKV_F16 || dt == DARTKV_BF16; }
bool fits_int(int64_t v) { return v < (1ll << 31); }

}  // namespace

// Groups along an axis whose columns lie next to each other (inner > 1, stride 1).  key_bits 0: mixed 2+2-bit keys.
// Returns 1 when the launch was made, 0 when the shape is not one of this file, a negative code on a failed launch.
int dartkv_quantize_columns_fast(const void* x, int dtype, int64_t outer, int64_t n, int64_t inner, int64_t so, int64_t sn,
                                 int key_bits, int group, int md, uint8_t* values, uint8_t* high, const int32_t* indices,
                                 int promoted, void* scale, void* zero, int32_t* nonfinite, cudaStream_t stream) {
  const int plane_bits = key_bits == 0 ? 2 : key_bits;
  if (!is16(dtype) || inner < 2 || inner % 2 || so % 2 || sn % 2 || (uintptr_t)x % 4 || (uintptr_t)values % 4 || (uintptr_t)high % 4)
    return 0;
  if ((int64_t)group * plane_bits % 32 || outer > 65535 || !fits_int(n + group) || !fits_int(inner)) return 0;
  const int64_t groups = ceil_div64(n, group), slabs = ceil_div64(inner, kSlab);
  if (slabs > 65535) return 0;
  const int words = (int)((int64_t)group * plane_bits / 32);
  const int splits = words % 4 == 0 ? 4 : words % 2 == 0 ? 2 : 1;
  ColumnArgs a{reinterpret_cast<const uint16_t*>(x), so, sn, (int)n, (int)inner, group, (int)groups,
               groups * (int64_t)words * 4, values, high, indices, promoted, md, scale, zero, nonfinite};
  const dim3 grid((unsigned)groups, (unsigned)slabs, (unsigned)outer);
  DARTKV_CUDA_OK(launch_following(dtype == DARTKV_F16 ? columns_variant<DARTKV_F16>(key_bits, group / splits)
                                                      : columns_variant<DARTKV_BF16>(key_bits, group / splits),
                                  grid, dim3(64 * splits), 0, stream, a));
  DARTKV_LAUNCH_OK("quantize_columns_kernel");
  return 1;
}

// ---------------------------------------------------------------------------- groups along contiguous elements
namespace {

// Eight elements per thread, group / 8 neighbouring lanes per group (a power of two up to a warp).
template <int DT, int VB>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const uint16_t* __restrict__ x, int64_t rows, int n, int64_t so,
                                                            int group, int md, uint8_t* __restrict__ values, void* scale_out,
                                                            void* zero_out, int32_t* nonfinite) {
  using P = Pack16<DT>;
  wait_previous();
  // the eighths of a row are numbered through all rows: whole groups in order, so neither the group's number nor this
  // lane's place in it needs a division, and the row only where rows are not contiguous
  const int per_row = n / 8, lanes = group / 8;
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = id < rows * per_row;
  int64_t at = live ? 8 * id : 0;
  if (so != n && live) {
    const int64_t row = id < (1ll << 31) ? (int64_t)((uint32_t)id / (uint32_t)per_row) : id / per_row;
    at = row * so + 8 * (id - row * per_row);
  }
  const uint4 raw = *reinterpret_cast<const uint4*>(x + at);
  const uint32_t v[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t mn2 = P::min2(P::min2(v[0], v[1]), P::min2(v[2], v[3])), mx2 = P::max2(P::max2(v[0], v[1]), P::max2(v[2], v[3]));
  for (int off = 1; off < lanes; off <<= 1) {
    mn2 = P::min2(mn2, __shfl_xor_sync(0xffffffffu, mn2, off));
    mx2 = P::max2(mx2, __shfl_xor_sync(0xffffffffu, mx2, off));
  }
  const bool odd = pair_nonfinite<DT>(mn2) || pair_nonfinite<DT>(mx2), odd_warp = __any_sync(0xffffffffu, odd);
  if (odd_warp) {   // Inf or NaN in the warp's groups: minimum and maximum leave the NaNs out, like quantize.cu
    mn2 = P::kInfinity; mx2 = P::kInfinity | 0x80008000u;
#pragma unroll
    for (int i = 0; i < 4; ++i) { mn2 = P::cap2(mn2, v[i]); mx2 = P::floor2(mx2, v[i]); }
    for (int off = 1; off < lanes; off <<= 1) {
      mn2 = P::cap2(mn2, __shfl_xor_sync(0xffffffffu, mn2, off));
      mx2 = P::floor2(mx2, __shfl_xor_sync(0xffffffffu, mx2, off));
    }
  }
  if (!live) return;   // groups lie wholly inside or outside
  const uint32_t mn1 = P::cap2(mn2, mn2 >> 16), mx1 = P::floor2(mx2, mx2 >> 16);
  const float mn = P::lo(mn1), mx = P::lo(mx1);
  constexpr float qmax = (float)((1 << VB) - 1);
  const float scale = scale_of<DT>(mn, mx, qmax), inv = inverse_scale(scale);
  const uint32_t mnp = (mn1 & 0xFFFFu) * 0x00010001u, cap2 = cap_pair<DT>(qmax, qmax);
  constexpr int PAIRS = 8 / VB, GATHERS = 4 / PAIRS;     // pairs per gathered 16 bits, gathers per thread
  constexpr uint32_t MAGIC = pair_magic<DT, VB>();
  constexpr uint32_t LOMASK = VB == 2 ? 0x3333u : VB == 4 ? 0x0F0Fu : 0x00FFu;
  uint32_t half_word[GATHERS];
#pragma unroll
  for (int g = 0; g < GATHERS; ++g) {
    uint32_t acc = 0u - magic_sum(MAGIC, PAIRS, 2 * VB);
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) acc = gather(acc, pair_codes<DT, VB>(v[g * PAIRS + i], mnp, scale, scale, inv, inv, cap2), 2 * VB * i);
    half_word[g] = (acc & LOMASK) | ((acc >> (16 - VB)) & (LOMASK << VB));
  }
  if (odd_warp || isinf(scale)) {
    // element by element: the packed arithmetic gives a NaN quotient (Inf / Inf too) the largest code, not code 0
    uint64_t codes = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      codes |= (uint64_t)group_code(P::lo(v[i]), mn, scale, qmax, DT) << (2 * i * VB);
      codes |= (uint64_t)group_code(P::hi(v[i]), mn, scale, qmax, DT) << ((2 * i + 1) * VB);
    }
#pragma unroll
    for (int g = 0; g < GATHERS; ++g) half_word[g] = (uint32_t)(codes >> (16 * g)) & 0xFFFFu;
  }
  if (VB == 2) reinterpret_cast<uint16_t*>(values)[id] = (uint16_t)half_word[0];
  else if (VB == 4) reinterpret_cast<uint32_t*>(values)[id] = half_word[0] | (half_word[GATHERS / 2] << 16);
  else reinterpret_cast<uint2*>(values)[id] = make_uint2(half_word[0] | (half_word[GATHERS > 1] << 16),
                                                         half_word[GATHERS / 2] | (half_word[GATHERS - 1] << 16));
  if (((int)id & (lanes - 1)) == 0) {   // a power of two, which divides the eighths of a row
    if (nonfinite && odd) *nonfinite = 1;
    const int64_t g = id >> (31 - __clz(lanes));
    store_f(scale_out, md, g, scale);
    store_f(zero_out, md, g, mn);
  }
}

template <int DT>
auto rows_variant(int bits) {
  return bits == 2 ? quantize_rows_kernel<DT, 2> : bits == 4 ? quantize_rows_kernel<DT, 4> : quantize_rows_kernel<DT, 8>;
}

}  // namespace

// Whole groups of 8..256 contiguous elements (a power of two); return value as above.
int dartkv_quantize_rows_fast(const void* x, int dtype, int64_t rows, int64_t n, int64_t so, int bits, int group, int md,
                              uint8_t* values, void* scale, void* zero, int32_t* nonfinite, cudaStream_t stream) {
  if (!is16(dtype) || group < 8 || group > 256 || (group & (group - 1)) || n % group || so % 8 || (uintptr_t)x % 16 ||
      (uintptr_t)values % 8 || !fits_int(n))
    return 0;
  const int64_t blocks = ceil_div64(rows * (n / 8), 256);
  if (!fits_int(blocks)) return 0;
  DARTKV_CUDA_OK(launch_following(dtype == DARTKV_F16 ? rows_variant<DARTKV_F16>(bits) : rows_variant<DARTKV_BF16>(bits),
                                  dim3((unsigned)blocks),
                                  dim3(256), 0, stream, reinterpret_cast<const uint16_t*>(x), rows, (int)n, so, group, md, values, scale,
                                  zero, nonfinite));
  DARTKV_LAUNCH_OK("quantize_rows_kernel");
  return 1;
}

// ---------------------------------------------------------------------------- channel scores and selection
namespace {

constexpr int kScoreSplits = 16, kScoreBlocks = 8;

// Promoted channels of one (batch, head): sum |k| per channel in double, scores rounded to the data dtype, rank by (score
// descending, channel ascending).  In fp16 the sum is exact in any order.  bf16 values can be further apart than a double
// has bits; the error is then some 2^-50 of the sum, which changes the score only where the sum lies that close to a
// boundary of the fp32 rounding that follows.  A cluster of blocks, each of 16 token splits x 64
// channel pairs, shares a row's tokens and meets in the first block's shared memory; scores (optional) are written too.
template <int DT>
__global__ void __launch_bounds__(64 * kScoreSplits) score_select_kernel(const uint16_t* __restrict__ keys, int64_t tokens, int d,
                                                                         int64_t sbh, int64_t st, int count,
                                                                         uint16_t* scores, int32_t* indices) {
  using P = Pack16<DT>;
  wait_previous();
  __shared__ double s_sum[kScoreSplits][2][64];
  __shared__ double s_all[kScoreBlocks][128];   // the blocks' sums, in the first one
  __shared__ uint32_t s_key[128];
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int blocks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int p = threadIdx.x & 63, split = threadIdx.x >> 6;
  const int64_t r = blockIdx.x / blocks;
  double lo = 0.0, hi = 0.0;
  if (2 * p < d) {
    // the blocks' tokens lie one after another: with a step that depends on the number of blocks the compiler tests the end
    // between the loads instead of requesting eight at a time ([32,8,4096,128] fp16, the whole call 283 us so, 214 here)
    const int64_t share = ceil_div64(tokens, blocks), end = min(tokens, (rank + 1) * share);
    const uint16_t* col = keys + r * sbh + 2 * p;
#pragma unroll 8
    for (int64_t t = rank * share + split; t < end; t += kScoreSplits) {
      const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(col + t * st));
      lo += (double)fabsf(P::lo(v));
      hi += (double)fabsf(P::hi(v));
    }
  }
  s_sum[split][0][p] = lo;
  s_sum[split][1][p] = hi;
  __syncthreads();
  const int c = threadIdx.x;
  uint32_t key = 0;
  double sum = 0.0;
  if (c < d) {
#pragma unroll
    for (int s = 0; s < kScoreSplits; ++s) sum += s_sum[s][c & 1][c >> 1];
  }
  if (blocks > 1) {
    cluster.sync();   // every block of the cluster has started
    if (c < d) *cluster.map_shared_rank(&s_all[rank][c], 0) = sum;
    cluster.sync();
    if (rank > 0) return;
    sum = 0.0;
    for (int k = 0; k < blocks && c < d; ++k) sum += s_all[k][c];
  }
  if (c < d) {
    const uint16_t bits = P::bits(__fdiv_rn((float)sum, (float)tokens));
    if (scores) scores[r * d + c] = bits;
    // scores are non-negative 16-bit floats: their bit patterns order like integers
    key = ((uint32_t)bits << 7) | (uint32_t)(127 - c);
    s_key[c] = key;
  }
  if (indices == nullptr) return;
  __syncthreads();
  if (c < d) {
    int rank = 0;
    for (int o = 0; o < d; ++o) rank += s_key[o] > key;
    if (rank < count) indices[r * count + rank] = c;
  }
}

}  // namespace

// keys [bh][tokens][d] with strides; scores and indices may be null.  Return value as above.
int dartkv_score_select_fast(const void* keys, int dtype, int64_t bh, int64_t tokens, int64_t d, int64_t sbh, int64_t st,
                             int count, void* scores, int32_t* indices, cudaStream_t stream) {
  if (!is16(dtype) || d > 128 || d % 2 || sbh % 2 || st % 2 || (uintptr_t)keys % 4 || !fits_int(bh)) return 0;
  const uint16_t* k = reinterpret_cast<const uint16_t*>(keys);
  uint16_t* s = reinterpret_cast<uint16_t*>(scores);
  // blocks per row: as many as the SMs hold at a time (two on each; with twice as many [8,8,512,128] takes 34.0 us instead of
  // 28.2, [8,8,4096,128] 68.4 instead of 65.1), with at least 128 tokens each ([4,8,512,128]: 25.2 us, with 64 tokens 27.1, one
  // block a row 26.5; [4,8,1024,128]: 28.3, one block a row 30.8; whole quantize_key_mixed calls)
  int blocks = 1;
  while (blocks < kScoreBlocks && bh * blocks * 2 <= 2 * dartkv_sm_count() && tokens >= 128 * blocks * 2) blocks *= 2;
  DARTKV_CUDA_OK(launch_clusters(blocks, dtype == DARTKV_F16 ? score_select_kernel<DARTKV_F16> : score_select_kernel<DARTKV_BF16>,
                                 dim3((unsigned)(bh * blocks)), dim3(64 * kScoreSplits), 0, stream, k, tokens, (int)d, sbh, st, count, s,
                                 indices));
  DARTKV_LAUNCH_OK("score_select_kernel");
  return 1;
}

// ---------------------------------------------------------------------------- dequantization
namespace {

struct RestoreArgs {
  const uint8_t *values, *high;
  const int32_t* indices;
  int promoted;
  const void *scale, *zero;
  int n, inner, group, groups, flavour;
  int64_t packed_bytes, so, sn;
  void* out;
};

// Groups along a strided axis: a thread restores the tokens of one code word for two neighbouring columns.
// grid (words / 4, slab of columns, outer), 256 threads = 64 column pairs x 4 words.  BITS 0: mixed keys.
template <int MD, int OUT, int BITS>
__global__ void __launch_bounds__(256) restore_columns_kernel(const __grid_constant__ RestoreArgs a) {
  constexpr int PB = BITS == 0 ? 2 : BITS, TOK = 32 / PB;
  wait_previous();
  __shared__ int s_slot[BITS == 0 ? kSlab : 1];
  const int64_t o = blockIdx.z;
  if (BITS == 0) {
    for (int i = threadIdx.x; i < kSlab; i += blockDim.x) s_slot[i] = -1;
    __syncthreads();
    for (int k = threadIdx.x; k < a.promoted; k += blockDim.x) {
      const int c = a.indices[o * a.promoted + k] - (int)blockIdx.y * kSlab;
      if (c >= 0 && c < kSlab) s_slot[c] = k;
    }
    __syncthreads();
  }
  const int p = threadIdx.x & 63, w = blockIdx.x * 4 + (threadIdx.x >> 6);
  const int c0 = blockIdx.y * kSlab + 2 * p, t0 = w * TOK;
  if (c0 >= a.inner || t0 >= a.n) return;
  const int g = t0 / a.group;
  const int64_t row = o * a.inner + c0;
  uint32_t code[2], high[2] = {0, 0}, s[2], z[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    code[i] = reinterpret_cast<const uint32_t*>(a.values + (row + i) * a.packed_bytes)[w];
    if (BITS == 0) {
      const int slot = s_slot[2 * p + i];
      if (slot >= 0) high[i] = reinterpret_cast<const uint32_t*>(a.high + (o * a.promoted + slot) * a.packed_bytes)[w];
    }
    s[i] = reinterpret_cast<const uint16_t*>(a.scale)[(row + i) * a.groups + g];
    z[i] = reinterpret_cast<const uint16_t*>(a.zero)[(row + i) * a.groups + g];
  }
  CodeConsts<MD> consts;
  consts.init();
  constexpr int PARTS = kColumnParts<BITS>, N = TOK / PARTS;
  uint16_t* out = reinterpret_cast<uint16_t*>(a.out) + o * a.so + (int64_t)t0 * a.sn + c0;
  auto restore = [&](auto affine) {
    affine.template init<0>(s[0] | (s[1] << 16), z[0] | (z[1] << 16));
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
      uint32_t v[N];
      restore_columns<MD, OUT, decltype(affine)::kFp32, BITS>(consts, code, high, affine, part, v);
#pragma unroll
      for (int u = 0; u < N; ++u, out += a.sn)
        if (t0 + part * N + u < a.n) *reinterpret_cast<uint32_t*>(out) = v[u];
    }
  };
  if (a.flavour == DARTKV_DEQUANT_PER_OP) restore(PairAffine<MD, OUT, false, true>());
  else restore(PairAffine<MD, OUT, true, true>());
}

// Groups along contiguous elements: a thread restores eight of them.
template <int MD, int OUT, int BITS>
__global__ void __launch_bounds__(256) restore_rows_kernel(const __grid_constant__ RestoreArgs a, int64_t total) {
  wait_previous();
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= total) return;
  // whole groups follow one another through all rows; divisions in 32 bits where they do
  const int eighths = a.group / 8;
  int64_t at = 8 * id, g;
  if (total < (1ll << 31)) {
    g = (uint32_t)id / (uint32_t)eighths;
    if (a.so != a.n) {
      const uint32_t row = (uint32_t)id / (uint32_t)(a.n / 8);
      at = row * a.so + 8 * ((uint32_t)id - row * (uint32_t)(a.n / 8));
    }
  } else {
    const int64_t row = id / (a.n / 8);
    g = id / eighths;
    at = row * a.so + 8 * (id - row * (a.n / 8));
  }
  uint64_t codes;
  if (BITS == 2) codes = reinterpret_cast<const uint16_t*>(a.values)[id];
  else if (BITS == 4) codes = reinterpret_cast<const uint32_t*>(a.values)[id];
  else codes = reinterpret_cast<const uint64_t*>(a.values)[id];
  const uint32_t s = reinterpret_cast<const uint16_t*>(a.scale)[g], z = reinterpret_cast<const uint16_t*>(a.zero)[g];
  CodeConsts<MD> consts;
  consts.init();
  uint32_t v[4];
  if (a.flavour == DARTKV_DEQUANT_PER_OP) restore_row<MD, OUT, false, BITS>(consts, codes, s, z, v);
  else restore_row<MD, OUT, true, BITS>(consts, codes, s, z, v);
  *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(a.out) + at) = make_uint4(v[0], v[1], v[2], v[3]);
}

template <int MD, int OUT>
cudaError_t launch_restore(bool columns, int bits, dim3 grid, cudaStream_t stream, const RestoreArgs& a, int64_t total) {
  if (columns)
    return launch_following(bits == 0   ? restore_columns_kernel<MD, OUT, 0>
                            : bits == 2 ? restore_columns_kernel<MD, OUT, 2>
                            : bits == 4 ? restore_columns_kernel<MD, OUT, 4>
                                        : restore_columns_kernel<MD, OUT, 8>,
                            grid, dim3(256), 0, stream, a);
  return launch_following(bits == 2   ? restore_rows_kernel<MD, OUT, 2>
                          : bits == 4 ? restore_rows_kernel<MD, OUT, 4>
                                      : restore_rows_kernel<MD, OUT, 8>,
                          grid, dim3(256), 0, stream, a, total);
}
cudaError_t launch_restore_typed(int md, int out_dtype, bool columns, int bits, dim3 grid, cudaStream_t stream, const RestoreArgs& a,
                                 int64_t total) {
  if (md == DARTKV_F16 && out_dtype == DARTKV_F16) return launch_restore<DARTKV_F16, DARTKV_F16>(columns, bits, grid, stream, a, total);
  if (md == DARTKV_F16) return launch_restore<DARTKV_F16, DARTKV_BF16>(columns, bits, grid, stream, a, total);
  if (out_dtype == DARTKV_F16) return launch_restore<DARTKV_BF16, DARTKV_F16>(columns, bits, grid, stream, a, total);
  return launch_restore<DARTKV_BF16, DARTKV_BF16>(columns, bits, grid, stream, a, total);
}

}  // namespace

// Inverse of dartkv_quantize_columns_fast; return value as above.
int dartkv_restore_columns_fast(const uint8_t* values, const uint8_t* high, const int32_t* indices, int promoted,
                                const void* scale, const void* zero, int md, int64_t outer, int64_t n, int64_t inner,
                                int key_bits, int group, int flavour, void* out, int out_dtype, int64_t so, int64_t sn,
                                cudaStream_t stream) {
  const int plane_bits = key_bits == 0 ? 2 : key_bits;
  if (!is16(md) || !is16(out_dtype) || inner < 2 || inner % 2 || so % 2 || sn % 2 || (uintptr_t)out % 4 || (uintptr_t)values % 4 ||
      (uintptr_t)high % 4 || (int64_t)group * plane_bits % 32 || outer > 65535 || !fits_int(n + group) || !fits_int(inner))
    return 0;
  const int64_t groups = ceil_div64(n, group), words = groups * (int64_t)group * plane_bits / 32, slabs = ceil_div64(inner, kSlab);
  if (slabs > 65535) return 0;
  RestoreArgs a{values, high, indices, promoted, scale, zero, (int)n, (int)inner, group, (int)groups, flavour, words * 4, so, sn, out};
  const dim3 grid((unsigned)ceil_div64(words, 4), (unsigned)slabs, (unsigned)outer);
  DARTKV_CUDA_OK(launch_restore_typed(md, out_dtype, true, key_bits, grid, stream, a, 0));
  DARTKV_LAUNCH_OK("restore_columns_kernel");
  return 1;
}

// Inverse of dartkv_quantize_rows_fast (any group that is a multiple of eight); return value as above.
int dartkv_restore_rows_fast(const uint8_t* values, const void* scale, const void* zero, int md, int64_t rows, int64_t n, int bits,
                             int group, int flavour, void* out, int out_dtype, int64_t so, cudaStream_t stream) {
  if (!is16(md) || !is16(out_dtype) || n % group || group % 8 || so % 8 || (uintptr_t)out % 16 || (uintptr_t)values % 8 || !fits_int(n))
    return 0;
  const int64_t total = rows * (n / 8), blocks = ceil_div64(total, 256);
  if (!fits_int(blocks)) return 0;
  RestoreArgs a{values, nullptr, nullptr, 0, scale, zero, (int)n, 1, group, (int)(n / group), flavour, 0, so, 1, out};
  DARTKV_CUDA_OK(launch_restore_typed(md, out_dtype, false, bits, dim3((unsigned)blocks), stream, a, total));
  DARTKV_LAUNCH_OK("restore_rows_kernel");
  return 1;
}
