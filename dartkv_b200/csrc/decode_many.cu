// Host side of decode_many.cuh: row groups, work split and the choice of the translation unit that has the kernels of the call's types.

#include "decode_many.cuh"

int dartkv_decode_many_bf16(const DecodeManyCall& call);
int dartkv_decode_many_bf16_f16(const DecodeManyCall& call);
int dartkv_decode_many_f16_bf16(const DecodeManyCall& call);
int dartkv_decode_many_f16(const DecodeManyCall& call);

// `rep` query rows per KV head run as this many groups of equal size (the last one may be smaller)
int dartkv_decode_many_groups(int rep) { return (rep + 31) / 32; }

// Blocks per work row (batch, KV head, row group) for that many pages.  Blocks run in waves of two per SM; a block costs its steps
// (pages, and for the dense tokens one or two more) and about two more for the query, the first page's latency and the partial.
int dartkv_decode_many_pieces(const dartkv_cache_desc* d, int rep, int pages) {
  const ManyGeom w = many_geometry(d, rep);
  const int per_sm = 2 * (many_smem(d, w) + 1024) <= 228 * 1024 ? 2 : 1;
  const long long rows = (long long)d->batch * d->kv_heads * w.groups, resident = (long long)per_sm * dartkv_sm_count();
  const int quads = (pages + 3) / 4;
  int best = 1;
  double best_cost = 1e30;
  for (int pieces = 1; pieces <= 16 && pieces <= quads; ++pieces) {
    const double share = (pages + 1 + pieces - 1) / pieces + 2.0;
    const double cost = share * ((rows * pieces + resident - 1) / resident);
    if (cost < best_cost - 1e-9) { best_cost = cost; best = pieces; }
  }
  return best;
}

int dartkv_decode_many_launch(const dartkv_cache_desc* d, const void* query, int query_heads, float scale, int pieces, int total_splits,
                              float* part_m, float* part_l, float* part_acc, int* status, const int32_t* row_start, cudaStream_t stream) {
  const DecodeManyCall call{d, query, query_heads, scale, pieces, total_splits, part_m, part_l, part_acc, status, row_start, stream};
  if (d->dtype == DARTKV_BF16) return d->md_dtype == DARTKV_BF16 ? dartkv_decode_many_bf16(call) : dartkv_decode_many_bf16_f16(call);
  return d->md_dtype == DARTKV_BF16 ? dartkv_decode_many_f16_bf16(call) : dartkv_decode_many_f16(call);
}
