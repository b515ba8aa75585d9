// decode_many_kernel for bf16 caches with bf16 metadata.

#include "decode_many.cuh"

int dartkv_decode_many_bf16(const DecodeManyCall& call) { return many_launch<DARTKV_BF16, DARTKV_BF16>(call); }
