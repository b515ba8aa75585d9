// decode_many_kernel for fp16 caches with bf16 metadata.

#include "decode_many.cuh"

int dartkv_decode_many_f16_bf16(const DecodeManyCall& call) { return many_launch<DARTKV_F16, DARTKV_BF16>(call); }
