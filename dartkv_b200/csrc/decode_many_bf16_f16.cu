// decode_many_kernel for bf16 caches with fp16 metadata.

#include "decode_many.cuh"

int dartkv_decode_many_bf16_f16(const DecodeManyCall& call) { return many_launch<DARTKV_BF16, DARTKV_F16>(call); }
