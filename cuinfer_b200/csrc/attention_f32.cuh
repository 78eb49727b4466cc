// The 32-bit attention of attention_f32.cu, as attention_generic.cu calls it.
#pragma once

#include "common.cuh"

namespace cib {

struct AttnF32 {
    const float* q; float* out; const float* cache; const int* block_table; const int* query_start_loc; const int* seq_lens;
    const int* token_request;
    int q_stride, out_stride, num_pages, page_size, table_stride, num_tokens, num_requests, nq, nkv, window;
    float scale;
};

// 1: launched, 0: not a call these kernels take (head sizes other than 64 and 128, rows off 16-byte boundaries), negative: an error.
int attention_f32_try(const AttnF32& p, int d, cudaStream_t stream);

}  // namespace cib
