// The prompt attention variant for launches of few CTAs (attention_tcgen05_wide.cu), as attention_tcgen05.cu calls it.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace cib {

// Keys of one tile, and at most of one box of `kv_map`: the map is made for the variant that is launched.
constexpr int kWideKeys = 128;

int attention_tcgen05_wide(const CUtensorMap& kv_map, int num_pages, const __nv_bfloat16* q, int q_stride, __nv_bfloat16* out,
                           int out_stride, int page_size, const int* block_table, int table_stride, const int* query_start_loc,
                           const int* seq_lens, int num_requests, int least_query, int num_tiles, int nq, int nkv, float scale_log2, int window,
                           int joined, const float* sinks, int* error_flag, cudaStream_t stream);

}  // namespace cib
