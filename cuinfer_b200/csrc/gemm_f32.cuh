// The order in which the 32-bit products add, and the products whose rows start on 16-byte boundaries (gemm_f32.cu).
//
// Every output is summed the same way whichever kernel computes it and however many rows the batch has: chains of
// kChain fused multiply-adds in the order of k; kSlice / kChain chains make a slice; the slices of a group add in order,
// and so do the groups, of which there are at most kMaxGroups.  How K divides into groups depends on K alone, so a kernel
// may give each group to a CTA of its own (a cluster then adds them) and each slice to a lane, and a row's result still
// has the same bits.  A sum of K = 1024 is 16 + 8 + 4 + 2 additions deep, of K = 3072 16 + 8 + 4 + 6.
#pragma once

#include "common.cuh"

namespace cib {

constexpr int kF32Chain = 16;
constexpr int kF32Slice = 128;
constexpr int kF32MaxGroups = 8;

__host__ __device__ inline int f32_slices(int K) { return (K + kF32Slice - 1) / kF32Slice; }
// slices of one group: four, or as many more as keep the groups at kF32MaxGroups
__host__ __device__ inline int f32_group_slices(int K) {
    const int per = (f32_slices(K) + kF32MaxGroups - 1) / kF32MaxGroups;
    return per < 4 ? 4 : per;
}
__host__ __device__ inline int f32_groups(int K) { return (f32_slices(K) + f32_group_slices(K) - 1) / f32_group_slices(K); }

struct GemmF32 {
    const float* a; const float* w; float* out;
    int lda, ldw, ldo, M, N, K;
    long long a_batch, w_batch, o_batch;
    bool w_constant;             // no kernel still in flight writes `w` (a model's loaded weights): it may be read before the wait
};

// Whether the kernels of gemm_f32.cu take these operands: every row of both starts on a 16-byte boundary.
bool gemm_f32_takes(const GemmF32& p, int batch);
// 0: launched, 1: the all-sizes kernel is the faster one for these sizes (it adds in the same order), negative: an error.
int gemm_f32_launch(const GemmF32& p, int batch, cudaStream_t stream);

}  // namespace cib
