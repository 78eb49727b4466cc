// out[M, N] = a[M, K] · w[N, K]^T on the ordinary 32-bit FMA pipe, for any M, N, K.
//
// The reference sends every projection to cuBLAS with 32-bit accumulation
// (csrc/ops/projection.cu:13-45).  This kernel is the fallback for shapes that the tensor-core kernels and the
// 32-bit kernels of gemm_f32.cu refuse (rows off 16-byte boundaries) or would be slower at.  Every output element of 32-bit
// operands adds in the order that gemm_f32.cuh lays down, so a row's result depends neither on how many other rows are in
// the batch nor on which kernel its address lets through; bfloat16 operands add chains of 16 values in the order of k.
#include "gemm_f32.cuh"

namespace cib {

constexpr int kBM = 64, kBN = 64, kBK = kF32Chain;

// GROUPS: 0: every chain of 16 joins one sum (bfloat16 operands: no other kernel has to give the same bits); 1 and 2: the order
// of gemm_f32.cuh for K of one group and of several.  The groups' sums, touched every 128 of K, lie in shared memory: in
// registers they left an SM two CTAs instead of four (467 x 4 095 x 1 023 in 32 bits: 190 us, so 183).
template <typename TI, typename TO, int GROUPS>
__global__ void __launch_bounds__(256)
gemm_generic_kernel(const TI* __restrict__ a, int lda, const TI* __restrict__ w, int ldw,
                    TO* __restrict__ out, int ldo, int M, int N, int K, long long a_batch, long long w_batch,
                    long long o_batch) {
    // blockIdx.z is the index of a batch of independent products (one per head, say): its operands lie the given
    // numbers of elements apart
    a += (size_t)blockIdx.z * a_batch;
    w += (size_t)blockIdx.z * w_batch;
    out += (size_t)blockIdx.z * o_batch;
    __shared__ float As[kBK][kBM + 4];
    __shared__ float Ws[kBK][kBN + 4];
    __shared__ float s_group[GROUPS > 0 ? 16 : 1][256], s_total[GROUPS > 1 ? 16 : 1][256];          // [output][thread]
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
    const int tx = tid & 15, ty = tid >> 4;       // 16 x 16 threads, 4 x 4 outputs each
    const int group_k = f32_group_slices(K) * kF32Slice;
    float slice[4][4] = {};
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        if (GROUPS > 0) s_group[e][tid] = 0.f;
        if (GROUPS > 1) s_total[e][tid] = 0.f;
    }

    // each thread loads 4 elements of each tile per step: row = tid / 4, k = (tid % 4) * 4 ..
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    for (int k0 = 0; k0 < K; k0 += kBK) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = k0 + lk + e;
            const int am = m0 + lrow, wn = n0 + lrow;
            As[lk + e][lrow] = (am < M && k < K) ? to_f32(a[(size_t)am * lda + k]) : 0.f;
            Ws[lk + e][lrow] = (wn < N && k < K) ? to_f32(w[(size_t)wn * ldw + k]) : 0.f;
        }
        __syncthreads();
        float part[4][4] = {};
#pragma unroll
        for (int kk = 0; kk < kBK; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j] = fmaf(av[i], wv[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) slice[i][j] += part[i][j];
        const int done = k0 + kBK;
        if (GROUPS > 0 && (done % kF32Slice == 0 || done >= K)) {
            const bool group_ends = GROUPS > 1 && (done % group_k == 0 || done >= K);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int e = i * 4 + j;
                    const float sum = s_group[e][tid] + slice[i][j];
                    slice[i][j] = 0.f;
                    s_group[e][tid] = group_ends ? 0.f : sum;
                    if (group_ends) s_total[e][tid] += sum;
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(GROUPS == 0 ? slice[i][j] : GROUPS == 1 ? s_group[i * 4 + j][tid] : s_total[i * 4 + j][tid]);
        }
    }
}

}  // namespace cib

using namespace cib;

static int gemm_generic_launch(const void* a, int lda, long long a_batch, const void* w, int ldw, long long w_batch,
                               int in_dtype, void* out, int ldo, long long o_batch, int out_dtype, int M, int N, int K,
                               int batch, int w_constant, cudaStream_t stream) {
    CIB_REQUIRE(M >= 0 && N > 0 && K > 0 && batch > 0, "gemm: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
    CIB_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm: leading dimensions too small (lda=%d ldw=%d ldo=%d)", lda, ldw, ldo);
    if (M == 0) return 0;
    if (in_dtype == kF32 && out_dtype == kF32) {
        const GemmF32 p{(const float*)a, (const float*)w, (float*)out, lda, ldw, ldo, M, N, K, a_batch, w_batch, o_batch, w_constant != 0};
        if (gemm_f32_takes(p, batch)) {
            const int rc = gemm_f32_launch(p, batch, stream);
            if (rc <= 0) return rc;
        }
    }
    dim3 grid((N + kBN - 1) / kBN, (M + kBM - 1) / kBM, batch);
    CIB_REQUIRE(grid.y <= 65535 && batch <= 65535, "gemm: M=%d or batch=%d too large for this kernel", M, batch);
    if (in_dtype == kF32 && out_dtype == kF32)
        (f32_groups(K) == 1 ? gemm_generic_kernel<float, float, 1> : gemm_generic_kernel<float, float, 2>)<<<grid, 256, 0, stream>>>((const float*)a, lda, (const float*)w, ldw, (float*)out, ldo, M, N, K, a_batch, w_batch, o_batch);
    else if (in_dtype == kBF16 && out_dtype == kBF16)
        gemm_generic_kernel<__nv_bfloat16, __nv_bfloat16, 0><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)a, lda, (const __nv_bfloat16*)w, ldw, (__nv_bfloat16*)out, ldo, M, N, K, a_batch, w_batch, o_batch);
    else if (in_dtype == kBF16 && out_dtype == kF32)
        gemm_generic_kernel<__nv_bfloat16, float, 0><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)a, lda, (const __nv_bfloat16*)w, ldw, (float*)out, ldo, M, N, K, a_batch, w_batch, o_batch);
    else
        CIB_REQUIRE(false, "gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
    CIB_LAUNCH_CHECK("gemm_generic");
    return 0;
}

// w_constant: no kernel still in flight in the stream writes `w`; without it a kernel launched early waits before it reads `w`.
extern "C" int cib_gemm_generic(const void* a, int lda, const void* w, int ldw, int in_dtype, void* out, int ldo,
                                int out_dtype, int M, int N, int K, int w_constant, cudaStream_t stream) {
    return gemm_generic_launch(a, lda, 0, w, ldw, 0, in_dtype, out, ldo, 0, out_dtype, M, N, K, 1, w_constant, stream);
}

// `batch` independent products out[b] = a[b] . w[b]^T whose operands lie a_batch / w_batch / o_batch elements apart
// (heads side by side inside wider rows: the batch stride is then smaller than the leading dimension).
extern "C" int cib_gemm_generic_batched(const void* a, int lda, long long a_batch, const void* w, int ldw,
                                        long long w_batch, int in_dtype, void* out, int ldo, long long o_batch,
                                        int out_dtype, int M, int N, int K, int batch, int w_constant, cudaStream_t stream) {
    return gemm_generic_launch(a, lda, a_batch, w, ldw, w_batch, in_dtype, out, ldo, o_batch, out_dtype, M, N, K, batch, w_constant, stream);
}
