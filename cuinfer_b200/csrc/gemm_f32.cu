// out[M, N] = a[M, K] · w[N, K]^T in true 32-bit arithmetic, for rows on 16-byte boundaries: a kernel for few rows, which
// is a stream over the weights, and one for many, which is bound by the fused multiply-adds.  Both add in the order that
// gemm_f32.cuh lays down, so a row's result does not depend on which of them computed it.
//
// Measured beside the kernel that took every size before (64 x 64 tiles of one CTA each, K in one piece, no copies ahead):
// a decode step of 3 rows of the 0.6B layer sizes 10 to 14 us a projection instead of 160, the output head of 622 MB 170 us
// (3.7 TB/s; 129 us at one row); 467 rows x 4096 x 1024 140 us (28 TFLOP/s).
#include "gemm_f32.cuh"
#include "mma_utils.cuh"

#include <cooperative_groups.h>
#include <stddef.h>

namespace cib {

// ---- few rows ----------------------------------------------------------------------------------------------------------
// A warp takes 8 output features x 512 of K: all of its 16 KB of weights are on their way to shared memory before it looks
// at the activations (with programmatic dependent launch, and where the caller says that nothing in flight writes the
// weights, before the kernel that computes the activations has ended), so an SM has its
// whole share of a projection in flight at once.  A lane then owns one feature and one slice of 128: its chains need no
// exchange with other lanes, and only the slices' sums meet in shared memory, once.  Rows of the weights lie 2 064 bytes
// apart and slices of the activations 528: eight lanes read eight weight rows without a bank conflict, and the warp's
// four slices of an activation row lie in four different banks.
constexpr int kFewFeatures = 8;
constexpr int kFewChunk = 512;                        // of K, per warp and round
constexpr int kFewWRow = kFewChunk * 4 + 16;          // bytes
constexpr int kFewARow = 4 * (kF32Slice * 4 + 16);    // bytes
constexpr int kFewMaxWarps = 6;
constexpr int kFewRows = 8;                           // rows of one pass

template <int MT>
__global__ void __launch_bounds__(kFewMaxWarps * 32, 2)
gemm_f32_few_kernel(const GemmF32 p, int rounds) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    unsigned char* s_w = smem + (size_t)warp * (kFewFeatures * kFewWRow + MT * kFewARow);
    unsigned char* s_a = s_w + kFewFeatures * kFewWRow;
    float* s_sum = reinterpret_cast<float*>(smem + (size_t)warps * (kFewFeatures * kFewWRow + MT * kFewARow));   // [slice][MT][8]
    const float* a = p.a + (size_t)blockIdx.y * p.a_batch;
    const float* w = p.w + (size_t)blockIdx.y * p.w_batch;
    float* out = p.out + (size_t)blockIdx.y * p.o_batch;
    const int n0 = blockIdx.x * kFewFeatures;
    const int feature = lane & 7, slice = lane >> 3;

    if (!p.w_constant) griddep_wait();
    for (int m0 = 0; m0 < p.M; m0 += MT) {
        for (int r = 0; r < rounds; ++r) {
            const int chunk = warp + r * warps, k0 = chunk * kFewChunk;
            if (m0 == 0 || rounds > 1) {
#pragma unroll
                for (int i = 0; i < kFewFeatures * 4; ++i) {
                    const int row = i >> 2, piece = (i & 3) * 32 + lane, k = k0 + piece * 4;
                    const bool in = n0 + row < p.N && k < p.K;
                    cp_async16(s_w + row * kFewWRow + piece * 16, in ? w + (size_t)(n0 + row) * p.ldw + k : w, in);
                }
            }
            if (m0 == 0 && r == 0) {
                griddep_launch();
                griddep_wait();                       // the activations come from the kernels before this one
            }
#pragma unroll
            for (int i = 0; i < MT * 4; ++i) {
                const int row = i >> 2, piece = (i & 3) * 32 + lane, k = k0 + piece * 4;
                const bool in = m0 + row < p.M && k < p.K;
                cp_async16(s_a + row * kFewARow + (i & 3) * (kF32Slice * 4 + 16) + lane * 16, in ? a + (size_t)(m0 + row) * p.lda + k : a, in);
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
            const float4* wl = reinterpret_cast<const float4*>(s_w + feature * kFewWRow + slice * kF32Slice * 4);
            const unsigned char* al = s_a + slice * (kF32Slice * 4 + 16);
            float acc[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[m] = 0.f;
#pragma unroll 2
            for (int c = 0; c < kF32Slice / kF32Chain; ++c) {
                float chain[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) chain[m] = 0.f;
#pragma unroll
                for (int q = 0; q < kF32Chain / 4; ++q) {
                    const float4 wv = wl[c * (kF32Chain / 4) + q];
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const float4 av = *reinterpret_cast<const float4*>(al + m * kFewARow + (c * (kF32Chain / 4) + q) * 16);
                        chain[m] = fmaf(av.x, wv.x, chain[m]);
                        chain[m] = fmaf(av.y, wv.y, chain[m]);
                        chain[m] = fmaf(av.z, wv.z, chain[m]);
                        chain[m] = fmaf(av.w, wv.w, chain[m]);
                    }
                }
#pragma unroll
                for (int m = 0; m < MT; ++m) acc[m] += chain[m];
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) s_sum[((chunk * 4 + slice) * MT + m) * kFewFeatures + feature] = acc[m];
            __syncwarp();                             // the next round or pass overwrites what other lanes may still read
        }
        __syncthreads();
        const int slices = f32_slices(p.K), per = f32_group_slices(p.K);
        for (int e = threadIdx.x; e < MT * kFewFeatures; e += blockDim.x) {
            const int m = m0 + e / kFewFeatures, n = n0 + e % kFewFeatures;
            float total = 0.f;
            for (int g = 0; g < slices; g += per) {
                float group = 0.f;
                const int end = min(slices, g + per);
#pragma unroll 4
                for (int s = g; s < end; ++s) group += s_sum[s * MT * kFewFeatures + e];
                total += group;
            }
            if (m < p.M && n < p.N) out[(size_t)m * p.ldo + n] = total;
        }
        __syncthreads();
    }
}

// ---- many rows ---------------------------------------------------------------------------------------------------------
// Tiles of 64 x 128 outputs, 128 threads of 8 x 8: paired multiply-adds (fma.rn.f32x2: the same rounding as two fmaf in
// half the issue slots) on operands read from shared memory one k ahead; a value of `a` becomes a pair of equal ones by
// register moves, which go into the free issue slots (pairs kept in shared memory took 12 of its cycles a warp and k instead of
// 8, with two warps a scheduler nearly as many as the multiply-adds: 467 x 4 096 x 1 024 167 us, 140 now; 2 048 rows 554 and 462).
// The next 16 of K come in through registers meanwhile.  A chain and a slice per output
// take 128 registers; the sums of the groups, touched every 128 of K, live in shared memory, which leaves room for two CTAs
// a SM.  With SPLIT the groups of K go to the CTAs of a cluster, which add their tiles in order through each other's shared
// memory: a product with fewer tiles than the SMs hold keeps them busy all the same.
constexpr int kTileM = 64, kTileN = 128, kTileThreads = 128;
constexpr int kTileCtas = 2 * 148;                              // resident at once

struct TileSmem {
    float a[2][kF32Chain][kTileM + 4];
    float w[2][kF32Chain][kTileN + 4];
    float part[64][kTileThreads];                               // the group's sum so far, [output][thread]; SPLIT: [64][128] at the end
    float total[64][kTileThreads];                              // the groups' sum (not with SPLIT)
};

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t twice(float v) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

template <bool SPLIT>
__global__ void __launch_bounds__(kTileThreads, 2)
gemm_f32_tile_kernel(const GemmF32 p) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem[];
    TileSmem& s = *reinterpret_cast<TileSmem*>(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int groups = f32_groups(p.K), group_k = f32_group_slices(p.K) * kF32Slice;
    const int group = SPLIT ? (int)(blockIdx.z % groups) : 0, batch = SPLIT ? (int)(blockIdx.z / groups) : (int)blockIdx.z;
    const float* a = p.a + (size_t)batch * p.a_batch;
    const float* w = p.w + (size_t)batch * p.w_batch;
    float* out = p.out + (size_t)batch * p.o_batch;
    const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;
    const int k_begin = group * group_k, k_end = SPLIT ? min(p.K, k_begin + group_k) : p.K;

    // loading: a thread has one weight row's 16 of k, and half of a row of `a`
    const int arow = tid & 63, aquad = (tid >> 6) * 2;
    const bool a_in = m0 + arow < p.M, w_in = n0 + tid < p.N;
    const float* ap = a + (size_t)(a_in ? m0 + arow : 0) * p.lda;
    const float* wp = w + (size_t)(w_in ? n0 + tid : 0) * p.ldw;
    float4 av[2], wv[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = k0 + (aquad + h) * 4;
            av[h] = a_in && k < p.K ? *reinterpret_cast<const float4*>(ap + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int k = k0 + h * 4;
            wv[h] = w_in && k < p.K ? __ldg(reinterpret_cast<const float4*>(wp + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](int buffer) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = (aquad + h) * 4;
            s.a[buffer][k][arow] = av[h].x;
            s.a[buffer][k + 1][arow] = av[h].y;
            s.a[buffer][k + 2][arow] = av[h].z;
            s.a[buffer][k + 3][arow] = av[h].w;
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            s.w[buffer][h * 4][tid] = wv[h].x;
            s.w[buffer][h * 4 + 1][tid] = wv[h].y;
            s.w[buffer][h * 4 + 2][tid] = wv[h].z;
            s.w[buffer][h * 4 + 3][tid] = wv[h].w;
        }
    };

    // outputs: rows i / 4 * 32 + ty * 4 + i % 4, columns tx * 4 + j and 64 + tx * 4 + j.  Neighbouring lanes share a place
    // of `w` and lanes two apart one of `a`: a 16-byte read by the warp is then two wavefronts (it is four where lanes 0 to
    // 7 read eight places, whatever the other lanes read).
    const int tx = ((lane >> 1) & 7) + 8 * (warp & 1), ty = ((lane >> 4) << 1 | (lane & 1)) + 4 * (warp >> 1);
    uint64_t slice[8][4];                                       // [row][pair of columns]
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) slice[i][j] = 0;
#pragma unroll
    for (int e = 0; e < 64; ++e) {
        s.part[e][tid] = 0.f;
        if (!SPLIT) s.total[e][tid] = 0.f;
    }

    griddep_launch();
    griddep_wait();
    fetch(k_begin);
    put(0);
    __syncthreads();
    int buffer = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += kF32Chain) {
        const bool more = k0 + kF32Chain < k_end;
        if (more) fetch(k0 + kF32Chain);
        uint64_t chain[8][4];
        float4 x[2][2];
        ulonglong2 y[2][2];
        auto operands = [&](int which, int k) {
#pragma unroll
            for (int i = 0; i < 2; ++i) x[which][i] = *reinterpret_cast<const float4*>(&s.a[buffer][k][i * 32 + ty * 4]);
            y[which][0] = *reinterpret_cast<const ulonglong2*>(&s.w[buffer][k][tx * 4]);
            y[which][1] = *reinterpret_cast<const ulonglong2*>(&s.w[buffer][k][64 + tx * 4]);
        };
        operands(0, 0);
#pragma unroll
        for (int k = 0; k < kF32Chain; ++k) {
            if (k + 1 < kF32Chain) operands((k + 1) & 1, k + 1);
            const float4* xk = x[k & 1];
            const ulonglong2* yk = y[k & 1];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t xi = twice((i & 3) == 0 ? xk[i / 4].x : (i & 3) == 1 ? xk[i / 4].y : (i & 3) == 2 ? xk[i / 4].z : xk[i / 4].w);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t yj = j & 1 ? yk[j / 2].y : yk[j / 2].x;
                    chain[i][j] = fma2(xi, yj, k == 0 ? 0ull : chain[i][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) slice[i][j] = add2(slice[i][j], chain[i][j]);
        const int done = k0 + kF32Chain;
        if (done % kF32Slice == 0 || !more) {
            const bool group_ends = !SPLIT && (done % group_k == 0 || !more);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 v = unpack2(slice[i][j]);
                    const int e = (i * 4 + j) * 2;
                    slice[i][j] = 0;
                    const float p0 = s.part[e][tid] + v.x, p1 = s.part[e + 1][tid] + v.y;
                    s.part[e][tid] = group_ends ? 0.f : p0;
                    s.part[e + 1][tid] = group_ends ? 0.f : p1;
                    if (group_ends) {
                        s.total[e][tid] += p0;
                        s.total[e + 1][tid] += p1;
                    }
                }
        }
        if (more) put(buffer ^ 1);
        __syncthreads();
        buffer ^= 1;
    }

    const bool wide = p.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    auto store4 = [&](int m, int n, float4 v) {
        if (m >= p.M) return;
        float* o = out + (size_t)m * p.ldo + n;
        if (wide && n + 3 < p.N) *reinterpret_cast<float4*>(o) = v;
        else {
            if (n < p.N) o[0] = v.x;
            if (n + 1 < p.N) o[1] = v.y;
            if (n + 2 < p.N) o[2] = v.z;
            if (n + 3 < p.N) o[3] = v.w;
        }
    };
    if (!SPLIT) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int e = i * 8 + h * 4;
                store4(m0 + i / 4 * 32 + ty * 4 + i % 4, n0 + 64 * h + tx * 4,
                       make_float4(s.total[e][tid], s.total[e + 1][tid], s.total[e + 2][tid], s.total[e + 3][tid]));
            }
        return;
    }
    float4 own[16];                                             // out of [output][thread] into rows of 128 that the cluster reads
#pragma unroll
    for (int q = 0; q < 16; ++q) own[q] = make_float4(s.part[q * 4][tid], s.part[q * 4 + 1][tid], s.part[q * 4 + 2][tid], s.part[q * 4 + 3][tid]);
    __syncthreads();
    float* s_part = &s.part[0][0];                              // [64][128]
#pragma unroll
    for (int q = 0; q < 16; ++q) *reinterpret_cast<float4*>(s_part + (q / 8 * 32 + ty * 4 + q / 2 % 4) * kTileN + 64 * (q & 1) + tx * 4) = own[q];
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int e = group * kTileThreads + tid; e < kTileM * kTileN / 4; e += kTileThreads * groups) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int g = 0; g < groups; ++g) {
            const float4 v = reinterpret_cast<const float4*>(cluster.map_shared_rank(s_part, g))[e];
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        store4(m0 + e / (kTileN / 4), n0 + e % (kTileN / 4) * 4, sum);
    }
    cluster.sync();                                             // a CTA's shared memory stays until the others have read it
}

// Rows up to which the few-rows kernel may be taken, where K fits one round of its warps.  Up to one pass of eight it always
// is; beyond, the three kernels' times are estimated (microseconds, fitted to 9 to 2 048 rows x 64 to 151 936 x 64 to 8 192
// within 30 %) and the smallest wins:
//   few rows: 2.5, and a pass of eight rows 1.5 and 0.57 for every warp that an SM has of it
//   tiles: 0.067 per value of a CTA's K for each CTA that an SM has, alone on it 0.096 (0.115 where every SM has one)
//   tiles and all sizes: 3 more
//   all sizes: 0.0535 per value of K for each CTA that an SM has, at least 0.075
// (64 x 151 936 x 1 024: 1 116, 597 and 972; 64 x 4 096 x 1 024: 44, 49 and 79; 64 x 6 144 x
// 1 024: 60, 52 and more; 64 x 64 x 64: 18, 8.8 and 7.8; 128 x 2 048 x
// 512, K a single group of which no cluster can share the work: tiles 51, all sizes 41.)
constexpr int kFewMaxRows = 64;

bool gemm_f32_takes(const GemmF32& p, int batch) {
    return p.K % 4 == 0 && p.lda % 4 == 0 && p.ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(p.a) & 15) == 0
        && (reinterpret_cast<uintptr_t>(p.w) & 15) == 0 && (batch == 1 || (p.a_batch % 4 == 0 && p.w_batch % 4 == 0));
}

template <int MT>
static int launch_few(const GemmF32& p, int batch, cudaStream_t stream) {
    const int chunks = (p.K + kFewChunk - 1) / kFewChunk;
    const int rounds = (chunks + kFewMaxWarps - 1) / kFewMaxWarps, warps = (chunks + rounds - 1) / rounds;
    const size_t smem = (size_t)warps * (kFewFeatures * kFewWRow + MT * kFewARow) + (size_t)rounds * warps * 4 * MT * kFewFeatures * 4;
    static SmemLimit limit;
    if (int rc = raise_smem_limit(limit, gemm_f32_few_kernel<MT>, 227 * 1024, "gemm")) return rc;
    const cudaError_t e = launch_pdl(gemm_f32_few_kernel<MT>, dim3((p.N + kFewFeatures - 1) / kFewFeatures, batch), dim3(warps * 32),
                                     smem, stream, prompt_pdl(), p, rounds);
    CIB_REQUIRE(e == cudaSuccess, "gemm: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

// K up to which the few-rows kernel is taken: the sums of five rounds' slices fit beside the weights and rows of six warps
constexpr int kFewMaxK = 5 * kFewMaxWarps * kFewChunk;
static_assert(kFewMaxWarps * (kFewFeatures * kFewWRow + kFewRows * kFewARow) + 5 * kFewMaxWarps * 4 * kFewRows * kFewFeatures * 4 <= 227 * 1024,
              "shared memory of the largest few-rows launch");

static long long per_sm(long long ctas) { return (ctas + 147) / 148; }

int gemm_f32_launch(const GemmF32& p, int batch, cudaStream_t stream) {
    CIB_REQUIRE((p.M + kTileM - 1) / kTileM <= 65535 && batch <= 65535, "gemm: M=%d or batch=%d too large for this kernel", p.M, batch);
    const int groups = f32_groups(p.K);
    const dim3 grid((p.N + kTileN - 1) / kTileN, (p.M + kTileM - 1) / kTileM, batch);
    // rounds of resident CTAs, in groups of K: a tile whole, or its groups apart where that fills the last round better (and
    // the launch's z extent holds them)
    const long long tiles = (long long)grid.x * grid.y * batch;
    const bool split = groups > 1 && (long long)batch * groups <= 65535 && (tiles * groups + kTileCtas - 1) / kTileCtas < (tiles + kTileCtas - 1) / kTileCtas * groups;

    bool few = p.K <= kFewMaxK && p.M <= kFewRows;
    if (!few) {
        const long long tile_ctas = tiles * (split ? groups : 1);
        const float tile_k = split ? (float)(f32_group_slices(p.K) * kF32Slice) : (float)p.K;
        const float t_tile = 3.f + tile_k * (tile_ctas <= 74 ? 0.096f : tile_ctas <= 148 ? 0.115f : 0.067f * per_sm(tile_ctas));
        const long long all_ctas = (long long)((p.N + 63) / 64) * ((p.M + 63) / 64) * batch;
        const float t_all = 3.f + p.K * fmaxf(0.075f, 0.0535f * per_sm(all_ctas));
        const int chunks = (p.K + kFewChunk - 1) / kFewChunk, passes = (p.M + kFewRows - 1) / kFewRows;
        const float t_few = 2.5f + passes * (1.5f + 0.57f * chunks * per_sm((long long)((p.N + kFewFeatures - 1) / kFewFeatures) * batch));
        few = p.M <= kFewMaxRows && chunks <= kFewMaxWarps && t_few <= fminf(t_tile, t_all);
        if (!few && t_all < t_tile) return 1;
    }
    if (few) {
        switch (p.M) {
            case 1: return launch_few<1>(p, batch, stream);
            case 2: return launch_few<2>(p, batch, stream);
            case 3: return launch_few<3>(p, batch, stream);
            case 4: return launch_few<4>(p, batch, stream);
            case 5: return launch_few<5>(p, batch, stream);
            case 6: return launch_few<6>(p, batch, stream);
            case 7: return launch_few<7>(p, batch, stream);
            default: return launch_few<8>(p, batch, stream);
        }
    }
    static SmemLimit limit_split, limit_whole;
    cudaError_t e;
    if (split) {
        if (int rc = raise_smem_limit(limit_split, gemm_f32_tile_kernel<true>, sizeof(TileSmem), "gemm")) return rc;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid.x, grid.y, batch * groups);
        cfg.blockDim = dim3(kTileThreads);
        cfg.dynamicSmemBytes = offsetof(TileSmem, total);
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = (unsigned)groups;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = prompt_pdl() ? 2 : 1;
        e = cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<true>, p);
    } else {
        if (int rc = raise_smem_limit(limit_whole, gemm_f32_tile_kernel<false>, sizeof(TileSmem), "gemm")) return rc;
        e = launch_pdl(gemm_f32_tile_kernel<false>, grid, dim3(kTileThreads), sizeof(TileSmem), stream, prompt_pdl(), p);
    }
    CIB_REQUIRE(e == cudaSuccess, "gemm: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

}  // namespace cib
