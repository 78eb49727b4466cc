// out[M, N] = act[M, K] · W[N, K]^T in bfloat16 for up to 128 rows: the weight matrix is the streamed operand.
//
// The reference sends every projection to cuBLAS (csrc/ops/projection.cu:32-44).  With few rows a projection is one
// pass over its weights, and what matters is how many bytes an SM keeps in flight, and how little lies between the end of the
// kernel before it and its own last store.  The few-rows kernel of this package (gemm_skinny.cu) has every CTA read all the
// activations of its share of K; from 17 rows on, and with large matrices, that is what bounds it.  Here the roles of the
// operands are swapped on the 5th-generation tensor cores instead:
//
//   * a CTA owns 128 output features: its weight rows are the 128-row A operand of `tcgen05.mma.kind::f16`, fetched by
//     TMA in 16 KB boxes (128 features x 64 k, 128-byte swizzle) through a ring of stages; the rows of the batch are the B
//     operand (N = 16, 32, 64 or 128, rows beyond M read as zeros); the accumulator, out^T, lives in tensor memory
//     (features = lanes, batch rows = columns);
//   * K is split over the 2, 4 or 8 CTAs of a cluster.  Every CTA finishes its share of the rows: the others send it their sums
//     of those rows (distributed shared memory, a region of its own), and it adds them in rank order, so results do not depend
//     on timing and a row's not on the rows beside it;
//   * the ring is kept small enough for two CTAs an SM (up to 64 rows): the next projection of a decode step is then resident,
//     its weights on their way (they do not wait for `griddepcontrol.wait`), while this one still runs;
//   * epilogues: bfloat16 or float32 rows, or silu(gate) * up for a weight of gate rows followed by up rows (a tile then
//     holds 64 gate features and the 64 matching up features), or the residual and the next norm's rows (`stream`: see
//     gemm_skinny.cu, whose description of a norm shared by two products holds here too).
//
// The engine takes it up to 64 rows; 65 to 128 rows (one CTA an SM) are for callers of the kernel itself: the library is faster there.
//
// Every mbarrier wait is bounded; on a time-out the kernel raises the error flag, frees its tensor memory and returns.  The CTA
// whose wait ran out stores nothing; the others of its cluster have its unfinished sums among theirs, so no row of a flagged launch
// counts, the residual's neither.
#include "tcgen05_utils.cuh"

#include "mma_utils.cuh"

namespace cib {
namespace ws {

enum Epilogue : int { kBf16 = 0, kF32 = 1, kSilu = 2, kStream = 3 };

constexpr int kWBytes = kTcBM * kTcBK * 2;          // a weight box: 128 features x 64 k

struct Args {
    void* out; int ldo; int M, N, K, up_offset;
    const float* squares_in; int squares_in_n; float eps;      // rows that carry a norm still to be applied, or null
    AnyVec gain; float* stream; float* squares_out;            // kStream; squares_out [M][ceil(N / 32)]
    const float* bias; int squared_relu;                       // kBf16, kF32: added to every row (or null), then relu(y)^2
    const void* warm; unsigned long long warm_bytes;           // what the kernel after this one reads first (or null)
    int* error_flag;
};

template <int BX, int S, int EPI>
struct Smem {
    static constexpr int kXBytes = BX * kTcBK * 2;
    static constexpr int kStageBytes = kWBytes + kXBytes;
    static constexpr int kStages = BX == 128 ? 5 : BX == 64 ? 3 : 4;
    static constexpr int kRing = kStages * kStageBytes;
    static constexpr int kRows = BX / S;                                       // rows a CTA finishes
    static constexpr int kInbox = (S - 1) * kRows * kTcBM * 4;                 // [source][row][feature]
    static constexpr int kTotal = kRing + kInbox + 1024 /* alignment slack */ + 256 /* barriers */ + BX * 4 /* factors */;
    static_assert(EPI != kSilu || kRows * 64 * 4 <= kRing, "the ups pass through the ring");
};

// C columns of this thread's lane of tensor memory
template <int C>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, float (&v)[C]) {
    static_assert(C == 2 || C == 4 || C == 8 || C == 16, "columns of one load");
    uint32_t r[C];
    if constexpr (C == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
    if constexpr (C == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
    if constexpr (C == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
    if constexpr (C == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                       "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr));
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < C; ++i) v[i] = __uint_as_float(r[i]);
}

// Grid: (128-feature tiles) x (cluster of S CTAs that split K).  192 threads: warp 0 TMA producer, warp 1 MMA issuer
// and tensor-memory owner, warps 2-5 epilogue (TMEM lanes 32 * (warp % 4) .. + 31 = features of the tile).
template <int BX, int S, int EPI>
__global__ void __launch_bounds__(192, BX == 128 ? 1 : 2)
gemm_wstream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Args a) {
    using Sm = Smem<BX, S, EPI>;
    constexpr int STAGES = Sm::kStages;
    constexpr int kTmemCols = BX < 32 ? 32 : BX;
    constexpr int R = Sm::kRows;
    constexpr int C = R < 16 ? R : 16;                       // rows of one piece of the epilogue
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* inbox = reinterpret_cast<float*>(ring + Sm::kRing);
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + Sm::kRing + Sm::kInbox);
    uint64_t* full = bars;                   // [STAGES] bytes of a stage have landed
    uint64_t* empty = bars + STAGES;         // [STAGES] the MMAs that read a stage are done
    uint64_t* acc_full = bars + 2 * STAGES;  // the accumulator holds this CTA's share
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
    float* s_factor = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(bars) + 256);
    __shared__ int s_abort;

    // "this CTA runs": its inbox may be written by the others of the cluster once all have said so
    if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = S > 1 ? (int)cluster_ctarank() : 0;
    const int tile = (int)(blockIdx.x / S);
    constexpr int kTileCols = EPI == kSilu ? 64 : 128;       // output features of a tile
    const int n0 = tile * kTileCols;
    const int steps_total = (a.K + kTcBK - 1) / kTcBK;
    const int steps_per = (steps_total + S - 1) / S;
    const int kb0 = rank * steps_per;
    const int nsteps = max(0, min(steps_total, kb0 + steps_per) - kb0);

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        warm_l2_share(a.warm, a.warm_bytes, blockIdx.x, gridDim.x);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    griddep_launch();          // (not before this CTA has its tensor memory: the next kernel's CTAs take theirs as they come)
    const uint32_t tmem_base = *tmem_slot;
    const bool epilogue_thread = warp >= 2;
    const int feature = (warp & 3) * 32 + lane;               // of the tile, for epilogue threads
    const int row0 = rank * R;                                // the rows this CTA finishes
    // kStream: this thread's column of the residual and its gain, fetched before the sums are there
    const int n = n0 + feature;
    float gain = 0.f, old[C];
    if (EPI == kStream && epilogue_thread && n < a.N) gain = a.gain[n];
    float bias = 0.f;
    if ((EPI == kBf16 || EPI == kF32) && a.bias != nullptr && epilogue_thread && n < a.N) bias = a.bias[n];
    auto fetch_old = [&](int c) {
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const int m = row0 + c + i;
            old[i] = m < a.M && n < a.N ? a.stream[(size_t)m * a.N + n] : 0.f;
        }
    };

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer ----
            auto load_w = [&](int i) {
                unsigned char* w_dst = ring + (size_t)(i % STAGES) * Sm::kStageBytes;
                const int k = (kb0 + i) * kTcBK;
                if (EPI == kSilu) {
                    tma_load_2d(w_dst, &map_w, &full[i % STAGES], k, n0);                              // 64 gate rows
                    tma_load_2d(w_dst + 64 * 128, &map_w, &full[i % STAGES], k, a.up_offset + n0);     // the 64 matching up rows
                } else {
                    tma_load_2d(w_dst, &map_w, &full[i % STAGES], k, n0);
                }
            };
            auto load_x = [&](int i) {
                tma_load_2d(ring + (size_t)(i % STAGES) * Sm::kStageBytes + kWBytes, &map_x, &full[i % STAGES], (kb0 + i) * kTcBK, 0);
            };
            // the weights of the first stages do not depend on the kernel before this one
            const int pre = min(STAGES, nsteps);
            for (int i = 0; i < pre; ++i) {
                mbar_expect_tx(&full[i], Sm::kStageBytes);
                load_w(i);
            }
            griddep_wait();
            for (int i = 0; i < pre; ++i) load_x(i);
            for (int i = pre; i < nsteps; ++i) {
                const int s = i % STAGES;
                if (!mbar_wait(&empty[s], (uint32_t)((i / STAGES - 1) & 1))) { atomicExch(a.error_flag, 31); s_abort = 1; break; }
                if (*(volatile int*)&s_abort) break;
                mbar_expect_tx(&full[s], Sm::kStageBytes);
                load_w(i);
                load_x(i);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer: D[128 features, BX rows] += W[128, 16 k] · X[BX, 16 k]^T ----
            constexpr uint32_t idesc = umma_idesc_bf16(kTcBM, BX);
            bool ok = true;
            for (int i = 0; i < nsteps; ++i) {
                const int s = i % STAGES;
                if (!mbar_wait(&full[s], (uint32_t)((i / STAGES) & 1))) { atomicExch(a.error_flag, 32); s_abort = 1; ok = false; break; }
                tcgen05_fence_after();
                const unsigned char* w_src = ring + (size_t)s * Sm::kStageBytes;
                const uint64_t adesc = umma_desc_k_major_sw128(w_src);
                const uint64_t bdesc = umma_desc_k_major_sw128(w_src + kWBytes);
#pragma unroll
                for (int k = 0; k < kTcBK / 16; ++k)
                    umma_bf16(tmem_base, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (i | k) != 0 ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            if (ok && nsteps > 0) umma_commit(acc_full);
            else mbar_arrive(acc_full);            // nothing to wait for: this CTA's share of K is empty (or it gave up)
        }
    } else {
        // ---- epilogue threads: what the results need beside the sums, then this CTA's sums of the others' rows to them ----
        griddep_wait();
        if (EPI == kStream) fetch_old(0);
        if (a.squares_in != nullptr) {
            for (int r = warp - 2; r < R; r += 4) {            // the factors of the rows this CTA finishes, a warp per row
                const int m = row0 + r;
                float ss = 0.f;
                if (m < a.M)
                    for (int p = lane; p < a.squares_in_n; p += 32) ss += a.squares_in[(size_t)m * a.squares_in_n + p];
                ss = warp_sum(ss);
                if (lane == 0) s_factor[r] = rsqrtf(ss / (float)a.K + a.eps);
            }
        }
        bool ok = mbar_wait(acc_full, 0);
        if (!ok && lane == 0) { atomicExch(a.error_flag, 33); s_abort = 1; }
        __syncwarp();
        tcgen05_fence_after();
    }
    __syncwarp();                                              // (the roles' lanes meet again before the barriers of whole warps)
    // (with an empty share of K the accumulator holds nothing: zeros stand for it)
    const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    auto sums_of = [&](int col, float (&v)[C]) {
        if (nsteps > 0) tmem_ld_cols<C>(lane_addr + (uint32_t)col, v);
        else {
#pragma unroll
            for (int i = 0; i < C; ++i) v[i] = 0.f;
        }
    };
    if constexpr (S > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");          // every CTA of the cluster runs
        if (epilogue_thread) {
#pragma unroll 1
            for (int d = 1; d < S; ++d) {
                const int to = (rank + d) % S;
                const uint32_t box = map_to_cta(inbox + (size_t)(rank < to ? rank : rank - 1) * R * kTcBM + feature, (uint32_t)to);
#pragma unroll 1
                for (int c = 0; c < R; c += C) {
                    float v[C];
                    sums_of(to * R + c, v);
#pragma unroll
                    for (int i = 0; i < C; ++i)
                        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(box + (uint32_t)((c + i) * kTcBM * 4)), "f"(v[i]) : "memory");
                }
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const bool healthy = !(*(volatile int*)&s_abort);
    if (epilogue_thread) {
        asm volatile("bar.sync 1, 128;" ::: "memory");        // the factors are there (and, gated, the ring is free)
        float* ups = reinterpret_cast<float*>(ring);          // kSilu: [R][64]
        // the rows' sums over K, in rank order
        auto total = [&](int c, float (&v)[C]) {
            float own[C];
            sums_of(row0 + c, own);
#pragma unroll
            for (int i = 0; i < C; ++i) v[i] = 0.f;
#pragma unroll
            for (int s = 0; s < S; ++s) {
#pragma unroll
                for (int i = 0; i < C; ++i) {
                    if (S == 1) v[i] = own[i];
                    else v[i] += s == rank ? own[i] : inbox[((size_t)(s < rank ? s : max(0, s - 1)) * R + c + i) * kTcBM + feature];
                }
            }
            if (a.squares_in != nullptr) {
#pragma unroll
                for (int i = 0; i < C; ++i) v[i] *= s_factor[c + i];
            }
        };
        if constexpr (EPI == kSilu) {
#pragma unroll 1
            for (int c = 0; c < R && feature >= 64; c += C) {
                float v[C];
                total(c, v);
#pragma unroll
                for (int i = 0; i < C; ++i) ups[(c + i) * 64 + feature - 64] = v[i];
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < R && feature < 64; c += C) {
                float v[C];
                total(c, v);
#pragma unroll
                for (int i = 0; i < C; ++i) {
                    const int m = row0 + c + i;
                    if (healthy && m < a.M && n < a.up_offset)
                        reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)m * a.ldo + n] =
                            __float2bfloat16_rn(v[i] / (1.f + expf(-v[i])) * ups[(c + i) * 64 + feature]);
                }
            }
        } else {
            const int parts = (a.N + 31) / 32;
#pragma unroll 1
            for (int c = 0; c < R; c += C) {
                if (row0 + c >= a.M) break;
                if (EPI == kStream && c > 0) fetch_old(c);
                float v[C];
                total(c, v);
#pragma unroll
                for (int i = 0; i < C; ++i) {
                    const int m = row0 + c + i;
                    const bool ok = healthy && m < a.M && n < a.N;
                    if constexpr (EPI == kStream) {
                        const float x = old[i] + v[i];
                        const float sq = warp_sum(ok ? x * x : 0.f);
                        if (ok) {
                            a.stream[(size_t)m * a.N + n] = x;
                            reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)m * a.ldo + n] = __float2bfloat16_rn(x * gain);
                            if (lane == 0) a.squares_out[(size_t)m * parts + n / 32] = sq;
                        }
                    } else if (ok) {
                        v[i] += bias;
                        if (a.squared_relu) {
                            v[i] = fmaxf(v[i], 0.f);
                            v[i] *= v[i];
                        }
                        if (EPI == kF32) reinterpret_cast<float*>(a.out)[(size_t)m * a.ldo + n] = v[i];
                        else reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)m * a.ldo + n] = __float2bfloat16_rn(v[i]);
                    }
                }
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
}

template <int BX, int S, int EPI>
static int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, int tiles, bool use_pdl, cudaStream_t stream) {
    auto kernel = gemm_wstream_kernel<BX, S, EPI>;
    constexpr int smem = Smem<BX, S, EPI>::kTotal;
    static_assert(smem <= (BX == 128 ? 227 : 113) * 1024, "one CTA an SM for 128 rows, two for fewer");
    static SmemLimit limit;
    if (int rc = raise_smem_limit(limit, kernel, smem, "gemm_wstream")) return rc;
    const cudaError_t e = launch_pdl_cluster(kernel, dim3(tiles * S), dim3(192), smem, stream, use_pdl, S, mw, mx, a);
    CIB_REQUIRE(e == cudaSuccess, "gemm_wstream: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

// K is split over the CTAs of a cluster until there is about a CTA for every SM, as long as there are two steps a CTA (the shares are
// rounded up, so the last CTAs may have less, or none: 17 steps over eight are 3, 3, 3, 3, 3, 2, 0, 0).  By the weight's sizes alone: a row's result does not depend on how many rows are beside it.
static int k_splits(int n_out, int K, bool pair) {
    const int tiles = (n_out + (pair ? 63 : 127)) / (pair ? 64 : 128), steps = (K + kTcBK - 1) / kTcBK;
    int s = 1;
    while (s < 8 && tiles * s < 140 && steps >= 4 * s) s *= 2;
    return s;
}

template <int BX, int EPI>
static int dispatch_splits(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, bool use_pdl, cudaStream_t stream) {
    const int n_out = EPI == kSilu ? a.up_offset : a.N, cols = EPI == kSilu ? 64 : 128, tiles = (n_out + cols - 1) / cols;
    switch (k_splits(n_out, a.K, EPI == kSilu)) {
        case 1: return launch<BX, 1, EPI>(mw, mx, a, tiles, use_pdl, stream);
        case 2: return launch<BX, 2, EPI>(mw, mx, a, tiles, use_pdl, stream);
        case 4: return launch<BX, 4, EPI>(mw, mx, a, tiles, use_pdl, stream);
        default: return launch<BX, 8, EPI>(mw, mx, a, tiles, use_pdl, stream);
    }
}

template <int BX>
static int dispatch(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, int epilogue, bool use_pdl, cudaStream_t stream) {
    switch (epilogue) {
        case kSilu: return dispatch_splits<BX, kSilu>(mw, mx, a, use_pdl, stream);
        case kF32: return dispatch_splits<BX, kF32>(mw, mx, a, use_pdl, stream);
        case kStream: return dispatch_splits<BX, kStream>(mw, mx, a, use_pdl, stream);
        default: return dispatch_splits<BX, kBf16>(mw, mx, a, use_pdl, stream);
    }
}

}  // namespace ws
}  // namespace cib

using namespace cib;

extern "C" int cib_gemm_wstream_supports(int M, int N, int K) {
    return M >= 1 && M <= 128 && N >= 8 && K >= 8 && K % 8 == 0;
}

// act: [M, K] bfloat16 rows (lda), w: [N, K] bfloat16 rows (ldw).  epilogue: 0 = bfloat16 out[M, N]; 1 = float32
// out[M, N]; 2 = rows [0, N / 2) of w are gates and rows [N / 2, N) the matching ups: out[M, N / 2] = silu(gate) * up in
// bfloat16; 3 = stream_rows[M, N] (32-bit, dense) += the product, out = bfloat16(stream_rows * gain), squares_out
// [M][ceil(N / 32)] = the sums of stream_rows^2 over 32 columns each.
// bias [N] (epilogues 0 and 1, or null) is added to every row; squared_relu: then y = relu(y)^2.
// squares_in: [M][squares_in_n] (or null): every result row is multiplied by rsqrt(sum(squares_in[row]) / K + eps).
// warm / warm_bytes: memory that the kernel after this one reads first, or null: fetched into the L2 meanwhile.
// error_flag: one zero int in device memory.
extern "C" int cib_gemm_wstream(const void* act, int lda, const void* w, int ldw, void* out, int ldo, int epilogue, int M,
                                int N, int K, const float* squares_in, int squares_in_n, float eps, float* stream_rows,
                                const void* gain, int gain_dtype, float* squares_out, const float* bias, int squared_relu,
                                const void* warm, long long warm_bytes, int use_pdl, int* error_flag, cudaStream_t stream) {
    CIB_REQUIRE(cib_gemm_wstream_supports(M, N, K), "gemm_wstream: M=%d N=%d K=%d is not taken (at most 128 rows, K a multiple of 8)", M, N, K);
    CIB_REQUIRE(lda >= K && ldw >= K && lda % 8 == 0 && ldw % 8 == 0 && ((uintptr_t)act % 16) == 0 && ((uintptr_t)w % 16) == 0,
                "gemm_wstream: rows must be 16-byte aligned");
    CIB_REQUIRE(epilogue >= 0 && epilogue <= 3 && error_flag != nullptr, "gemm_wstream: bad arguments");
    CIB_REQUIRE(epilogue != ws::kSilu || N % 2 == 0, "gemm_wstream: a gate/up weight has an even number of rows");
    CIB_REQUIRE(ldo >= (epilogue == ws::kSilu ? N / 2 : N), "gemm_wstream: ldo too small");
    CIB_REQUIRE(epilogue != ws::kStream || (stream_rows != nullptr && gain != nullptr && squares_out != nullptr),
                "gemm_wstream: the stream epilogue needs the residual, the norm's gains and room for the squares");
    CIB_REQUIRE((bias == nullptr && !squared_relu) || epilogue == ws::kBf16 || epilogue == ws::kF32, "gemm_wstream: a bias goes with plain rows");
    CIB_REQUIRE(squares_in == nullptr || squares_in_n > 0, "gemm_wstream: sums of squares without parts");
    CUtensorMap mw, mx;
    if (tc_make_map(&mw, w, N, K, ldw, epilogue == ws::kSilu ? 64 : 128, "gemm_wstream") != 0) return -1;
    const int bx = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
    if (tc_make_map(&mx, act, M, K, lda, bx, "gemm_wstream") != 0) return -1;
    if (((uintptr_t)warm % 16) != 0 || warm_bytes <= 0) { warm = nullptr; warm_bytes = 0; }
    const ws::Args a = {out, ldo, M, N, K, N / 2, squares_in, squares_in_n, eps, AnyVec{gain, gain_dtype == kBF16}, stream_rows, squares_out,
                        bias, squared_relu, warm, (unsigned long long)warm_bytes, error_flag};
    switch (bx) {
        case 16: return ws::dispatch<16>(mw, mx, a, epilogue, use_pdl != 0, stream);
        case 32: return ws::dispatch<32>(mw, mx, a, epilogue, use_pdl != 0, stream);
        case 64: return ws::dispatch<64>(mw, mx, a, epilogue, use_pdl != 0, stream);
        default: return ws::dispatch<128>(mw, mx, a, epilogue, use_pdl != 0, stream);
    }
}
