// out[M, N] = a[M, K] · w[N, K]^T in bfloat16 on the 5th-generation tensor cores: TMA-fed, TMEM-accumulated.
//
// The reference calls cuBLAS for every projection (csrc/ops/projection.cu:32-44).  This is the prompt-sized
// replacement (many rows).  The kernel is persistent: one CTA per SM walks over 128 x BN output tiles, K in
// 64-element steps, and two accumulators in tensor memory let the epilogue of one tile run under the MMAs of the next.
//
//   warp 0, one thread : TMA producer.  Per step two `cp.async.bulk.tensor.2d` loads (an activation tile 128 x 64 and
//                        a weight tile BN x 64, both K-major, 128-byte swizzle) into a ring of shared-memory stages,
//                        completion counted in bytes on the stage's "full" mbarrier.  No multicast.
//   warp 1, one thread : MMA issuer.  Waits for "full", issues four `tcgen05.mma.cta_group::1.kind::f16`
//                        (128 x BN x 16 each) whose accumulator lives in tensor memory, then `tcgen05.commit` to the
//                        stage's "empty" mbarrier; after the last step a commit to the "accumulator ready" mbarrier.
//   warps 2-5          : epilogue.  Each warp owns the 32 TMEM lanes (= output rows) its rank allows, reads them with
//                        `tcgen05.ld.32x32b`, converts and stores rows to global memory (bfloat16 or float32).
//
// Rows beyond M, features beyond N and the tail of K read as zeros (TMA out-of-bounds fill) and are not stored.
// Every mbarrier wait is bounded: if a limit is hit the kernel raises a flag in global memory, stops issuing,
// drains what it started, frees its tensor memory and returns, so a fault in this kernel cannot hang the device.
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

#include <stdlib.h>

namespace cib {

// The stream epilogue (see the kernel): kStreamBufs pieces of the residual, 32 columns of 32-bit values each, and two panels of 64
// bfloat16 columns.
constexpr int kStreamBufs = 2;
constexpr int kStreamPiece = kTcBM * 128;

template <int BN, int STAGES, bool PAIR = false, bool STREAM = false>
struct TcSmem {
    static constexpr int kABytes = kTcBM * kTcBK * 2;
    static constexpr int kBBytes = (PAIR ? BN / 2 : BN) * kTcBK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    // 128 rows x 128 bfloat16 columns for the TMA store (two panels of 64), and the pieces of the residual
    static constexpr int kStagingBytes = kTcBM * 128 * 2 + (STREAM ? kStreamBufs * kStreamPiece : 0);
    static constexpr int kTotal = STAGES * kStageBytes + kStagingBytes + 1024 /* alignment slack */ + 512 /* barriers */ + (STREAM ? 1024 : 0) /* gains */;
};

// TMA_STORE: bfloat16 results leave through a 128-byte-swizzled staging buffer and `cp.async.bulk.tensor` stores
// (whole 128-byte lines per row; tails clipped by the tensor map).  Otherwise every thread stores its row itself.
// SILU: the weight rows are (gate, up) halves, rows [0, up_offset) and [up_offset, 2 up_offset); a tile multiplies BN / 2
// gate rows and the matching BN / 2 up rows (two weight boxes per stage) and stores silu(gate) * up, BN / 2 columns wide,
// straight from the 32-bit accumulators: the activation kernel and the round trip of the gate/up matrix are gone.
// PAIR: launched as clusters of two CTAs that share each 256 x BN tile (see the helpers above).  Per 64-k step a CTA
// then fetches 16 KB of activations and BN / 2 weight rows instead of BN: the kernel is bound by what an SM can fetch
// from the L2, so fewer bytes per flop is what makes it faster.
// STREAM: the result joins the 32-bit residual (`extra.res`, updated in place) and what is stored to `out` is the new residual times
// the next norm's gains; `squares_out` [M][tiles along N] gets the sums of the new residual's squares over a tile's columns.  A
// norm kernel of its own read and wrote 100 MB for 8 192 rows of 1 024 (21 us alone); here 84 of them pass under the MMAs, in pieces of 32
// columns that a seventh warp brings by TMA before the epilogue needs them and stores behind it.  The product after the norm gets
// those sums (`squares_in`; NORMED) and multiplies its rows by rsqrt(mean square + eps).
struct TcNorm {
    const float* squares_in; int squares_in_n; float eps;      // null: rows without a norm
    AnyVec gain; float* squares_out;                           // STREAM
};

// what a kernel gets beside its operands: nothing for a plain product, whose parameters stay as short as they are
template <bool STREAM, bool NORMED> struct TcExtra { TcNorm norm; };
template <> struct TcExtra<true, false> { CUtensorMap res; TcNorm norm; };
template <> struct TcExtra<false, false> {};

template <int BN, int STAGES, bool F32OUT, bool TMA_STORE, int SILU = 0, bool PAIR = false, bool STREAM = false, bool NORMED = false>
__global__ void __launch_bounds__(STREAM ? 224 : 192)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_out, const __grid_constant__ TcExtra<STREAM, NORMED> extra,
                    void* __restrict__ out, int ldo, int M, int N, int K, int up_offset, int* __restrict__ error_flag) {
    using Smem = TcSmem<BN, STAGES, PAIR, STREAM>;
    static_assert(!STREAM || (TMA_STORE && !F32OUT && !SILU && kStreamBufs == 2), "the stream epilogue's panels are free again when its pieces are");
    static_assert(!SILU || (BN == 256 && TMA_STORE && !F32OUT), "the gated epilogue is built for 256-wide tiles stored by TMA");
    constexpr int kOutCols = SILU ? BN / 2 : BN;      // output columns of a tile
    extern __shared__ unsigned char smem_raw[];
    // stages must start on a 1024-byte boundary (one swizzle atom)
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* staging = tiles + STAGES * Smem::kStageBytes;      // 1024-byte aligned as well
    uint64_t* bars = reinterpret_cast<uint64_t*>(staging + Smem::kStagingBytes);
    uint64_t* full = bars;                     // [STAGES]  bytes of a stage have landed
    uint64_t* empty = bars + STAGES;           // [STAGES]  the MMAs that read a stage are done
    uint64_t* acc_full = bars + 2 * STAGES;    // [2]       an accumulator holds a finished tile
    uint64_t* acc_empty = bars + 2 * STAGES + 2;  // [2]    the epilogue has read an accumulator
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    uint64_t* res_full = bars + 2 * STAGES + 5;   // [kStreamBufs] a piece of the residual has landed
    uint64_t* res_done = res_full + kStreamBufs;  // [kStreamBufs] the epilogue has added to it
    unsigned char* pieces = staging + kTcBM * 128 * 2;
    float* s_gain = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(bars) + 512);     // [4 warps][2][32]
    __shared__ int s_abort;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_steps = (K + kTcBK - 1) / kTcBK;
    constexpr int kTileRows = PAIR ? 2 * kTcBM : kTcBM;       // rows of a tile (of the pair's tile)
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;       // 0: the CTA that issues the MMAs
    const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int n_out = SILU ? up_offset : N;
    const int n_blocks = (n_out + kOutCols - 1) / kOutCols, m_blocks = (M + kTileRows - 1) / kTileRows;
    const int num_tiles = n_blocks * m_blocks;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], PAIR ? 8 : 4); }
        if (STREAM)
            for (int b = 0; b < kStreamBufs; ++b) { mbar_init(&res_full[b], 1); mbar_init(&res_done[b], 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"((uint32_t)(2 * BN)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"((uint32_t)(2 * BN)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();          // the other CTA's barriers exist before anything arrives on them
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // set-up (barriers, tensor memory) may run under the tail of the kernel before this one; its results may not be read
    // nor this kernel's written before it has ended
    griddep_launch();
    griddep_wait();

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer: one running step counter over all tiles of this CTA ----
            int step = 0;
            bool ok = true;
            for (int tile = worker; tile < num_tiles && ok; tile += workers) {
                const int m0 = (tile / n_blocks) * kTileRows + (int)rank * kTcBM, n0 = (tile % n_blocks) * kOutCols;
                for (int kb = 0; kb < k_steps; ++kb, ++step) {
                    const int s = step % STAGES;
                    const uint32_t phase = (step / STAGES) & 1;
                    if (!mbar_wait(&empty[s], phase ^ 1)) { atomicExch(error_flag, 1); s_abort = 1; ok = false; break; }
                    if (*(volatile int*)&s_abort) { ok = false; break; }
                    unsigned char* a_dst = tiles + (size_t)s * Smem::kStageBytes;
                    unsigned char* b_dst = a_dst + Smem::kABytes;
                    if constexpr (PAIR) {
                        // both CTAs' bytes are counted on the first CTA's barrier; it expects them all
                        const uint32_t bar = map_to_cta(&full[s], 0);
                        if (rank == 0) mbar_expect_tx(&full[s], 2 * Smem::kStageBytes);
                        tma_load_2d_pair(a_dst, &map_a, bar, kb * kTcBK, m0);
                        // this CTA's half of the tile's weight rows (gated: the first CTA the gates, the second the ups)
                        const int w_row = SILU ? (rank == 0 ? n0 : up_offset + n0) : n0 + (int)rank * (BN / 2);
                        tma_load_2d_pair(b_dst, &map_w, bar, kb * kTcBK, w_row);
                        continue;
                    }
                    mbar_expect_tx(&full[s], Smem::kStageBytes);
                    tma_load_2d(a_dst, &map_a, &full[s], kb * kTcBK, m0);
                    if (SILU) {
                        // gate rows, then the matching up rows: accumulator columns [0, BN/2) and [BN/2, BN)
                        tma_load_2d(b_dst, &map_w, &full[s], kb * kTcBK, n0);
                        tma_load_2d(b_dst + (BN / 2) * 128, &map_w, &full[s], kb * kTcBK, up_offset + n0);
                    } else {
                        tma_load_2d(b_dst, &map_w, &full[s], kb * kTcBK, n0);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // ---- MMA issuer (of the pair) ----
            constexpr uint32_t idesc = umma_idesc_bf16(kTileRows, BN);
            int step = 0, local = 0;
            bool ok = true;
            for (int tile = worker; tile < num_tiles && ok; tile += workers, ++local) {
                const int buf = local & 1;
                const uint32_t acc_phase = (local >> 1) & 1;
                if (!mbar_wait(&acc_empty[buf], acc_phase ^ 1)) { atomicExch(error_flag, 4); s_abort = 1; ok = false; break; }
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
                for (int kb = 0; kb < k_steps; ++kb, ++step) {
                    const int s = step % STAGES;
                    const uint32_t phase = (step / STAGES) & 1;
                    if (!mbar_wait(&full[s], phase)) { atomicExch(error_flag, 2); s_abort = 1; ok = false; break; }
                    tcgen05_fence_after();
                    const unsigned char* a_src = tiles + (size_t)s * Smem::kStageBytes;
                    const unsigned char* b_src = a_src + Smem::kABytes;
                    const uint64_t adesc = umma_desc_k_major_sw128(a_src);
                    const uint64_t bdesc = umma_desc_k_major_sw128(b_src);
#pragma unroll
                    for (int k = 0; k < kTcBK / 16; ++k) {
                        // 16 elements of K = 32 bytes further inside the swizzle atom: +2 in 16-byte units
                        if (PAIR) umma_bf16_pair(tmem_d, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
                        else umma_bf16(tmem_d, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
                    }
                    if (PAIR) umma_commit_pair(&empty[s]);
                    else umma_commit(&empty[s]);   // frees the stage when these MMAs have read it
                }
                if (PAIR) umma_commit_pair(&acc_full[buf]);
                else umma_commit(&acc_full[buf]);  // arrives when every MMA issued so far has finished
            }
        }
    } else if (STREAM && warp == 6) {
        if constexpr (STREAM) if (lane == 0) {
            // ---- mover of the residual's pieces: two ahead of the epilogue in, behind it out.  A piece's buffer is loaded
            // again once every store so far has read its shared memory, which frees the panel of rows two pieces back too ----
            constexpr int kPieces = BN / 32;
            const int my_tiles = worker < num_tiles ? (num_tiles - 1 - worker) / workers + 1 : 0;
            const int total = my_tiles * kPieces;
            auto load = [&](int i) {
                const int tile = worker + i / kPieces * workers, b = i % kStreamBufs;
                mbar_expect_tx(&res_full[b], kStreamPiece);
                tma_load_2d(pieces + (size_t)b * kStreamPiece, &extra.res, &res_full[b], (tile % n_blocks) * kOutCols + i % kPieces * 32,
                            (tile / n_blocks) * kTileRows + (int)rank * kTcBM);
            };
            for (int i = 0; i < kStreamBufs && i < total; ++i) load(i);
            for (int i = 0; i < total; ++i) {
                const int tile = worker + i / kPieces * workers, b = i % kStreamBufs;
                const int m0 = (tile / n_blocks) * kTileRows + (int)rank * kTcBM, n0 = (tile % n_blocks) * kOutCols + i % kPieces * 32;
                if (!mbar_wait(&res_done[b], (uint32_t)((i / kStreamBufs) & 1))) { atomicExch(error_flag, 5); s_abort = 1; break; }
                if (*(volatile int*)&s_abort) break;
                if (m0 < M) {
                    if (n0 < N) tma_store_2d(&extra.res, pieces + (size_t)b * kStreamPiece, n0, m0);
                    if ((i & 1) && n0 - 32 < N) tma_store_2d(&map_out, staging + (size_t)((i >> 1) & 1) * (kTcBM * 128), n0 - 32, m0);
                }
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                if (i + kStreamBufs < total) {
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    load(i + kStreamBufs);
                }
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else {
        // ---- epilogue: warps 2..5 own TMEM lanes 32 * (warp % 4) .. +31 ----
        const int quarter = warp & 3;
        int local = 0;
        bool ok = true;
        // the accumulator goes back to the CTA that issues the MMAs
        auto release_accumulator = [&](int buf) {
            if (PAIR) mbar_arrive_cluster(map_to_cta(&acc_empty[buf], 0));
            else mbar_arrive(&acc_empty[buf]);
        };
        // the sums of squares of this thread's row of the next tile: on their way while this tile's results are stored (read at the
        // tile's start they cost the epilogue, which the gated product waits for, a microsecond a tile)
        bool few_parts = false;
        if constexpr (NORMED) few_parts = extra.norm.squares_in_n <= 16 && extra.norm.squares_in_n % 4 == 0;
        float4 parts[4];
        auto fetch_parts = [&](int tile) {
            const int row = (tile / n_blocks) * kTileRows + (int)rank * kTcBM + quarter * 32 + lane;
            if constexpr (NORMED) if (few_parts && tile < num_tiles && row < M) {
                const TcNorm& norm = extra.norm;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q * 4 < norm.squares_in_n) parts[q] = reinterpret_cast<const float4*>(norm.squares_in + (size_t)row * norm.squares_in_n)[q];
            }
        };
        fetch_parts(worker);
        for (int tile = worker; tile < num_tiles && ok; tile += workers, ++local) {
            const int buf = local & 1;
            const uint32_t acc_phase = (local >> 1) & 1;
            const int m0 = (tile / n_blocks) * kTileRows + (int)rank * kTcBM, n0 = (tile % n_blocks) * kOutCols;
            const int row = m0 + quarter * 32 + lane;
            float factor = 1.f;
            if constexpr (NORMED) if (row < M) {
                const TcNorm& norm = extra.norm;
                float ss = 0.f;
                if (few_parts) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (q * 4 < norm.squares_in_n) ss += (parts[q].x + parts[q].y) + (parts[q].z + parts[q].w);
                } else {
                    for (int p = 0; p < norm.squares_in_n; ++p) ss += norm.squares_in[(size_t)row * norm.squares_in_n + p];
                }
                factor = rsqrtf(ss / (float)K + norm.eps);
            }
            ok = mbar_wait(&acc_full[buf], acc_phase);
            if (!ok && lane == 0) { atomicExch(error_flag, 3); s_abort = 1; }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0 && !(*(volatile int*)&s_abort);
            if (!ok) break;
            tcgen05_fence_after();
            fetch_parts(tile + workers);
            if constexpr (SILU) {
                const int r_local = quarter * 32 + lane;
                const bool store_thread = threadIdx.x == 64;
                if (store_thread) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // staging is free again
                epilogue_barrier();
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    uint32_t gv[32], uv[32];
                    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c * 32);
                    tmem_ld_32x32b_x32(taddr, gv);
                    tmem_ld_32x32b_x32(taddr + (uint32_t)(BN / 2), uv);
                    tmem_ld_wait();
                    if (c == 3) {
                        tcgen05_fence_before();
                        if (lane == 0) release_accumulator(buf);     // the accumulator has been read completely
                    }
                    unsigned char* panel = staging + (size_t)(c >> 1) * (kTcBM * 128) + (size_t)r_local * 128;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float y[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float g = NORMED ? __uint_as_float(gv[8 * j + e]) * factor : __uint_as_float(gv[8 * j + e]);
                            const float u = NORMED ? __uint_as_float(uv[8 * j + e]) * factor : __uint_as_float(uv[8 * j + e]);
                            // silu(g) = g / (1 + 2^(-g log2 e)) with the hardware's ex2 and reciprocal: the exact expf
                            // and division, with four epilogue warps, took longer than the tile's MMAs (a 2048 x 6144 x
                            // 1024 product went from 26 to 40 us).  The two approximations are good to about 2^-21
                            // relative, far inside the 2^-9 of the bfloat16 rounding that follows; exp overflowing to
                            // infinity for g < -88 gives g / inf = -0, the limit
                            // SILU == 2: the tanh form of GELU, g (1 + tanh z) / 2 = g / (1 + exp(-2 z)) with
                            // z = sqrt(2 / pi) (g + 0.044715 g^3): the same shape with another exponent
                            const float arg = SILU == 2 ? -2.f * 0.7978845608028654f * fmaf(0.044715f * g * g, g, g) : -g;
                            float ex;
                            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex) : "f"(arg * 1.4426950408889634f));
                            y[e] = __fdividef(g, 1.f + ex) * u;
                        }
                        uint4 pk;
                        __nv_bfloat162 t0 = __floats2bfloat162_rn(y[0], y[1]), t1 = __floats2bfloat162_rn(y[2], y[3]);
                        __nv_bfloat162 t2 = __floats2bfloat162_rn(y[4], y[5]), t3 = __floats2bfloat162_rn(y[6], y[7]);
                        pk.x = *reinterpret_cast<uint32_t*>(&t0); pk.y = *reinterpret_cast<uint32_t*>(&t1);
                        pk.z = *reinterpret_cast<uint32_t*>(&t2); pk.w = *reinterpret_cast<uint32_t*>(&t3);
                        const int chunk = ((c & 1) * 4 + j) ^ (r_local & 7);       // 128-byte swizzle
                        *reinterpret_cast<uint4*>(panel + chunk * 16) = pk;
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                epilogue_barrier();
                if (store_thread) {
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const int col = n0 + p * 64;
                        if (col < n_out) tma_store_2d(&map_out, staging + (size_t)p * (kTcBM * 128), col, m0);
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else if constexpr (STREAM) {
                const TcNorm& norm = extra.norm;
                const int r_local = quarter * 32 + lane;
                float sq = 0.f;
                float gain = n0 + lane < N ? norm.gain[n0 + lane] : 0.f;         // a lane's column of the next 32
#pragma unroll 1
                for (int c = 0; c < BN / 32 && ok; ++c) {
                    const int piece = local * (BN / 32) + c, b = piece % kStreamBufs;
                    ok = mbar_wait(&res_full[b], (uint32_t)((piece / kStreamBufs) & 1));
                    if (!ok && lane == 0) { atomicExch(error_flag, 6); s_abort = 1; }
                    ok = __all_sync(0xffffffffu, ok) != 0;
                    if (!ok) break;
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c * 32), v);
                    // (two rows of gains in turn: a lane that writes the third has passed the warp's barrier behind the first)
                    float* gains = s_gain + ((warp - 2) * 2 + (c & 1)) * 32;
                    gains[lane] = gain;
                    __syncwarp();
                    const int next = n0 + (c + 1) * 32 + lane;
                    gain = c + 1 < BN / 32 && next < N ? norm.gain[next] : 0.f;
                    tmem_ld_wait();
                    if (c == BN / 32 - 1) {
                        tcgen05_fence_before();
                        if (lane == 0) release_accumulator(buf);
                    }
                    // 32 columns: eight 16-byte chunks of the residual's row, four of the bfloat16 panel's
                    unsigned char* res_row = pieces + (size_t)b * kStreamPiece + (size_t)r_local * 128;
                    unsigned char* panel = staging + (size_t)((piece >> 1) & 1) * (kTcBM * 128) + (size_t)r_local * 128;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t pk[4];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float4* at = reinterpret_cast<float4*>(res_row + ((2 * j + h) ^ (r_local & 7)) * 16);
                            float4 x = *at;
                            const float4 gw = *reinterpret_cast<const float4*>(gains + j * 8 + h * 4);
                            x.x += __uint_as_float(v[8 * j + 4 * h]); x.y += __uint_as_float(v[8 * j + 4 * h + 1]);
                            x.z += __uint_as_float(v[8 * j + 4 * h + 2]); x.w += __uint_as_float(v[8 * j + 4 * h + 3]);
                            sq += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
                            *at = x;
                            pk[2 * h] = pack_bf16(x.x * gw.x, x.y * gw.y);
                            pk[2 * h + 1] = pack_bf16(x.z * gw.z, x.w * gw.w);
                        }
                        *reinterpret_cast<uint4*>(panel + (((c & 1) * 4 + j) ^ (r_local & 7)) * 16) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&res_done[b]);
                }
                if (row < M && ok) norm.squares_out[(size_t)row * n_blocks + tile % n_blocks] = sq;
            } else if constexpr (TMA_STORE) {
                const int r_local = quarter * 32 + lane;                 // row of the tile = TMEM lane
                const bool store_thread = threadIdx.x == 64;
#pragma unroll 1
                for (int half = 0; half < BN / 128; ++half) {
                    if (store_thread) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // staging is free again
                    epilogue_barrier();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t v[32];
                        tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + half * 128 + c * 32), v);
                        tmem_ld_wait();
                        if (half == BN / 128 - 1 && c == 3) {
                            tcgen05_fence_before();
                            if (lane == 0) release_accumulator(buf);     // the accumulator has been read completely
                        }
                        if (NORMED) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * factor);
                        }
                        // 32 columns = 64 bytes = four 16-byte chunks of this row, in panel c / 2, chunks (c % 2) * 4 ..
                        unsigned char* panel = staging + (size_t)(c >> 1) * (kTcBM * 128) + (size_t)r_local * 128;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint4 pk;
                            __nv_bfloat162 t0 = __floats2bfloat162_rn(__uint_as_float(v[8 * j]), __uint_as_float(v[8 * j + 1]));
                            __nv_bfloat162 t1 = __floats2bfloat162_rn(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
                            __nv_bfloat162 t2 = __floats2bfloat162_rn(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
                            __nv_bfloat162 t3 = __floats2bfloat162_rn(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
                            pk.x = *reinterpret_cast<uint32_t*>(&t0); pk.y = *reinterpret_cast<uint32_t*>(&t1);
                            pk.z = *reinterpret_cast<uint32_t*>(&t2); pk.w = *reinterpret_cast<uint32_t*>(&t3);
                            const int chunk = ((c & 1) * 4 + j) ^ (r_local & 7);       // 128-byte swizzle
                            *reinterpret_cast<uint4*>(panel + chunk * 16) = pk;
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    epilogue_barrier();
                    if (store_thread) {
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const int col = n0 + half * 128 + p * 64;
                            if (col < N) tma_store_2d(&map_out, staging + (size_t)p * (kTcBM * 128), col, m0);
                        }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
            } else {
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c0), v);
                tmem_ld_wait();
                if (NORMED) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * factor);
                }
                if (c0 + 32 >= BN) {
                    // the accumulator has been read completely: hand it back before the stores
                    tcgen05_fence_before();
                    if (lane == 0) release_accumulator(buf);
                }
                if (row < M) {
                    const int n = n0 + c0;
                    if (F32OUT) {
                        float* dst = reinterpret_cast<float*>(out) + (size_t)row * ldo + n;
                        if (n + 32 <= N && (ldo % 4) == 0) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4)
                                *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                                  __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (n + j < N) dst[j] = __uint_as_float(v[j]);
                        }
                    } else {
                        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out) + (size_t)row * ldo + n;
                        if (n + 32 <= N && (ldo % 8) == 0) {
#pragma unroll
                            for (int j = 0; j < 32; j += 8) {
                                uint4 pk;
                                __nv_bfloat162 t0 = __floats2bfloat162_rn(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                                __nv_bfloat162 t1 = __floats2bfloat162_rn(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                                __nv_bfloat162 t2 = __floats2bfloat162_rn(__uint_as_float(v[j + 4]), __uint_as_float(v[j + 5]));
                                __nv_bfloat162 t3 = __floats2bfloat162_rn(__uint_as_float(v[j + 6]), __uint_as_float(v[j + 7]));
                                pk.x = *reinterpret_cast<uint32_t*>(&t0); pk.y = *reinterpret_cast<uint32_t*>(&t1);
                                pk.z = *reinterpret_cast<uint32_t*>(&t2); pk.w = *reinterpret_cast<uint32_t*>(&t3);
                                *reinterpret_cast<uint4*>(dst + j) = pk;
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (n + j < N) dst[j] = __float2bfloat16_rn(__uint_as_float(v[j]));
                        }
                    }
                }
            }
            }
        }
    }
    // ---- teardown: everything issued has been waited for on the normal path; free the tensor memory ----
    if (TMA_STORE && !STREAM && threadIdx.x == 64) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    tcgen05_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();          // neither CTA leaves while the other may still arrive on its barriers
    if (warp == 1) {
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * BN)) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * BN)) : "memory");
    }
}

// CUINFER_B200_GEMM_PAIR=0 keeps one CTA per tile, for comparisons (and no product adds to the residual: that takes pairs).
static bool pair_allowed() {
    static const bool allowed = [] { const char* e = getenv("CUINFER_B200_GEMM_PAIR"); return !(e && e[0] == '0'); }();
    return allowed;
}

static int make_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows) {
    return tc_make_map(map, base, rows, K, ld, box_rows, "gemm_tcgen05");
}

template <int BN, int STAGES, bool F32OUT, bool TMA_STORE, int SILU = 0, bool PAIR = false, bool STREAM = false, bool NORMED = false>
static int launch_tc(const CUtensorMap& ma, const CUtensorMap& mw, const CUtensorMap& mo, const TcNorm& norm, void* out, int ldo, int M,
                     int N, int K, int* error_flag, cudaStream_t stream, int up_offset = 0, const CUtensorMap* mr = nullptr) {
    // (a kernel of its own for rows that carry a norm: two more multiplications a value cost the gated epilogue, which its tiles wait
    // for, 1.6 us a layer at 2 048 rows.  All stores and tile forms have it: a reader of such rows may have few features, a number of
    // them that is not a multiple of eight, or 32-bit results)
    if constexpr (!NORMED && !STREAM)
        if (norm.squares_in != nullptr)
            return launch_tc<BN, STAGES, F32OUT, TMA_STORE, SILU, PAIR, STREAM, true>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream, up_offset, mr);
    auto kernel = gemm_tcgen05_kernel<BN, STAGES, F32OUT, TMA_STORE, SILU, PAIR, STREAM, NORMED>;
    constexpr int smem = TcSmem<BN, STAGES, PAIR, STREAM>::kTotal;
    constexpr int threads = STREAM ? 224 : 192;
    TcExtra<STREAM, NORMED> extra;
    if constexpr (STREAM) extra.res = *mr;
    if constexpr (STREAM || NORMED) extra.norm = norm;
    static_assert(smem <= 227 * 1024, "a CTA has 227 KB of shared memory");
    static SmemLimit limit;
    if (int rc = raise_smem_limit(limit, kernel, smem, "gemm_tcgen05")) return rc;
    static int num_sms = 0;
    if (num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || num_sms <= 0) num_sms = 148;
    }
    const int out_cols = SILU ? BN / 2 : BN, n_out = SILU ? up_offset : N;
    const int tile_rows = PAIR ? 2 * kTcBM : kTcBM;
    const int tiles = ((n_out + out_cols - 1) / out_cols) * ((M + tile_rows - 1) / tile_rows);
    if (!PAIR) {
        dim3 grid(tiles < num_sms ? tiles : num_sms);
        cudaError_t e = launch_pdl(kernel, grid, dim3(threads), (size_t)smem, stream, prompt_pdl(), ma, mw, mo, extra, out, ldo, M, N, K, up_offset, error_flag);
        if (e != cudaSuccess) {
            set_error("gemm_tcgen05: launch failed: %s", cudaGetErrorString(e));
            return -2;
        }
        return 0;
    }
    // clusters of two CTAs, one pair per tile at a time
    const int pairs = tiles < num_sms / 2 ? tiles : num_sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = prompt_pdl() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mw, mo, extra, out, ldo, M, N, K, up_offset, error_flag);
    if (e != cudaSuccess) {
        set_error("gemm_tcgen05: launch of CTA pairs failed: %s", cudaGetErrorString(e));
        return -2;
    }
    return 0;
}

}  // namespace cib

using namespace cib;

extern "C" int cib_gemm_tcgen05_supports(int M, int N, int K) {
    return M >= 1 && N >= 8 && K >= 8 && K % 8 == 0;
}

// The columns of a tile of the product that adds to the residual (squares_out has ceil(N / that) sums a row), or 0 where it does not
// take the shape: it runs as pairs of CTAs.
extern "C" int cib_gemm_tcgen05_stream_cols(int M, int N, int K) {
    if (!cib_gemm_tcgen05_supports(M, N, K) || !pair_allowed() || M < 256 || N % 8 != 0) return 0;
    const int m_pairs = (M + 255) / 256;
    if (m_pairs * ((N + 127) / 128) < 74) return 0;
    return N % 256 == 0 && (N / 256) * m_pairs >= 60 ? 256 : 128;
}

// a: [M, K] bfloat16 rows (lda), w: [N, K] bfloat16 rows (ldw), out: [M, N] bfloat16 (out_f32 = 0) or float32.
// error_flag: one int in device memory, zero before the call; non-zero afterwards means a bounded wait gave up.
// silu_pair: w holds N / 2 gate rows followed by N / 2 up rows and out is [M, N / 2] bfloat16 = act(a gate^T) * (a up^T),
// act = SiLU (1) or the tanh form of GELU (2).
// squares_in: [M][squares_in_n] (or null): every result row is multiplied by rsqrt(sum(squares_in[row]) / K + eps).
// stream_rows: 32-bit [M, N], dense (or null): it grows by the product, out = bfloat16(stream_rows * gain), squares_out
// [M][ceil(N / cib_gemm_tcgen05_stream_cols)] = the sums of stream_rows^2 over a tile's columns.
extern "C" int cib_gemm_tcgen05(const void* a, int lda, const void* w, int ldw, void* out, int ldo, int out_f32, int silu_pair,
                                int M, int N, int K, const float* squares_in, int squares_in_n, float eps, float* stream_rows,
                                const void* gain, int gain_dtype, float* squares_out, int* error_flag, cudaStream_t stream) {
    CIB_REQUIRE(cib_gemm_tcgen05_supports(M, N, K), "gemm_tcgen05: M=%d N=%d K=%d is not taken (K must be a multiple of 8)", M, N, K);
    CIB_REQUIRE(lda >= K && ldw >= K && lda % 8 == 0 && ldw % 8 == 0, "gemm_tcgen05: row strides must be multiples of 8 elements");
    CIB_REQUIRE(((uintptr_t)a % 16) == 0 && ((uintptr_t)w % 16) == 0, "gemm_tcgen05: operands must be 16-byte aligned");
    CIB_REQUIRE(ldo >= (silu_pair ? N / 2 : N) && error_flag != nullptr, "gemm_tcgen05: bad output arguments");
    CIB_REQUIRE(squares_in == nullptr || (squares_in_n > 0 && ((uintptr_t)squares_in % 16) == 0), "gemm_tcgen05: sums of squares without parts, or not on 16 bytes");
    const TcNorm norm = {squares_in, squares_in_n, eps, AnyVec{gain, gain_dtype == kBF16}, squares_out};
    CUtensorMap ma, mw;
    // From 256 rows on, pairs of CTAs share 256-row tiles
    // (only when there are enough 256-row tiles for every pair of SMs: with fewer, one CTA per 128-row tile measured faster)
    const int pair_tiles = ((M + 255) / 256) * (((silu_pair ? N / 2 : N) + 127) / 128);
    const bool pair = pair_allowed() && M >= 256 && pair_tiles >= 74;
    if (stream_rows != nullptr) {
        const int bn = cib_gemm_tcgen05_stream_cols(M, N, K);
        CIB_REQUIRE(bn > 0 && !out_f32 && !silu_pair && gain != nullptr && squares_out != nullptr && ldo % 8 == 0 && ((uintptr_t)out % 16) == 0 &&
                        ((uintptr_t)stream_rows % 16) == 0,
                    "gemm_tcgen05: the stream epilogue does not take M=%d N=%d K=%d or its arguments", M, N, K);
        CUtensorMap mo3, mr;
        if (make_map(&ma, a, M, K, lda, kTcBM) != 0 || make_map(&mw, w, N, K, ldw, bn / 2) != 0 || make_map(&mo3, out, M, N, ldo, kTcBM) != 0 ||
            encode_tensor_map_f32_2d(&mr, stream_rows, M, N, N, 32, kTcBM, "gemm_tcgen05") != 0)
            return -1;
        if (bn == 256) return launch_tc<256, 5, false, true, 0, true, true>(ma, mw, mo3, norm, out, ldo, M, N, K, error_flag, stream, 0, &mr);
        return launch_tc<128, 6, false, true, 0, true, true>(ma, mw, mo3, norm, out, ldo, M, N, K, error_flag, stream, 0, &mr);
    }
    if (silu_pair) {
        const int half = N / 2;
        CIB_REQUIRE(N % 2 == 0 && !out_f32 && ldo % 8 == 0 && ((uintptr_t)out % 16) == 0,
                    "gemm_tcgen05: the gated epilogue stores bfloat16 rows that are 16-byte aligned, N even");
        CUtensorMap mo;
        if (make_map(&ma, a, M, K, lda, kTcBM) != 0 || make_map(&mw, w, N, K, ldw, 128) != 0 ||
            make_map(&mo, out, M, half, ldo, kTcBM) != 0)
            return -1;
        if (silu_pair == 2) {       // the gate is the tanh form of GELU
            if (pair) return launch_tc<256, 6, false, true, 2, true>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream, half);
            return launch_tc<256, 4, false, true, 2>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream, half);
        }
        if (pair) return launch_tc<256, 6, false, true, 1, true>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream, half);
        return launch_tc<256, 4, false, true, 1>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream, half);
    }
    if (pair) {
        // 256 x 256 tiles when those still give most pairs a tile, else 256 x 128; a CTA loads half of a tile's weight rows
        const int m_pairs = (M + 255) / 256;
        const int bn2 = (N % 256 == 0 && (N / 256) * m_pairs >= 60) ? 256 : 128;
        const bool tma_out2 = !out_f32 && ldo % 8 == 0 && ((uintptr_t)out % 16) == 0;
        CUtensorMap mo2;
        if (make_map(&ma, a, M, K, lda, kTcBM) != 0 || make_map(&mw, w, N, K, ldw, bn2 / 2) != 0) return -1;
        mo2 = ma;
        if (tma_out2 && make_map(&mo2, out, M, N, ldo, kTcBM) != 0) return -1;
        if (bn2 == 256) {
            if (out_f32) return launch_tc<256, 6, true, false, false, true>(ma, mw, mo2, norm, out, ldo, M, N, K, error_flag, stream);
            if (tma_out2) return launch_tc<256, 6, false, true, false, true>(ma, mw, mo2, norm, out, ldo, M, N, K, error_flag, stream);
            return launch_tc<256, 6, false, false, false, true>(ma, mw, mo2, norm, out, ldo, M, N, K, error_flag, stream);
        }
        if (out_f32) return launch_tc<128, 8, true, false, false, true>(ma, mw, mo2, norm, out, ldo, M, N, K, error_flag, stream);
        if (tma_out2) return launch_tc<128, 8, false, true, false, true>(ma, mw, mo2, norm, out, ldo, M, N, K, error_flag, stream);
        return launch_tc<128, 8, false, false, false, true>(ma, mw, mo2, norm, out, ldo, M, N, K, error_flag, stream);
    }
    // Tile width: 256 when that still gives most SMs a tile, else 128.
    const int m_blocks = (M + 127) / 128;
    int bn = 128;
    if (N % 256 == 0 && (N / 256) * m_blocks >= 120) bn = 256;
    if (make_map(&ma, a, M, K, lda, kTcBM) != 0) return -1;
    if (make_map(&mw, w, N, K, ldw, bn) != 0) return -1;
    // bfloat16 results with 16-byte aligned rows leave by TMA store; anything else is stored by the threads
    const bool tma_out = !out_f32 && ldo % 8 == 0 && ((uintptr_t)out % 16) == 0;
    CUtensorMap mo = ma;
    if (tma_out && make_map(&mo, out, M, N, ldo, kTcBM) != 0) return -1;
    if (bn == 256) {
        if (out_f32) return launch_tc<256, 4, true, false>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream);
        if (tma_out) return launch_tc<256, 4, false, true>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream);
        return launch_tc<256, 4, false, false>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream);
    }
    if (out_f32) return launch_tc<128, 5, true, false>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream);
    if (tma_out) return launch_tc<128, 5, false, true>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream);
    return launch_tc<128, 5, false, false>(ma, mw, mo, norm, out, ldo, M, N, K, error_flag, stream);
}
