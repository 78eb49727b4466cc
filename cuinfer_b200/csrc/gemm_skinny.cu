// out[M, N] = act[M, K] · W[N, K]^T for a handful of rows (M <= 16): the decode-step projections, bfloat16.
//
// The reference sends these to cuBLAS one by one, with a norm kernel before and an activation kernel after
// (csrc/model/layers/attention.cpp:44-105, csrc/model/layers/mlp.cpp:21-27, csrc/ops/projection.cu:32-44).
// With few rows the product is a single pass over the weights, and a decode step is a chain of such passes that is bound by
// what each of them needs between the end of the kernel before it and its own last store.  So:
//
//   * the weight matrix is the A operand of mma.sync m16n8k16 (16 output features x 16 k), the rows of the batch are the B
//     operand (k x 8 rows): "swap A/B".  Every lane reads its A fragments straight from global memory as 16-byte loads
//     (8 consecutive k of one weight row), which fixes a permutation of k inside each 32-k step; every weight byte is read
//     exactly once.  The loads of the first 2 048 / RW values of K are issued before `griddepcontrol.wait`: with programmatic
//     dependent launch a projection's weights arrive while the kernel before it is still running;
//   * the eight warps of a CTA each take an eighth of its K, so the activations a warp needs are its own: it reads its B
//     fragments straight from global memory too, with the same permutation of k (one round trip to the L2 after the wait,
//     no shared memory and no barrier before the MMAs);
//   * slices are summed in shared memory in a fixed order, so results do not depend on timing or on the other rows;
//   * a norm between two projections costs no kernel and no pass of its own: the projection before it (`stream` epilogue) adds
//     its result to the 32-bit residual, stores the rows times the norm's gains in bfloat16 and the squares' sum over each
//     16 columns; the projection after it multiplies those rows and applies rsqrt(mean square + eps) per row to its 32-bit
//     sums.  (Both see one rounding of a row to bfloat16, as when the factor is applied first.)
//   * other epilogues: rows come in (gate, up) pairs and act(gate) * up is stored; or the result is stored in 32 bits.
//
// A second kernel keeps the norm of 32-bit rows in its prologue, for rows that no projection of this file produced.
#include "mma_utils.cuh"

namespace cib {

constexpr int kSkWarps = 8;
constexpr int kSkU = 4;           // 32-k steps whose weight loads are in flight together

enum SkinnyEpilogue : int { kStoreBf16 = 0, kStoreF32 = 1, kSiluPair = 2, kStream = 3 };

struct SkinnyArgs {
    const __nv_bfloat16* w; int ldw; int N; int K;
    const __nv_bfloat16* act; int lda;                       // plain activations, or
    const float* res_in; const void* pending; int pending_bf16; AnyVec norm_w; float eps; float* res_out;
    void* out; int ldo; int M;
    int up_offset;                                           // kSiluPair: first row of the "up" half
    int act_stride;                                          // norm prologue: shared-memory row stride in elements
    const void* warm; unsigned long long warm_bytes;         // the weights of the kernel after this one (or null): fetched into L2
    int norm_w_offset;                                       // norm prologue: byte offset of the gains' copy in shared memory
    int gate_gelu;                                           // kSiluPair: the gate is the tanh form of GELU instead of SiLU
    // rows that carry a norm still to be applied: sums of squares [M][squares_in_n] of the rows before their gains (or null)
    const float* squares_in; int squares_in_n;
    // kStream: residual [M, N] in 32 bits, updated in place; out then receives the new rows times norm_w, squares_out [M][tiles]
    // their squares' sums over 16 columns each
    float* stream; float* squares_out; int squares_out_n;
};

__device__ __forceinline__ uint4 ldg_stream16(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// Rows normed in the prologue.  A CTA has 8 warps: RT tiles of 16 output features x KS slices of K.
template <int MT, int RT, int KS, int EPI>
__global__ void __launch_bounds__(kSkWarps * 32)
skinny_norm_gemm_kernel(const SkinnyArgs a) {
    const int tile_block = (int)blockIdx.x;
    static_assert(RT * KS == kSkWarps, "a CTA has 8 warps");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16* s_act = reinterpret_cast<__nv_bfloat16*>(smem_raw);                  // [MT*8][act_stride]
    float* s_red = reinterpret_cast<float*>(smem_raw + (size_t)MT * 8 * a.act_stride * 2); // [KS][RT][16][MT*8]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = lane & 3, qrow = lane >> 2;
    const int rt = warp % RT, ks = warp / RT;

    // rows of this warp's tile
    int tile_row0;
    if (EPI == kSiluPair) tile_row0 = (rt == 0 ? 0 : a.up_offset) + tile_block * 16;
    else tile_row0 = (tile_block * RT + rt) * 16;
    const int row_limit = (EPI == kSiluPair) ? (rt == 0 ? a.up_offset : a.N) : a.N;
    const int r0 = tile_row0 + qrow, r1 = r0 + 8;
    const bool ok0 = r0 < row_limit, ok1 = r1 < row_limit;
    const __nv_bfloat16* w0 = a.w + (size_t)(ok0 ? r0 : 0) * a.ldw;
    const __nv_bfloat16* w1 = a.w + (size_t)(ok1 ? r1 : 0) * a.ldw;

    // k range of this warp's slice, in 32-k steps
    const int steps_total = (a.K + 31) / 32;
    const int steps_per = (steps_total + KS - 1) / KS;
    const int step_begin = ks * steps_per;
    const int step_end = min(steps_total, step_begin + steps_per);

    // two register buffers of kSkU steps each, named apart so that every index is a compile-time constant
    uint4 waA[kSkU], wbA[kSkU], waB[kSkU], wbB[kSkU];
    auto load_chunk = [&](uint4 (&wa)[kSkU], uint4 (&wb)[kSkU], int step0) {
#pragma unroll
        for (int u = 0; u < kSkU; ++u) {
            const int k = (step0 + u) * 32 + quad * 8;
            const bool in = step0 + u < step_end && k < a.K;
            wa[u] = (in && ok0) ? ldg_stream16(w0 + k) : make_uint4(0, 0, 0, 0);
            wb[u] = (in && ok1) ? ldg_stream16(w1 + k) : make_uint4(0, 0, 0, 0);
        }
    };
    load_chunk(waA, wbA, step_begin);   // weights do not depend on the kernel before this one
    if (tid == 0) warm_l2_share(a.warm, a.warm_bytes, blockIdx.x, gridDim.x);
    // neither do the norm's gains: they wait in shared memory (read from global memory in the second pass of the norm,
    // eight dependent round trips per row, they were a third of this kernel's time)
    float* s_nw = reinterpret_cast<float*>(smem_raw + a.norm_w_offset);
    for (int k = tid; k < a.K; k += kSkWarps * 32) s_nw[k] = a.norm_w[k];
    griddep_launch();
    griddep_wait();                     // from here on the previous kernel's results may be read
    __syncthreads();                    // the gains' copy is complete

    // ---- normed rows -> shared memory (bfloat16, padded) ----
    const int rows_pad = MT * 8;
    {
        float* s_x = reinterpret_cast<float*>(s_red);               // un-normalised 32-bit rows [rows][K]
        for (int row = warp; row < rows_pad; row += kSkWarps) {
            float ss = 0.f;
            if (row < a.M) {
                const float* rp = a.res_in + (size_t)row * a.K;
                // eight independent 16-byte loads of the residual (and of the delta) are in flight per lane
                for (int k0 = lane * 4; k0 < a.K; k0 += 128 * 8) {
                    float4 x[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int k = k0 + u * 128;
                        x[u] = k < a.K ? *reinterpret_cast<const float4*>(rp + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    if (a.pending) {
                        if (a.pending_bf16) {
                            uint2 pv[8];
                            const __nv_bfloat16* pp = reinterpret_cast<const __nv_bfloat16*>(a.pending) + (size_t)row * a.K;
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                const int k = k0 + u * 128;
                                pv[u] = k < a.K ? *reinterpret_cast<const uint2*>(pp + k) : make_uint2(0u, 0u);
                            }
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                const __nv_bfloat162 p01 = *reinterpret_cast<const __nv_bfloat162*>(&pv[u].x);
                                const __nv_bfloat162 p23 = *reinterpret_cast<const __nv_bfloat162*>(&pv[u].y);
                                x[u].x += __low2float(p01); x[u].y += __high2float(p01);
                                x[u].z += __low2float(p23); x[u].w += __high2float(p23);
                            }
                        } else {
                            const float* pp = reinterpret_cast<const float*>(a.pending) + (size_t)row * a.K;
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                const int k = k0 + u * 128;
                                if (k < a.K) {
                                    const float4 pv = *reinterpret_cast<const float4*>(pp + k);
                                    x[u].x += pv.x; x[u].y += pv.y; x[u].z += pv.z; x[u].w += pv.w;
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int k = k0 + u * 128;
                        if (k < a.K) {
                            ss += x[u].x * x[u].x + x[u].y * x[u].y + x[u].z * x[u].z + x[u].w * x[u].w;
                            if (tile_block == 0 && a.res_out) *reinterpret_cast<float4*>(a.res_out + (size_t)row * a.K + k) = x[u];
                            *reinterpret_cast<float4*>(s_x + (size_t)row * a.K + k) = x[u];
                        }
                    }
                }
                ss = warp_sum(ss);
            }
            const float factor = row < a.M ? rsqrtf(ss / (float)a.K + a.eps) : 0.f;
            __syncwarp();
            for (int k = lane * 4; k < a.K; k += 128) {
                float4 x = row < a.M ? *reinterpret_cast<const float4*>(s_x + (size_t)row * a.K + k)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 gw = *reinterpret_cast<const float4*>(s_nw + k);
                const float n0 = x.x * factor * gw.x, n1 = x.y * factor * gw.y;
                const float n2 = x.z * factor * gw.z, n3 = x.w * factor * gw.w;
                uint2 pk;
                pk.x = pack_bf16(n0, n1);
                pk.y = pack_bf16(n2, n3);
                *reinterpret_cast<uint2*>(s_act + (size_t)row * a.act_stride + k) = pk;
            }
        }
    }
    __syncthreads();

    // ---- main loop over this warp's k slice ----
    // two accumulators per row tile, one for each half of a 32-k step: a warp's MMAs then form two chains of half the
    // length instead of one (the k slices are short, so the chain's latency is most of the loop; four chains measured
    // no better); summed at the end
    float acc[MT][4], acc2[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = acc2[i][e] = 0.f;
    }
    auto compute_chunk = [&](const uint4 (&wa)[kSkU], const uint4 (&wb)[kSkU], int step0) {
#pragma unroll
        for (int u = 0; u < kSkU; ++u) {
            if (step0 + u < step_end) {
                const int k = (step0 + u) * 32 + quad * 8;
                const uint32_t a1[4] = {wa[u].x, wb[u].x, wa[u].y, wb[u].y};
                const uint32_t a2[4] = {wa[u].z, wb[u].z, wa[u].w, wb[u].w};
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    uint4 bv = make_uint4(0, 0, 0, 0);
                    if (k < a.K) bv = *reinterpret_cast<const uint4*>(s_act + (size_t)(nt * 8 + qrow) * a.act_stride + k);
                    mma_bf16_16816(acc[nt], a1, bv.x, bv.y);
                    mma_bf16_16816(acc2[nt], a2, bv.z, bv.w);
                }
            }
        }
    };
    for (int step0 = step_begin; step0 < step_end; step0 += 2 * kSkU) {
        load_chunk(waB, wbB, step0 + kSkU);
        compute_chunk(waA, wbA, step0);
        load_chunk(waA, wbA, step0 + 2 * kSkU);
        compute_chunk(waB, wbB, step0 + kSkU);
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] += acc2[i][e];
    }

    // ---- sum the k slices (fixed order), then the epilogue ----
    __syncthreads();                       // the activations (and the norm's scratch) are no longer needed
    constexpr int kCols = MT * 8;
    float* red = reinterpret_cast<float*>(smem_raw);                                    // [KS][RT][16][kCols]
#pragma unroll
    for (int nt = 0; nt < MT; ++nt) {
        float* base = red + (((size_t)ks * RT + rt) * 16) * kCols + nt * 8 + quad * 2;
        base[(size_t)qrow * kCols] = acc[nt][0];
        base[(size_t)qrow * kCols + 1] = acc[nt][1];
        base[(size_t)(qrow + 8) * kCols] = acc[nt][2];
        base[(size_t)(qrow + 8) * kCols + 1] = acc[nt][3];
    }
    __syncthreads();
    if (EPI == kSiluPair) {
        for (int idx = tid; idx < 16 * kCols; idx += kSkWarps * 32) {
            const int token = idx / 16, nl = idx % 16;
            if (token >= a.M) continue;
            float gsum = 0.f, usum = 0.f;
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                gsum += red[(((size_t)s * RT + 0) * 16 + nl) * kCols + token];
                usum += red[(((size_t)s * RT + 1) * 16 + nl) * kCols + token];
            }
            const int n = tile_block * 16 + nl;
            if (n < a.up_offset)
                reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)token * a.ldo + n] = __float2bfloat16_rn(
                    (a.gate_gelu ? 0.5f * gsum * (1.f + tanhf(0.7978845608028654f * (gsum + 0.044715f * gsum * gsum * gsum)))
                                 : gsum / (1.f + expf(-gsum))) * usum);
        }
    } else {
        for (int idx = tid; idx < RT * 16 * kCols; idx += kSkWarps * 32) {
            const int token = idx / (RT * 16), nl = idx % (RT * 16);
            if (token >= a.M) continue;
            const int t = nl / 16, r = nl % 16;
            float sum = 0.f;
#pragma unroll
            for (int s = 0; s < KS; ++s) sum += red[(((size_t)s * RT + t) * 16 + r) * kCols + token];
            const int n = tile_block * RT * 16 + nl;
            if (n < a.N) {
                if (EPI == kStoreF32) reinterpret_cast<float*>(a.out)[(size_t)token * a.ldo + n] = sum;
                else reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)token * a.ldo + n] = __float2bfloat16_rn(sum);
            }
        }
    }
}

// Plain rows, or rows that carry a norm (`squares_in`).  All 8 warps split K; every warp multiplies the CTA's RW row tiles of 16
// output features (kSiluPair: the first half gates, the second half the matching ups), so it reads its activations once.
// CS > 1: a cluster of CS CTAs shares the row tiles, each CTA taking 1/CS of K; the partial sums meet in the shared memory of
// the cluster's first CTA (distributed shared memory), which stores the result.
// PRE: a warp's slice of K fits into this many chunks of kSkU / RW 32-k steps (1 or 2), all of which are asked for up front; 0: it
// may be longer, and the two buffers go round.
template <int MT, int RW, int EPI, int CS, int PRE>
__global__ void __launch_bounds__(kSkWarps * 32, 2)
skinny_gemm_kernel(const SkinnyArgs a) {
    constexpr int KS = kSkWarps;
    // 32-k steps of a chunk: two chunks of weights (64 registers, or 48 beside sixteen rows' activations) are in flight
    constexpr int U = MT == 2 && RW == 1 && PRE == 0 ? 3 : kSkU / RW;
    constexpr int kCols = MT * 8;
    constexpr int kRows = RW * 16;            // output features of the CTA
    constexpr int kPad = kCols + 1;           // floats between two features' sums: the epilogue reads along the features
    __shared__ float s_part[KS][kRows * kPad];
    __shared__ float s_factor[kCols];
    __shared__ float s_inbox[CS > 1 ? (CS - 1) * kRows * kCols : 1];
    const int crank = CS > 1 ? (int)(blockIdx.x % CS) : 0;
    const int tile_block = CS > 1 ? (int)(blockIdx.x / CS) : (int)blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = lane & 3, qrow = lane >> 2;
    // "this CTA runs": its shared memory may be written by the others of the cluster once all have said so
    if (CS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

    // first feature of row tile t, and the features' end
    auto tile_row = [&](int t) {
        if (EPI == kSiluPair) return (t < RW / 2 ? 0 : a.up_offset) + (tile_block * (RW / 2) + t % (RW > 1 ? RW / 2 : 1)) * 16;
        return (tile_block * RW + t) * 16;
    };
    const __nv_bfloat16* w0[RW];
    const __nv_bfloat16* w1[RW];
    bool ok0[RW], ok1[RW];
#pragma unroll
    for (int t = 0; t < RW; ++t) {
        const int limit = EPI == kSiluPair && t < RW / 2 ? a.up_offset : a.N;
        const int r0 = tile_row(t) + qrow, r1 = r0 + 8;
        ok0[t] = r0 < limit;
        ok1[t] = r1 < limit;
        w0[t] = a.w + (size_t)(ok0[t] ? r0 : 0) * a.ldw + quad * 8;
        w1[t] = a.w + (size_t)(ok1[t] ? r1 : 0) * a.ldw + quad * 8;
    }
    // this warp's slice of K, in 32-k steps
    const int steps_total = (a.K + 31) / 32;
    const int steps_per = (steps_total + KS * CS - 1) / (KS * CS);
    const int step_begin = (crank * KS + warp) * steps_per;
    const int step_end = min(steps_total, step_begin + steps_per);

    struct Chunk { uint4 w[U][RW][2]; };
    auto load_w = [&](Chunk& c, int step0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = (step0 + u) * 32;
            const bool in = step0 + u < step_end && k + quad * 8 < a.K;
#pragma unroll
            for (int t = 0; t < RW; ++t) {
                c.w[u][t][0] = (in && ok0[t]) ? ldg_stream16(w0[t] + k) : make_uint4(0, 0, 0, 0);
                c.w[u][t][1] = (in && ok1[t]) ? ldg_stream16(w1[t] + k) : make_uint4(0, 0, 0, 0);
            }
        }
    };
    struct Rows { uint4 b[U][MT]; };
    const __nv_bfloat16* x0[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) x0[i] = a.act + (size_t)min(i * 8 + qrow, a.M - 1) * a.lda + quad * 8;
    auto load_b = [&](Rows& r, int step0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = (step0 + u) * 32;
            const bool in = step0 + u < step_end && k + quad * 8 < a.K;
#pragma unroll
            for (int i = 0; i < MT; ++i)
                r.b[u][i] = in && i * 8 + qrow < a.M ? *reinterpret_cast<const uint4*>(x0[i] + k) : make_uint4(0, 0, 0, 0);
        }
    };
    Chunk wA, wB;                       // two buffers named apart, so that every index is a compile-time constant
    load_w(wA, step_begin);             // weights do not depend on the kernel before this one
    if (PRE != 1) load_w(wB, step_begin + U);
    if (tid == 0) warm_l2_share(a.warm, a.warm_bytes, blockIdx.x, gridDim.x);
    constexpr int kOut = (EPI == kSiluPair ? kRows / 2 : kRows) * kCols;      // values that leave the CTA
    constexpr int kPer = (kOut + kSkWarps * 32 - 1) / (kSkWarps * 32);        // of them a thread's
    float gain[kPer], old[kPer];
    if (EPI == kStream && crank == 0) {
#pragma unroll
        for (int p = 0; p < kPer; ++p) {
            const int n = tile_block * kRows + (tid + p * kSkWarps * 32) % kRows;
            gain[p] = n < a.N ? a.norm_w[n] : 0.f;
        }
    }
    griddep_launch();
    griddep_wait();                     // from here on the previous kernel's results may be read
    Rows xA, xB;
    load_b(xA, step_begin);
    constexpr bool kTwoRows = MT == 1 || RW > 1;       // (sixteen rows of a row tile alone: one buffer of activations fits the registers)
    if (PRE == 2 && kTwoRows) load_b(xB, step_begin + U);
    if (EPI == kStream && crank == 0) {
#pragma unroll
        for (int p = 0; p < kPer; ++p) {
            const int idx = tid + p * kSkWarps * 32, n = tile_block * kRows + idx % kRows, token = idx / kRows;
            old[p] = n < a.N && token < a.M ? a.stream[(size_t)token * a.N + n] : 0.f;
        }
    }
    if (a.squares_in != nullptr && crank == 0) {
        // a row's factor, a warp per row; the first loads of the activations are on their way meanwhile
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int row = i * 8 + warp;
            float ss = 0.f;
            if (row < a.M)
                for (int p = lane; p < a.squares_in_n; p += 32) ss += a.squares_in[(size_t)row * a.squares_in_n + p];
            ss = warp_sum(ss);
            if (lane == 0) s_factor[row] = rsqrtf(ss / (float)a.K + a.eps);
        }
    }

    // with one row tile, two accumulators, one for each half of a 32-k step: a warp's MMAs then form two chains of half the length
    // instead of one; summed at the end
    constexpr int kChains = RW == 1 ? 2 : 1;
    float acc[kChains][RW][MT][4];
#pragma unroll
    for (int c = 0; c < kChains; ++c)
#pragma unroll
        for (int t = 0; t < RW; ++t)
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[c][t][i][e] = 0.f;
    auto compute = [&](const Chunk& c, const Rows& r, int step0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (step0 + u < step_end) {
#pragma unroll
                for (int t = 0; t < RW; ++t) {
                    const uint4 p = c.w[u][t][0], q = c.w[u][t][1];
                    const uint32_t a1[4] = {p.x, q.x, p.y, q.y}, a2[4] = {p.z, q.z, p.w, q.w};
#pragma unroll
                    for (int i = 0; i < MT; ++i) {
                        mma_bf16_16816(acc[0][t][i], a1, r.b[u][i].x, r.b[u][i].y);
                        mma_bf16_16816(acc[kChains - 1][t][i], a2, r.b[u][i].z, r.b[u][i].w);
                    }
                }
            }
        }
    };
    if constexpr (PRE != 0) {
        compute(wA, xA, step_begin);
        if (PRE == 2 && !kTwoRows) load_b(xA, step_begin + U);
        if (PRE == 2) compute(wB, kTwoRows ? xB : xA, step_begin + U);
    } else {
        for (int step0 = step_begin; step0 < step_end; step0 += 2 * U) {
            if (kTwoRows) load_b(xB, step0 + U);
            compute(wA, xA, step0);
            load_w(wA, step0 + 2 * U);
            load_b(xA, step0 + (kTwoRows ? 2 : 1) * U);
            compute(wB, kTwoRows ? xB : xA, step0 + U);
            load_w(wB, step0 + 3 * U);
            if (!kTwoRows) load_b(xA, step0 + 2 * U);
        }
    }

    // ---- sum the k slices (fixed order) ----
#pragma unroll
    for (int t = 0; t < RW; ++t)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                s_part[warp][(t * 16 + qrow + (e >> 1) * 8) * kPad + i * 8 + quad * 2 + (e & 1)] = kChains == 2 ? acc[0][t][i][e] + acc[kChains - 1][t][i][e] : acc[0][t][i][e];
    __syncthreads();
    auto slices = [&](int feature, int token) {
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s < KS; ++s) sum += s_part[s][feature * kPad + token];
        return sum;
    };
    if constexpr (CS > 1) {
        // every CTA sums its own slices; the others then write their sums into slots of the first CTA's shared memory, say so
        // with a release and leave; the first CTA waits for them and sums in rank order
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");       // every CTA of the cluster runs
        if (crank != 0) {
            uint32_t inbox;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(inbox) : "r"(smem_u32(s_inbox + (crank - 1) * kRows * kCols)), "r"(0));
            for (int idx = tid; idx < kRows * kCols; idx += kSkWarps * 32)
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(inbox + (uint32_t)idx * 4), "f"(slices(idx % kRows, idx / kRows)) : "memory");
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            return;
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    float sum[kPer], up[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
        const int idx = tid + p * kSkWarps * 32;
        sum[p] = up[p] = 0.f;
        if (idx < kOut) {
            constexpr int cols = EPI == kSiluPair ? kRows / 2 : kRows;
            sum[p] = slices(idx % cols, idx / cols);
            if (EPI == kSiluPair) up[p] = slices(idx % cols + kRows / 2, idx / cols);
        }
    }
    if constexpr (CS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
        const int idx = tid + p * kSkWarps * 32;
        if (kOut % (kSkWarps * 32) != 0 && idx >= kOut) break;      // (whole warps: kOut is a multiple of 128)
        constexpr int cols = EPI == kSiluPair ? kRows / 2 : kRows;
        const int token = idx / cols, col = idx % cols, n = tile_block * cols + col;
        const bool ok = token < a.M && n < (EPI == kSiluPair ? a.up_offset : a.N);
#pragma unroll
        for (int c = 1; c < CS; ++c) sum[p] += s_inbox[(c - 1) * kRows * kCols + idx];
        const float factor = a.squares_in != nullptr && ok ? s_factor[token] : 1.f;
        const float v = sum[p] * factor;
        if (EPI == kSiluPair) {
            if (ok)
                reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)token * a.ldo + n] = __float2bfloat16_rn(
                    (a.gate_gelu ? 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v))) : v / (1.f + expf(-v))) *
                    (up[p] * factor));
        } else if (EPI == kStream) {
            const float x = old[p] + v;
            float sq = ok ? x * x : 0.f;
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
            if (ok) {
                a.stream[(size_t)token * a.N + n] = x;
                reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)token * a.ldo + n] = __float2bfloat16_rn(x * gain[p]);
                if (n % 16 == 0) a.squares_out[(size_t)token * a.squares_out_n + n / 16] = sq;
            }
        } else if (ok) {
            if (EPI == kStoreF32) reinterpret_cast<float*>(a.out)[(size_t)token * a.ldo + n] = v;
            else reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)token * a.ldo + n] = __float2bfloat16_rn(v);
        }
    }
}

template <typename Kernel>
static int launch_skinny(Kernel kernel, const SkinnyArgs& a, int grid, int cluster, size_t smem, int use_pdl, cudaStream_t stream) {
    const cudaError_t e = launch_pdl_cluster(kernel, dim3(grid * cluster), dim3(kSkWarps * 32), smem, stream, use_pdl != 0, cluster, a);
    CIB_REQUIRE(e == cudaSuccess, "gemm_skinny: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

static int act_stride_for(int K) {
    // row stride (elements) such that consecutive rows start 16 banks apart: 16-byte reads of two rows never collide
    const int words = K / 2;
    const int pad_words = ((16 - words % 32) % 32 + 32) % 32;
    return K + pad_words * 2;
}

// the kernel that norms 32-bit rows in its prologue
template <int MT, int RT, int KS, int EPI>
static int launch_norm(SkinnyArgs& a, int grid, int use_pdl, cudaStream_t stream) {
    a.act_stride = act_stride_for(a.K);
    const size_t act_bytes = (size_t)MT * 8 * a.act_stride * 2;
    const size_t norm_bytes = (size_t)MT * 8 * a.K * 4;                  // un-normalised 32-bit rows during the prologue
    const size_t red_bytes = (size_t)KS * RT * 16 * MT * 8 * 4;
    size_t smem = act_bytes + (norm_bytes > red_bytes ? norm_bytes : red_bytes);
    smem = (smem + 15) & ~size_t(15);
    a.norm_w_offset = (int)smem;
    smem += (size_t)a.K * 4;
    CIB_REQUIRE(smem <= 200 * 1024, "gemm_skinny: %d rows x K=%d need %zu bytes of shared memory", a.M, a.K, smem);
    auto kernel = skinny_norm_gemm_kernel<MT, RT, KS, EPI>;
    static SmemLimit limit;
    if (int rc = raise_smem_limit(limit, kernel, 200 * 1024, "gemm_skinny")) return rc;
    return launch_skinny(kernel, a, grid, 1, smem, use_pdl, stream);
}

template <int MT>
static int dispatch_norm(SkinnyArgs& a, int epilogue, int use_pdl, cudaStream_t stream) {
    if (epilogue == kSiluPair) return launch_norm<MT, 2, 4, kSiluPair>(a, (a.up_offset + 15) / 16, use_pdl, stream);
    // As few 16-row tiles per CTA as keep the launch within one round of CTAs (two fit on each of the 148 SMs);
    // the warps that are not needed for rows split K instead.
    const int tiles = (a.N + 15) / 16;
    int rt = 1;
    while (rt < 8 && (tiles + rt - 1) / rt > 296) rt *= 2;
    const int grid = (tiles + rt - 1) / rt;
#define CIB_SKINNY_CASE(RTV, KSV)                                                                 \
    if (rt == RTV) {                                                                              \
        if (epilogue == kStoreF32) return launch_norm<MT, RTV, KSV, kStoreF32>(a, grid, use_pdl, stream); \
        return launch_norm<MT, RTV, KSV, kStoreBf16>(a, grid, use_pdl, stream);                   \
    }
    CIB_SKINNY_CASE(1, 8)
    CIB_SKINNY_CASE(2, 4)
    CIB_SKINNY_CASE(4, 2)
    CIB_SKINNY_CASE(8, 1)
#undef CIB_SKINNY_CASE
    return -1;
}

template <int MT, int RW, int EPI, int CS>
static int launch_rows(SkinnyArgs& a, int grid, int use_pdl, cudaStream_t stream) {
    const int steps = ((a.K + 31) / 32 + kSkWarps * CS - 1) / (kSkWarps * CS);       // of a warp
    if (steps <= kSkU / RW) return launch_skinny(skinny_gemm_kernel<MT, RW, EPI, CS, 1>, a, grid, CS, 0, use_pdl, stream);
    if (steps <= 2 * kSkU / RW) return launch_skinny(skinny_gemm_kernel<MT, RW, EPI, CS, 2>, a, grid, CS, 0, use_pdl, stream);
    return launch_skinny(skinny_gemm_kernel<MT, RW, EPI, CS, 0>, a, grid, CS, 0, use_pdl, stream);
}

template <int MT, int EPI>
static int dispatch_rows(SkinnyArgs& a, int use_pdl, cudaStream_t stream) {
    if constexpr (EPI == kSiluPair) {
        return launch_rows<MT, 2, EPI, 1>(a, (a.up_offset + 15) / 16, use_pdl, stream);
    } else {
        const int tiles = (a.N + 15) / 16;
        // Few output features and a long K: four CTAs of a cluster share each tile so that most SMs stream, and each reads a quarter
        // of the activations.  (Two CTAs: a step of one row 625 us instead of 607, of twelve 826 instead of 789, of eight 692 instead
        // of 698; none: 643, 997 and 730.  The split may not depend on the rows: a row's result does not depend on its neighbours.)
        // From 75 tiles on a CTA a tile fills half of the SMs, and the cluster's merge costs more than the others bring: 8 rows of 2 048 x
        // 2 048 4.7 us in clusters, 2.8 without.
        if (tiles <= 74 && a.K >= 2048) return launch_rows<MT, 1, EPI, 4>(a, tiles, use_pdl, stream);
        // one row tile a CTA as long as two CTAs an SM hold them all (with two tiles from 101 on: 620 us instead of 607, 806 of 789)
        if (tiles <= 296) return launch_rows<MT, 1, EPI, 1>(a, tiles, use_pdl, stream);
        return launch_rows<MT, 2, EPI, 1>(a, (tiles + 1) / 2, use_pdl, stream);
    }
}

template <int MT>
static int dispatch_skinny(SkinnyArgs& a, int epilogue, int use_pdl, cudaStream_t stream) {
    if (a.res_in != nullptr) return dispatch_norm<MT>(a, epilogue, use_pdl, stream);
    switch (epilogue) {
        case kSiluPair: return dispatch_rows<MT, kSiluPair>(a, use_pdl, stream);
        case kStoreF32: return dispatch_rows<MT, kStoreF32>(a, use_pdl, stream);
        case kStream: return dispatch_rows<MT, kStream>(a, use_pdl, stream);
        default: return dispatch_rows<MT, kStoreBf16>(a, use_pdl, stream);
    }
}

}  // namespace cib

using namespace cib;

// with_norm: the activations are normalised in the kernel, which keeps them in shared memory, the 32-bit rows as well.  Plain
// rows need no such room; the limit on their K (about 6 000 for 16 rows, 12 000 for 8) is part of what callers of the kernel
// rely on being refused; the engine gives it 4 096 at most (more only for fewer than eight features).
extern "C" int cib_gemm_skinny_supports(int M, int N, int K, int with_norm) {
    if (!(M >= 1 && M <= 16 && N >= 1 && K >= 32 && K % 8 == 0)) return 0;
    const size_t rows = M <= 8 ? 8 : 16;
    const size_t bytes = rows * (K + 64) * 2 + (with_norm ? rows * K * 4 + (size_t)K * 4 + 16 : (size_t)kSkWarps * 16 * rows * 4);
    return bytes <= 200 * 1024 && (!with_norm || K % 4 == 0);
}

// act: [M, K] bfloat16 rows (lda), or null when res_in is given: then the activations are
// RMSNorm(res_in + pending) * norm_w computed in the kernel, and res_out (if not null) receives res_in + pending.
// epilogue: 0 = bfloat16 out[M, N]; 1 = float32 out[M, N]; 2 = rows [0, up_offset) are gates and rows
// [up_offset, N) the matching ups: out[M, up_offset] = silu(gate) * up in bfloat16; 3 = the same with gelu_tanh(gate);
// 4 = stream[M, N] (32-bit, dense) += the product, out = bfloat16(stream * norm_w), squares_out[M][ceil(N / 16)] = the sums of
// stream^2 over 16 columns each.
// squares_in: [M][squares_in_n] (or null): every result row is multiplied by rsqrt(sum(squares_in[row]) / K + eps) (with act only).
// warm / warm_bytes: memory that the kernel after this one reads first (its weights), or null: fetched into the L2 meanwhile.
extern "C" int cib_gemm_skinny(const void* w, int ldw, int N, int K, const void* act, int lda, const float* res_in,
                               const void* pending, int pending_dtype, const void* norm_w, int norm_w_dtype, float eps,
                               float* res_out, void* out, int ldo, int M, int epilogue, int up_offset, int use_pdl,
                               const void* warm, long long warm_bytes, const float* squares_in, int squares_in_n, float* stream_rows,
                               float* squares_out, cudaStream_t stream) {
    CIB_REQUIRE(cib_gemm_skinny_supports(M, N, K, res_in != nullptr), "gemm_skinny: M=%d N=%d K=%d is not taken by this kernel (M <= 16, K a multiple of 8)", M, N, K);
    CIB_REQUIRE(ldw >= K && ldw % 8 == 0 && ((uintptr_t)w % 16) == 0, "gemm_skinny: weight rows must be 16-byte aligned");
    CIB_REQUIRE((act != nullptr) != (res_in != nullptr), "gemm_skinny: give plain activations or a residual to normalise");
    CIB_REQUIRE(act == nullptr || (lda >= K && lda % 8 == 0 && ((uintptr_t)act % 16) == 0), "gemm_skinny: activation rows must be 16-byte aligned");
    CIB_REQUIRE(res_in == nullptr || (norm_w != nullptr && K % 4 == 0 && res_out != res_in), "gemm_skinny: the norm needs its weight and a second residual buffer");
    CIB_REQUIRE(epilogue >= 0 && epilogue <= 4, "gemm_skinny: unknown epilogue %d", epilogue);
    const int gate_gelu = epilogue == 3;           // 3: as 2 with the tanh form of GELU as the gate
    if (gate_gelu) epilogue = kSiluPair;
    else if (epilogue == 4) epilogue = kStream;
    CIB_REQUIRE(epilogue != kSiluPair || (up_offset > 0 && 2 * up_offset == N && ldo >= up_offset), "gemm_skinny: a gate/up pair needs N = 2 * up_offset");
    CIB_REQUIRE(epilogue == kSiluPair || ldo >= N, "gemm_skinny: ldo too small");
    CIB_REQUIRE(epilogue != kStream || (res_in == nullptr && stream_rows != nullptr && squares_out != nullptr && norm_w != nullptr),
                "gemm_skinny: the stream epilogue needs plain rows, the residual, the norm's gains and room for the squares");
    CIB_REQUIRE(squares_in == nullptr || (act != nullptr && squares_in_n > 0), "gemm_skinny: sums of squares go with plain rows");
    SkinnyArgs a;
    a.w = (const __nv_bfloat16*)w; a.ldw = ldw; a.N = N; a.K = K;
    a.act = (const __nv_bfloat16*)act; a.lda = lda;
    a.res_in = res_in; a.pending = pending; a.pending_bf16 = pending_dtype == kBF16;
    a.norm_w = AnyVec{norm_w, norm_w_dtype == kBF16}; a.eps = eps; a.res_out = res_out;
    a.out = out; a.ldo = ldo; a.M = M; a.up_offset = up_offset; a.act_stride = 0; a.norm_w_offset = 0; a.gate_gelu = gate_gelu;
    a.warm = ((uintptr_t)warm % 16) == 0 && warm_bytes > 0 ? warm : nullptr;
    a.warm_bytes = a.warm ? (unsigned long long)warm_bytes : 0;
    a.squares_in = squares_in; a.squares_in_n = squares_in_n;
    a.stream = stream_rows; a.squares_out = squares_out; a.squares_out_n = (N + 15) / 16;
    if (M <= 8) return dispatch_skinny<1>(a, epilogue, use_pdl, stream);
    return dispatch_skinny<2>(a, epilogue, use_pdl, stream);
}
