// Paged causal attention in 32 bits for head sizes 64 and 128: the steps of a float32 engine.
//
// Scores, exponential, weights and sums are 32-bit as in attention_generic.cu (which stays for every other head size);
// what differs is who reads what.  There one warp walks a query's keys alone, each lane a key of its own: 32 cache lines
// a load instruction, and keys and values read again for every query.  Here
//   * a step of few tokens gives each (token, kv head) a cluster of CTAs whose warps share out the keys in eights; eight
//     lanes read one key together and the heads of the group use it while it is in registers;
//   * a step of more tokens gives each (16 query rows of one request and kv head) a CTA that stages tiles of 32 keys and values in
//     shared memory with asynchronous copies, a tile ahead; a lane scores one key for four rows.
// Measured per layer of 16 heads over 8 kv heads of 128: 3 requests with 200 to 300 keys 6.4 us instead of 200, one
// request with 4 000 keys 18 us; 467 prompt tokens of three requests 53 us.
// A key that a row may not see is never used for it, not even with weight zero (its value may be infinite).
//
// Cache layout of one layer: [page][0 = keys, 1 = values][kv head][slot in page][d].
#include "attention_f32.cuh"
#include "mma_utils.cuh"

#include <cooperative_groups.h>

namespace cib {

// ---- few tokens ----------------------------------------------------------------------------------------------------------
constexpr int kFewAttnWarps = 8, kFewAttnKeys = 8;                 // keys a warp has in flight, with their values
constexpr int kFewAttnMaxSplit = 8;

// HB heads of one kv head for one token.  The warps of a cluster's CTAs take eight keys each in turn; all of a key's and its
// value's bytes are asked for before the scores, so a round costs one trip to memory.  The cluster's first CTA merges.
template <int D, int HB>
__global__ void __launch_bounds__(kFewAttnWarps * 32)
attention_f32_few_kernel(const AttnF32 p, int splits) {
    namespace cg = cooperative_groups;
    constexpr int Q4 = D / 32;            // float4 of a key per lane of a group of eight
    constexpr int VD = D / 32;            // values per lane
    __shared__ float s_m[kFewAttnWarps][HB], s_l[kFewAttnWarps][HB];
    __shared__ float s_acc[kFewAttnWarps][HB][D];
    __shared__ float s_top[HB], s_sum[HB], s_out[HB][D];           // of this CTA
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, of = lane >> 3;
    const int blocks = p.nq / p.nkv / HB;                          // blocks of heads per kv head
    const int t = blockIdx.x, kvh = blockIdx.y / blocks, part = blockIdx.z;
    const int head0 = kvh * (p.nq / p.nkv) + blockIdx.y % blocks * HB;
    griddep_launch();
    griddep_wait();
    const int r = p.token_request[t], q0 = p.query_start_loc[r];
    const int pos = p.seq_lens[r] - (p.query_start_loc[r + 1] - q0) + (t - q0);
    const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    const int* table = p.block_table + (size_t)r * p.table_stride;
    const size_t head_stride = (size_t)p.page_size * D, page_stride = 2 * p.nkv * head_stride;
    const float* base = p.cache + kvh * head_stride;
    const size_t v_off = p.nkv * head_stride;

    float4 q[HB][Q4];
#pragma unroll
    for (int h = 0; h < HB; ++h)
#pragma unroll
        for (int i = 0; i < Q4; ++i) {
            float4 v = *reinterpret_cast<const float4*>(p.q + (size_t)t * p.q_stride + (size_t)(head0 + h) * D + (i * 8 + sub) * 4);
            q[h][i] = make_float4(v.x * p.scale, v.y * p.scale, v.z * p.scale, v.w * p.scale);
        }
    float acc[HB][VD], m[HB], l[HB];
#pragma unroll
    for (int h = 0; h < HB; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < VD; ++i) acc[h][i] = 0.f;
    }
    const int stride = kFewAttnWarps * kFewAttnKeys * splits;
    for (int c = lo + (part * kFewAttnWarps + warp) * kFewAttnKeys; c <= pos; c += stride) {
        const int j = c + sub;
        long long row = -1;                                        // where key c + (lane % 8) lies, in elements; -1: nowhere
        if (j <= pos) {
            const int page = table[j / p.page_size];
            if (page >= 0 && page < p.num_pages) row = (long long)(page * page_stride + (size_t)(j % p.page_size) * D);
        }
        float4 k[2][Q4];
        __align__(16) float v[kFewAttnKeys][VD];
        bool in[2];
#pragma unroll
        for (int step = 0; step < 2; ++step) {
            const long long kr = __shfl_sync(0xffffffffu, row, step * 4 + of);
            in[step] = kr >= 0;
#pragma unroll
            for (int i = 0; i < Q4; ++i)
                k[step][i] = kr >= 0 ? *reinterpret_cast<const float4*>(base + kr + (i * 8 + sub) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int jj = 0; jj < kFewAttnKeys; ++jj) {
            const long long vr = __shfl_sync(0xffffffffu, row, jj);
            if (VD == 4) *reinterpret_cast<float4*>(v[jj]) = vr >= 0 ? *reinterpret_cast<const float4*>(base + v_off + vr + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            else *reinterpret_cast<float2*>(v[jj]) = vr >= 0 ? *reinterpret_cast<const float2*>(base + v_off + vr + lane * 2) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int h = 0; h < HB; ++h) {
            float w[2];
#pragma unroll
            for (int step = 0; step < 2; ++step) {
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < Q4; ++i) {
                    s = fmaf(q[h][i].x, k[step][i].x, s);
                    s = fmaf(q[h][i].y, k[step][i].y, s);
                    s = fmaf(q[h][i].z, k[step][i].z, s);
                    s = fmaf(q[h][i].w, k[step][i].w, s);
                }
                s += __shfl_xor_sync(0xffffffffu, s, 4);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                w[step] = in[step] ? s : -INFINITY;                // the score of key step * 4 + of
            }
            float top = fmaxf(w[0], w[1]);
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
            const float m_new = fmaxf(m[h], top);
            float corr = 1.f;
            if (m_new != -INFINITY) {
                w[0] = w[0] == -INFINITY ? 0.f : expf(w[0] - m_new);
                w[1] = w[1] == -INFINITY ? 0.f : expf(w[1] - m_new);
                corr = m[h] == -INFINITY ? 0.f : expf(m[h] - m_new);
            } else {
                w[0] = w[1] = 0.f;
            }
            float sum = w[0] + w[1];
            sum += __shfl_xor_sync(0xffffffffu, sum, 8);
            sum += __shfl_xor_sync(0xffffffffu, sum, 16);
            l[h] = l[h] * corr + sum;
            m[h] = m_new;
#pragma unroll
            for (int i = 0; i < VD; ++i) acc[h][i] *= corr;
#pragma unroll
            for (int jj = 0; jj < kFewAttnKeys; ++jj) {
                const float wj = __shfl_sync(0xffffffffu, w[jj / 4], (jj % 4) * 8);
#pragma unroll
                for (int i = 0; i < VD; ++i) acc[h][i] = fmaf(wj, v[jj][i], acc[h][i]);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < HB; ++h) {
        if (lane == 0) { s_m[warp][h] = m[h]; s_l[warp][h] = l[h]; }
#pragma unroll
        for (int i = 0; i < VD; ++i) s_acc[warp][h][lane * VD + i] = acc[h][i];
    }
    __syncthreads();
    const bool alone = splits == 1;
    for (int e = threadIdx.x; e < HB * D; e += kFewAttnWarps * 32) {
        const int h = e / D, i = e % D;
        float top = -INFINITY;
#pragma unroll
        for (int w = 0; w < kFewAttnWarps; ++w) top = fmaxf(top, s_m[w][h]);
        float sum = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < kFewAttnWarps; ++w) {
            if (s_m[w][h] == -INFINITY) continue;                  // a warp without keys
            const float f = expf(s_m[w][h] - top);
            sum = fmaf(f, s_l[w][h], sum);
            o = fmaf(f, s_acc[w][h][i], o);
        }
        if (alone) p.out[(size_t)t * p.out_stride + (size_t)(head0 + h) * D + i] = o * (sum > 0.f ? 1.f / sum : 0.f);
        else {
            s_out[h][i] = o;
            if (i == 0) { s_top[h] = top; s_sum[h] = sum; }
        }
    }
    if (alone) return;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (part == 0) {
        for (int e = threadIdx.x; e < HB * D; e += kFewAttnWarps * 32) {
            const int h = e / D, i = e % D;
            float tops[kFewAttnMaxSplit], top = -INFINITY;
#pragma unroll
            for (int c = 0; c < kFewAttnMaxSplit; ++c) {
                tops[c] = c < splits ? *cluster.map_shared_rank(&s_top[h], c) : -INFINITY;
                top = fmaxf(top, tops[c]);
            }
            float sum = 0.f, o = 0.f;
#pragma unroll
            for (int c = 0; c < kFewAttnMaxSplit; ++c) {
                if (tops[c] == -INFINITY) continue;
                const float f = expf(tops[c] - top);
                sum = fmaf(f, *cluster.map_shared_rank(&s_sum[h], c), sum);
                o = fmaf(f, *cluster.map_shared_rank(&s_out[h][i], c), o);
            }
            p.out[(size_t)t * p.out_stride + (size_t)(head0 + h) * D + i] = o * (sum > 0.f ? 1.f / sum : 0.f);
        }
    }
    cluster.sync();                                                // the others' shared memory stays until it has been read
}

// ---- more tokens -----------------------------------------------------------------------------------------------------------
constexpr int kTileRows = 16, kTileKeys = 32, kTileWarps = 4, kWarpRows = kTileRows / kTileWarps;

// (three CTAs of head size 128 fill an SM's shared memory to the last byte)
template <int D>
struct AttnF32Smem {
    float k[2][kTileKeys][D + 4];                                   // + 4: eight lanes that read eight keys hit different banks
    float v[2][kTileKeys][D];
    float q[kTileRows][D];
    float p[kTileRows][kTileKeys];
};

// kTileRows query rows of one request: kTileRows / HB tokens with HB heads of one kv head each.  A request's last tile may be
// short, so that no tile walks one request's keys after another's: decoded tokens beside a prompt, sixteen to a tile in
// turn, took 885 us (20 of 500 keys and 200 prompt tokens, 8 heads of 64) where a CTA for each takes 55.
template <int D, int HB>
__global__ void __launch_bounds__(kTileWarps * 32)
attention_f32_tile_kernel(const AttnF32 p) {
    constexpr int VD = D / 32;
    constexpr int TT = kTileRows / HB;                              // tokens of a tile
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AttnF32Smem<D>& s = *reinterpret_cast<AttnF32Smem<D>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int blocks = p.nq / p.nkv / HB;
    const int kvh = blockIdx.y / blocks, head0 = kvh * (p.nq / p.nkv) + blockIdx.y % blocks * HB;
    int* s_at = reinterpret_cast<int*>(&s.p[0][0]);                 // request and first token, until the weights lie there
    const size_t head_stride = (size_t)p.page_size * D, page_stride = 2 * p.nkv * head_stride;
    const float* base = p.cache + kvh * head_stride;
    const size_t v_off = p.nkv * head_stride;
    griddep_launch();
    griddep_wait();
    if (warp == 0) {                                                // which request and which of its tiles, 32 requests at a time
        int tile = blockIdx.x, request = -1, first = 0;
        for (int r0 = 0; r0 < p.num_requests; r0 += 32) {
            const int r = r0 + lane, q0 = r < p.num_requests ? p.query_start_loc[r] : 0;
            const int tiles = r < p.num_requests ? (p.query_start_loc[r + 1] - q0 + TT - 1) / TT : 0;
            int upto = tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int before = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += before;
            }
            const unsigned int hit = __ballot_sync(0xffffffffu, tile < upto);
            if (hit != 0u) {
                const int at = __ffs(hit) - 1;
                request = r0 + at;
                first = __shfl_sync(0xffffffffu, q0, at) + (tile - __shfl_sync(0xffffffffu, upto - tiles, at)) * TT;
                break;
            }
            tile -= __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) { s_at[0] = request; s_at[1] = first; }
    }
    __syncthreads();
    const int r = s_at[0], t0 = s_at[1];
    if (r < 0 || (unsigned)t0 >= (unsigned)p.num_tokens) return;    // the launch is sized for the worst split of its tokens
    const int q0 = p.query_start_loc[r], q1 = min(p.num_tokens, p.query_start_loc[r + 1]);
    const int t1 = min(t0 + TT, q1);                                // this tile's tokens: [t0, t1)
    const int pos0 = p.seq_lens[r] - (p.query_start_loc[r + 1] - q0) + (t0 - q0);     // position of token t0
    const int last = pos0 + (t1 - 1 - t0);                          // of the last one
    const int first = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
    const int* table = p.block_table + (size_t)r * p.table_stride;

    for (int e = tid; e < kTileRows * D / 4; e += kTileWarps * 32) {
        const int row = e / (D / 4), i = e % (D / 4) * 4, t = t0 + row / HB;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < t1) v = *reinterpret_cast<const float4*>(p.q + (size_t)t * p.q_stride + (size_t)(head0 + row % HB) * D + i);
        *reinterpret_cast<float4*>(&s.q[row][i]) = make_float4(v.x * p.scale, v.y * p.scale, v.z * p.scale, v.w * p.scale);
    }

    auto fetch = [&](int buffer, int c) {                       // keys c .. c + 31; what has no page or lies behind `last` is zero
#pragma unroll 4
        for (int e = tid; e < kTileKeys * D / 4; e += kTileWarps * 32) {
            const int key = e / (D / 4), i = e % (D / 4) * 4, j = c + key;
            int page = -1;
            if (j <= last) page = table[j / p.page_size];
            const bool in = page >= 0 && page < p.num_pages;
            const float* src = in ? base + page * page_stride + (size_t)(j % p.page_size) * D + i : p.cache;
            cp_async16(&s.k[buffer][key][i], src, in);
            cp_async16(&s.v[buffer][key][i], in ? src + v_off : src, in);
        }
        cp_async_commit();
    };

    float acc[kWarpRows][VD], m[kWarpRows], l[kWarpRows];
    int low[kWarpRows], high[kWarpRows];                        // the keys a row sees; high < low: not a token of this tile
    int warp_low = 0, warp_high = 0x7fffffff;                   // the keys that all of them see
    bool any = false;
#pragma unroll
    for (int k = 0; k < kWarpRows; ++k) {
        const int t = t0 + (warp * kWarpRows + k) / HB;
        m[k] = -INFINITY;
        l[k] = 0.f;
#pragma unroll
        for (int i = 0; i < VD; ++i) acc[k][i] = 0.f;
        high[k] = t < t1 ? pos0 + (t - t0) : -1;
        low[k] = p.window > 0 ? max(0, high[k] - p.window + 1) : 0;
        if (high[k] < 0) low[k] = 0;
        any = any || high[k] >= 0;
        warp_low = max(warp_low, low[k]);
        warp_high = min(warp_high, high[k]);
    }
    if (first <= last) fetch(0, first);
    int buffer = 0;
    for (int c = first; c <= last; c += kTileKeys, buffer ^= 1) {
        if (c + kTileKeys <= last) {
            fetch(buffer ^ 1, c + kTileKeys);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        if (any) {
            const int j = c + lane;
            bool readable = false;
            if (j <= last) {
                const int page = table[j / p.page_size];
                readable = page >= 0 && page < p.num_pages;
            }
            float score[kWarpRows] = {};
            const float4* kp = reinterpret_cast<const float4*>(&s.k[buffer][lane][0]);
#pragma unroll 8
            for (int i = 0; i < D / 4; ++i) {
                const float4 kv = kp[i];
#pragma unroll
                for (int k = 0; k < kWarpRows; ++k) {
                    const float4 qv = *reinterpret_cast<const float4*>(&s.q[warp * kWarpRows + k][i * 4]);
                    score[k] = fmaf(qv.x, kv.x, score[k]);
                    score[k] = fmaf(qv.y, kv.y, score[k]);
                    score[k] = fmaf(qv.z, kv.z, score[k]);
                    score[k] = fmaf(qv.w, kv.w, score[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < kWarpRows; ++k) {
                const float sc = readable && j >= low[k] && j <= high[k] ? score[k] : -INFINITY;
                const float m_new = fmaxf(m[k], warp_max(sc));
                float w = 0.f, corr = 1.f;
                if (m_new != -INFINITY) {
                    w = sc == -INFINITY ? 0.f : expf(sc - m_new);
                    corr = m[k] == -INFINITY ? 0.f : expf(m[k] - m_new);
                }
                l[k] = l[k] * corr + warp_sum(w);
                m[k] = m_new;
#pragma unroll
                for (int i = 0; i < VD; ++i) acc[k][i] *= corr;
                s.p[warp * kWarpRows + k][lane] = w;
            }
            __syncwarp();
            const bool all = c >= warp_low && c + kTileKeys - 1 <= warp_high;
#pragma unroll 2
            for (int j4 = 0; j4 < kTileKeys; j4 += 4) {
                float4 w4[kWarpRows];
#pragma unroll
                for (int k = 0; k < kWarpRows; ++k) w4[k] = *reinterpret_cast<const float4*>(&s.p[warp * kWarpRows + k][j4]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    __align__(16) float v[VD];
                    const float* vp = &s.v[buffer][j4 + u][lane * VD];
                    if (VD == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(vp);
                    else *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(vp);
                    const int key = c + j4 + u;
#pragma unroll
                    for (int k = 0; k < kWarpRows; ++k) {
                        const float w = u == 0 ? w4[k].x : u == 1 ? w4[k].y : u == 2 ? w4[k].z : w4[k].w;
                        if (all || (key >= low[k] && key <= high[k])) {
#pragma unroll
                            for (int i = 0; i < VD; ++i) acc[k][i] = fmaf(w, v[i], acc[k][i]);
                        }
                    }
                }
            }
        }
        __syncthreads();                                        // the next fetch overwrites this buffer
    }
#pragma unroll
    for (int k = 0; k < kWarpRows; ++k) {
        const int row = warp * kWarpRows + k, t = t0 + row / HB;
        if (t >= t1) continue;
        const float inv = l[k] > 0.f ? 1.f / l[k] : 0.f;
        float* o = p.out + (size_t)t * p.out_stride + (size_t)(head0 + row % HB) * D + lane * VD;
#pragma unroll
        for (int i = 0; i < VD; ++i) o[i] = acc[k][i] * inv;
    }
}

// Few tokens: while a CTA per (token, block of heads) is at most two for each SM, and for as many tokens as
// requests (a step of decoded tokens: 32 requests of 1 000 keys, 12 heads of 64 over 4, 40 us, 1 760 in tiles of several
// requests); beyond, a key is read for one token where the tile kernel reads it for several.  As many CTAs to a cluster as
// the SMs have room for without a second round.
constexpr int kFewAttnCtas = 296;

template <int D, int HB>
static int launch_attention_f32(const AttnF32& p, cudaStream_t stream) {
    const int head_blocks = p.nq / HB;
    const long long ctas = (long long)p.num_tokens * head_blocks;
    cudaError_t e;
    if (ctas <= kFewAttnCtas || p.num_tokens <= p.num_requests) {
        int splits = 1;
        while (splits < kFewAttnMaxSplit && ctas * splits * 2 <= 148) splits *= 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(p.num_tokens, head_blocks, splits);
        cfg.blockDim = dim3(kFewAttnWarps * 32);
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = (unsigned)splits;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = prompt_pdl() ? 2 : 1;
        e = cudaLaunchKernelEx(&cfg, attention_f32_few_kernel<D, HB>, p, splits);
    } else {
        static SmemLimit limit;
        if (int rc = raise_smem_limit(limit, attention_f32_tile_kernel<D, HB>, sizeof(AttnF32Smem<D>), "paged_attention")) return rc;
        constexpr int TT = kTileRows / HB;
        e = launch_pdl(attention_f32_tile_kernel<D, HB>, dim3(p.num_tokens / TT + p.num_requests, head_blocks), dim3(kTileWarps * 32),
                       sizeof(AttnF32Smem<D>), stream, prompt_pdl(), p);
    }
    CIB_REQUIRE(e == cudaSuccess, "paged_attention: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

int attention_f32_try(const AttnF32& p, int d, cudaStream_t stream) {
    const auto aligned = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
    if ((d != 64 && d != 128) || p.q_stride % 4 || !aligned(p.q) || !aligned(p.cache) || p.nq > 65535) return 0;
    const int per = p.nq / p.nkv, hb = per % 4 == 0 ? 4 : per % 2 == 0 ? 2 : 1;
    int rc;
    if (d == 64) rc = hb == 4 ? launch_attention_f32<64, 4>(p, stream) : hb == 2 ? launch_attention_f32<64, 2>(p, stream) : launch_attention_f32<64, 1>(p, stream);
    else rc = hb == 4 ? launch_attention_f32<128, 4>(p, stream) : hb == 2 ? launch_attention_f32<128, 2>(p, stream) : launch_attention_f32<128, 1>(p, stream);
    return rc ? rc : 1;
}

}  // namespace cib
