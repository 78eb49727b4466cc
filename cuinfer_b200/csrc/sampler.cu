// Next-token sampling from 32-bit logits: greedy, temperature, top-k, top-p.  A cluster of up to eight CTAs per row.
//
// Meaning of the options follows the reference's sampler (csrc/ops/sampler.cu:134-387):
//   temperature == 0   -> argmax, ties to the lowest id (:207-212)
//   top_k  in (0, V)   -> keep the values >= the exact k-th largest, ties at the edge kept (:216-250)
//   top_p  in (0, 1)   -> the smallest set of most probable kept tokens whose mass reaches top_p
//   weight_i = exp((x_i - max) / temperature) (:252-281)
// The reference draws with Philox inside the kernel and accepts or rejects candidates; here the
// uniform number u in [0, 1) of every row is an input (the host derives it from seed, request and
// output index), and the kept set is found exactly by a radix descent, so the kernel is a pure
// function of (logits, options, u) and needs no scratch memory.
//
// Masses are summed as 32.32 fixed-point integers: q_i = floor(weight_i * 2^32) (at most 2^32 - 1), so
// that every sum is exact and independent of the order in which threads add.
#include "common.cuh"

#include <cooperative_groups.h>

namespace cib {

// A cluster of up to eight CTAs takes a row, a share of the vocabulary each, kept in shared memory: the logits are read from
// device memory once, the exponentials are taken once, and every level of a descent walks shared memory.  What bounds it
// is the chain of levels (a histogram of the share, a cluster barrier, a scan of 256 sums), not the bytes.  Two things keep
// the histograms from serialising on one bin: the lowest digit's sum is never needed (it is what is left when no other digit
// reaches the goal), and it is the digit that nearly every token of a large vocabulary has; and a warp whose lanes all have
// one digit adds once.  The masses go into the histogram as two 32-bit halves of 16 bits each, whose sums over a share of up
// to 65 536 tokens fit 32 bits, because shared memory has no 64-bit add (a compare-and-swap loop stands in for it).
// Rows of 151 936 tokens, microseconds with the L2 flushed, against one CTA a row with 64-bit sums of every digit: 32 rows
// with top_p 0.9 55 (10 749), 1 row 39 (10 699), 128 rows 184 (10 770); 32 rows with top_k 50 59 (1 912), with neither 29
// (141); 32 rows of 400 000 tokens, which shared memory does not hold, 363 (5 273).
constexpr int kSampleCtas = 8;                  // at most
constexpr int kSampleThreads = 512;
constexpr int kSampleWarps = kSampleThreads / 32;
constexpr int kSampleShareMax = 49152;          // tokens of a share that shared memory holds (192 KB); longer ones are re-read
constexpr int kSampleShareFour = 12800;         // tokens of a share with which four CTAs fit an SM, all its threads

// CTAs of a row: as few as leave an SM four of them, since every CTA of a large batch costs its start and its part of every
// barrier; more, down to 512 tokens each, while the whole batch still has at most two for each SM.  (With eight at every
// size 512 rows of 128 tokens took 29 us greedily and 193 with top_p, one CTA each 5 and 15; 128 rows of 8 192 with
// top_p 58, now 20.)
inline int sample_ctas(int rows, int vocab) {
    int ctas = 1;
    while (ctas < kSampleCtas && vocab > ctas * kSampleShareFour) ctas *= 2;
    while (ctas < kSampleCtas && (long long)rows * ctas * 2 <= 2 * 148 && vocab >= 2 * ctas * 512) ctas *= 2;
    return ctas;
}

struct SampleParams {
    float temperature;
    int top_k;
    float top_p;
    float u;
};

__device__ __forceinline__ uint32_t order_key(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ uint32_t mass_of(float x, float mx, float temperature, uint32_t key_min) {
    if (order_key(x) < key_min) return 0u;
    const float w = expf((x - mx) / temperature);
    const float scaled = w * 4294967296.f;
    return scaled >= 4294967040.f ? 0xffffffffu : (uint32_t)scaled;
}

__device__ __forceinline__ void take_better(float& best, int& best_i, float v, int i) {
    if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
}

typedef unsigned long long u64;

__device__ __forceinline__ u64 warp_sum_u64(u64 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// What the CTAs of a row tell one another.  Everything but the histograms is pushed: rank r writes its number into slot r of
// every CTA and all meet at a cluster barrier, after which each reads its own copy; a slot array is used once a launch.
struct SampleShared {
    float best[kSampleCtas];
    int best_i[kSampleCtas];
    u64 total[kSampleCtas], kept[kSampleCtas];
    unsigned int hist[2][2][256];               // by parity of the level: low and high halves (or both words of a 64-bit sum)
    u64 warp_part[kSampleWarps];
    float warp_best[kSampleWarps];
    int warp_best_i[kSampleWarps];
    unsigned int bin;
    u64 above;
};

template <int CTAS>
__device__ __forceinline__ void cluster_barrier() {
    if (CTAS == 1) { __syncthreads(); return; }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// `p`, a place in this CTA's shared memory, in that of CTA `rank` of the row.
template <int CTAS, typename T>
__device__ __forceinline__ T* of_rank(T* p, int rank) {
    return CTAS == 1 ? p : cooperative_groups::this_cluster().map_shared_rank(p, rank);
}

// One level of a descent: the sums of this CTA's histogram and its peers' are joined by every CTA for itself, and the highest
// digit d is found with above + sum of the digits >= d reaching `need` (0 if none does).  `above` becomes the sum of the
// digits above it.  kWide: the two words of the histogram are one 64-bit sum.
template <int CTAS, bool kWide>
__device__ __forceinline__ unsigned int descend(SampleShared& s, int parity, u64 need, u64& above) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    cluster_barrier<CTAS>();                                     // every CTA's histogram is complete
    u64 suffix = 0ull;
    if (tid < 256) {
        u64 v = 0ull;
#pragma unroll
        for (int r = 0; r < CTAS; ++r) {
            const unsigned int* h = of_rank<CTAS>(&s.hist[parity][0][0], r);
            v += kWide ? reinterpret_cast<const u64*>(h)[tid] : (u64)h[tid] + ((u64)h[256 + tid] << 16);
        }
        suffix = v;                                              // sum over the digits >= tid of this warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 up = __shfl_down_sync(0xffffffffu, suffix, o);
            if (lane + o < 32) suffix += up;
        }
        if (lane == 0) s.warp_part[warp] = suffix;
    }
    __syncthreads();
    if (tid < 256) {
        u64 base = above;
        for (int w = warp + 1; w < 8; ++w) base += s.warp_part[w];
        const u64 here = base + suffix;
        u64 next = __shfl_down_sync(0xffffffffu, here, 1);       // with the digits above this one only
        if (lane == 31) next = base;
        const bool reaches = tid == 0 || here >= need;
        const bool above_reaches = tid < 255 && next >= need;
        if (reaches && !above_reaches) { s.bin = (unsigned int)tid; s.above = next; }
    }
    __syncthreads();
    above = s.above;
    return s.bin;
}

// kCached: the share lies in shared memory (logits first, masses in their place later); else the row is re-read and the
// masses are taken again at every level.
template <int CTAS, bool kCached>
__global__ void __launch_bounds__(kSampleThreads)
sample_cluster_kernel(const float* __restrict__ logits, int ld, int vocab, int share, const SampleParams* __restrict__ params,
                      int* __restrict__ out_ids) {
    extern __shared__ __align__(16) float s_row[];
    __shared__ SampleShared s;
    const int row = blockIdx.x / CTAS, rank = blockIdx.x % CTAS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (CTAS > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // remote stores come after every CTA runs
    const float* x = logits + (size_t)row * ld;
    const int begin = min(vocab, rank * share), end = min(vocab, begin + share), count = end - begin;
    const SampleParams p = params[row];

    // ---- max and argmax (lowest index wins ties) ----
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {            // a share is a multiple of four tokens
        const float4* x4 = reinterpret_cast<const float4*>(x + begin);
#pragma unroll 4
        for (int g = tid; g < count / 4; g += kSampleThreads) {
            const float4 v = x4[g];
            if (kCached) reinterpret_cast<float4*>(s_row)[g] = v;
            const int i = begin + 4 * g;
            take_better(best, best_i, v.x, i); take_better(best, best_i, v.y, i + 1);
            take_better(best, best_i, v.z, i + 2); take_better(best, best_i, v.w, i + 3);
        }
        for (int i = (count & ~3) + tid; i < count; i += kSampleThreads) {
            const float v = x[begin + i];
            if (kCached) s_row[i] = v;
            take_better(best, best_i, v, begin + i);
        }
    } else {
#pragma unroll 8
        for (int i = tid; i < count; i += kSampleThreads) {
            const float v = x[begin + i];
            if (kCached) s_row[i] = v;
            take_better(best, best_i, v, begin + i);
        }
    }
    for (int o = 16; o > 0; o >>= 1)
        take_better(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
    if (lane == 0) { s.warp_best[warp] = best; s.warp_best_i[warp] = best_i; }
    for (int i = tid; i < 2 * 2 * 256; i += kSampleThreads) (&s.hist[0][0][0])[i] = 0u;
    if (CTAS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        best = lane < kSampleWarps ? s.warp_best[lane] : -INFINITY;
        best_i = lane < kSampleWarps ? s.warp_best_i[lane] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1)
            take_better(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
        if (lane < CTAS) {
            *of_rank<CTAS>(&s.best[rank], lane) = best;
            *of_rank<CTAS>(&s.best_i[rank], lane) = best_i;
        }
    }
    cluster_barrier<CTAS>();
    best = s.best[0];
    best_i = s.best_i[0];
#pragma unroll
    for (int r = 1; r < CTAS; ++r) take_better(best, best_i, s.best[r], s.best_i[r]);
    const float mx = best;
    const int argmax = best_i == 0x7fffffff ? 0 : best_i;
    if (!(p.temperature > 0.f) || p.top_k == 1) {                // the same for every CTA of the row; no peer reads this one's memory any more
        if (rank == 0 && tid == 0) out_ids[row] = argmax;
        return;
    }

    int level = 0;
    const int rounds = (count + kSampleThreads - 1) / kSampleThreads;
    // ---- top-k: exact k-th largest key by radix descent over the order-preserving bits ----
    uint32_t key_min = 0u;
    if (p.top_k > 0 && p.top_k < vocab) {
        uint32_t prefix = 0u, mask = 0u;
        u64 above = 0ull;
        for (int shift = 24; shift >= 0; shift -= 8, ++level) {
            unsigned int* hist = &s.hist[level & 1][0][0];
            for (int n = 0; n < rounds; ++n) {                   // whole warps: the lanes are matched below
                const int i = n * kSampleThreads + tid;
                uint32_t digit = 0u;
                if (i < count) {
                    const uint32_t k = order_key(kCached ? s_row[i] : x[begin + i]);
                    if ((k & mask) == prefix) digit = (k >> shift) & 0xffu;
                }
                // few different digits at the first level (a sign and seven bits of exponent): one add a digit and warp
                const unsigned int same = __match_any_sync(0xffffffffu, digit);
                if (digit != 0u && lane == __ffs(same) - 1) {
                    if (kCached) atomicAdd(&hist[digit], (unsigned int)__popc(same));
                    else atomicAdd(reinterpret_cast<u64*>(hist) + digit, (u64)__popc(same));
                }
            }
            const uint32_t digit = descend<CTAS, !kCached>(s, level & 1, (u64)p.top_k, above);
            prefix |= digit << shift;
            mask |= 0xffu << shift;
            // the other parity's histogram was read before the barrier that this level has passed
            for (int i = tid; i < 512; i += kSampleThreads) (&s.hist[(level + 1) & 1][0][0])[i] = 0u;
            __syncthreads();
        }
        key_min = prefix;
    }

    // ---- total mass of the kept tokens ----
    u64 part = 0ull;
#pragma unroll 4
    for (int i = tid; i < count; i += kSampleThreads) {
        const uint32_t q = mass_of(kCached ? s_row[i] : x[begin + i], mx, p.temperature, key_min);
        if (kCached) s_row[i] = __uint_as_float(q);
        part += q;
    }
    const auto mass = [&](int i) { return kCached ? __float_as_uint(s_row[i]) : mass_of(x[begin + i], mx, p.temperature, key_min); };

    // ---- top-p: largest mass threshold whose kept set still reaches top_p of the total ----
    uint32_t q_min = 0u;
    if (p.top_p > 0.f && p.top_p < 1.f) {
        part = warp_sum_u64(part);
        if (lane == 0) s.warp_part[warp] = part;
        __syncthreads();
        if (warp == 0) {
            part = warp_sum_u64(lane < kSampleWarps ? s.warp_part[lane] : 0ull);
            if (lane < CTAS) *of_rank<CTAS>(&s.total[rank], lane) = part;
        }
        cluster_barrier<CTAS>();
        u64 total = 0ull;
#pragma unroll
        for (int r = 0; r < CTAS; ++r) total += s.total[r];
        const double want = (double)p.top_p * (double)total;
        u64 need = (u64)want;
        if ((double)need < want) ++need;
        need = need > total ? total : (need == 0ull ? 1ull : need);
        uint32_t prefix = 0u, mask = 0u;
        u64 above = 0ull;
        for (int shift = 24; shift >= 0; shift -= 8, ++level) {
            unsigned int* hist = &s.hist[level & 1][0][0];
            for (int n = 0; n < rounds; ++n) {
                const int i = n * kSampleThreads + tid;
                const uint32_t q = i < count ? mass(i) : 0u;
                const uint32_t digit = (q & mask) == prefix ? (q >> shift) & 0xffu : 0u;
                if (!kCached) {
                    if (digit != 0u) atomicAdd(reinterpret_cast<u64*>(hist) + digit, (u64)q);
                    continue;
                }
                const unsigned int busy = __ballot_sync(0xffffffffu, digit != 0u);
                if (busy == 0u) continue;
                const uint32_t first = __shfl_sync(0xffffffffu, digit, __ffs(busy) - 1);
                if (__popc(busy) > 8 && __all_sync(0xffffffffu, digit == 0u || digit == first)) {
                    const unsigned int lo = __reduce_add_sync(0xffffffffu, digit ? q & 0xffffu : 0u);
                    const unsigned int hi = __reduce_add_sync(0xffffffffu, digit ? q >> 16 : 0u);
                    if (lane == 0) { atomicAdd(&hist[first], lo); atomicAdd(&hist[256 + first], hi); }
                } else if (digit != 0u) {
                    atomicAdd(&hist[digit], q & 0xffffu);
                    atomicAdd(&hist[256 + digit], q >> 16);
                }
            }
            const uint32_t digit = descend<CTAS, !kCached>(s, level & 1, need, above);
            prefix |= digit << shift;
            mask |= 0xffu << shift;
            for (int i = tid; i < 512; i += kSampleThreads) (&s.hist[(level + 1) & 1][0][0])[i] = 0u;
            __syncthreads();
        }
        q_min = prefix;
    }

    // ---- draw: the first index whose running kept mass exceeds u * kept mass ----
    // a warp's segment is a run of tokens, so that the sums are in the order of the vocabulary
    const int segment = ((count + kSampleWarps - 1) / kSampleWarps + 31) & ~31;
    const int seg_begin = min(warp * segment, count), seg_end = min(seg_begin + segment, count);
    __syncthreads();                                             // another thread took the mass, with no descent in between
    part = 0ull;
    for (int i = seg_begin + lane; i < seg_end; i += 32) {
        const uint32_t q = mass(i);
        if (q >= q_min) part += q;
    }
    part = warp_sum_u64(part);
    if (lane == 0) s.warp_part[warp] = part;
    __syncthreads();
    if (warp == 0) {
        const u64 all = warp_sum_u64(lane < kSampleWarps ? s.warp_part[lane] : 0ull);
        if (lane < CTAS) *of_rank<CTAS>(&s.kept[rank], lane) = all;
    }
    cluster_barrier<CTAS>();                                           // the last access to a peer's memory lies before it
    u64 kept = 0ull, run = 0ull;
#pragma unroll
    for (int r = 0; r < CTAS; ++r) {
        if (r < rank) run += s.kept[r];
        kept += s.kept[r];
    }
    if (kept == 0ull) {
        if (rank == 0 && tid == 0) out_ids[row] = argmax;
        return;
    }
    float u = p.u;
    u = u < 0.f ? 0.f : (u >= 1.f ? 0.99999994f : u);
    u64 target = (u64)((double)u * (double)kept);
    if (target >= kept) target = kept - 1ull;
    for (int w = 0; w < warp; ++w) run += s.warp_part[w];
    if (target < run || target >= run + part) return;            // another warp's, or another CTA's
    for (int i0 = seg_begin; i0 < seg_end; i0 += 32) {
        const int i = i0 + lane;
        const uint32_t q = i < seg_end ? mass(i) : 0u;
        u64 upto = q >= q_min ? (u64)q : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 before = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += before;
        }
        const unsigned int past = __ballot_sync(0xffffffffu, run + upto > target);
        if (past != 0u) {
            if (lane == 0) out_ids[row] = begin + i0 + __ffs(past) - 1;
            return;
        }
        run += __shfl_sync(0xffffffffu, upto, 31);
    }
}

// ---- every row greedy: a cluster of eight CTAs per row, each over an eighth of the vocabulary ----
// One CTA walking a row of 150 k logits is bound by what one SM fetches from the L2 (about 15 us); eight of them take
// an eighth each and meet in the first CTA's shared memory.  The largest value wins, ties go to the lowest id, values
// that are not numbers never win: the same answer as the kernel above, whatever the order of the comparisons.
constexpr int kArgmaxCtas = 8;
constexpr int kArgmaxThreads = 512;

__global__ void __launch_bounds__(kArgmaxThreads)
argmax_cluster_kernel(const float* __restrict__ logits, int ld, int vocab, int* __restrict__ out_ids) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float s_val[kArgmaxThreads / 32];
    __shared__ int s_idx[kArgmaxThreads / 32];
    __shared__ float s_part_val[kArgmaxCtas];
    __shared__ int s_part_idx[kArgmaxCtas];
    const int row = blockIdx.x / kArgmaxCtas, rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* x = logits + (size_t)row * ld;
    // Distributed shared memory may only be touched once every CTA of the cluster runs: arrive here, wait before the
    // remote store, so that the scan hides the barrier.
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int chunk = ((vocab + kArgmaxCtas - 1) / kArgmaxCtas + 3) & ~3;
    const int begin = min(vocab, rank * chunk), end = min(vocab, begin + chunk);
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        // begin is a multiple of four: whole float4 groups, then the tail
        const int groups = (end - begin) / 4;
        const float4* x4 = reinterpret_cast<const float4*>(x + begin);
        for (int g = tid; g < groups; g += kArgmaxThreads) {
            const float4 v = x4[g];
            const int i = begin + 4 * g;
            take_better(best, best_i, v.x, i); take_better(best, best_i, v.y, i + 1);
            take_better(best, best_i, v.z, i + 2); take_better(best, best_i, v.w, i + 3);
        }
        for (int i = begin + 4 * groups + tid; i < end; i += kArgmaxThreads) take_better(best, best_i, x[i], i);
    } else {
        for (int i = begin + tid; i < end; i += kArgmaxThreads) take_better(best, best_i, x[i], i);
    }
    for (int o = 16; o > 0; o >>= 1)
        take_better(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
    if (lane == 0) { s_val[warp] = best; s_idx[warp] = best_i; }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        best = lane < kArgmaxThreads / 32 ? s_val[lane] : -INFINITY;
        best_i = lane < kArgmaxThreads / 32 ? s_idx[lane] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1)
            take_better(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
        if (lane == 0) {
            // every CTA of the cluster has started (the barrier above the scan): its shared memory may be written
            *cluster.map_shared_rank(&s_part_val[rank], 0) = best;
            *cluster.map_shared_rank(&s_part_idx[rank], 0) = best_i;
        }
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
        best = -INFINITY; best_i = 0x7fffffff;
        for (int r = 0; r < kArgmaxCtas; ++r) take_better(best, best_i, s_part_val[r], s_part_idx[r]);
        out_ids[row] = best_i == 0x7fffffff ? 0 : best_i;
    }
}

}  // namespace cib

using namespace cib;

// Every row greedy (temperature 0): out_ids[r] = argmax of logits[r], ties to the lowest id.
extern "C" int cib_argmax_rows(const float* logits, int ld, int rows, int vocab, int* out_ids, cudaStream_t stream) {
    CIB_REQUIRE(rows >= 0 && vocab > 0 && ld >= vocab, "argmax_rows: bad sizes rows=%d V=%d ld=%d", rows, vocab, ld);
    if (rows == 0) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows * kArgmaxCtas);
    cfg.blockDim = dim3(kArgmaxThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kArgmaxCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, argmax_cluster_kernel, logits, ld, vocab, out_ids);
    if (e != cudaSuccess) {
        set_error("argmax_rows: launch failed: %s", cudaGetErrorString(e));
        return -2;
    }
    return 0;
}

// params: [rows] of {float temperature, int top_k, float top_p, float u}.
extern "C" int cib_sample(const float* logits, int ld, int rows, int vocab, const void* params, int* out_ids,
                          cudaStream_t stream) {
    CIB_REQUIRE(rows >= 0 && vocab > 0 && ld >= vocab, "sample: bad sizes rows=%d V=%d ld=%d", rows, vocab, ld);
    if (rows == 0) return 0;
    const int ctas = sample_ctas(rows, vocab), share = ((vocab + ctas - 1) / ctas + 3) & ~3;
    const bool cached = share <= kSampleShareMax;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows * ctas);
    cfg.blockDim = dim3(kSampleThreads);
    cfg.dynamicSmemBytes = cached ? share * sizeof(float) : 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctas > 1 ? 1 : 0;
    static SmemLimit limits[4];
    const auto launch = [&](auto kernel, SmemLimit& limit) -> int {
        if (cached && raise_smem_limit(limit, kernel, kSampleShareMax * sizeof(float), "sample") != 0) return -2;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, logits, ld, vocab, share, (const SampleParams*)params, out_ids);
        if (e == cudaSuccess) return 0;
        set_error("sample: launch failed: %s", cudaGetErrorString(e));
        return -2;
    };
    if (!cached) return launch(sample_cluster_kernel<kSampleCtas, false>, limits[0]);      // such a row has eight
    switch (ctas) {
        case 1: return launch(sample_cluster_kernel<1, true>, limits[0]);
        case 2: return launch(sample_cluster_kernel<2, true>, limits[1]);
        case 4: return launch(sample_cluster_kernel<4, true>, limits[2]);
        default: return launch(sample_cluster_kernel<8, true>, limits[3]);
    }
}
