// Paged causal attention for prompt portions on the 5th-generation tensor cores (head size 128, bfloat16).
//
// Same contract as csrc/ops/paged_attention.cu:133-383 of the reference (queries are the last n positions of a
// request, keys 0..position come from its pages, rows of a tile are query token x query head of one kv head), on
// Blackwell's own path instead of mma.sync:
//
//   * a CTA owns a 128-row query tile (128 / g tokens x g heads of one kv head) and walks over 64-key tiles; two CTAs share
//     an SM (256 columns of tensor memory and 97 KB of shared memory each), so that one takes exponentials while the other
//     starts, waits for its first keys or stores (8 prompts of 1 024 tokens, 16 heads over 8: 72 us a layer, 475 TFLOP/s,
//     where one CTA an SM, 128-key tiles and sixteen softmax warps took 89; one of 8 192: 275 us, 1 000 TFLOP/s, for 328).
//     Launches of few CTAs run that other variant (attention_tcgen05_wide.cu);
//   * keys and values come page by page through TMA (`cp.async.bulk.tensor.2d`, one box of 64 columns x one page per
//     copy, 128-byte swizzle: the layout the tensor cores read), issued by the lanes of the producer warps,
//     double-buffered, completion counted in bytes on mbarriers (four buffers each changed nothing).  (Copies issued by
//     ordinary loads or `cp.async` kept too few bytes in flight per SM: a tile took longer to arrive than its softmax takes.)
//     The page size must be a power of two of at least 8 slots, so that a box starts on a 1024-byte swizzle atom;
//   * S = Q K^T and O += P V are `tcgen05.mma.cta_group::1.kind::f16` with accumulators in tensor memory; K is a
//     K-major operand, V an MN-major one, straight from the page layout; P is the A operand of P V straight from tensor
//     memory (bfloat16, written with `tcgen05.st` over the scores it was made from), so it never touches shared memory;
//   * key tiles alternate between two buffers of S: S of tile j+1 is computed while the four softmax warps take the
//     exponentials of tile j.  A thread owns a row (TMEM lane = row): no exchange with other threads; it keeps the running
//     maximum in base 2 and raises it only when it grows by more than 8 (so O is rescaled rarely, with
//     `tcgen05.ld`/`tcgen05.st`);
//   * a fifth warp's first lane issues the MMAs.
//
// Two options serve attention layers that keep a token's key and value side by side in one cache row and put a learned
// number per head into the softmax's denominator: `joined` (the cache is [pages][kv heads][slots][key 128 | value 128];
// keys and values are boxes of the same tensor map, 128 columns apart) and `sinks` (32-bit, one per query head: at the
// end exp(sink) joins the denominator once, with no value).
//
// Every mbarrier wait is bounded; on a time-out the kernel raises the error flag, stops, frees its tensor memory
// and returns.
#include "attention_tcgen05_wide.cuh"
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

namespace cib {
namespace fa {

constexpr int kD = 128;          // head size
constexpr int kM = 128;          // rows per CTA
constexpr int kN = 64;           // keys per tile
constexpr int kPanel = kM * 128; // bytes of one 64-column panel of the 128 query rows
constexpr int kKvPanel = kN * 128;

// MN-major operand (values: [key][d], d contiguous), 128-byte swizzle: 64-element panels `panel_bytes` apart (leading
// offset), 8-key groups 1024 bytes apart (stride offset).
__device__ __forceinline__ uint64_t desc_mnmajor(const void* smem, uint32_t panel_bytes) {
    return (uint64_t)((tc_smem_u32(smem) & 0x3ffff) >> 4) | ((uint64_t)(panel_bytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// D = F32, A = B = BF16, M = 128; b_mn: B is MN-major.
__host__ __device__ constexpr uint32_t idesc(bool b_mn, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tst32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tst_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// shared memory: Q | K0 | K1 | V0 | V1; Q has 128 rows x 128 columns bf16 = 32 KB as two 64-column panels, a key or value tile
// 64 rows = 16 KB
constexpr int kQBytes = 2 * kPanel, kTileBytes = 2 * kKvPanel;
constexpr int kKBufs = 2, kVBufs = 2;
constexpr int kSmemBytes = kQBytes + (kKBufs + kVBufs) * kTileBytes + 1024 + 256;
constexpr int kTmemCols = 256;                     // S of buffer 0 | S of buffer 1 | O

constexpr int kMmaWarp = 4;                        // warps 0-3: the softmax, a thread per row
constexpr int kThreads = (kMmaWarp + 3) * 32;      // + the MMA warp, a producer warp for keys and one for values

// A operand from tensor memory (P, bfloat16, two keys to a column), B from shared memory
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a_tmem), "l"(b), "r"(id), "r"(acc) : "memory");
}

__global__ void __launch_bounds__(kThreads, 2)
attention_tcgen05_kernel(const __grid_constant__ CUtensorMap kv_map, int num_pages, const __nv_bfloat16* __restrict__ q, int q_stride,
                         __nv_bfloat16* __restrict__ out, int out_stride, int page_size,
                         const int* __restrict__ block_table, int table_stride, const int* __restrict__ query_start_loc,
                         const int* __restrict__ seq_lens, int num_requests, int least_query, int nq, int nkv, float scale_log2, int window,
                         int joined, const float* __restrict__ sinks, int* __restrict__ error_flag) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* sQ = base;
    unsigned char* sK = base + kQBytes;                         // kKBufs buffers: tile j in buffer j % kKBufs
    unsigned char* sV = sK + kKBufs * kTileBytes;         // kVBufs buffers
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kVBufs * kTileBytes);
    // one barrier per buffer; key tile j uses key, value and score buffer j % 2
    uint64_t* k_full = bars;           // [kKBufs <= 3] a key tile has landed (bytes counted)
    uint64_t* v_full = bars + 3;       // [2] a value tile has landed
    uint64_t* s_full = bars + 5;       // [2] S of a tile is in tensor memory
    uint64_t* p_ready = bars + 7;      // [2] P of a tile is in tensor memory (the softmax warps arrive)
    uint64_t* pv_done = bars + 9;      // [2] O includes a tile
    // With two key and two value buffers, tile j's buffers are free again exactly when s_full[j % 2] (S has read the
    // keys) and pv_done[j % 2] (P V has read the values) complete: the producers wait on those, and the thread that
    // issues the MMAs, which every tile waits for in turn, has two commits fewer per tile to issue.
    static_assert(kKBufs == 2 && kVBufs == 2, "the producers take s_full and pv_done for the buffers' release");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    __shared__ int s_req, s_tile, s_abort, s_q0, s_n, s_seq;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = blockIdx.x;     // heads vary fastest: every head's longest tile starts before any shorter one
    const int g = nq / nkv;

    const int g_shift = 31 - __clz(g);      // g divides 128: a power of two

    if (warp == 0) {
        // which request and which of its row tiles: the whole warp looks, 32 requests at a time (one thread walking up
        // to 64 requests took 6 us, and nothing else of the tile can start before this is known)
        int t = gridDim.y - 1 - blockIdx.y;     // later (longer) tiles first
        int req = num_requests, tile = 0;
        for (int r0 = 0; r0 < num_requests; r0 += 32) {
            const int r = r0 + lane;
            int tiles = 0;
            if (r < num_requests) {
                const int n = query_start_loc[r + 1] - query_start_loc[r];
                tiles = n < least_query ? 0 : (n * g + kM - 1) / kM;
            }
            int upto = tiles;                   // tiles of the requests r0 .. r
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += o;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, r < num_requests && t < upto);
            if (hit) {
                const int first = __ffs(hit) - 1;
                req = r0 + first;
                tile = t - (__shfl_sync(0xffffffffu, upto, first) - __shfl_sync(0xffffffffu, tiles, first));
                break;
            }
            t -= __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) {
            s_req = req; s_tile = tile; s_abort = 0;
            if (req < num_requests) {   // read here once, so that the other threads need no round trip of their own after the barrier
                s_q0 = query_start_loc[req];
                s_n = query_start_loc[req + 1] - query_start_loc[req];
                s_seq = seq_lens[req];
            }
            asm volatile("prefetch.tensormap [%0];" ::"l"(&kv_map) : "memory");
        }
    } else if (warp == 1 && lane < 16) {
        // a thread per barrier: p_ready (at 7 and 8) counts the softmax warps, all others one arrival
        mbar_init(&bars[lane], lane == 7 || lane == 8 ? kMmaWarp : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // stale values must at least be finite: rows of a tile that no page covers are multiplied by P = 0 (stale keys need not
    // be: their scores are replaced, not multiplied)
    for (int i = tid; i < kVBufs * kTileBytes / 16; i += blockDim.x) reinterpret_cast<uint4*>(sV)[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // before the bulk copies write the same bytes
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    // everything so far read only what the host wrote for this step; queries, keys and values come from the kernel before
    griddep_launch();
    griddep_wait();
    const uint32_t tmem = *tmem_slot;
    const int r = s_req;
    const bool active = r < num_requests;

    int q0 = 0, n = 0, seq_len = 0, row0 = 0, rows_total = 0, num_tiles = 0, k_lo = 0;
    if (active) {
        q0 = s_q0;
        n = s_n;
        seq_len = s_seq;
        rows_total = n * g;
        row0 = s_tile * kM;
        const int last_row = min(row0 + kM, rows_total) - 1;
        const int pos_first = seq_len - n + (row0 >> g_shift), pos_last = seq_len - n + (last_row >> g_shift);
        k_lo = window > 0 ? max(0, pos_first - window + 1) / kN * kN : 0;
        num_tiles = (pos_last + 1 - k_lo + kN - 1) / kN;
    }

    if (active && warp < kMmaWarp) {
        // ---- the query tile: row = token_local * g + head_in_group, two swizzled 64-column panels ----
        // (a thread's loads are all on their way before the first is stored: one round trip)
        constexpr int kPer = kM * 16 / (kMmaWarp * 32);
        uint4 v[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int idx = tid + u * kMmaWarp * 32;
            const int row = idx >> 4, c = idx & 15;
            const int grow = row0 + row;
            v[u] = make_uint4(0, 0, 0, 0);
            if (grow < rows_total) {
                const int tl = grow >> g_shift, hi = grow & (g - 1);
                v[u] = *reinterpret_cast<const uint4*>(q + (size_t)(q0 + tl) * q_stride + (size_t)(kvh * g + hi) * kD + c * 8);
            }
        }
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int idx = tid + u * kMmaWarp * 32;
            const int row = idx >> 4, c = idx & 15;
            *reinterpret_cast<uint4*>(sQ + (c >> 3) * kPanel + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = v[u];
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // the MMA warp waits for the query tile; the producer warps do not, so that the first keys and values are on their
    // way while the queries are still being copied
    if (warp <= kMmaWarp) asm volatile("bar.sync 10, %0;" ::"r"((kMmaWarp + 1) * 32) : "memory");

    // tensor memory: S of buffer 0 | S of buffer 1, 64 columns each, | O, 128 columns; P (bfloat16, two keys to a column)
    // takes the first 32 columns of its S once the softmax holds S in registers
    if (active && warp == kMmaWarp) {
        // ---- the MMAs: the whole warp walks the loop, lane 0 issues ----
        auto issue_s = [&](int j) {
            if (lane != 0) return;
            const int b = j & 1;
            const uint64_t qd = umma_desc_k_major_sw128(sQ), kd = umma_desc_k_major_sw128(sK + (j % kKBufs) * kTileBytes);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint64_t q_off = (uint64_t)(((k >> 2) * kPanel + (k & 3) * 32) >> 4), k_off = (uint64_t)(((k >> 2) * kKvPanel + (k & 3) * 32) >> 4);
                umma_bf16(tmem + (uint32_t)(b * kN), qd + q_off, kd + k_off, idesc(false, kN), k != 0);
            }
            umma_commit(&s_full[b]);            // also: the key buffer can be refilled
        };
        auto wait_all = [&](uint64_t* bar, uint32_t parity, int code) {
            bool ok = mbar_wait(bar, parity);
            if (!ok && lane == 0) { atomicExch(error_flag, code); s_abort = 1; }
            return __all_sync(0xffffffffu, ok);
        };
        bool ok = true;
        ok = wait_all(&k_full[0], 0, 11);
        if (ok) { tcgen05_fence_after(); issue_s(0); }
        for (int j = 0; j < num_tiles && ok; ++j) {
            const int b = j & 1;
            const uint32_t parity = (j >> 1) & 1;
            if (j + 1 < num_tiles) {
                // S(j+1) overwrites S and P of tile j-1 (same buffer): P V(j-1) was issued before, and the tensor pipe
                // runs what one thread issues in order
                ok = wait_all(&k_full[(j + 1) % kKBufs], ((j + 1) / kKBufs) & 1, 12);
                if (!ok) break;
                tcgen05_fence_after();
                issue_s(j + 1);
            }
            ok = wait_all(&p_ready[b], parity, 13) && wait_all(&v_full[b], parity, 14);
            if (!ok) break;
            {
                // the last page of the request came whole: value rows past its last token may hold anything, and
                // 0 x NaN is NaN, so they are cleared (their columns of P are 0)
                const int valid_rows = seq_len - (k_lo + j * kN);
                if (valid_rows < kN) {
                    const int box_rows = min(page_size, kN);
                    const int end = min(kN, (valid_rows + box_rows - 1) / box_rows * box_rows);
                    unsigned char* vb = sV + b * kTileBytes;
                    for (int idx = valid_rows * 16 + lane; idx < end * 16; idx += 32) {
                        const int row = idx >> 4, c = idx & 15;
                        *reinterpret_cast<uint4*>(vb + (c >> 3) * kKvPanel + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = make_uint4(0, 0, 0, 0);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                }
            }
            tcgen05_fence_after();
            if (lane == 0) {
                // O += P V: P is the A operand straight from tensor memory (16 keys = 8 columns per step)
#pragma unroll
                for (int k = 0; k < kN / 16; ++k) {
                    const uint64_t vd = desc_mnmajor(sV + b * kTileBytes + k * 16 * 128, kKvPanel);
                    mma_ts(tmem + (uint32_t)(2 * kN), tmem + (uint32_t)(b * kN + k * 8), vd, idesc(true, kD), j > 0 || k != 0);
                }
                umma_commit(&pv_done[b]);        // also: the value buffer can be refilled
            }
            __syncwarp();
        }
    } else if (active && warp > kMmaWarp) {
        // ---- producer warps (first: keys, second: values): a lane issues one TMA copy per (page
        // of the tile, 64-column panel); keys of tile j+2 as soon as S(j) has read its buffer, values of tile j+2 after P V(j).  Rows of a tile past the
        // request's last page are not copied: their columns of S are masked and P is 0 there.  A page number outside the
        // pool turns into a row outside the tensor map, which reads as zeros and still counts its bytes. ----
        const int* table = block_table + (size_t)r * table_stride;
        const int box_rows = min(page_size, kN);
        const int boxes = kN / box_rows;
        // joined: a token's key and value lie side by side in one row of 2 x 128 values (one plane), else in two planes
        const long long total_rows = (long long)num_pages * (joined ? 1 : 2) * nkv * page_size;
        // a tile has at most 16 boxes (8 pages of 8 slots x 2 panels): lane = box * 2 + panel.  The page number of
        // a lane's box is fetched a tile ahead, so that no copy waits for a round trip to the table.
        const int kv = warp - kMmaWarp - 1;
        const int box = lane >> 1, panel = lane & 1;
        int page = -1;
        auto lookup = [&](int t) {
            const int key = k_lo + t * kN + box * box_rows;
            page = t < num_tiles && box < boxes && key < seq_len ? __ldg(table + key / page_size) : -1;
        };
        const int depth = kv ? kVBufs : kKBufs;
        auto fill = [&](int t) {
            const int b = t % depth;
            const int key0 = k_lo + t * kN;
            uint64_t* bar = kv ? &v_full[b] : &k_full[b];
            const int nvalid = min(boxes, max(0, (seq_len - key0 + box_rows - 1) / box_rows));
            if (lane == 0) mbar_expect_tx(bar, (uint32_t)(nvalid * 2 * box_rows * 128));
            __syncwarp();
            if (box < nvalid) {
                const int off = (key0 + box * box_rows) % page_size;        // not 0 only for pages longer than a tile
                const long long row = page >= 0 && page < num_pages
                                          ? (joined ? ((long long)page * nkv + kvh) * page_size + off
                                                    : (((long long)page * 2 + kv) * nkv + kvh) * page_size + off)
                                          : total_rows;
                tma_load_2d((kv ? sV : sK) + b * kTileBytes + panel * kKvPanel + box * box_rows * 128, &kv_map, bar,
                            (joined ? kv * kD : 0) + panel * 64, (int)row);
            }
        };
        auto wait_all = [&](uint64_t* bar, uint32_t parity, int code) {
            bool ok = mbar_wait(bar, parity);
            if (!ok && lane == 0) { atomicExch(error_flag, code); s_abort = 1; }
            return __all_sync(0xffffffffu, ok);
        };
        uint64_t* free_bar = kv ? pv_done : s_full;
        for (int t = 0; t < depth && t < num_tiles; ++t) {
            lookup(t);
            fill(t);
        }
        lookup(depth);
        for (int j = 0; j + depth < num_tiles; ++j) {
            if (!wait_all(&free_bar[j % depth], (j / depth) & 1, 18 + kv)) break;      // S(j) / P V(j) has read the buffer
            fill(j + depth);
            lookup(j + depth + 1);
        }
    } else if (active && warp < kMmaWarp) {
        // ---- softmax: a thread per row (TMEM lane 32 * warp + lane); S of the next tile is computed meanwhile ----
        const int row_local = tid;
        const int grow = row0 + row_local;
        const bool row_ok = grow < rows_total;
        const int pos = row_ok ? seq_len - n + (grow >> g_shift) : -1;
        const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16), o_addr = lane_addr + 2 * kN;
        float m_used = -INFINITY, l = 0.f;
        bool ok = true;
        auto wait_here = [&](uint64_t* bar, uint32_t parity, int code) {       // false if the wait ran out
            bool good = mbar_wait(bar, parity);
            if (!good && lane == 0) { atomicExch(error_flag, code); s_abort = 1; }
            return __all_sync(0xffffffffu, good) != 0;
        };
        for (int j = 0; j < num_tiles; ++j) {
            const int b = j & 1;
            const int key0 = k_lo + j * kN;
            ok = wait_here(&s_full[b], (uint32_t)((j >> 1) & 1), 15);
            ok = __all_sync(0xffffffffu, ok && !(*(volatile int*)&s_abort)) != 0;
            if (!ok) break;
            tcgen05_fence_after();
            const bool need_mask = key0 + kN - 1 > pos || window > 0;
            const int hi = pos - key0;                              // columns <= hi are visible ...
            const int lo = window > 0 ? hi - window : -1;           // ... and > lo
            // the row's 64 scores, read from tensor memory once; masked ones become -inf here, so that the
            // maximum (the scale is positive: applied afterwards) and the exponentials need no second look at the mask
            uint32_t v[2][32];
            tmem_ld_32x32b_x32(lane_addr + (uint32_t)(b * kN), v[0]);
            tmem_ld_32x32b_x32(lane_addr + (uint32_t)(b * kN + 32), v[1]);
            tmem_ld_wait();
            if (need_mask) {
#pragma unroll
                for (int e = 0; e < kN; ++e)
                    if (!(e <= hi && e > lo)) v[e / 32][e % 32] = __float_as_uint(-INFINITY);
            }
            float part[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < kN; ++e) part[e & 3] = fmaxf(part[e & 3], __uint_as_float(v[e / 32][e % 32]));
            const float mx = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3])) * scale_log2;
            // raise the reference maximum only when it would grow by more than 8 (values stay below 2^8) — but whenever it grows
            // over the first 256 keys, so that a short context's largest weight is 1 and not rounded
            float corr = 1.f;
            bool rescale = false;
            if (mx > m_used + (j < 256 / kN ? 0.f : 8.f) || (m_used == -INFINITY && mx != -INFINITY)) {
                corr = m_used == -INFINITY ? 0.f : exp2f(m_used - mx);
                m_used = mx;
                l *= corr;
                rescale = j > 0;
            }
            // P = 2^(s * scale - m): one fused multiply-add and one ex2 per score, packed two to a register.  The sum is of the
            // weights as they are multiplied, rounded: the reference maximum lags behind, so that even a row's largest weight
            // is rounded, and only a sum that has the same rounding takes it out again
            const float m_eff = m_used == -INFINITY ? 0.f : m_used;
            uint32_t p[32];
            float sums[2] = {0.f, 0.f};
#pragma unroll
            for (int e = 0; e < kN; e += 2) {
                float pe[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float x = fmaf(__uint_as_float(v[e / 32][e % 32 + u]), scale_log2, -m_eff);
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(pe[u]) : "f"(x));
                }
                p[e / 2] = pack_bf16(pe[0], pe[1]);
                sums[0] += __uint_as_float(p[e / 2] << 16);
                sums[1] += __uint_as_float(p[e / 2] & 0xffff0000u);
            }
            l += sums[0] + sums[1];
            // O is only touched once P V of the tile before has finished
            if (j > 0 && __any_sync(0xffffffffu, rescale)) {
                ok = wait_here(&pv_done[b ^ 1], (uint32_t)(((j - 1) >> 1) & 1), 16);
                if (!ok) break;
                tcgen05_fence_after();
#pragma unroll 1
                for (int c = 0; c < kD; c += 32) {
                    uint32_t o[32];
                    tmem_ld_32x32b_x32(o_addr + (uint32_t)c, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
                    tst32(o_addr + (uint32_t)c, o);
                }
            }
            // P (bfloat16, two keys to a column) over the scores, which this row's thread holds in registers
            tst32(lane_addr + (uint32_t)(b * kN), p);
            tst_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[b]);
        }
        // every thread waits for the last P V itself: behind it no MMA reads shared or tensor memory
        if (ok && num_tiles > 0) ok = wait_here(&pv_done[(num_tiles - 1) & 1], (uint32_t)(((num_tiles - 1) >> 1) & 1), 17);
        tcgen05_fence_after();
        if (!(*(volatile int*)&s_abort) && num_tiles > 0) {
            float total = l;
            // a sink is a score of the row's head without key or value: it joins the denominator once, unscaled
            float keep = 1.f;
            if (sinks != nullptr && row_ok) {
                const float sink = sinks[kvh * g + (grow & (g - 1))] * 1.4426950408889634f;
                const float top = fmaxf(m_used, sink);
                keep = m_used == -INFINITY ? 0.f : exp2f(m_used - top);
                total = total * keep + exp2f(sink - top);
            }
            // (total is at least 2^-8 for a row with a visible key and at most a few thousand)
            const float f = keep * (total > 0.f ? __fdividef(1.f, total) : 0.f);
            // into the query tile's shared memory (every S has read it), a row's 256 bytes together, its 16-byte pieces
            // swapped by the row number so that neither these stores nor the loads below meet in a bank
#pragma unroll 1
            for (int c = 0; c < kD; c += 32) {
                uint32_t o[32];
                tmem_ld_32x32b_x32(o_addr + (uint32_t)c, o);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; e += 8) {
                    uint4 pk;
                    pk.x = pack_bf16(__uint_as_float(o[e]) * f, __uint_as_float(o[e + 1]) * f);
                    pk.y = pack_bf16(__uint_as_float(o[e + 2]) * f, __uint_as_float(o[e + 3]) * f);
                    pk.z = pack_bf16(__uint_as_float(o[e + 4]) * f, __uint_as_float(o[e + 5]) * f);
                    pk.w = pack_bf16(__uint_as_float(o[e + 6]) * f, __uint_as_float(o[e + 7]) * f);
                    const int piece = (c + e) >> 3;
                    *reinterpret_cast<uint4*>(sQ + row_local * 256 + ((piece ^ (row_local & 15)) << 4)) = pk;
                }
            }
        }
        // out to global memory sixteen threads to a row: a thread that stored its own row's pieces sent 32 partial
        // sectors with every instruction, and the tile's 2 048 of them took 1.5 us
        asm volatile("bar.sync 9, %0;" ::"r"(kMmaWarp * 32) : "memory");
        if (!(*(volatile int*)&s_abort) && num_tiles > 0) {
#pragma unroll
            for (int u = 0; u < kM * 16 / (kMmaWarp * 32); ++u) {
                const int idx = tid + u * kMmaWarp * 32;
                const int row = idx >> 4, c = idx & 15;
                const int grow_out = row0 + row;
                if (grow_out < rows_total) {
                    const uint4 pk = *reinterpret_cast<const uint4*>(sQ + row * 256 + ((c ^ (row & 15)) << 4));
                    const int tl = grow_out >> g_shift, hh = grow_out & (g - 1);
                    *reinterpret_cast<uint4*>(out + (size_t)(q0 + tl) * out_stride + (size_t)(kvh * g + hh) * kD + c * 8) = pk;
                }
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemCols) : "memory");
}

}  // namespace fa
}  // namespace cib

using namespace cib;


extern "C" int cib_attention_tcgen05_supports(int head_dim, int nq, int nkv, int page_size) {
    if (head_dim != 128 || nkv <= 0 || nq % nkv != 0) return 0;
    const int g = nq / nkv;
    return 128 % g == 0 && page_size >= 8 && (page_size & (page_size - 1)) == 0;
}

// num_tiles = sum over requests of ceil(tokens_r * (nq / nkv) / 128), or more: CTAs that find no tile leave.  least_tiles: how many
// of them the step has at least, which decides between the two variants (a recorded step is launched for the worst split of
// its tokens over its requests).  least_query: requests that bring fewer tokens have no tiles (1: all have; 2: those of one token are
// left to another kernel).  error_flag: one zero int in device memory.
extern "C" int cib_attention_tcgen05(const void* q, int q_stride, void* out, int out_stride, const void* cache, int num_pages,
                                     int page_size, const int* block_table, int table_stride, const int* query_start_loc,
                                     const int* seq_lens, int num_requests, int num_tiles, int least_tiles, int least_query, int nq, int nkv,
                                     int head_dim, float scale, int window, int joined, const float* sinks, int* error_flag,
                                     cudaStream_t stream) {
    CIB_REQUIRE(cib_attention_tcgen05_supports(head_dim, nq, nkv, page_size),
                "attention_tcgen05: head_dim %d, %d/%d heads, page size %d are not taken (head size 128, heads per kv head dividing 128, pages of 8, 16, 32, ... slots)",
                head_dim, nq, nkv, page_size);
    CIB_REQUIRE(num_requests >= 0 && num_tiles >= 0 && num_tiles <= 65535 && least_tiles <= num_tiles && num_pages > 0 && table_stride > 0,
                "attention_tcgen05: bad sizes");
    CIB_REQUIRE(q_stride % 8 == 0 && ((uintptr_t)q % 16) == 0 && out_stride % 8 == 0 && ((uintptr_t)out % 16) == 0 && ((uintptr_t)cache % 16) == 0,
                "attention_tcgen05: rows must be 16-byte aligned");
    CIB_REQUIRE(error_flag != nullptr, "attention_tcgen05: error flag missing");
    if (num_requests == 0 || num_tiles == 0) return 0;
    // the cache as rows of one head's slot: [pages * 2 * kv heads * page_size, 128], or, joined, [pages * kv heads *
    // page_size, 256] with the key in the first and the value in the second half of a row; a box is one page x 64 columns
    const long long total_rows = (long long)num_pages * (joined ? 1 : 2) * nkv * page_size;
    CIB_REQUIRE(total_rows < (1ll << 31), "attention_tcgen05: %lld cache rows do not fit a 32-bit coordinate", total_rows);
    // few CTAs: the variant that has an SM alone (attention_tcgen05_wide.cu says why the line lies here)
    const bool wide = (long long)nkv * least_tiles <= 3 * 148;
    const int tile_keys = wide ? kWideKeys : fa::kN;
    CUtensorMap kv_map;
    const int row_values = joined ? 2 * fa::kD : fa::kD;
    if (encode_tensor_map_bf16_2d(&kv_map, cache, (unsigned long long)total_rows, row_values, row_values, 64,
                                  page_size < tile_keys ? page_size : tile_keys, "attention_tcgen05") != 0)
        return -1;
    const float scale_log2 = scale * 1.4426950408889634f;
    if (wide)
        return attention_tcgen05_wide(kv_map, num_pages, (const __nv_bfloat16*)q, q_stride, (__nv_bfloat16*)out, out_stride, page_size, block_table,
                                      table_stride, query_start_loc, seq_lens, num_requests, least_query, num_tiles, nq, nkv, scale_log2, window, joined,
                                      sinks, error_flag, stream);
    static SmemLimit limit;
    if (int rc = raise_smem_limit(limit, fa::attention_tcgen05_kernel, fa::kSmemBytes, "attention_tcgen05")) return rc;
    const cudaError_t e = launch_pdl(fa::attention_tcgen05_kernel, dim3(nkv, num_tiles), dim3(fa::kThreads), (size_t)fa::kSmemBytes, stream,
                                     prompt_pdl(), kv_map, num_pages, (const __nv_bfloat16*)q, q_stride, (__nv_bfloat16*)out, out_stride,
                                     page_size, block_table, table_stride, query_start_loc, seq_lens, num_requests, least_query, nq, nkv, scale_log2,
                                     window, joined, sinks, error_flag);
    CIB_REQUIRE(e == cudaSuccess, "attention_tcgen05: launch failed: %s", cudaGetErrorString(e));
    return 0;
}
