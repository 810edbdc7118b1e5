// Split-K flash-decode grouped-query attention over the paged KV cache.
//
// Work item = (query row, KV head): the G = heads / kv_heads query heads that share a KV head are processed
// together, so every K/V byte is read once per item.  The key range of an item is cut into splits of
// `pages_per_split` pages (grid.y); each CTA produces a partial (max, sum, accumulator) triple per head in the
// caller's scratch buffer and a second small kernel merges the splits.  The work is KV streaming (HBM-bound).
// Chunks of several positions per sequence (prefill) put 16 / G consecutive positions into one item of the fast path:
// the 16 fragment rows of the tensor-core products are positions x heads, each row with its own causal key count,
// so the K/V bytes of a sequence are streamed 16 / G times less often than with one item per position.
//
// Fast path (bf16 pools, 64-token pages, head_dim 64 or 128): a producer warp stages K and V pages with
// non-multicast TMA (cp.async.bulk.tensor, 128-byte swizzle) through a ring of shared-memory stages guarded by
// mbarriers; eight consumer warps in two groups (a group per page, 16 tokens per warp) compute Q.K^T and P.V with bf16 mma.sync
// (m16n8k16, f32 accumulation, fragments fetched with ldmatrix from the swizzled tiles), keep an online softmax
// per row, reduce row maxima and sums with quad shuffles and merge through shared memory.
//
// Generic path (f32 pools, other head sizes or page sizes): one (row, head) per CTA with plain loads and f32
// FMAs -- this is the path the f32 parity configuration runs on.
//
// Reference semantics: src/ops/attention.cpp:65-95 (scores * f32(1/sqrt(hd)), softmax, P.V) with the causal rule
// key_pos <= query_pos (src/ops/attention.cpp:52-57) expressed as a per-row key count.
#include "common.cuh"
#include "kv_cache.cuh"

#include <cmath>
#include <map>
#include <mutex>
#include <utility>

namespace b200 {
namespace {

struct AttnParams {
    const float* q;    // [rows, heads, head_dim]
    int rows, tokens_per_sequence, heads, causal;
    int positions_per_item;   // tensor-core kernel: consecutive positions of one sequence that share a CTA (1 in decode)
    KvView kv;
    int pages_per_split, num_splits;
    int items;         // persistent tensor-core kernel: items the grid walks (grid x otherwise)
    float* part_o;     // [rows*heads, num_splits, head_dim]
    float* part_ml;    // [rows*heads, num_splits, 2]
    float* out;        // [rows, heads*head_dim]
    __nv_bfloat16 *out_hi, *out_lo;  // optional: result as a shadow (bf16 hi + lo planes) instead of `out`
    float scale;
    int32_t* status;
};

struct SplitPlan { int pages_total, pages_per_split, num_splits; };

SplitPlan plan_splits(int64_t rows, int kv_heads, int max_length, int page_size) {
    SplitPlan s{};
    s.pages_total = (max_length + page_size - 1) / page_size;
    if (s.pages_total < 1) s.pages_total = 1;
    const int64_t items = rows * kv_heads;
    // Enough CTAs to fill the SMs about three times (the scheduler evens out unequal items), but 8 to 16 pages
    // (128 to 512 KB of K and V) per CTA: a shorter stream is mostly pipeline ramp.
    const int64_t fill = 444;
    const int64_t want_splits = (fill + items - 1) / items;
    int64_t pps = s.pages_total / want_splits;
    if (pps < 8) pps = 8;
    if (pps > 16) pps = 16;
    if (items * ((s.pages_total + pps - 1) / pps) > 32768) pps = s.pages_total;
    // short contexts: one CTA per (row, KV head), no merge kernel - also up to 32 pages once the items alone give every SM a
    // CTA (a decode step is a chain of dependent launches: the merge launch costs more than the shorter streams save)
    if (s.pages_total <= 16 || (s.pages_total <= 32 && items >= 148)) pps = s.pages_total;
    if (pps > s.pages_total) pps = s.pages_total;
    s.pages_per_split = static_cast<int>(pps);
    s.num_splits = (s.pages_total + s.pages_per_split - 1) / s.pages_per_split;
    return s;
}

// Final attention value: f32, or the shadow planes when the caller asked for them.
__device__ __forceinline__ void store_result(const AttnParams& p, int64_t at, float value) {
    if (p.out_hi) {
        const __nv_bfloat16 hi = __float2bfloat16_rn(value);
        p.out_hi[at] = hi;
        p.out_lo[at] = __float2bfloat16_rn(value - __bfloat162float(hi));
    } else {
        p.out[at] = value;
    }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kConsumerWarps = 8;   // two groups of four: group g takes pages g, g+2, ... so two pages are in the
constexpr int kGroupWarps = 4;      // tensor-core pipeline at a time; a warp owns 16 tokens of its group's page
constexpr int kFastThreads = (kConsumerWarps + 1) * 32;
constexpr int kHalfTileBytes = 64 * 128;  // one TMA box: 64 tokens x 64 bf16
constexpr int kFastControlBytes = 256;    // behind the ring: full / empty barriers (at most 128 bytes), the give-up flag at 192

template <int HD, int STAGES> struct FastShape {
    static constexpr int halves = HD / 64;
    static constexpr int tile_bytes = halves * kHalfTileBytes;  // K or V page
    static constexpr int stage_bytes = 2 * tile_bytes;
    static constexpr int stages = STAGES;  // 6 x 32 KB (head_dim 128) or 8 / 6 x 16 KB (head_dim 64) of K and V in flight per CTA
    static constexpr int smem_bytes = stages * stage_bytes + 1024 + kFastControlBytes;   // 1024: slack of the 1024-byte alignment
};

// Byte offset of 16-byte chunk `chunk` (8 features) of token `token` inside a swizzled K or V page.
__device__ __forceinline__ uint32_t tile_offset(int token, int chunk) {
    return static_cast<uint32_t>((chunk >> 3) * kHalfTileBytes + token * 128 + (((chunk & 7) ^ (token & 7)) << 4));
}

// Barrier over the consumer warps only (the producer warp keeps streaming).
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumerWarps * 32) : "memory"); }

// Pages per split for a sequence of `pages` cached pages: the splits the sequence needs at the planned size share its
// pages evenly (17 pages planned as 16 + 1 become 9 + 8).
__device__ __forceinline__ int balanced_pages_per_split(int pages, int planned) {
    const int needed = (pages + planned - 1) / planned;
    return needed > 0 ? (pages + needed - 1) / needed : planned;
}

constexpr int kMostClustered = 8;   // CTAs of a cluster, the largest portable size

// MULTI: items of several positions (prefill chunks); the decode instantiation keeps one position per item and one key
// count for all of its rows.
// CLUSTERED: the splits of an item (grid y) are a thread-block cluster that merges them through distributed shared memory, in the order and
// arithmetic of attention_combine_kernel; every CTA stays to the end, with pages or without.
template <int HD, int STAGES, bool MULTI, bool CLUSTERED>
__global__ void __launch_bounds__(kFastThreads) attention_mma_kernel(const __grid_constant__ CUtensorMap kmap,
                                                                     const __grid_constant__ CUtensorMap vmap,
                                                                     const AttnParams p) {
    using S = FastShape<HD, STAGES>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::stages * S::stage_bytes);
    uint64_t* empty = full + S::stages;

    grid_dependency_wait();   // q, the cache and the lengths come from the preceding kernels
    grid_launch_dependents();
    // An item is (sequence, block of consecutive positions, KV head).  The 16 fragment rows of a warp hold the block's
    // positions times the head group: row r = position r / group, query head r % group.  Decode: one position, rows =
    // the group.  Prefill: 16 / group positions share every K/V byte the CTA streams.
    const int item = blockIdx.x, split = blockIdx.y;
    const int kvh = item % p.kv.kv_heads, block = item / p.kv.kv_heads;
    const int positions = MULTI ? p.positions_per_item : 1;
    const int blocks_per_sequence = (p.tokens_per_sequence + positions - 1) / positions;
    const int sequence = block / blocks_per_sequence;
    const int t_first = (block - sequence * blocks_per_sequence) * positions;
    const int t_count = MULTI ? min(positions, p.tokens_per_sequence - t_first) : 1;
    const int row = sequence * p.tokens_per_sequence + t_first;   // first activation row of the item
    const int base_len = p.kv.lengths[sequence];
    const int kv_len = base_len + (p.causal ? t_first + t_count : 0);   // keys the item's last position sees
    int page_end = (kv_len + kFastPageSize - 1) / kFastPageSize;
    const int per_split = balanced_pages_per_split(page_end, p.pages_per_split);
    const int filled = CLUSTERED ? min((page_end + per_split - 1) / per_split, static_cast<int>(gridDim.y)) : 0;   // splits that have pages
    const int page_begin = split * per_split;
    if (page_end > page_begin + per_split) page_end = page_begin + per_split;
    if (!CLUSTERED && page_begin >= page_end) return;  // uniform for the CTA
    const int pages = page_end - page_begin;
    const int group = p.heads / p.kv.kv_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kGroupWarps);
        }
        mbar_fence_init();
    }
    __syncthreads();

    float m_row[2] = {-INFINITY, -INFINITY}, l_row[2] = {0.0f, 0.0f};
    float o[HD / 8][4];
#pragma unroll
    for (int j = 0; j < HD / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f;

    if (warp == kConsumerWarps) {
        // ---- producer: all lanes walk the loop together, lane 0 waits and issues ----
        if (lane == 0) { tma_prefetch_descriptor(&kmap); tma_prefetch_descriptor(&vmap); }
        const int32_t* table = p.kv.page_table + static_cast<int64_t>(sequence) * p.kv.pages_per_seq + page_begin;
        bool alive = true;
        for (int i = 0; i < pages && alive; ++i) {
            if (lane == 0) {
                const int s = i % S::stages;
                const uint32_t phase = (i / S::stages) & 1;
                if (!mbar_wait(&empty[s], phase ^ 1)) {
                    atomicExch(p.status, B200_DEVICE_TIMEOUT);
                    alive = false;
                } else {
                    const int page = table[i];
                    const int y = (page * p.kv.kv_heads + kvh) * kFastPageSize;
                    uint8_t* kdst = smem + s * S::stage_bytes;
                    uint8_t* vdst = kdst + S::tile_bytes;
                    mbar_expect_tx(&full[s], S::stage_bytes);
#pragma unroll
                    for (int h = 0; h < S::halves; ++h) {
                        tma_load_2d(kdst + h * kHalfTileBytes, &kmap, h * 64, y, &full[s]);
                        tma_load_2d(vdst + h * kHalfTileBytes, &vmap, h * 64, y, &full[s]);
                    }
                }
            }
            alive = __shfl_sync(0xffffffffu, alive, 0);
        }
    } else {
        // ---- consumers ----
        const int g = lane >> 2, t = lane & 3;
        uint32_t qa[HD / 16][4];
        // this thread's two fragment rows: position and head inside the item, and the keys each may see
        const int pos0 = MULTI ? g / group : 0, pos1 = MULTI ? (g + 8) / group : 0;
        const bool v0 = g < group * t_count, v1 = g + 8 < group * t_count;
        const int limit0 = MULTI ? (v0 ? base_len + (p.causal ? t_first + pos0 + 1 : 0) : 0) : kv_len;
        const int limit1 = MULTI ? (v1 ? base_len + (p.causal ? t_first + pos1 + 1 : 0) : 0) : kv_len;
        {
            const float* q0 = p.q + (static_cast<int64_t>(row + pos0) * p.heads + kvh * group + (g - pos0 * group)) * HD;
            const float* q1 = p.q + (static_cast<int64_t>(row + pos1) * p.heads + kvh * group + (g + 8 - pos1 * group)) * HD;
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk) {
                const int c = kk * 16 + 2 * t;
                qa[kk][0] = v0 ? pack_bf16(q0[c], q0[c + 1]) : 0u;
                qa[kk][1] = v1 ? pack_bf16(q1[c], q1[c + 1]) : 0u;
                qa[kk][2] = v0 ? pack_bf16(q0[c + 8], q0[c + 9]) : 0u;
                qa[kk][3] = v1 ? pack_bf16(q1[c + 8], q1[c + 9]) : 0u;
            }
        }
        const int tok0 = (warp & (kGroupWarps - 1)) * 16;
        const int group_index = warp / kGroupWarps;
        const int mi = lane >> 3, ri = lane & 7;
        bool alive = true;
        for (int i = group_index; i < pages && alive; i += kConsumerWarps / kGroupWarps) {
            const int s = i % S::stages;
            const uint32_t phase = (i / S::stages) & 1;
            if (!mbar_wait(&full[s], phase)) {
                if (lane == 0) atomicExch(p.status, B200_DEVICE_TIMEOUT);
                alive = false;
                break;
            }
            const uint32_t kbase = smem_u32(smem + s * S::stage_bytes);
            const uint32_t vbase = kbase + S::tile_bytes;

            float sc[2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.0f;
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk) {
                uint32_t r[4];
                ldmatrix_x4(r, kbase + tile_offset(tok0 + (mi >> 1) * 8 + ri, 2 * kk + (mi & 1)));
                mma_bf16(sc[0], qa[kk], r[0], r[1]);
                mma_bf16(sc[1], qa[kk], r[2], r[3]);
            }
            // scale, mask keys at or beyond the row's key count, online softmax per row (g and g+8)
            const int token_base = (page_begin + i) * kFastPageSize + tok0 + 2 * t;
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int token = token_base + n * 8 + (e & 1);
                    const float v = token < (MULTI ? ((e >> 1) ? limit1 : limit0) : kv_len) ? sc[n][e] * p.scale : -INFINITY;
                    sc[n][e] = v;
                    mx[e >> 1] = fmaxf(mx[e >> 1], v);
                }
            float corr[2], safe[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
                const float m_new = fmaxf(m_row[h], mx[h]);
                safe[h] = m_new == -INFINITY ? 0.0f : m_new;
                corr[h] = expf(m_row[h] - safe[h]);
                m_row[h] = m_new;
            }
            float sum[2] = {0.0f, 0.0f};
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sc[n][e] = expf(sc[n][e] - safe[e >> 1]);
                    sum[e >> 1] += sc[n][e];
                }
            l_row[0] = l_row[0] * corr[0] + sum[0];
            l_row[1] = l_row[1] * corr[1] + sum[1];
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) {
                o[j][0] *= corr[0]; o[j][1] *= corr[0];
                o[j][2] *= corr[1]; o[j][3] *= corr[1];
            }
            uint32_t pa[4];
            pa[0] = pack_bf16(sc[0][0], sc[0][1]);
            pa[1] = pack_bf16(sc[0][2], sc[0][3]);
            pa[2] = pack_bf16(sc[1][0], sc[1][1]);
            pa[3] = pack_bf16(sc[1][2], sc[1][3]);
#pragma unroll
            for (int j = 0; j < HD / 8; j += 2) {
                uint32_t r[4];
                ldmatrix_x4_trans(r, vbase + tile_offset(tok0 + (mi & 1) * 8 + ri, j + (mi >> 1)));
                mma_bf16(o[j], pa, r[0], r[1]);
                mma_bf16(o[j + 1], pa, r[2], r[3]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            l_row[h] += __shfl_xor_sync(0xffffffffu, l_row[h], 1);
            l_row[h] += __shfl_xor_sync(0xffffffffu, l_row[h], 2);
        }
    }
    __syncthreads();  // every page has been consumed: the stage memory can be reused for the merge

    float* merge_o = reinterpret_cast<float*>(smem);                       // [warps][group][HD]
    float* merge_ml = merge_o + kConsumerWarps * 16 * HD;                   // [warps][16][2]
    float* split_o = merge_ml + kConsumerWarps * 16 * 2;                    // CLUSTERED: what the CTA adds to the item, [group][HD], and
    float* split_ml = split_o + 16 * HD;                                    //   [group][2] (max, sum)
    static_assert((kConsumerWarps + 1) * 16 * (HD + 2) * 4 <= S::stages * S::stage_bytes);
    if (warp < kConsumerWarps) {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = g + 8 * h;
            if (r < group * t_count) {
                float* dst = merge_o + (warp * 16 + r) * HD + 2 * t;
#pragma unroll
                for (int j = 0; j < HD / 8; ++j) {
                    dst[j * 8] = o[j][2 * h];
                    dst[j * 8 + 1] = o[j][2 * h + 1];
                }
                if (t == 0) {
                    merge_ml[(warp * 16 + r) * 2] = m_row[h];
                    merge_ml[(warp * 16 + r) * 2 + 1] = l_row[h];
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < group * t_count * HD; i += kFastThreads) {
        const int r = i / HD, d = i - r * HD;
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) m = fmaxf(m, merge_ml[(w * 16 + r) * 2]);
        float acc = 0.0f, l = 0.0f;
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) {
            const float mw = merge_ml[(w * 16 + r) * 2];
            const float weight = mw == -INFINITY ? 0.0f : expf(mw - m);
            acc += weight * merge_o[(w * 16 + r) * HD + d];
            l += weight * merge_ml[(w * 16 + r) * 2 + 1];
        }
        if constexpr (CLUSTERED) {
            split_o[i] = acc;
            if (d == 0) { split_ml[2 * r] = m; split_ml[2 * r + 1] = l; }
            continue;
        }
        const int position = MULTI ? r / group : 0;
        const int64_t head_item = static_cast<int64_t>(row + position) * p.heads + kvh * group + (r - position * group);
        if (p.num_splits == 1) {
            store_result(p, head_item * HD + d, acc / l);
        } else {
            p.part_o[(head_item * p.num_splits + split) * HD + d] = acc;
            if (d == 0) {
                p.part_ml[(head_item * p.num_splits + split) * 2] = m;
                p.part_ml[(head_item * p.num_splits + split) * 2 + 1] = l;
            }
        }
    }
    if constexpr (CLUSTERED) {
        cluster_sync_all();   // every split's sums are in its CTA's shared memory; each CTA finishes a share of the item
        const uint32_t o_at = smem_u32(split_o), ml_at = smem_u32(split_ml);
        for (int i = split * kFastThreads + threadIdx.x; i < group * HD; i += gridDim.y * kFastThreads) {
            const int r = i / HD, d = i - r * HD;
            float value[kMostClustered], m = -INFINITY, acc = 0.0f, l = 0.0f;
            float2 ml[kMostClustered];
#pragma unroll
            for (int c = 0; c < kMostClustered; ++c) {
                const bool there = c < filled;
                const uint32_t pair = map_peer_shared(ml_at + r * 8, there ? c : 0), at = map_peer_shared(o_at + i * 4, there ? c : 0);
                ml[c] = there ? make_float2(load_cluster_float(pair), load_cluster_float(pair + 4)) : make_float2(-INFINITY, 0.0f);
                value[c] = there ? load_cluster_float(at) : 0.0f;
            }
#pragma unroll
            for (int c = 0; c < kMostClustered; ++c) m = fmaxf(m, ml[c].x);
#pragma unroll
            for (int c = 0; c < kMostClustered; ++c) {
                if (c >= filled) break;
                l += expf(ml[c].x - m) * ml[c].y;
                acc += expf(ml[c].x - m) * value[c];
            }
            // (a row that sees no key is left as it is)
            if (filled > 0) store_result(p, (static_cast<int64_t>(row) * p.heads + kvh * group + r) * HD + d, acc / l);
        }
        cluster_sync_all();   // nobody leaves while a peer reads its shared memory
    }
}

// The same kernel for decode with more units of work (item, split of its pages) than resident CTAs: a CTA walks the units
// blockIdx.x, + gridDim.x, ... and its
// producer warp runs ahead into the next item's pages while the consumers finish the current one, so the K/V stream of an
// SM does not stop at item boundaries (an item of 17 pages is ~290 KB: a sixth of its time was pipeline ramp).  The
// cross-warp merge then has its own shared memory behind the ring instead of re-using drained stages.
template <int HD, int STAGES>
__global__ void __launch_bounds__(kFastThreads) attention_persistent_kernel(const __grid_constant__ CUtensorMap kmap,
                                                                     const __grid_constant__ CUtensorMap vmap,
                                                                     const AttnParams p) {
    using S = FastShape<HD, STAGES>;
    constexpr bool MULTI = false, PERSIST = true;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::stages * S::stage_bytes);
    uint64_t* empty = full + S::stages;
    volatile int* gave_up = reinterpret_cast<volatile int*>(smem + S::stages * S::stage_bytes + 192);   // a consumer's wait ran out

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    grid_dependency_wait();   // q, the cache and the lengths come from the preceding kernels
    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < S::stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kGroupWarps);
        }
        *gave_up = 0;
        mbar_fence_init();
    }
    __syncthreads();

    // An item is (sequence, block of consecutive positions, KV head).  The 16 fragment rows of a warp hold the block's
    // positions times the head group: row r = position r / group, query head r % group.  Decode: one position, rows =
    // the group.  Prefill: 16 / group positions share every K/V byte the CTA streams.
    const int group = p.heads / p.kv.kv_heads;
    const int positions = MULTI ? p.positions_per_item : 1;
    const int blocks_per_sequence = (p.tokens_per_sequence + positions - 1) / positions;
    // units of work: (item, split of its pages); without PERSIST the grid has one CTA per unit
    const int units = PERSIST ? p.items * p.num_splits : static_cast<int>(blockIdx.x) + 1;
    // the cross-warp merge: [warps][16][HD] partial outputs and [warps][16][2] (max, sum); PERSIST keeps only the rows of a
    // decode item ([warps][group][...]) in its own memory behind the barriers
    float* merge_o = PERSIST ? reinterpret_cast<float*>(smem + S::stages * S::stage_bytes + kFastControlBytes) : reinterpret_cast<float*>(smem);
    const int merge_rows = PERSIST ? group : 16;
    float* merge_ml = merge_o + kConsumerWarps * merge_rows * HD;
    int walked = 0;   // pages this CTA has been through before the current item: stage and phase follow from it

    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int item = PERSIST ? unit / p.num_splits : unit;
        const int split = PERSIST ? unit - item * p.num_splits : static_cast<int>(blockIdx.y);
        const int kvh = item % p.kv.kv_heads, block = item / p.kv.kv_heads;
        const int sequence = block / blocks_per_sequence;
        const int t_first = (block - sequence * blocks_per_sequence) * positions;
        const int t_count = MULTI ? min(positions, p.tokens_per_sequence - t_first) : 1;
        const int row = sequence * p.tokens_per_sequence + t_first;   // first activation row of the item
        const int base_len = p.kv.lengths[sequence];
        const int kv_len = base_len + (p.causal ? t_first + t_count : 0);   // keys the item's last position sees
        int page_end = (kv_len + kFastPageSize - 1) / kFastPageSize;
        const int per_split = balanced_pages_per_split(page_end, p.pages_per_split);
        const int page_begin = split * per_split;
        if (page_end > page_begin + per_split) page_end = page_begin + per_split;
        if (page_begin >= page_end) continue;  // uniform for the CTA (a sequence without keys writes nothing, as before)
        const int pages = page_end - page_begin;

        if (warp == kConsumerWarps) {
            // ---- producer: all lanes walk the loop together, lane 0 waits and issues ----
            if (lane == 0 && walked == 0) { tma_prefetch_descriptor(&kmap); tma_prefetch_descriptor(&vmap); }
            const int32_t* table = p.kv.page_table + static_cast<int64_t>(sequence) * p.kv.pages_per_seq + page_begin;
            bool alive = true;
            for (int i = 0; i < pages && alive; ++i) {
                if (lane == 0) {
                    const int n = walked + i;
                    const int s = n % S::stages;
                    const uint32_t phase = (n / S::stages) & 1;
                    if (!mbar_wait(&empty[s], phase ^ 1)) {
                        atomicExch(p.status, B200_DEVICE_TIMEOUT);
                        alive = false;
                    } else {
                        const int page = table[i];
                        const int y = (page * p.kv.kv_heads + kvh) * kFastPageSize;
                        uint8_t* kdst = smem + s * S::stage_bytes;
                        uint8_t* vdst = kdst + S::tile_bytes;
                        mbar_expect_tx(&full[s], S::stage_bytes);
#pragma unroll
                        for (int h = 0; h < S::halves; ++h) {
                            tma_load_2d(kdst + h * kHalfTileBytes, &kmap, h * 64, y, &full[s]);
                            tma_load_2d(vdst + h * kHalfTileBytes, &vmap, h * 64, y, &full[s]);
                        }
                    }
                }
                alive = __shfl_sync(0xffffffffu, alive, 0);
            }
            walked += pages;
            if (!alive) break;   // the consumers run into their own bounded waits
            continue;
        }

        // ---- consumers ----
        float m_row[2] = {-INFINITY, -INFINITY}, l_row[2] = {0.0f, 0.0f};
        float o[HD / 8][4];
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f;
        const int g = lane >> 2, t = lane & 3;
        uint32_t qa[HD / 16][4];
        // this thread's two fragment rows: position and head inside the item, and the keys each may see
        const int pos0 = MULTI ? g / group : 0, pos1 = MULTI ? (g + 8) / group : 0;
        const bool v0 = g < group * t_count, v1 = g + 8 < group * t_count;
        const int limit0 = MULTI ? (v0 ? base_len + (p.causal ? t_first + pos0 + 1 : 0) : 0) : kv_len;
        const int limit1 = MULTI ? (v1 ? base_len + (p.causal ? t_first + pos1 + 1 : 0) : 0) : kv_len;
        {
            const float* q0 = p.q + (static_cast<int64_t>(row + pos0) * p.heads + kvh * group + (g - pos0 * group)) * HD;
            const float* q1 = p.q + (static_cast<int64_t>(row + pos1) * p.heads + kvh * group + (g + 8 - pos1 * group)) * HD;
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk) {
                const int c = kk * 16 + 2 * t;
                qa[kk][0] = v0 ? pack_bf16(q0[c], q0[c + 1]) : 0u;
                qa[kk][1] = v1 ? pack_bf16(q1[c], q1[c + 1]) : 0u;
                qa[kk][2] = v0 ? pack_bf16(q0[c + 8], q0[c + 9]) : 0u;
                qa[kk][3] = v1 ? pack_bf16(q1[c + 8], q1[c + 9]) : 0u;
            }
        }
        const int tok0 = (warp & (kGroupWarps - 1)) * 16;
        const int group_index = warp / kGroupWarps;
        const int mi = lane >> 3, ri = lane & 7;
        bool alive = true;
        // the two warp groups alternate over the CTA's pages as a whole, not per item: stage n belongs to group n % 2
        for (int i = (group_index + walked) & 1; i < pages && alive; i += kConsumerWarps / kGroupWarps) {
            const int n = walked + i;
            const int s = n % S::stages;
            const uint32_t phase = (n / S::stages) & 1;
            if (!mbar_wait(&full[s], phase)) {
                if (lane == 0) { atomicExch(p.status, B200_DEVICE_TIMEOUT); *gave_up = 1; }
                alive = false;
                break;
            }
            const uint32_t kbase = smem_u32(smem + s * S::stage_bytes);
            const uint32_t vbase = kbase + S::tile_bytes;

            float sc[2][4];
#pragma unroll
            for (int n2 = 0; n2 < 2; ++n2) sc[n2][0] = sc[n2][1] = sc[n2][2] = sc[n2][3] = 0.0f;
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk) {
                uint32_t r[4];
                ldmatrix_x4(r, kbase + tile_offset(tok0 + (mi >> 1) * 8 + ri, 2 * kk + (mi & 1)));
                mma_bf16(sc[0], qa[kk], r[0], r[1]);
                mma_bf16(sc[1], qa[kk], r[2], r[3]);
            }
            // scale, mask keys at or beyond the row's key count, online softmax per row (g and g+8)
            const int token_base = (page_begin + i) * kFastPageSize + tok0 + 2 * t;
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int n2 = 0; n2 < 2; ++n2)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int token = token_base + n2 * 8 + (e & 1);
                    const float v = token < (MULTI ? ((e >> 1) ? limit1 : limit0) : kv_len) ? sc[n2][e] * p.scale : -INFINITY;
                    sc[n2][e] = v;
                    mx[e >> 1] = fmaxf(mx[e >> 1], v);
                }
            float corr[2], safe[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
                const float m_new = fmaxf(m_row[h], mx[h]);
                safe[h] = m_new == -INFINITY ? 0.0f : m_new;
                corr[h] = expf(m_row[h] - safe[h]);
                m_row[h] = m_new;
            }
            float sum[2] = {0.0f, 0.0f};
#pragma unroll
            for (int n2 = 0; n2 < 2; ++n2)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sc[n2][e] = expf(sc[n2][e] - safe[e >> 1]);
                    sum[e >> 1] += sc[n2][e];
                }
            l_row[0] = l_row[0] * corr[0] + sum[0];
            l_row[1] = l_row[1] * corr[1] + sum[1];
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) {
                o[j][0] *= corr[0]; o[j][1] *= corr[0];
                o[j][2] *= corr[1]; o[j][3] *= corr[1];
            }
            uint32_t pa[4];
            pa[0] = pack_bf16(sc[0][0], sc[0][1]);
            pa[1] = pack_bf16(sc[0][2], sc[0][3]);
            pa[2] = pack_bf16(sc[1][0], sc[1][1]);
            pa[3] = pack_bf16(sc[1][2], sc[1][3]);
#pragma unroll
            for (int j = 0; j < HD / 8; j += 2) {
                uint32_t r[4];
                ldmatrix_x4_trans(r, vbase + tile_offset(tok0 + (mi & 1) * 8 + ri, j + (mi >> 1)));
                mma_bf16(o[j], pa, r[0], r[1]);
                mma_bf16(o[j + 1], pa, r[2], r[3]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
        walked += pages;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            l_row[h] += __shfl_xor_sync(0xffffffffu, l_row[h], 1);
            l_row[h] += __shfl_xor_sync(0xffffffffu, l_row[h], 2);
        }
        // Every consumer warp is through its pages: without PERSIST the whole ring is drained and serves the merge; with it
        // the merge has its own memory, which the previous item's readers have left (second barrier below).
        consumer_barrier();
        if (*gave_up) break;   // the same for every consumer warp after the barrier: nobody is left waiting at the next one
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = g + 8 * h;
            if (r < group * t_count) {
                float* dst = merge_o + (warp * merge_rows + r) * HD + 2 * t;
#pragma unroll
                for (int j = 0; j < HD / 8; ++j) {
                    dst[j * 8] = o[j][2 * h];
                    dst[j * 8 + 1] = o[j][2 * h + 1];
                }
                if (t == 0) {
                    merge_ml[(warp * merge_rows + r) * 2] = m_row[h];
                    merge_ml[(warp * merge_rows + r) * 2 + 1] = l_row[h];
                }
            }
        }
        consumer_barrier();
        for (int i = threadIdx.x; i < group * t_count * HD; i += kConsumerWarps * 32) {
            const int r = i / HD, d = i - r * HD;
            float m = -INFINITY;
#pragma unroll
            for (int w = 0; w < kConsumerWarps; ++w) m = fmaxf(m, merge_ml[(w * merge_rows + r) * 2]);
            float acc = 0.0f, l = 0.0f;
#pragma unroll
            for (int w = 0; w < kConsumerWarps; ++w) {
                const float mw = merge_ml[(w * merge_rows + r) * 2];
                const float weight = mw == -INFINITY ? 0.0f : expf(mw - m);
                acc += weight * merge_o[(w * merge_rows + r) * HD + d];
                l += weight * merge_ml[(w * merge_rows + r) * 2 + 1];
            }
            const int position = MULTI ? r / group : 0;
            const int64_t head_item = static_cast<int64_t>(row + position) * p.heads + kvh * group + (r - position * group);
            if (p.num_splits == 1) {
                store_result(p, head_item * HD + d, acc / l);
            } else {
                p.part_o[(head_item * p.num_splits + split) * HD + d] = acc;
                if (d == 0) {
                    p.part_ml[(head_item * p.num_splits + split) * 2] = m;
                    p.part_ml[(head_item * p.num_splits + split) * 2 + 1] = l;
                }
            }
        }
    }
}

// Passes of many positions per sequence (prefill): the arithmetic of attention_mma_kernel - a warp takes 16 tokens of every second page, with a running
// maximum, sum and accumulator of its own, and the eight of them are merged in the end, so that a row's result does not hang on the
// kernel, bit for bit - for two blocks of 16 fragment rows per CTA: a page is staged and its fragments are fetched once for both, whose
// chains of dependent instructions run side by side.  Every row sees the keys of its own position: a page behind those adds nothing.
// Blocks of late positions, which see the most pages, come first.  Bound by the chain of a page (products, softmax, products), of which 16 warps
// per SM (8 with heads of 128) hide a part, and by what stands around the pages, 5 us of a CTA's 14 at 1024 positions.  us, attention_mma_kernel
// | here: 8 prompts of 1024 positions, 32 / 8 heads of 64 598 | 388; 16 of 549, 12 / 4 heads 207 | 127; 2 of 4096, heads of 128 2619 | 2146.
// (With 16 rows per warp through whole pages, 128 a CTA, the first took 149 us, but then the weights, rounded to bf16, are relative to one maximum
// instead of eight: 18 % further from 64 bits, with peaked scores twice as far.)
constexpr int kPrefillThreads = kConsumerWarps * 32, kPrefillBlocks = 2, kPrefillStages = 6;   // 96 KB of pages: two CTAs per SM; 192 KB: one
template <int HD> struct PrefillShape : FastShape<HD, kPrefillStages> {
    using Base = FastShape<HD, kPrefillStages>;
    static constexpr int q_bytes = kPrefillBlocks * (HD / 16) * 32 * 16;   // q as fragments of the products
    static constexpr int smem_bytes = Base::smem_bytes + q_bytes;
    static constexpr int pitch = HD + 8;   // merge area: [blocks][warps][16][pitch], then (max, sum) and weights
    static constexpr int units = kPrefillBlocks * kConsumerWarps * 16;
    static_assert(units * (pitch + 3) * 4 + kPrefillBlocks * 16 * 4 <= Base::stages * Base::stage_bytes);
};

template <int HD>
__global__ void __launch_bounds__(kPrefillThreads, HD == 64 ? 2 : 1) attention_prefill_kernel(const __grid_constant__ CUtensorMap kmap,
                                                                                           const __grid_constant__ CUtensorMap vmap, const AttnParams p) {
    using S = PrefillShape<HD>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int gave_up;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::stages * S::stage_bytes);
    uint64_t* empty = full + S::stages;
    uint4* q_fragments = reinterpret_cast<uint4*>(smem + S::stages * S::stage_bytes + kFastControlBytes);   // [blocks][HD / 16][lanes]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S::stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kGroupWarps);
        }
        gave_up = 0;
        mbar_fence_init();
    }
    __syncthreads();
    grid_dependency_wait();   // q, the cache and the lengths come from the preceding kernels
    grid_launch_dependents();

    const int group = p.heads / p.kv.kv_heads, positions = p.positions_per_item, span = kPrefillBlocks * positions;
    const int streams = p.kv.sequences * p.kv.kv_heads;   // (sequence, KV head)
    const int spans = (p.tokens_per_sequence + span - 1) / span;
    const int stream = blockIdx.x % streams, t_first = (spans - 1 - static_cast<int>(blockIdx.x) / streams) * span;
    const int sequence = stream / p.kv.kv_heads, kvh = stream - sequence * p.kv.kv_heads;
    const int t_count = min(span, p.tokens_per_sequence - t_first);
    const int base_len = p.kv.lengths[sequence];
    const int pages = (base_len + (p.causal ? t_first + t_count : 0) + kFastPageSize - 1) / kFastPageSize;
    if (pages == 0) return;   // a row that sees no key is left as it is

    // The first lane of warp 0 requests the pages: a ring's worth here, later ones kLag pages after their stage was last read.
    constexpr int kLag = 4;
    const int32_t* table = p.kv.page_table + static_cast<int64_t>(sequence) * p.kv.pages_per_seq;
    int requested = 0;
    auto request = [&] {
        const int s = requested % S::stages, y = (table[requested] * p.kv.kv_heads + kvh) * kFastPageSize;
        uint8_t* kdst = smem + s * S::stage_bytes;
        uint8_t* vdst = kdst + S::tile_bytes;
        mbar_expect_tx(&full[s], S::stage_bytes);
#pragma unroll
        for (int h = 0; h < S::halves; ++h) {
            tma_load_2d(kdst + h * kHalfTileBytes, &kmap, h * 64, y, &full[s]);
            tma_load_2d(vdst + h * kHalfTileBytes, &vmap, h * 64, y, &full[s]);
        }
        ++requested;
    };
    if (threadIdx.x == 0)
        while (requested < min(pages, S::stages)) request();

    const int g = lane >> 2, t = lane & 3, mi = lane >> 3, ri = lane & 7;
    // fragment row r of block b: position b * positions + r / group, query head r % group
    auto rows_of = [&](int b) { return group * max(0, min(positions, t_count - b * positions)); };
    auto row_at = [&](int b, int r) {
        const int position = r / group;
        return (static_cast<int64_t>(sequence) * p.tokens_per_sequence + t_first + b * positions + position) * p.heads + kvh * group + (r - position * group);
    };
    for (int f = warp; f < kPrefillBlocks * (HD / 16); f += kConsumerWarps) {
        const int b = f / (HD / 16), c = (f - b * (HD / 16)) * 16 + 2 * t;
        uint32_t q[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (g + 8 * h < rows_of(b)) {
                const float* from = p.q + row_at(b, g + 8 * h) * HD + c;
                q[h] = pack_bf16(from[0], from[1]);
                q[2 + h] = pack_bf16(from[8], from[9]);
            }
        q_fragments[f * 32 + lane] = make_uint4(q[0], q[1], q[2], q[3]);
    }
    int limit[kPrefillBlocks][2];   // keys that this thread's two rows of a block see
#pragma unroll
    for (int b = 0; b < kPrefillBlocks; ++b)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = g + 8 * h;
            limit[b][h] = r < rows_of(b) ? base_len + (p.causal ? t_first + b * positions + r / group + 1 : 0) : 0;
        }
    const int seen_by_all = base_len + (p.causal ? t_first + 1 : 0);   // keys that every row of the CTA sees
    __syncthreads();

    float m_row[kPrefillBlocks][2], l_row[kPrefillBlocks][2], o[kPrefillBlocks][HD / 8][4];
#pragma unroll
    for (int b = 0; b < kPrefillBlocks; ++b) {
        m_row[b][0] = m_row[b][1] = -INFINITY;
        l_row[b][0] = l_row[b][1] = 0.0f;
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) o[b][j][0] = o[b][j][1] = o[b][j][2] = o[b][j][3] = 0.0f;
    }
    const int tok0 = (warp & (kGroupWarps - 1)) * 16;
    for (int i = warp / kGroupWarps; i < pages; i += kConsumerWarps / kGroupWarps) {
        const int s = i % S::stages;
        if (threadIdx.x == 0)
            for (int j = i - kLag; j < i - kLag + 2; ++j) {   // (a wait that runs out leaves a page unrequested: everyone's wait for it runs out too)
                if (j < 0 || j + S::stages >= pages) continue;
                if (requested == j + S::stages && mbar_wait(&empty[j % S::stages], (j / S::stages) & 1)) request();
            }
        __syncwarp();
        if (!mbar_wait(&full[s], (i / S::stages) & 1)) {
            if (lane == 0) atomicExch(p.status, B200_DEVICE_TIMEOUT);
            *static_cast<volatile int*>(&gave_up) = 1;
            break;
        }
        const uint32_t kbase = smem_u32(smem + s * S::stage_bytes), vbase = kbase + S::tile_bytes;
        float sc[kPrefillBlocks][2][4];
#pragma unroll
        for (int b = 0; b < kPrefillBlocks; ++b)
#pragma unroll
            for (int n = 0; n < 2; ++n) sc[b][n][0] = sc[b][n][1] = sc[b][n][2] = sc[b][n][3] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
            uint32_t r[4];
            ldmatrix_x4(r, kbase + tile_offset(tok0 + (mi >> 1) * 8 + ri, 2 * kk + (mi & 1)));
#pragma unroll
            for (int b = 0; b < kPrefillBlocks; ++b) {
                const uint4 packed = q_fragments[(b * (HD / 16) + kk) * 32 + lane];
                const uint32_t q[4] = {packed.x, packed.y, packed.z, packed.w};
                mma_bf16(sc[b][0], q, r[0], r[1]);
                mma_bf16(sc[b][1], q, r[2], r[3]);
            }
        }
        const bool masked = (i + 1) * kFastPageSize > seen_by_all;
        const int token = i * kFastPageSize + tok0 + 2 * t;
        uint32_t pa[kPrefillBlocks][4];
#pragma unroll
        for (int b = 0; b < kPrefillBlocks; ++b) {
            // scale, mask keys at or beyond the row's key count, online softmax per row (g and g + 8)
            float mx[2] = {-INFINITY, -INFINITY}, corr[2], safe[2], sum[2] = {0.0f, 0.0f};
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float v = sc[b][n][e] * p.scale;
                    if (masked && token + n * 8 + (e & 1) >= limit[b][e >> 1]) v = -INFINITY;
                    sc[b][n][e] = v;
                    mx[e >> 1] = fmaxf(mx[e >> 1], v);
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
                const float m_new = fmaxf(m_row[b][h], mx[h]);
                safe[h] = m_new == -INFINITY ? 0.0f : m_new;
                corr[h] = expf(m_row[b][h] - safe[h]);
                m_row[b][h] = m_new;
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sc[b][n][e] = expf(sc[b][n][e] - safe[e >> 1]);
                    sum[e >> 1] += sc[b][n][e];
                }
            l_row[b][0] = l_row[b][0] * corr[0] + sum[0];
            l_row[b][1] = l_row[b][1] * corr[1] + sum[1];
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) {
                o[b][j][0] *= corr[0]; o[b][j][1] *= corr[0];
                o[b][j][2] *= corr[1]; o[b][j][3] *= corr[1];
            }
            pa[b][0] = pack_bf16(sc[b][0][0], sc[b][0][1]);
            pa[b][1] = pack_bf16(sc[b][0][2], sc[b][0][3]);
            pa[b][2] = pack_bf16(sc[b][1][0], sc[b][1][1]);
            pa[b][3] = pack_bf16(sc[b][1][2], sc[b][1][3]);
        }
#pragma unroll
        for (int j = 0; j < HD / 8; j += 2) {
            uint32_t r[4];
            ldmatrix_x4_trans(r, vbase + tile_offset(tok0 + (mi & 1) * 8 + ri, j + (mi >> 1)));
#pragma unroll
            for (int b = 0; b < kPrefillBlocks; ++b) {
                mma_bf16(o[b][j], pa[b], r[0], r[1]);
                mma_bf16(o[b][j + 1], pa[b], r[2], r[3]);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    }
    __syncthreads();   // every page has been consumed: the stages can be reused for the merge
    if (gave_up) {     // ... unless a wait ran out: pages that are on their way get the same time again before the CTA leaves
        if (threadIdx.x == 0)
            for (int j = max(0, requested - S::stages); j < requested; ++j) mbar_wait(&full[j % S::stages], (j / S::stages) & 1);
        __syncthreads();
        return;
    }

    float* merge_o = reinterpret_cast<float*>(smem);                     // [blocks][warps][16][pitch]
    float* merge_ml = merge_o + S::units * S::pitch;                       // [blocks][warps][16][2]
    float* weights = merge_ml + S::units * 2;                              // [blocks][16][warps]
    float* sums = weights + S::units;                                      // [blocks][16]
#pragma unroll
    for (int b = 0; b < kPrefillBlocks; ++b)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float l = l_row[b][h];
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            const int unit = (b * kConsumerWarps + warp) * 16 + g + 8 * h;
            float* to = merge_o + unit * S::pitch + 2 * t;
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) *reinterpret_cast<float2*>(to + j * 8) = make_float2(o[b][j][2 * h], o[b][j][2 * h + 1]);
            if (t == 0) {
                merge_ml[2 * unit] = m_row[b][h];
                merge_ml[2 * unit + 1] = l;
            }
        }
    __syncthreads();
    {   // eight adjacent lanes are the eight warps' parts of one row
        static_assert(S::units == kPrefillThreads);
        const int row = threadIdx.x >> 3, w = threadIdx.x & 7, unit = ((row >> 4) * kConsumerWarps + w) * 16 + (row & 15);
        const float mw = merge_ml[2 * unit], lw = merge_ml[2 * unit + 1];
        float m = mw;
#pragma unroll
        for (int x = 1; x < 8; x <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
        const float weight = mw == -INFINITY ? 0.0f : expf(mw - m);
        float l = 0.0f;
#pragma unroll
        for (int x = 0; x < 8; ++x) l += __shfl_sync(0xffffffffu, weight, (lane & 24) + x) * __shfl_sync(0xffffffffu, lw, (lane & 24) + x);
        weights[threadIdx.x] = weight;
        if (w == 0) sums[row] = l;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < kPrefillBlocks; ++b)
        for (int i = threadIdx.x; i < rows_of(b) * HD; i += kPrefillThreads) {
            const int r = i / HD, d = i - r * HD;
            const float* part = merge_o + (b * kConsumerWarps * 16 + r) * S::pitch + d;
            const float* weight = weights + (b * 16 + r) * kConsumerWarps;
            float acc = 0.0f;
#pragma unroll
            for (int w = 0; w < kConsumerWarps; ++w) acc += weight[w] * part[w * 16 * S::pitch];
            store_result(p, row_at(b, r) * HD + d, acc / sums[b * 16 + r]);
        }
}

// Generic path: one (row, head) per CTA, eight warps that take kGenericTokens tokens of the split at a time.  Bound by latency (the f32 byte
// decoder at context 64: 8 CTAs), so the loads and the reductions of a batch of tokens are independent of each other and only one
// softmax update follows a batch; with four warps and a token at a time the launch took 13.5 us there, now 5.4.
constexpr int kGenericThreads = 256, kGenericWarps = kGenericThreads / 32, kGenericTokens = 8;
constexpr int kMaxDimsPerLane = 8;  // head_dim <= 256

__global__ void __launch_bounds__(kGenericThreads) attention_generic_kernel(const AttnParams p) {
    __shared__ float merge_ml[kGenericWarps][2];
    extern __shared__ float merge_o[];  // [warps][head_dim]
    grid_dependency_wait();
    grid_launch_dependents();
    const int hd = p.kv.head_dim;
    const int item = blockIdx.x, split = blockIdx.y;
    const int row = item / p.heads, head = item % p.heads;
    const int kvh = head / (p.heads / p.kv.kv_heads);
    const int sequence = row / p.tokens_per_sequence;
    const int kv_len = p.kv.lengths[sequence] + (p.causal ? row % p.tokens_per_sequence + 1 : 0);
    const int per_split = balanced_pages_per_split((kv_len + p.kv.page_size - 1) / p.kv.page_size, p.pages_per_split);
    const int begin = split * per_split * p.kv.page_size;
    int end = begin + per_split * p.kv.page_size;
    if (end > kv_len) end = kv_len;
    if (begin >= end) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* q = p.q + (static_cast<int64_t>(row) * p.heads + head) * hd;
    float qv[kMaxDimsPerLane], acc[kMaxDimsPerLane];
#pragma unroll
    for (int i = 0; i < kMaxDimsPerLane; ++i) {
        const int d = lane + 32 * i;
        qv[i] = d < hd ? q[d] : 0.0f;
        acc[i] = 0.0f;
    }
    float m = -INFINITY, l = 0.0f;
    for (int first = begin + warp * kGenericTokens; first < end; first += kGenericWarps * kGenericTokens) {
        int64_t at[kGenericTokens];
        float score[kGenericTokens];
#pragma unroll
        for (int u = 0; u < kGenericTokens; ++u) {   // tokens past the end repeat the last one and get no weight
            at[u] = kv_offset(p.kv, sequence, min(first + u, end - 1), kvh);
            score[u] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kMaxDimsPerLane; ++i) {
            const int d = lane + 32 * i;
            if (d >= hd) break;
#pragma unroll
            for (int u = 0; u < kGenericTokens; ++u) score[u] = fmaf(qv[i], kv_load(p.kv, 0, at[u] + d), score[u]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < kGenericTokens; ++u) score[u] += __shfl_xor_sync(0xffffffffu, score[u], o);
        float m_new = m;
#pragma unroll
        for (int u = 0; u < kGenericTokens; ++u) {
            score[u] = first + u < end ? score[u] * p.scale : -INFINITY;
            m_new = fmaxf(m_new, score[u]);
        }
        const float corr = expf(m - m_new);
        l *= corr;
#pragma unroll
        for (int u = 0; u < kGenericTokens; ++u) {
            score[u] = first + u < end ? expf(score[u] - m_new) : 0.0f;
            l += score[u];
        }
#pragma unroll
        for (int i = 0; i < kMaxDimsPerLane; ++i) {
            const int d = lane + 32 * i;
            if (d >= hd) break;
            acc[i] *= corr;
#pragma unroll
            for (int u = 0; u < kGenericTokens; ++u)
                acc[i] = first + u < end ? fmaf(score[u], kv_load(p.kv, 1, at[u] + d), acc[i]) : acc[i];
        }
        m = m_new;
    }
#pragma unroll
    for (int i = 0; i < kMaxDimsPerLane; ++i) {
        const int d = lane + 32 * i;
        if (d < hd) merge_o[warp * hd + d] = acc[i];
    }
    if (lane == 0) { merge_ml[warp][0] = m; merge_ml[warp][1] = l; }
    __syncthreads();
    const int64_t head_item = static_cast<int64_t>(row) * p.heads + head;
    for (int d = threadIdx.x; d < hd; d += kGenericThreads) {
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < kGenericWarps; ++w) mm = fmaxf(mm, merge_ml[w][0]);
        float a = 0.0f, ll = 0.0f;
#pragma unroll
        for (int w = 0; w < kGenericWarps; ++w) {
            const float weight = merge_ml[w][0] == -INFINITY ? 0.0f : expf(merge_ml[w][0] - mm);
            a += weight * merge_o[w * hd + d];
            ll += weight * merge_ml[w][1];
        }
        if (p.num_splits == 1) {
            store_result(p, head_item * hd + d, a / ll);
        } else {
            p.part_o[(head_item * p.num_splits + split) * hd + d] = a;
            if (d == 0) {
                p.part_ml[(head_item * p.num_splits + split) * 2] = mm;
                p.part_ml[(head_item * p.num_splits + split) * 2 + 1] = ll;
            }
        }
    }
}

// Merge of the split partials: one (row, head) per CTA.
__global__ void attention_combine_kernel(const AttnParams p) {
    grid_dependency_wait();
    grid_launch_dependents();
    const int hd = p.kv.head_dim;
    const int64_t head_item = blockIdx.x;
    const int row = static_cast<int>(head_item / p.heads);
    const int sequence = row / p.tokens_per_sequence;
    const int kv_len = p.kv.lengths[sequence] + (p.causal ? row % p.tokens_per_sequence + 1 : 0);
    const int pages = (kv_len + p.kv.page_size - 1) / p.kv.page_size;
    const int per_split = balanced_pages_per_split(pages, p.pages_per_split);
    int valid = (pages + per_split - 1) / per_split;   // splits whose CTA had pages and wrote a partial
    if (valid > p.num_splits) valid = p.num_splits;
    if (valid == 0) return;   // a row that sees no key is left as it is, as without splits
    const float* ml = p.part_ml + head_item * p.num_splits * 2;
    float m = -INFINITY;
    for (int s = 0; s < valid; ++s) m = fmaxf(m, ml[2 * s]);
    float l = 0.0f;
    for (int s = 0; s < valid; ++s) l += expf(ml[2 * s] - m) * ml[2 * s + 1];
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {
        float acc = 0.0f;
        for (int s = 0; s < valid; ++s) acc += expf(ml[2 * s] - m) * p.part_o[(head_item * p.num_splits + s) * hd + d];
        store_result(p, head_item * hd + d, acc / l);
    }
}

// Whether a pass takes the prefill kernel: where its half as many CTAs save rounds over the SMs.  A round costs about 8 + pages us there, 8 +
// 0.53 pages with attention_mma_kernel (the results are the same); CTAs with heads of 64, two per SM, gain little from having an SM to
// themselves.  us, attention_mma_kernel | prefill kernel: 48 positions behind 1000, heads of 64, 1 sequence 12.6 | 18.0, 4 sequences 26.9 | 24.2,
// 16 83.8 | 67.4; 100 positions behind 4000, heads of 128, 1 sequence 80 | 69, 200 positions 120 | 138.  Over 180 sizes up to 13 % from the better one.
bool takes_prefill(int64_t items, int64_t ctas, int pages, int head_dim, int sms) {
    auto rounds = [&](int64_t n) {
        const double whole = static_cast<double>((n + sms - 1) / sms);
        return head_dim == 64 && whole < 1.45 ? 1.45 : whole;
    };
    return rounds(ctas) * (8.0 + pages) < rounds(items) * (8.0 + 0.53 * pages);
}

int64_t prefill_ctas(const AttnParams& p) {
    const int span = kPrefillBlocks * p.positions_per_item;
    return static_cast<int64_t>(p.kv.sequences) * p.kv.kv_heads * ((p.tokens_per_sequence + span - 1) / span);
}

template <int HD> int launch_prefill(const b200_kv_cache* cache, const AttnParams& p, cudaStream_t stream) {
    auto kernel = attention_prefill_kernel<HD>;
    B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PrefillShape<HD>::smem_bytes));
    return cuda_status(launch_dependent(kernel, dim3(static_cast<unsigned>(prefill_ctas(p))), dim3(kPrefillThreads), PrefillShape<HD>::smem_bytes, stream,
                                        *kv_tensor_map(cache, 0), *kv_tensor_map(cache, 1), p), "attention_prefill_kernel launch");
}

// Clusters of `splits` CTAs that the device holds at once; asked of the runtime once per device and size, and kept.
template <int HD, int STAGES> int resident_clusters(int splits, int device) {
    static std::mutex mutex;
    static std::map<std::pair<int, int>, int> known;
    std::lock_guard<std::mutex> lock(mutex);
    const auto [at, first] = known.try_emplace({device, splits}, 0);
    if (!first) return at->second;
    auto kernel = attention_mma_kernel<HD, STAGES, false, true>;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(1, static_cast<unsigned>(splits));
    config.blockDim = dim3(kFastThreads);
    config.dynamicSmemBytes = FastShape<HD, STAGES>::smem_bytes;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = 1; attribute.val.clusterDim.y = static_cast<unsigned>(splits); attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FastShape<HD, STAGES>::smem_bytes) != cudaSuccess
        || cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
        cudaGetLastError();
        clusters = 0;
    }
    return at->second = clusters;
}

template <int HD, int STAGES> int launch_fast(const b200_kv_cache* cache, AttnParams p, bool& merged, cudaStream_t stream) {
    using S = FastShape<HD, STAGES>;
    const int blocks_per_sequence = (p.tokens_per_sequence + p.positions_per_item - 1) / p.positions_per_item;
    const int items = (p.rows / p.tokens_per_sequence) * blocks_per_sequence * p.kv.kv_heads;
    int device = 0;
    B200_CUDA(cudaGetDevice(&device));
    // Decode with more units of work than the SMs hold at once: persistent CTAs that stream across unit boundaries.
    const int group = p.heads / p.kv.kv_heads;
    const int merge_bytes = kConsumerWarps * group * (HD + 2) * static_cast<int>(sizeof(float));
    const int persist_bytes = S::smem_bytes + merge_bytes;   // the merge area follows the control block
    // Splits of decode items merge inside a cluster where the device holds all of them at once: the merge kernel's launch and the partials' way through
    // memory are saved (8 items of 24 pages, three splits, inside a decode step: 9.3 -> 7.5 us); a second wave would cost more than that.
    if (p.num_splits > 1 && p.num_splits <= kMostClustered && p.positions_per_item == 1 && p.tokens_per_sequence == 1
        && items <= resident_clusters<HD, STAGES>(p.num_splits, device)) {
        auto kernel = attention_mma_kernel<HD, STAGES, false, true>;
        B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::smem_bytes));
        const unsigned splits = static_cast<unsigned>(p.num_splits);
        merged = true;
        return cuda_status(launch_dependent_cluster(kernel, dim3(static_cast<unsigned>(items), splits), dim3(kFastThreads), S::smem_bytes, stream,
                                                    dim3(1, splits, 1), *kv_tensor_map(cache, 0), *kv_tensor_map(cache, 1), p),
                           "attention_mma_kernel launch");
    }
    // With split items the units are dealt out in turn, which only balances when the sequences are equally long (what
    // the cache's owner knows on the host); ragged split batches keep one CTA per unit and the hardware's scheduling.
    if (p.positions_per_item == 1 && persist_bytes <= 232448 && static_cast<int64_t>(items) * p.num_splits > sm_count(device)
        && (p.num_splits == 1 || cache->even_lengths)) {
        auto kernel = attention_persistent_kernel<HD, STAGES>;
        B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, persist_bytes));
        int per_sm = 0;   // CTAs of this kernel an SM holds at once, asked of the runtime (1 if it cannot say)
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kFastThreads, static_cast<size_t>(persist_bytes)) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        const int resident = per_sm * sm_count(device);
        p.items = items;
        if (items * p.num_splits <= resident) {   // every unit has a CTA of its own anyway
            return cuda_status(launch_dependent(kernel, dim3(static_cast<unsigned>(items * p.num_splits)), dim3(kFastThreads),
                                                static_cast<size_t>(persist_bytes), stream, *kv_tensor_map(cache, 0), *kv_tensor_map(cache, 1), p),
                               "attention_mma_kernel launch");
        }
        p.items = items;
        return cuda_status(launch_dependent(kernel, dim3(static_cast<unsigned>(resident)), dim3(kFastThreads), static_cast<size_t>(persist_bytes),
                                            stream, *kv_tensor_map(cache, 0), *kv_tensor_map(cache, 1), p), "attention_mma_kernel launch");
    }
    auto kernel = p.positions_per_item > 1 ? attention_mma_kernel<HD, STAGES, true, false> : attention_mma_kernel<HD, STAGES, false, false>;
    B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::smem_bytes));
    const dim3 grid(static_cast<unsigned>(items), p.num_splits);
    return cuda_status(launch_dependent(kernel, grid, dim3(kFastThreads), S::smem_bytes, stream, *kv_tensor_map(cache, 0),
                                        *kv_tensor_map(cache, 1), p), "attention_mma_kernel launch");
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" size_t b200_attention_scratch_bytes(int64_t rows, int32_t heads, int32_t kv_heads, int32_t head_dim,
                                               int32_t max_length, int32_t page_size) {
    if (rows <= 0 || heads <= 0 || kv_heads <= 0 || head_dim <= 0 || max_length <= 0 || page_size <= 0) return 0;
    const SplitPlan s = plan_splits(rows, kv_heads, max_length, page_size);
    if (s.num_splits == 1) return 256;
    return static_cast<size_t>(rows) * heads * s.num_splits * (head_dim + 2) * sizeof(float) + 256;
}

namespace {
int attention_launch(const float* q, int64_t rows, int32_t tokens_per_sequence, int32_t heads, const b200_kv_cache* cache,
                     int32_t max_length, int32_t causal, void* scratch, size_t scratch_bytes, float* out, __nv_bfloat16* out_hi,
                     __nv_bfloat16* out_lo, void* stream) {
    if (!q || !cache || (!out && !(out_hi && out_lo)) || rows <= 0 || tokens_per_sequence <= 0 || heads <= 0 || heads % cache->kv_heads
        || rows != static_cast<int64_t>(cache->sequences) * tokens_per_sequence || max_length <= 0) {
        set_error("b200_attention_decode: bad pointer, size or head grouping");
        return B200_BAD_ARGUMENT;
    }
    if (cache->head_dim > 32 * kMaxDimsPerLane) { set_error("b200_attention_decode: head_dim above 256 is not supported"); return B200_UNSUPPORTED; }
    {   // the kernels run on the current device: it must be the one that holds the cache (and, for the static entry, the scratch)
        int current = -1;
        B200_CUDA(cudaGetDevice(&current));
        if (current != cache->device) {
            set_error("b200_attention_decode: the cache lives on device %d, the current device is %d", cache->device, current);
            return B200_BAD_ARGUMENT;
        }
    }
    if (max_length > cache->capacity) max_length = cache->capacity;
    const int group = heads / cache->kv_heads;
    const bool fast = kv_tensor_map(cache, 0) && group <= 16 && (cache->head_dim == 64 || cache->head_dim == 128);
    // Chunks of several positions (prefill) on the tensor-core kernel: 16 / group consecutive positions share a CTA and one
    // CTA walks all pages of its item (the split sizes of the merge kernel are per row, the items' are per block).
    const int positions = fast && tokens_per_sequence > 1 ? (16 / group > 0 ? 16 / group : 1) : 1;
    SplitPlan plan = plan_splits(rows, cache->kv_heads, max_length, cache->page_size);
    if (positions > 1) {
        plan.pages_per_split = plan.pages_total;
        plan.num_splits = 1;
    }
    const size_t need = b200_attention_scratch_bytes(rows, heads, cache->kv_heads, cache->head_dim, max_length, cache->page_size);
    if (plan.num_splits > 1 && (!scratch || scratch_bytes < need)) {
        set_error("b200_attention_decode: scratch of %zu bytes needed, %zu given", need, scratch_bytes);
        return B200_BAD_ARGUMENT;
    }
    AttnParams p{};
    p.q = q; p.rows = static_cast<int>(rows); p.tokens_per_sequence = tokens_per_sequence; p.heads = heads; p.causal = causal;
    p.positions_per_item = positions;
    p.kv = kv_view(cache);
    p.pages_per_split = plan.pages_per_split; p.num_splits = plan.num_splits;
    p.part_o = static_cast<float*>(scratch);
    p.part_ml = p.part_o ? p.part_o + static_cast<size_t>(rows) * heads * plan.num_splits * cache->head_dim : nullptr;
    p.out = out; p.out_hi = out_hi; p.out_lo = out_lo;
    p.scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(cache->head_dim)));
    p.status = device_status_word(cache->device);
    if (!p.status) { set_error("b200_attention_decode: the device status word could not be allocated"); return B200_NO_DEVICE; }
    cudaStream_t s = as_stream(stream);
    int status;
    bool merged = plan.num_splits == 1;   // nothing is left to the merge kernel
    if (fast) {
        int device = 0;
        B200_CUDA(cudaGetDevice(&device));
        // head_dim 64 with more CTAs than SMs: a 96 KB ring lets two CTAs share an SM, so one CTA's pipeline ramp and
        // drain overlap the other's streaming; with fewer CTAs each keeps the deeper ring to itself.
        const int64_t ctas = (static_cast<int64_t>(p.rows) / tokens_per_sequence) * ((tokens_per_sequence + positions - 1) / positions)
                             * p.kv.kv_heads * p.num_splits;
        if (tokens_per_sequence > 1 && takes_prefill(ctas, prefill_ctas(p), plan.pages_total, cache->head_dim, sm_count(device)))
            return cache->head_dim == 128 ? launch_prefill<128>(cache, p, s) : launch_prefill<64>(cache, p, s);
        if (cache->head_dim == 128) status = launch_fast<128, 6>(cache, p, merged, s);
        else if (ctas > sm_count(device)) status = launch_fast<64, 6>(cache, p, merged, s);
        else status = launch_fast<64, 8>(cache, p, merged, s);
    } else {
        const dim3 grid(static_cast<unsigned>(rows) * heads, plan.num_splits);
        status = cuda_status(launch_dependent(attention_generic_kernel, grid, dim3(kGenericThreads), sizeof(float) * kGenericWarps * cache->head_dim, s, p),
                             "attention_generic_kernel launch");
    }
    if (status != B200_OK || merged) return status;
    return cuda_status(launch_dependent(attention_combine_kernel, dim3(static_cast<unsigned>(rows) * heads), dim3(128), 0, s, p),
                       "attention_combine_kernel launch");
}
}  // namespace

extern "C" int b200_attention_decode(const float* q, int64_t rows, int32_t tokens_per_sequence, int32_t heads,
                                     const b200_kv_cache* cache, int32_t max_length, int32_t causal, void* scratch,
                                     size_t scratch_bytes, float* out, void* stream) {
    if (!out) { set_error("b200_attention_decode: bad pointer, size or head grouping"); return B200_BAD_ARGUMENT; }
    return attention_launch(q, rows, tokens_per_sequence, heads, cache, max_length, causal, scratch, scratch_bytes, out, nullptr, nullptr, stream);
}

extern "C" int b200_attention_decode_shadow(const float* q, int64_t rows, int32_t tokens_per_sequence, int32_t heads,
                                            const b200_kv_cache* cache, int32_t max_length, int32_t causal, void* scratch,
                                            size_t scratch_bytes, void* out_hi, void* out_lo, void* stream) {
    if (!out_hi || !out_lo) { set_error("b200_attention_decode_shadow: shadow planes missing"); return B200_BAD_ARGUMENT; }
    return attention_launch(q, rows, tokens_per_sequence, heads, cache, max_length, causal, scratch, scratch_bytes, nullptr,
                            static_cast<__nv_bfloat16*>(out_hi), static_cast<__nv_bfloat16*>(out_lo), stream);
}

// ---- allocation-free variant ------------------------------------------------------------------------------
// Split partials live in this fixed array of the library image instead of a caller workspace.  In host code the
// name below is only a handle for the runtime: the device address comes from cudaGetSymbolAddress, looked up once
// per device with that device current, and that address is what the kernels receive.
static __device__ __align__(256) unsigned char attention_static_scratch[B200_STATIC_SCRATCH_BYTES];

namespace {
std::mutex static_scratch_mutex;
void* static_scratch_address[64];

int static_scratch_for(int device, void** address) {
    std::lock_guard<std::mutex> lock(static_scratch_mutex);
    if (device < 0 || device >= 64) { set_error("b200_attention_decode_static: device %d out of range", device); return B200_BAD_ARGUMENT; }
    if (!static_scratch_address[device]) {
        int current = -1;
        B200_CUDA(cudaGetDevice(&current));
        if (current != device) B200_CUDA(cudaSetDevice(device));
        void* found = nullptr;
        const cudaError_t status = cudaGetSymbolAddress(&found, attention_static_scratch);
        if (current != device) cudaSetDevice(current);
        if (status != cudaSuccess || !found) return cuda_status(status == cudaSuccess ? cudaErrorInvalidSymbol : status,
                                                                "cudaGetSymbolAddress(attention_static_scratch)");
        static_scratch_address[device] = found;
    }
    *address = static_scratch_address[device];
    return B200_OK;
}
}  // namespace

extern "C" int b200_attention_decode_static(const float* q, int64_t rows, int32_t tokens_per_sequence, int32_t heads,
                                            const b200_kv_cache* cache, int32_t max_length, int32_t causal, float* out,
                                            void* stream) {
    if (!cache || rows <= 0 || heads <= 0 || max_length <= 0) {
        set_error("b200_attention_decode_static: bad pointer or size");
        return B200_BAD_ARGUMENT;
    }
    const int32_t bounded = max_length > cache->capacity ? cache->capacity : max_length;
    const size_t need = b200_attention_scratch_bytes(rows, heads, cache->kv_heads, cache->head_dim, bounded, cache->page_size);
    if (need > B200_STATIC_SCRATCH_BYTES) {
        set_error("b200_attention_decode_static: this shape needs %zu bytes of split partials, the built-in array holds %u; "
                  "call b200_attention_decode with a workspace of your own", need, static_cast<unsigned>(B200_STATIC_SCRATCH_BYTES));
        return B200_BAD_ARGUMENT;
    }
    if (!device_status_word_if_allocated(cache->device)) {
        set_error("b200_attention_decode_static: no status word on device %d (create the KV cache through b200_kv_cache_create)", cache->device);
        return B200_BAD_ARGUMENT;
    }
    void* scratch = nullptr;
    const int status = static_scratch_for(cache->device, &scratch);
    if (status != B200_OK) return status;
    return b200_attention_decode(q, rows, tokens_per_sequence, heads, cache, max_length, causal, scratch,
                                 B200_STATIC_SCRATCH_BYTES, out, stream);
}
