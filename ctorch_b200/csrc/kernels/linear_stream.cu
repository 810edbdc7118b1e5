// Skinny linears for bf16 weights and up to 16 activation rows (decode batches): y = epilogue(rmsnorm?(x) @ W^T).  Two kernels:
//   * linear_stream_kernel: activations that arrive as two bf16 planes - every linear of a bf16 decode step;
//   * linear_staged_kernel: f32 activation rows, normalised and split while they are staged (logits behind a prefill, plain linears).
#include "linear_common.cuh"
#include "mma.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>


namespace b200 {
namespace {

constexpr int kConsumers = 8;
constexpr int kThreads = (kConsumers + 1) * 32;
constexpr int kRows = 16;
constexpr int kMaxIn = 2048;

struct StreamParams {
    LinearParams base;
    int tile_features;   // TF: 8, 16, 32 or 64
    int slots;           // ring depth, one whole tile [TF][in_padded + 8] per slot
    int tiles;           // ceil(out / TF)
    int in_padded;       // in rounded up to 64
    int32_t* status;
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void ldmatrix_x2(uint32_t (&r)[2], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(address));
}
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers * 32) : "memory"); }

// ---- streaming kernel: activations as bf16 planes ---------------------------------------------------------------------------
// Bound by weight streaming, so nothing stands between memory and the tensor cores: 16 bytes of a weight row are a lane's fragment of
// mma.m16n8k16 as they lie.  Lane (g, t) of a warp fetches entries [8t, 8t + 8) of a 32-column chunk of weight rows g and g + 8, and of
// activation row g; the products of a chunk take the columns in an order of their own (product 0: entries 8t .. 8t + 3 of every lane,
// product 1: 8t + 4 .. 8t + 7), the same on both sides, so nothing is shuffled.  Weights are the M side (16 features), activation rows
// the N side (8 or 16 tokens, two planes).
//   * A group of warps (8 or 16, see few_groups) owns tiles of 16 features and shares out the chunks of K.  Every lane has a ring of its own
//     in shared memory, filled by cp.async and read back by the same lane: no barrier, and 128 KB in flight per SM across tile borders,
//     started before the wait for the predecessor (6.5 TB/s over 148 SMs need about 45 KB at a microsecond of latency; a ring of 80 KB
//     in half the registers, so that two kernels share an SM, spilled and was a quarter slower).
//   * Activations stay in registers over all tiles where a warp has at most kFewKeep chunks (in <= 2048), all requested at once.
//   * The warps' partial sums meet in shared memory, in two buffers, so that a tile costs one barrier; the first 64 * NT threads finish
//     it (one row, two adjacent features each) while the other warps are in the next tile.
// Measured back to back, weights from memory, 1 | 16 rows, against a ring of whole tiles of 8 - 32 features with all activations staged first
// and two barriers a tile: 2048 -> 16384 SwiGLU 31.5 | 22.6 -> 12.8 | 15.6 us (5.2 | 4.3 TB/s), 2048 -> 32000 argmax 54.0 | 43.9 -> 21.9 |
// 26.1 us (6.0 TB/s), 2048 -> 3072 15.4 | 6.9 -> 5.0 | 6.1, 768 -> 768 6.6 | 3.9 -> 2.7 | 3.1, 768 -> 32000 18.3 | 14.5 -> 10.8 | 13.6.
struct FewParams {
    LinearParams base;
    int tiles;   // ceil(out / 16)
};
constexpr int kFewFeatures = 16, kFewKeep = 4, kFewDepth = 8, kFewWarps = 16;

template <int NT, int WARPS, int EPI>
__global__ void __launch_bounds__(kFewWarps * 32, 1) linear_stream_kernel(const __grid_constant__ FewParams fp) {
    constexpr int kPitch = 8 * NT + 1, kGroups = kFewWarps / WARPS, kSpan = WARPS * 32;   // kSpan: columns that a group takes side by side
    const LinearParams& p = fp.base;
    extern __shared__ __align__(16) uint4 ring[];   // [warps][kFewDepth][2][32]
    __shared__ float partial[kGroups][2][WARPS][kFewFeatures * kPitch];
    __shared__ float slices[kGroups][WARPS * 4 / NT][8 * NT];   // sums of squares: slices of the producer's partials x rows
    const int groups = blockDim.x / kSpan, group = threadIdx.x / kSpan, thread = threadIdx.x % kSpan;
    const int warp = thread >> 5, lane = thread & 31, g = lane >> 2, t = lane & 3;
    const int first_tile = blockIdx.x * groups + group, tile_step = gridDim.x * groups;
    const int per_tile = (p.in + kSpan - 1) / kSpan, column0 = warp * 32 + 8 * t;
    const uint4 zeros = make_uint4(0u, 0u, 0u, 0u);

    const uint4* mine = ring + (threadIdx.x >> 5) * (kFewDepth * 64) + lane;
    const uint32_t ring_at = smem_u32(mine);
    // the next chunk of this warp, zeros where there is none
    int load_feature = first_tile * kFewFeatures + g, load_column = column0, load_slot = 0;
    const auto* load_from = static_cast<const __nv_bfloat16*>(p.weight) + static_cast<int64_t>(load_feature) * p.in + column0;
    const int64_t upper_rows = static_cast<int64_t>(8) * p.in, next_tile = static_cast<int64_t>(tile_step * kFewFeatures) * p.in - (per_tile - 1) * kSpan;
    auto load = [&] {
        const bool live = load_column < p.in && load_feature < p.out, upper = load_column < p.in && load_feature + 8 < p.out;
        const uint32_t to = ring_at + load_slot * 1024;
        copy_async_16(to, live ? load_from : p.weight, live);
        copy_async_16(to + 512, upper ? load_from + upper_rows : p.weight, upper);
        asm volatile("cp.async.commit_group;" ::: "memory");
        load_slot = load_slot + 1 == kFewDepth ? 0 : load_slot + 1;
        load_column += kSpan;
        if (load_column - column0 < per_tile * kSpan) {
            load_from += kSpan;
        } else {
            load_column = column0;
            load_feature += tile_step * kFewFeatures;
            load_from += next_tile;
        }
    };
#pragma unroll
    for (int i = 0; i < kFewDepth; ++i) load();

    // Weights are constants; the activations (and residual, cache, q) come from the preceding kernels.
    grid_dependency_wait();
    uint4 hi[kFewKeep][NT], lo[kFewKeep][NT];
    auto load_x = [&](int step0) {   // this warp's activations of chunks step0 .. step0 + kFewKeep - 1
#pragma unroll
        for (int u = 0; u < kFewKeep; ++u) {
            const int column = (step0 + u) * kSpan + column0;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const bool live = n * 8 + g < p.rows && column < p.in;
                const int64_t at = static_cast<int64_t>(n * 8 + g) * p.in + column;
                hi[u][n] = live ? *reinterpret_cast<const uint4*>(p.x_hi + at) : zeros;
                lo[u][n] = live && p.x_lo ? *reinterpret_cast<const uint4*>(p.x_lo + at) : zeros;
            }
        }
    };
    load_x(0);
    constexpr int kSlices = WARPS * 4 / NT;
    if (p.sumsq_in) {   // read again behind the first tile's barrier
        const int r = thread & (8 * NT - 1), slice = thread / (8 * NT);
        float sum = 0.0f;
        if (r < p.rows)
#pragma unroll 4
            for (int i = slice; i < p.parts_in; i += kSlices) sum += __ldg(p.sumsq_in + static_cast<int64_t>(i) * p.rows + r);
        slices[group][slice][r] = sum;
    }
    grid_launch_dependents();

    // this thread's share of a tile's epilogue
    const int my_row = thread >> 3, my_pair = (thread & 7) * 2;
    const bool finishes = thread < 64 * NT;
    float row_scale = 1.0f;
    bool scaled = p.sumsq_in == nullptr;
    Candidate running{-INFINITY, INT32_MAX};
    float carried[2] = {0.0f, 0.0f};
    float acc[NT][4], rest[NT][4];   // sums of the hi and of the lo plane: two chains of products
    int parity = 0, slot = 0;
    auto finish = [&](int tile) {
        float* mine = partial[group][parity][warp];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            mine[g * kPitch + n * 8 + 2 * t] = acc[n][0] + rest[n][0];
            mine[g * kPitch + n * 8 + 2 * t + 1] = acc[n][1] + rest[n][1];
            mine[(g + 8) * kPitch + n * 8 + 2 * t] = acc[n][2] + rest[n][2];
            mine[(g + 8) * kPitch + n * 8 + 2 * t + 1] = acc[n][3] + rest[n][3];
        }
        asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kSpan) : "memory");
        if (finishes) {   // whole warps
            if (!scaled) {
                float sum = 0.0f;
                for (int slice = 0; slice < kSlices; ++slice) sum += slices[group][slice][my_row];
                row_scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, static_cast<float>(p.in)), static_cast<float>(p.eps))));
                scaled = true;
            }
            float a = 0.0f, b = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                a += partial[group][parity][w][my_pair * kPitch + my_row];
                b += partial[group][parity][w][(my_pair + 1) * kPitch + my_row];
            }
            a *= row_scale;
            b *= row_scale;
            const int row = my_row, feature0 = tile * kFewFeatures + my_pair;
            const bool live = row < p.rows && feature0 < p.out, second = feature0 + 1 < p.out;
            if constexpr (EPI == B200_EPI_RESIDUAL) {
                if (live) {
                    const int64_t at = static_cast<int64_t>(row) * p.out + feature0;
                    a = __fadd_rn(carried[0], a);
                    b = second ? __fadd_rn(carried[1], b) : 0.0f;
                    p.y[at] = a;
                    if (second) p.y[at + 1] = b;
                    store_copies(p, at, a, b, second);
                }
                // a, b are the new residual-stream values: shadow for the consumer, row sums of squares for its norm
                float square = live ? a * a + b * b : 0.0f;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) square += __shfl_xor_sync(0xffffffffu, square, o);
                if (p.sumsq_out && my_pair == 0 && row < p.rows) p.sumsq_out[static_cast<int64_t>(tile) * p.rows + row] = square;
                if (p.out_hi && live) {   // out is even here
                    float wa = 1.0f, wb = 1.0f;
                    if (p.out_norm_weight) {
                        if (p.out_norm_dtype == B200_BF16) {
                            const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(p.out_norm_weight) + feature0;
                            wa = __bfloat162float(w[0]);
                            wb = __bfloat162float(w[1]);
                        } else {
                            const float* w = static_cast<const float*>(p.out_norm_weight) + feature0;
                            wa = w[0];
                            wb = w[1];
                        }
                    }
                    const float va = out_norm_value(p, a, wa, p.out_norm_bias ? p.out_norm_bias[feature0] : 0.0f);
                    const float vb = out_norm_value(p, b, wb, p.out_norm_bias ? p.out_norm_bias[feature0 + 1] : 0.0f);
                    uint32_t h, l;
                    pack_planes(va, vb, h, l);
                    const int64_t at = static_cast<int64_t>(row) * p.out + feature0;
                    *reinterpret_cast<uint32_t*>(p.out_hi + at) = h;
                    *reinterpret_cast<uint32_t*>(p.out_lo + at) = l;
                }
            } else if constexpr (EPI == B200_EPI_ARGMAX) {
                if (live) {
                    const Candidate best = pair_candidate(feature0, a, b, p.out);
                    if (preferred(best, running)) running = best;
                }
            } else if (live) {
                linear_epilogue<EPI>(p, row, feature0, a, b);
                if constexpr (EPI == B200_EPI_SWIGLU) {
                    if (p.out_hi) {
                        const __nv_bfloat16 h = __float2bfloat16_rn(a);
                        const int64_t at = row * p.out_stride + (feature0 >> 1);
                        p.out_hi[at] = h;
                        p.out_lo[at] = __float2bfloat16_rn(a - __bfloat162float(h));
                    }
                }
            }
        }
        parity ^= 1;   // (a warp reaches this buffer again only past the next tile's barrier, which the readers pass afterwards)
    };
    for (int tile = first_tile; tile < fp.tiles; tile += tile_step) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = rest[n][i] = 0.0f;
        if constexpr (EPI == B200_EPI_RESIDUAL) {   // the values that the epilogue adds, requested under the products
            const int feature0 = tile * kFewFeatures + my_pair;
            if (finishes && my_row < p.rows && feature0 < p.out) {
                const float* from = p.residual + static_cast<int64_t>(my_row) * p.out + feature0;
                carried[0] = from[0];
                carried[1] = feature0 + 1 < p.out ? from[1] : 0.0f;
            }
        }
        for (int step0 = 0; step0 < per_tile; step0 += kFewKeep) {
            if (per_tile > kFewKeep && (step0 > 0 || tile != first_tile)) load_x(step0);
#pragma unroll
            for (int u = 0; u < kFewKeep; ++u) {
                if (step0 + u >= per_tile) break;
                asm volatile("cp.async.wait_group %0;" ::"n"(kFewDepth - 1) : "memory");
                const uint4 w0 = mine[slot * 64], w1 = mine[slot * 64 + 32];
                const uint32_t first[4] = {w0.x, w1.x, w0.y, w1.y}, second[4] = {w0.z, w1.z, w0.w, w1.w};
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    mma_16816(acc[n], first, hi[u][n].x, hi[u][n].y);
                    mma_16816(rest[n], first, lo[u][n].x, lo[u][n].y);
                    mma_16816(acc[n], second, hi[u][n].z, hi[u][n].w);
                    mma_16816(rest[n], second, lo[u][n].z, lo[u][n].w);
                }
                slot = slot + 1 == kFewDepth ? 0 : slot + 1;
                load();   // into the slot that was just read
            }
        }
        finish(tile);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if constexpr (EPI == B200_EPI_ARGMAX) {   // one candidate per row and group
        if (finishes) {
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const Candidate other{__shfl_xor_sync(0xffffffffu, running.value, o), __shfl_xor_sync(0xffffffffu, running.index, o)};
                if (preferred(other, running)) running = other;
            }
            if (my_pair == 0 && my_row < p.rows) {
                p.best_value[static_cast<int64_t>(first_tile) * p.rows + my_row] = running.value;
                p.best_index[static_cast<int64_t>(first_tile) * p.rows + my_row] = running.index;
            }
        }
    }
}

// How a launch is cut.  Up to 1024 columns, eight warps hold their activations in registers as well as sixteen do, and two groups of eight
// cover each other's barriers and epilogues (768 -> 32000, one row: 14.3 us with one group of sixteen, 10.8 with two of eight); a second
// group only where there is more than a tile per SM.
struct FewGroups {
    int warps, per_cta, ctas;
    int total() const { return per_cta * ctas; }
};
FewGroups few_groups(int in, int out, int sms) {
    const int tiles = (out + kFewFeatures - 1) / kFewFeatures, warps = in <= kFewKeep * 8 * 32 ? 8 : kFewWarps;
    const int per_cta = warps == 8 && tiles > sms ? 2 : 1;
    return {warps, per_cta, std::min((tiles + per_cta - 1) / per_cta, sms)};
}

// Rows up to which inner sizes beyond 2048 take the streaming kernel too.  There a group fetches its activations again for every tile (4 bytes
// a value and row for every 32 bytes of weights).  1 | 4 rows, here against linear_decode_kernel: 8192 -> 2048 9.9 | 10.2 us against
// 12.1 | 12.5, 4096 -> 28672 39.0 | 40.5 against 41.9 | 42.1; with 8 rows the activations are a fifth of the traffic and the lead is gone.
constexpr int kFewWideRows = 4;

template <int NT, int WARPS> int launch_few(const FewParams& fp, int epilogue, const FewGroups& cut, cudaStream_t stream) {
    auto go = [&](auto kernel) {
        const int threads = cut.per_cta * WARPS * 32;
        B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewDepth * kFewWarps * 1024));
        return cuda_status(launch_dependent(kernel, dim3(cut.ctas), dim3(threads), threads * kFewDepth * 32, stream, fp), "linear_stream_kernel launch");
    };
    switch (epilogue) {
    case B200_EPI_STORE: return go(linear_stream_kernel<NT, WARPS, B200_EPI_STORE>);
    case B200_EPI_RESIDUAL: return go(linear_stream_kernel<NT, WARPS, B200_EPI_RESIDUAL>);
    case B200_EPI_SWIGLU: return go(linear_stream_kernel<NT, WARPS, B200_EPI_SWIGLU>);
    case B200_EPI_QKV: return go(linear_stream_kernel<NT, WARPS, B200_EPI_QKV>);
    case B200_EPI_ARGMAX: return go(linear_stream_kernel<NT, WARPS, B200_EPI_ARGMAX>);
    }
    return B200_UNSUPPORTED;
}

// ---- staged kernel: f32 activation rows -----------------------------------------------------------------------------------
// Persistent CTAs (one per SM) walk feature tiles of TF rows of W; a producer warp streams every tile through a ring of shared-memory
// slots with bulk TMA copies (one per weight row, mbarrier completion, no multicast) and runs ahead across tile boundaries.  The
// activation rows are staged once per CTA: RMSNorm (src/kernels/cpu/normalization.cpp:39-51 of the reference), then split into bf16
// hi + lo.  Eight consumer warps split K, fragments via ldmatrix (padded rows: no bank conflicts), and add their partial sums through
// shared memory before the shared epilogue.  Rows beyond 16 are covered by blockIdx.y (weights then come from L2).
// Shapes it does not take (f32 weights, in > 2048 or in % 8 != 0) stay on the CUDA-core kernel.
// Shared memory map (offsets from a 128-byte aligned base):
//   [0, slots * slot_bytes)         weight tiles, [TF rows][in_padded + 8] bf16 each (row stride = 16 mod 128 bytes)
//   then x_hi, x_lo                 [16][in_padded + 8] bf16 each
//   then partial sums               [8 warps][16 rows][TF] f32
//   then mbarriers                  full[slots], empty[slots]
template <int TF, int EPI>
__global__ void __launch_bounds__(kThreads, 2) linear_staged_kernel(const StreamParams sp) {
    constexpr int NT = TF / 8;  // n-tiles of 8 features
    const LinearParams& p = sp.base;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    const int x_stride = sp.in_padded + 8;  // bf16 elements per staged row (activations and weights)
    const int slot_bytes = TF * x_stride * 2;
    uint8_t* slot_base = smem;
    __nv_bfloat16* x_hi = reinterpret_cast<__nv_bfloat16*>(smem + sp.slots * slot_bytes);
    __nv_bfloat16* x_lo = x_hi + kRows * x_stride;
    float* partial = reinterpret_cast<float*>(x_lo + kRows * x_stride);
    uint64_t* full = reinterpret_cast<uint64_t*>(partial + kConsumers * kRows * TF);
    uint64_t* empty = full + sp.slots;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = blockIdx.y * kRows;
    const int my_tiles = (sp.tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);

    // A bounded wait may run out in one consumer warp and not in another.  The warps therefore never leave on their own:
    // the one that gave up raises this flag, still arrives at the next barrier of the consumers, and all of them test the
    // flag behind that barrier and leave together.
    __shared__ int consumers_gave_up;
    if (threadIdx.x == 0) {
        for (int s = 0; s < sp.slots; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kConsumers);
        }
        consumers_gave_up = 0;
        mbar_fence_init();
    }
    // Columns in .. in_padded+8 of the weight slots are never written by the copies; the last k-step may read up to
    // 8 of them, so they are cleared once (stale bit patterns could be NaN, and 0 * NaN is NaN).
    if (p.in & 15) {
        for (int i = threadIdx.x; i < sp.slots * TF; i += kThreads) {
            __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(slot_base) + static_cast<size_t>(i) * x_stride;
            for (int k = p.in; k < x_stride; ++k) row[k] = __float2bfloat16_rn(0.0f);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy stores before async-proxy copies
    }
    __syncthreads();

    if (warp == kConsumers) {
        // ---- producer: lane i requests rows i, i+32, ... of every tile; lane 0 owns the barriers ----
        bool alive = true;
        for (int t = 0; t < my_tiles && alive; ++t) {
            const int tile = blockIdx.x + t * gridDim.x;
            const int s = t % sp.slots;
            const uint32_t phase = (t / sp.slots) & 1;
            int rows = p.out - tile * TF;
            if (rows > TF) rows = TF;
            if (lane == 0) {
                if (!mbar_wait(&empty[s], phase ^ 1)) {
                    atomicExch(sp.status, B200_DEVICE_TIMEOUT);
                    alive = false;
                } else {
                    mbar_expect_tx(&full[s], static_cast<uint32_t>(rows * p.in * 2));
                }
            }
            alive = __shfl_sync(0xffffffffu, alive, 0);
            if (!alive) break;
            const __nv_bfloat16* source = static_cast<const __nv_bfloat16*>(p.weight) + static_cast<int64_t>(tile) * TF * p.in;
            uint8_t* dst = slot_base + s * slot_bytes;
            for (int r = lane; r < rows; r += 32)
                bulk_load(dst + r * x_stride * 2, source + static_cast<int64_t>(r) * p.in, static_cast<uint32_t>(p.in * 2), &full[s]);
        }
        return;
    }

    // Weights are constants; the activations (and residual, cache, q) come from the preceding kernels.
    grid_dependency_wait();
    // ---- consumers: stage the activations (the weight stream is already in flight) ----
    // Warp w owns rows w and w+8.  Both rows are read with independent 16-byte loads into registers (one L2 round
    // trip), reduced to their RMS (f32 squares per lane, f64 across lanes and for the square root), normalised,
    // split into bf16 hi + lo and written to shared memory.  Rows longer than 1024 are handled one after the other.
    {
        const int vectors = p.in >> 2;             // float4 per row (in % 8 == 0)
        const int per_lane = (vectors + 31) >> 5;  // float4 per lane and row, at most 16
        auto stage_rows = [&](auto count_tag, int first_row) {
            constexpr int ROWS = decltype(count_tag)::value;  // rows handled together by this warp
            constexpr int MAXV = ROWS == 2 ? 8 : 16;
            float4 v[ROWS][MAXV];
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const int r = first_row + q * kConsumers;
                const bool valid = row0 + r < p.rows;
                const float4* source = reinterpret_cast<const float4*>(p.x + static_cast<int64_t>(valid ? row0 + r : 0) * p.in);
#pragma unroll
                for (int u = 0; u < MAXV; ++u) {
                    const int at = u * 32 + lane;
                    v[q][u] = (u < per_lane && valid && at < vectors) ? __ldg(source + at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            }
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const int r = first_row + q * kConsumers;
                float scale = 1.0f;
                if (p.norm_weight) {
                    float squares = 0.0f;
#pragma unroll
                    for (int u = 0; u < MAXV; ++u)
                        if (u < per_lane) squares += v[q][u].x * v[q][u].x + v[q][u].y * v[q][u].y + v[q][u].z * v[q][u].z + v[q][u].w * v[q][u].w;
                    const float total = warp_sum(squares);
                    scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(p.in)), static_cast<float>(p.eps))));
                }
#pragma unroll
                for (int u = 0; u < MAXV; ++u) {
                    const int k = (u * 32 + lane) * 4;
                    if (u >= per_lane || k >= sp.in_padded) continue;
                    float e[4] = {v[q][u].x, v[q][u].y, v[q][u].z, v[q][u].w};
                    if (p.norm_weight && k < p.in) {
                        float w[4];
                        if (p.norm_dtype == B200_BF16) {
                            const uint2 packed = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p.norm_weight) + k));
                            w[0] = bf16_lo(packed.x); w[1] = bf16_hi(packed.x); w[2] = bf16_lo(packed.y); w[3] = bf16_hi(packed.y);
                        } else {
                            const float4 f = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p.norm_weight) + k));
                            w[0] = f.x; w[1] = f.y; w[2] = f.z; w[3] = f.w;
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) e[i] = __fmul_rn(__fmul_rn(e[i], scale), w[i]);
                    }
                    const __nv_bfloat162 h0 = __floats2bfloat162_rn(e[0], e[1]), h1 = __floats2bfloat162_rn(e[2], e[3]);
                    const __nv_bfloat162 l0 = __floats2bfloat162_rn(e[0] - __low2float(h0), e[1] - __high2float(h0));
                    const __nv_bfloat162 l1 = __floats2bfloat162_rn(e[2] - __low2float(h1), e[3] - __high2float(h1));
                    uint2 hi, lo;
                    hi.x = *reinterpret_cast<const uint32_t*>(&h0); hi.y = *reinterpret_cast<const uint32_t*>(&h1);
                    lo.x = *reinterpret_cast<const uint32_t*>(&l0); lo.y = *reinterpret_cast<const uint32_t*>(&l1);
                    *reinterpret_cast<uint2*>(x_hi + r * x_stride + k) = hi;
                    *reinterpret_cast<uint2*>(x_lo + r * x_stride + k) = lo;
                }
            }
        };
        // in_padded beyond in: the tail columns of a row are written as zeros by the lanes that own them
        if (per_lane <= 8) {
            stage_rows(std::integral_constant<int, 2>{}, warp);
        } else {
            stage_rows(std::integral_constant<int, 1>{}, warp);
            stage_rows(std::integral_constant<int, 1>{}, warp + kConsumers);
        }
        consumer_barrier();
        grid_launch_dependents();
    }

    const int mi = lane >> 3, ri = lane & 7;
    // ldmatrix row address of the activation fragment: matrices (rows 0-7, k 0-7), (rows 8-15, k 0-7), (rows 0-7, k 8-15), (rows 8-15, k 8-15)
    const uint32_t a_lane = static_cast<uint32_t>((((mi & 1) * 8 + ri) * x_stride + (mi >> 1) * 8) * 2);
    const uint32_t a_hi = smem_u32(x_hi) + a_lane, a_lo = smem_u32(x_lo) + a_lane;
    const int ksteps = (p.in + 15) >> 4;

    bool alive = true;
    for (int t = 0; t < my_tiles && alive; ++t) {
        const int tile = blockIdx.x + t * gridDim.x;
        float acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
        {
            const int s = t % sp.slots;
            const uint32_t phase = (t / sp.slots) & 1;
            if (!mbar_wait(&full[s], phase)) {
                if (lane == 0) atomicExch(sp.status, B200_DEVICE_TIMEOUT);
                *static_cast<volatile int*>(&consumers_gave_up) = 1;
                alive = false;
            }
            const uint32_t slot = smem_u32(slot_base + s * slot_bytes);
            // ldmatrix row addresses of the weight fragments: x4 = (features n*8.., k 0-7), (same, k 8-15),
            // (features (n+1)*8.., k 0-7), (same, k 8-15); x2 = the first two
            const uint32_t b_lane = slot + static_cast<uint32_t>((((NT == 1 ? 0 : (mi >> 1)) * 8 + ri) * x_stride + (mi & 1) * 8) * 2);
            for (int j = warp; alive && j < ksteps; j += kConsumers) {
                uint32_t ah[4], al[4];
                const uint32_t column_bytes = static_cast<uint32_t>(j * 32);
                ldmatrix_x4(ah, a_hi + column_bytes);
                ldmatrix_x4(al, a_lo + column_bytes);
                if constexpr (NT == 1) {
                    uint32_t b[2];
                    ldmatrix_x2(b, b_lane + column_bytes);
                    mma_16816(acc[0], ah, b[0], b[1]);
                    mma_16816(acc[0], al, b[0], b[1]);
                } else {
#pragma unroll
                    for (int n = 0; n < NT; n += 2) {
                        uint32_t b[4];
                        ldmatrix_x4(b, b_lane + static_cast<uint32_t>(n * 8 * x_stride * 2) + column_bytes);
                        mma_16816(acc[n], ah, b[0], b[1]);
                        mma_16816(acc[n], al, b[0], b[1]);
                        mma_16816(acc[n + 1], ah, b[2], b[3]);
                        mma_16816(acc[n + 1], al, b[2], b[3]);
                    }
                }
            }
            __syncwarp();
            if (alive && lane == 0) mbar_arrive(&empty[s]);
        }
        // ---- add the eight K-slices and finish the tile ----
        {
            const int g = lane >> 2, tq = lane & 3;
            float* mine = partial + warp * kRows * TF;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                *reinterpret_cast<float2*>(mine + g * TF + n * 8 + 2 * tq) = make_float2(acc[n][0], acc[n][1]);
                *reinterpret_cast<float2*>(mine + (g + 8) * TF + n * 8 + 2 * tq) = make_float2(acc[n][2], acc[n][3]);
            }
        }
        consumer_barrier();
        if (*static_cast<volatile int*>(&consumers_gave_up)) break;   // a weight tile never arrived: every consumer warp leaves here
        // items of one row are TF/2 consecutive threads of a warp: thread i finishes the feature pair (r, f)
#pragma unroll
        for (int base = 0; base < kRows * (TF / 2); base += kConsumers * 32) {
            const int i = base + threadIdx.x;
            const int r = i / (TF / 2), f = (i - r * (TF / 2)) * 2;
            const bool in_tile = i < kRows * (TF / 2);
            float a = 0.0f, b = 0.0f;
            if (in_tile) {
#pragma unroll
                for (int w = 0; w < kConsumers; ++w) {
                    const float2 v = *reinterpret_cast<const float2*>(partial + (w * kRows + r) * TF + f);
                    a += v.x;
                    b += v.y;
                }
            }
            const int row = row0 + r, feature0 = tile * TF + f;
            const bool live = in_tile && row < p.rows && feature0 < p.out;
            if (live) linear_epilogue<EPI>(p, row, feature0, a, b);
        }
        consumer_barrier();
    }
}

template <int TF, int EPI> int launch_tile(const StreamParams& sp, size_t smem, int ctas, int row_tiles, cudaStream_t stream) {
    auto kernel = linear_staged_kernel<TF, EPI>;
    B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    return cuda_status(launch_dependent(kernel, dim3(ctas, row_tiles), dim3(kThreads), smem, stream, sp), "linear_staged_kernel launch");
}

template <int EPI> int pick_tile(const StreamParams& sp, size_t smem, int ctas, int row_tiles, cudaStream_t stream) {
    switch (sp.tile_features) {
    case 8: return launch_tile<8, EPI>(sp, smem, ctas, row_tiles, stream);
    case 16: return launch_tile<16, EPI>(sp, smem, ctas, row_tiles, stream);
    case 32: return launch_tile<32, EPI>(sp, smem, ctas, row_tiles, stream);
    default: return launch_tile<64, EPI>(sp, smem, ctas, row_tiles, stream);
    }
}

// Tile size, ring depth and shared-memory size for a weight matrix [out, in]; false when nothing fits.
bool choose_tiling(int in, int out, int sms, StreamParams& sp, size_t& smem) {
    sp.in_padded = (in + 63) & ~63;
    const size_t row_bytes = static_cast<size_t>(sp.in_padded + 8) * 2;
    // Smallest tile with which one round of CTAs covers the matrix (every further tile of a CTA costs a reduction
    // round).  Half of the shared memory is preferred (two CTAs per SM: this kernel's tail next to the early-started
    // successor), the whole when a ring of two tiles does not fit in half, a smaller tile when it does not fit at all.
    const size_t half = 110 * 1024, whole = 220 * 1024;
    int tf = 8;
    while (tf < 64 && (out + tf - 1) / tf > sms) tf <<= 1;
    size_t fixed = 0;
    int slots = 0;
    for (;; tf >>= 1) {
        fixed = 2 * kRows * row_bytes + static_cast<size_t>(kConsumers) * kRows * tf * 4 + 128 + 1536;
        slots = fixed < half ? static_cast<int>((half - fixed) / (tf * row_bytes)) : 0;
        if (slots < 2) slots = fixed < whole ? static_cast<int>((whole - fixed) / (tf * row_bytes)) : 0;
        if (slots >= 2 || tf == 8) break;
    }
    if (slots < 2) return false;
    if (slots > 8) slots = 8;
    sp.tile_features = tf;
    sp.slots = slots;
    sp.tiles = (out + tf - 1) / tf;
    smem = fixed + static_cast<size_t>(slots) * tf * row_bytes;
    return true;
}

}  // namespace

bool linear_stream_takes(int rows, int in) { return rows < kGemmRows && (in <= kMaxIn || rows <= kFewWideRows); }

int linear_stream_parts(int rows, int in, int out) {
    if ((in & 7) || in <= 0 || out <= 0) return 0;
    return linear_stream_takes(rows, in) ? (out + kFewFeatures - 1) / kFewFeatures : linear_gemm_parts(rows, in, out, true);
}

int linear_argmax_parts(int rows, int in, int out) {
    if ((in & 7) || in <= 0 || out <= 0) return 0;
    if (!linear_stream_takes(rows, in)) return linear_gemm_parts(rows, in, out, false);
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess) { cudaGetLastError(); device = -1; }   // no device: the figures of a 148-SM part
    return few_groups(in, out, sm_count(device)).total();   // one candidate slice per group
}

// ---- thin outputs (adapter down-projections: a few dozen output features) for passes the dense kernel would serve ----
// A 128-wide tensor-core tile would be one mostly empty tile with a K split of four CTAs at the kernel's latency floor.
// Here a CTA takes one activation row and eight output features: 256 threads stride over K with 16-byte loads (eight
// activation values from the hi (+ lo) planes, eight weights per feature), f32 FMAs, then a block reduction.  The
// operands are a few hundred KB that every CTA finds in L2.
constexpr int kThinFeatures = 8, kThinThreads = 256, kThinMaxOut = 64;

__global__ void __launch_bounds__(kThinThreads) linear_thin_kernel(const LinearParams p) {
    __shared__ float partial[kThinThreads / 32][kThinFeatures];
    grid_dependency_wait();
    grid_launch_dependents();
    const int row = blockIdx.x, feature0 = blockIdx.y * kThinFeatures;
    const auto* weight = static_cast<const __nv_bfloat16*>(p.weight);
    float squares = 0.0f;   // the partial sums of the row's norm, fetched by the first warp's lanes side by side
    if (p.sumsq_in && threadIdx.x < 32)
        for (int i = threadIdx.x; i < p.parts_in; i += 32) squares += __ldg(p.sumsq_in + static_cast<int64_t>(i) * p.rows + row);
    float acc[kThinFeatures];
#pragma unroll
    for (int f = 0; f < kThinFeatures; ++f) acc[f] = 0.0f;
    for (int k = threadIdx.x * 8; k < p.in; k += kThinThreads * 8) {
        const uint4 hi = *reinterpret_cast<const uint4*>(p.x_hi + static_cast<int64_t>(row) * p.in + k);
        uint4 lo = make_uint4(0u, 0u, 0u, 0u);
        if (p.x_lo) lo = *reinterpret_cast<const uint4*>(p.x_lo + static_cast<int64_t>(row) * p.in + k);
        const uint32_t h[4] = {hi.x, hi.y, hi.z, hi.w}, l[4] = {lo.x, lo.y, lo.z, lo.w};
        float x[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[2 * i] = bf16_lo(h[i]) + bf16_lo(l[i]);
            x[2 * i + 1] = bf16_hi(h[i]) + bf16_hi(l[i]);
        }
#pragma unroll
        for (int f = 0; f < kThinFeatures; ++f) {
            // (features past the end repeat the last one: a branch here would make the eight loads a chain)
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(weight + static_cast<int64_t>(min(feature0 + f, p.out - 1)) * p.in + k));
            const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[f] = fmaf(x[2 * i], bf16_lo(v[i]), fmaf(x[2 * i + 1], bf16_hi(v[i]), acc[f]));
        }
    }
#pragma unroll
    for (int f = 0; f < kThinFeatures; ++f) acc[f] = warp_sum(acc[f]);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int f = 0; f < kThinFeatures; ++f) partial[threadIdx.x >> 5][f] = acc[f];
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    squares = warp_sum(squares);
    if (threadIdx.x < kThinFeatures && feature0 + threadIdx.x < p.out) {
        float total = 0.0f;
#pragma unroll
        for (int w = 0; w < kThinThreads / 32; ++w) total += partial[w][threadIdx.x];
        float scale = 1.0f;
        if (p.sumsq_in)
            scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(squares, static_cast<float>(p.in)), static_cast<float>(p.eps))));
        p.y[static_cast<int64_t>(row) * p.out + feature0 + threadIdx.x] = total * scale;
    }
}

bool linear_thin_takes(int rows, int in, int64_t out) { return (rows >= kGemmRows || in > kMaxIn) && out <= kThinMaxOut && rows <= 512; }

int launch_linear_thin(const LinearParams& p, cudaStream_t stream) {
    const dim3 grid(static_cast<unsigned>(p.rows), static_cast<unsigned>((p.out + kThinFeatures - 1) / kThinFeatures));
    return cuda_status(launch_dependent(linear_thin_kernel, grid, dim3(kThinThreads), 0, stream, p), "linear_thin_kernel launch");
}

int launch_linear_stream(const LinearParams& p, int epilogue, cudaStream_t stream) {
    if (p.x_hi && epilogue == B200_EPI_STORE && linear_thin_takes(p.rows, p.in, p.out) && p.weight_dtype == B200_BF16 && (p.in & 7) == 0
        && ((reinterpret_cast<uintptr_t>(p.weight) | reinterpret_cast<uintptr_t>(p.x_hi) | reinterpret_cast<uintptr_t>(p.x_lo)) & 15) == 0)
        return launch_linear_thin(p, stream);
    if (p.x_hi) {
        if (!linear_stream_takes(p.rows, p.in)) return launch_linear_gemm(p, epilogue, stream);
        if (p.weight_dtype != B200_BF16 || (p.in & 7) || (p.out_hi && (p.out & 1))
            || ((reinterpret_cast<uintptr_t>(p.weight) | reinterpret_cast<uintptr_t>(p.x_hi) | reinterpret_cast<uintptr_t>(p.x_lo)) & 15))
            return B200_UNSUPPORTED;
        if (!p.x_lo && p.in <= kMaxIn) return B200_UNSUPPORTED;   // one plane: a form of the tensor-core kernels only
        int device = 0;
        B200_CUDA(cudaGetDevice(&device));
        const FewParams fp{p, (p.out + kFewFeatures - 1) / kFewFeatures};
        const FewGroups cut = few_groups(p.in, p.out, sm_count(device));
        if (p.rows <= 8) return cut.warps == 8 ? launch_few<1, 8>(fp, epilogue, cut, stream) : launch_few<1, 16>(fp, epilogue, cut, stream);
        return cut.warps == 8 ? launch_few<2, 8>(fp, epilogue, cut, stream) : launch_few<2, 16>(fp, epilogue, cut, stream);
    }
    if (p.weight_dtype != B200_BF16 || p.in > kMaxIn || (p.in & 7) || (reinterpret_cast<uintptr_t>(p.weight) & 15)
        || (reinterpret_cast<uintptr_t>(p.x) & 15))
        return B200_UNSUPPORTED;
    int device = 0;
    B200_CUDA(cudaGetDevice(&device));
    const int sms = sm_count(device);

    StreamParams sp{};
    sp.base = p;
    sp.status = device_status_word(device);
    if (!sp.status) { set_error("the device status word could not be allocated"); return B200_NO_DEVICE; }
    size_t smem = 0;
    if (!choose_tiling(p.in, p.out, sms, sp, smem)) return B200_UNSUPPORTED;

    const int row_tiles = (p.rows + kRows - 1) / kRows;
    const int ctas = sp.tiles < sms ? sp.tiles : sms;
    switch (epilogue) {
    case B200_EPI_STORE: return pick_tile<B200_EPI_STORE>(sp, smem, ctas, row_tiles, stream);
    case B200_EPI_RESIDUAL: return pick_tile<B200_EPI_RESIDUAL>(sp, smem, ctas, row_tiles, stream);
    case B200_EPI_SWIGLU: return pick_tile<B200_EPI_SWIGLU>(sp, smem, ctas, row_tiles, stream);
    case B200_EPI_QKV: return pick_tile<B200_EPI_QKV>(sp, smem, ctas, row_tiles, stream);
    }
    return B200_UNSUPPORTED;
}

}  // namespace b200

