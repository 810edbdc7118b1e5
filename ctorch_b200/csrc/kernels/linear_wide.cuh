// Register epilogue of the kernels with 128 x 256 tiles: a thread finishes one token row, 32 features at a time.
#pragma once

#include "linear_rows.cuh"
#include "tcgen05.cuh"

namespace b200 {

constexpr int kWideN = 256, kWideThreads = 320;   // features of a tile; producer warp, issuing warp, two epilogue warps per lane quarter

// What a CTA has under way: K blocks requested and multiplied, and whether a bounded wait ran out.
struct WideFlight { int loads, products, gave_up; };
// After a wait that ran out, before the CTA leaves: copies and products that are under way get the same time again (one thread).
__device__ __forceinline__ void wide_drain(const WideFlight& flight, uint64_t* full, uint64_t* empty, int stages) {
    for (int j = max(0, flight.loads - stages); j < flight.loads; ++j) mbar_wait(&full[j % stages], (j / stages) & 1);
    for (int j = max(0, flight.products - stages); j < flight.products; ++j) mbar_wait(&empty[j % stages], (j / stages) & 1);
}

__device__ __forceinline__ void pack_eight(const float* v, uint4& hi, uint4& lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i] - __low2float(a), v[2 * i + 1] - __high2float(a));
        h[i] = *reinterpret_cast<const uint32_t*>(&a);
        l[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// 32 adjacent features from `feature` on of one token row; the accumulators are in tensor memory at `address`.  Features end on a multiple of 8
// (SwiGLU: 16, q|k|v: 32), so what is stored at a time is there or not as a whole.
template <int EPI>
__device__ __forceinline__ void finish_chunk(const LinearParams& p, int row, int feature, uint32_t address, float scale, const int2& place, float& squares) {
    const bool live = row < p.rows && feature < p.out;
    const int64_t at = static_cast<int64_t>(row) * p.out + feature;
    float4 carried[8];
    if constexpr (EPI == B200_EPI_RESIDUAL) {
#pragma unroll
        for (int i = 0; i < 8; ++i) carried[i] = live && feature + 4 * i < p.out ? *reinterpret_cast<const float4*>(p.residual + at + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    uint32_t r[32];
    tmem_load_32(address, r);
    if (!live) return;
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * scale;
    if constexpr (EPI == B200_EPI_STORE || EPI == B200_EPI_RESIDUAL) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (feature + 4 * i >= p.out) break;
            float4 t = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            if constexpr (EPI == B200_EPI_RESIDUAL) {
                t = make_float4(__fadd_rn(carried[i].x, t.x), __fadd_rn(carried[i].y, t.y), __fadd_rn(carried[i].z, t.z), __fadd_rn(carried[i].w, t.w));
                squares += t.x * t.x + t.y * t.y;
                squares += t.z * t.z + t.w * t.w;
                v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
            }
            *reinterpret_cast<float4*>(p.y + at + 4 * i) = t;
            store_copies(p, at + 4 * i, t);
        }
        if constexpr (EPI == B200_EPI_RESIDUAL) {
            if (p.out_hi) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    if (feature + i >= p.out) break;
                    float w[8] = {1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f}, b[8] = {};
                    if (p.out_norm_weight && p.out_norm_dtype == B200_BF16) {
                        const uint4 q = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.out_norm_weight) + feature + i));
                        const uint32_t pairs[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) { w[2 * k] = bf16_lo(pairs[k]); w[2 * k + 1] = bf16_hi(pairs[k]); }
                    } else if (p.out_norm_weight) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) w[k] = __ldg(static_cast<const float*>(p.out_norm_weight) + feature + i + k);
                    }
                    if (p.out_norm_bias) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) b[k] = __ldg(p.out_norm_bias + feature + i + k);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) w[k] = out_norm_value(p, v[i + k], w[k], b[k]);
                    uint4 hi, lo;
                    pack_eight(w, hi, lo);
                    *reinterpret_cast<uint4*>(p.out_hi + at + i) = hi;
                    *reinterpret_cast<uint4*>(p.out_lo + at + i) = lo;
                }
            }
        }
    } else if constexpr (EPI == B200_EPI_SWIGLU) {
        // (gate_j, up_j) of the interleaved weight rows; the shadow input makes this a bf16 model (see silu_fast)
        const int j = feature >> 1;
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = gated_unit(p, v[2 * i], v[2 * i + 1], true);
        if (p.y) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                if (feature + 2 * i < p.out) *reinterpret_cast<float4*>(p.y + static_cast<int64_t>(row) * (p.out >> 1) + j + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        if (p.out_hi) {
            const int64_t to = row * p.out_stride + j;
#pragma unroll
            for (int i = 0; i < 16; i += 8) {
                if (feature + 2 * i >= p.out) break;
                uint4 hi, lo;
                pack_eight(v + i, hi, lo);
                *reinterpret_cast<uint4*>(p.out_hi + to + i) = hi;
                *reinterpret_cast<uint4*>(p.out_lo + to + i) = lo;
            }
        }
    } else if constexpr (EPI == B200_EPI_GELU) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = gelu_exact(v[i]);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            if (feature + i >= p.out) break;
            uint4 hi, lo;
            pack_eight(v + i, hi, lo);
            *reinterpret_cast<uint4*>(p.out_hi + at + i) = hi;
            *reinterpret_cast<uint4*>(p.out_lo + at + i) = lo;
        }
    } else {
        // q | k | v (src/nn/decoder.cpp:77-88; src/ops/contraction.cpp:44-49; src/nn/kv_cache.cpp:24-28): the 32 features lie in one head
        const int D = p.heads * p.head_dim, KV = p.kv_heads * p.head_dim;
        int region = 0, local = feature;
        if (local >= D) { region = 1; local -= D; }
        if (region == 1 && local >= KV) { region = 2; local -= KV; }
        const int head = local / p.head_dim, inside = local - head * p.head_dim;
        if (region != 2 && static_cast<unsigned>(place.x) < static_cast<unsigned>(p.context)) {
            const int64_t angle = static_cast<int64_t>(place.x) * (p.head_dim >> 1) + (inside >> 1);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 c4 = __ldg(reinterpret_cast<const float4*>(p.cosine + angle + i)), s4 = __ldg(reinterpret_cast<const float4*>(p.sine + angle + i));
                const float c[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {   // adjacent-pair rotation, each product rounded before the add
                    const float even = v[2 * (i + k)], odd = v[2 * (i + k) + 1];
                    v[2 * (i + k)] = __fsub_rn(__fmul_rn(even, c[k]), __fmul_rn(odd, sn[k]));
                    v[2 * (i + k) + 1] = __fadd_rn(__fmul_rn(even, sn[k]), __fmul_rn(odd, c[k]));
                }
            }
        }
        if (region == 0 || p.kv.dtype != B200_BF16) {
            float* to = p.q_out + static_cast<int64_t>(row) * D + local;
            if (region != 0)
                to = static_cast<float*>(p.kv.pool[region - 1])
                    + ((static_cast<int64_t>(place.y) * p.kv.kv_heads + head) * p.kv.page_size + place.x % p.kv.page_size) * p.kv.head_dim + inside;
#pragma unroll
            for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(to + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        } else {
            auto* to = static_cast<__nv_bfloat16*>(p.kv.pool[region - 1])
                + ((static_cast<int64_t>(place.y) * p.kv.kv_heads + head) * p.kv.page_size + place.x % p.kv.page_size) * p.kv.head_dim + inside;
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
                uint32_t h[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const __nv_bfloat162 a = __floats2bfloat162_rn(v[i + 2 * k], v[i + 2 * k + 1]);
                    h[k] = *reinterpret_cast<const uint32_t*>(&a);
                }
                *reinterpret_cast<uint4*>(to + i) = make_uint4(h[0], h[1], h[2], h[3]);
            }
        }
    }
}

}  // namespace b200
