// Split-K merge of decode attention: combines the per-partition (max, sum, un-normalised output)
// partials of one query head and applies the inverse rotation of the output.  Used by the stand-alone
// merge kernel and by the last CTA of a KV head inside the tensor-core decode kernel, so both produce
// identical bits.  Follows tq_fused_attention_reduce (src/cache/cuda/kernels/tq_attention_kernel.cu:299-332),
// with the inverse block rotation (src/cache/wht_tensor.rs:27-65) applied once per output block.
#pragma once
#include <float.h>

#include "tqb_common.cuh"

namespace tqb {

struct MergeArgs {
    const float* partial_out;   // [hq, P, D]
    const float* partial_max;   // [hq, P]  natural-log units
    const float* partial_sum;   // [hq, P]
    const float* dev_signs;     // legacy entry point (else nullptr)
    void* out;
    float* lse_out;             // nullptr, or [hq, 2]: out stays un-normalised and (max, sum) go here
    int head_dim, nblk, num_partitions, rotate;
    int out_dtype;
    float sign_mag;
    // merge_group128 only: when num_copies > 0 the un-normalised f32 result and the (max, sum) pairs go to these
    // record buffers ([num_q_heads, 128] floats, then [num_q_heads, 2]) instead of out / lse_out
    int num_copies, num_q_heads;
    float* copy_rec[kMaxPeers];
    // merge_group128<GROUP = true> only: where an intermediate partial goes
    float* group_out;
    float* group_max;
    float* group_sum;
};

// Two-level merge of the tensor-core decode kernels: partitions are merged in groups of kMergeGroup by the CTA that
// finishes a group, the group results by the CTA that finishes the last group of a KV head.  With P > 16 partitions the
// serial tail is two merges of about kMergeGroup and P / kMergeGroup slots instead of one of P slots by one CTA.
constexpr int kMergeGroup = 8;
__host__ __device__ inline int merge_groups(int num_partitions) {
    // up to two chunks of eight a single merge is shorter than two levels with their extra ticket round
    return num_partitions <= 2 * kMergeGroup ? 0 : (num_partitions + kMergeGroup - 1) / kMergeGroup;
}

namespace merge_detail {
__device__ __forceinline__ float sum32(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float wht32(float v, int lane) {
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
        float other = __shfl_xor_sync(0xffffffffu, v, h);
        v = (lane & h) ? (other - v) : (v + other);
    }
    return v;
}
__device__ __forceinline__ void store_out(void* out, int dtype, size_t i, float v) {
    if (dtype == TQB_F32) reinterpret_cast<float*>(out)[i] = v;
    else if (dtype == TQB_F16) reinterpret_cast<__half*>(out)[i] = __float2half_rn(v);
    else reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(v);
}
}  // namespace merge_detail

// All threads of a CTA of `nwarps` warps call this for one query head; warp w handles output blocks
// w, w + nwarps, ...; lane = element of the block.  Partials are read past L1 (they may have been
// written by other CTAs of the same launch).
__device__ __forceinline__ void merge_head(const MergeArgs& a, int head, int lane, int warp, int nwarps) {
    using namespace merge_detail;
    const int D = a.head_dim, P = a.num_partitions;
    const float* pm = a.partial_max + (size_t)head * P;
    const float* ps = a.partial_sum + (size_t)head * P;
    // Lane p keeps (max, sum) of partition p; both loads are issued before either is used, and the partial
    // outputs below are fetched eight at a time, so the merge costs a few trips to L2, not one per partition.
    float pmv = -FLT_MAX, psv = 0.0f;
    if (lane < P) {
        pmv = __ldcg(pm + lane);
        psv = __ldcg(ps + lane);
    }
    float M = pmv;
    for (int p = lane + 32; p < P; p += 32) M = fmaxf(M, __ldcg(pm + p));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    const float wl = lane < P ? expf(pmv - M) : 0.0f;   // weight of partition `lane`
    float L = lane < P ? psv * wl : 0.0f;
    for (int p = lane + 32; p < P; p += 32) L += __ldcg(ps + p) * expf(__ldcg(pm + p) - M);
    L = sum32(L);
    const float inv_sqrt = 1.0f / sqrtf((float)kBlock);
    const uint32_t neg = 0xB1A6D4B2u;   // src/cache/precomputed/rotation.rs:16-20
    const float sg = a.dev_signs ? a.dev_signs[lane] : (((neg >> lane) & 1u) ? -a.sign_mag : a.sign_mag);
    const float inv_l = L > 0.0f ? 1.0f / L : 0.0f;
    for (int b = warp; b < a.nblk; b += nwarps) {
        const float* po = a.partial_out + (size_t)head * P * D + b * 32 + lane;
        float acc = 0.0f;   // sum over partitions in ascending order
        if (P <= 32) {
            for (int p0 = 0; p0 < P; p0 += 8) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = p0 + i < P ? __ldcg(po + (size_t)(p0 + i) * D) : 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (p0 + i < P) acc = fmaf(v[i], __shfl_sync(0xffffffffu, wl, p0 + i), acc);
            }
        } else {
            for (int p = 0; p < P; ++p) acc = fmaf(__ldcg(po + (size_t)p * D), expf(__ldcg(pm + p) - M), acc);
        }
        if (a.rotate) acc = wht32(acc * sg, lane) * inv_sqrt;
        if (a.lse_out == nullptr) acc *= inv_l;
        store_out(a.out, a.out_dtype, (size_t)head * D + b * 32 + lane, acc);
    }
    if (a.lse_out != nullptr && lane == 0 && warp == 0) {
        a.lse_out[head * 2] = M;
        a.lse_out[head * 2 + 1] = L;
    }
}

// The same merge for ALL g <= 8 query heads of one KV head by one CTA of 128 threads, head_dim 128: warp w owns heads w and
// w + 4, lane = element of each of the four blocks.  All loads of a warp - up to eight slots of both heads and their
// (max, sum) pairs - are in flight together, so a merge costs one trip to L2 and the arithmetic, and no warp waits for another.
// (A thread per element going through all heads needs either 64 loads and as much code, which runs once and is fetched cold,
// or a trip a head: 8 heads x 131,072 tokens in 74 partitions 70 or 75 us a launch.)
//
// Source: slots [first, first + count) of arrays laid out [head][head_stride][...] (a.partial_*).
// Destination, GROUP = true: one more partial - un-normalised sum, max and sum of slot `gslot` of the group arrays
// (a.group_*, [head][group_stride][...]), still in the rotated domain.  GROUP = false: the final result as merge_head
// writes it (or, with num_copies > 0, the record copies).  Sums run over the slots in ascending order.
// All 128 threads must call; there is no block-wide barrier inside.
template <bool GROUP>
__device__ __forceinline__ void merge_group128(const MergeArgs& a, int head0, int g, int tid, int first, int count, int head_stride,
                                               int gslot = 0, int group_stride = 0) {
    using namespace merge_detail;
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int D = 128;
    const float inv_sqrt = 1.0f / sqrtf((float)kBlock);
    const uint32_t neg = 0xB1A6D4B2u;   // src/cache/precomputed/rotation.rs:16-20
    const float sg = a.dev_signs ? a.dev_signs[lane] : (((neg >> lane) & 1u) ? -a.sign_mag : a.sign_mag);
    float v[2][8][4], pm[2], pl[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const bool on = warp + 4 * t < g;
        const size_t at = (size_t)(head0 + (on ? warp + 4 * t : 0)) * head_stride + first;
        const float* po = a.partial_out + at * D + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int b = 0; b < 4; ++b) v[t][i][b] = (on && i < count) ? __ldcg(po + (size_t)i * D + 32 * b) : 0.0f;
        pm[t] = (on && lane < count) ? __ldcg(a.partial_max + at + lane) : -FLT_MAX;
        pl[t] = (on && lane < count) ? __ldcg(a.partial_sum + at + lane) : 0.0f;
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int head = head0 + warp + 4 * t;
        if (warp + 4 * t >= g) break;
        const size_t at = (size_t)head * head_stride + first;
        float M = pm[t];
        for (int p = lane + 32; p < count; p += 32) M = fmaxf(M, __ldcg(a.partial_max + at + p));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        const float wl = lane < count ? expf(pm[t] - M) : 0.0f;
        float L = pl[t] * wl;
        for (int p = lane + 32; p < count; p += 32) L += __ldcg(a.partial_sum + at + p) * expf(__ldcg(a.partial_max + at + p) - M);
        L = sum32(L);
        float r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float w = __shfl_sync(0xffffffffu, wl, i);   // (0 past `count`)
#pragma unroll
            for (int b = 0; b < 4; ++b) r[b] = fmaf(v[t][i][b], w, r[b]);
        }
#pragma unroll 1
        for (int p0 = 8; p0 < count; p0 += 8) {
            const float* po = a.partial_out + (at + p0) * D + lane;
            float u[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int b = 0; b < 4; ++b) u[i][b] = p0 + i < count ? __ldcg(po + (size_t)i * D + 32 * b) : 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int p = p0 + i;
                float w = __shfl_sync(0xffffffffu, wl, p & 31);
                if (p >= 32) w = p < count ? expf(__ldcg(a.partial_max + at + p) - M) : 0.0f;
#pragma unroll
                for (int b = 0; b < 4; ++b) r[b] = fmaf(u[i][b], w, r[b]);
            }
        }
        if (GROUP) {
            const size_t gi = (size_t)head * group_stride + gslot;
#pragma unroll
            for (int b = 0; b < 4; ++b) a.group_out[gi * D + 32 * b + lane] = r[b];
            if (lane == 0) {
                a.group_max[gi] = M;
                a.group_sum[gi] = L;
            }
            continue;
        }
        const float norm = (a.num_copies == 0 && a.lse_out == nullptr) ? (L > 0.0f ? 1.0f / L : 0.0f) : 1.0f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (a.rotate) r[b] = wht32(r[b] * sg, lane) * inv_sqrt;
            r[b] *= norm;
        }
        if (a.num_copies > 0) {
            // (constant indices only: a run-time index would move the argument block to local memory)
#pragma unroll
            for (int c = 0; c < kMaxPeers; ++c)
                if (c < a.num_copies) {
#pragma unroll
                    for (int b = 0; b < 4; ++b) a.copy_rec[c][(size_t)head * D + 32 * b + lane] = r[b];
                    if (lane == 0) {
                        float* lse = a.copy_rec[c] + (size_t)a.num_q_heads * D;
                        lse[head * 2] = M;
                        lse[head * 2 + 1] = L;
                    }
                }
            continue;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) store_out(a.out, a.out_dtype, (size_t)head * D + 32 * b + lane, r[b]);
        if (a.lse_out != nullptr && lane == 0) {
            a.lse_out[head * 2] = M;
            a.lse_out[head * 2 + 1] = L;
        }
    }
}

}  // namespace tqb
