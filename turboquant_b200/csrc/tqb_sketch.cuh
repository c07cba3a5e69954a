// Sign sketch: the sequential row products, and the launchers of the kernels in tqb_sketch.cu.
#pragma once
#include "tqb_common.cuh"

namespace tqb {

// Sequential Rademacher row products of one vector held in shared memory.
// Lane handles rows lane, lane+32, ...; s_rb has row stride W+1 words.
template <int EPL>
__device__ __forceinline__ void rademacher_rows(const float* vec, const uint32_t* s_rb, int lane, float inv_sqrt_d,
                                                float (&proj)[EPL]) {
    constexpr int W = EPL;
    float s[EPL];
#pragma unroll
    for (int k = 0; k < EPL; ++k) s[k] = 0.0f;
#pragma unroll 1
    for (int cw = 0; cw < W; ++cw) {
        uint32_t rb[EPL];
#pragma unroll
        for (int k = 0; k < EPL; ++k) rb[k] = s_rb[(lane + 32 * k) * (W + 1) + cw];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            const uint32_t val = __float_as_uint(vec[cw * 32 + c]);
#pragma unroll
            for (int k = 0; k < EPL; ++k)
                s[k] = s[k] + __uint_as_float(val ^ ((rb[k] << (31 - c)) & 0x80000000u));
        }
    }
#pragma unroll
    for (int k = 0; k < EPL; ++k) proj[k] = s[k] * inv_sqrt_d;
}

// Signs [n, dim / 8] and residual norms [n] (f16 bits) of vectors whose codes and scales are stored already.
// bits: 2 or 3 (the polar width); x 16-byte aligned.
int launch_whole_sketch(int dim, int bits, const float* x, const uint8_t* packed, const uint16_t* scales, long long n,
                        const uint32_t* rbits, uint8_t* signs, uint16_t* norms, const Codebook& cb, int seed_odd, float inv_sqrt_d,
                        cudaStream_t s);

// The same for given reconstructions xhat (f32); x of `dtype`; both 16-byte aligned.  Row i is stored at
// (i / rows_per_group) * group_stride + row_offset + i % rows_per_group (rows_per_group 0: i).
int launch_residual_sketch(int dim, const void* x, int dtype, const float* xhat, long long n, const uint32_t* rbits, uint8_t* signs,
                           uint16_t* norms, long long rows_per_group, long long group_stride, long long row_offset, float inv_sqrt_d,
                           cudaStream_t s);

constexpr long long kProjTileMin = 2048;   // below, one query per warp fills the chip
// Projections of nq queries of `dtype`: f32 queries bit for bit as projections_kernel gives them, 16-bit ones on the tensor cores.
int launch_projections_tile(int dim, const void* q, int dtype, long long nq, const uint32_t* rbits, float* rq, float inv_sqrt_d,
                            cudaStream_t s);

// One decode step's input of the TQ cache in one launch (head_dim 32 W; MaxNorm, every block on the normal codebook): the new K and V
// rows [heads, D] quantized into row `row` of their heads, the key's sign sketch and residual norm, and the projections
// rq [nq, D] of the queries.  Everything 16-byte aligned.  TQB_ERR_UNSUPPORTED: take the separate kernels.
struct TqAppend {
    const void *k, *v, *q;
    int dtype, bits, dim, heads;
    long long nq;
    const uint32_t* rbits;
    uint8_t *ki, *vi, *signs;
    uint16_t *ks, *vs, *norms;
    long long cap, sketch_cap, row;   // rows per head of the code and sketch arrays, the row written
    float* rq;
};
int launch_tq_append(const TqAppend& a, cudaStream_t s);

// QuantizedKVCache on short lists (tqb_whole.cu): one launch, host-mapped results.
int launch_scores_query(const tqb_config* cfg, const uint32_t* rbits, const float* q_host, const uint8_t* packed,
                        const uint16_t* scales, const uint8_t* signs, const uint16_t* rnorms, long long n, float* scores,
                        cudaStream_t s);
int launch_weighted_values_one(const tqb_config* cfg, const float* w, const uint8_t* packed, const uint16_t* scales, long long n,
                               float* out, float* partial, unsigned* ticket, cudaStream_t s);

}  // namespace tqb
