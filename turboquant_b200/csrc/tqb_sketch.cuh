// Launchers of the sign-sketch kernels in tqb_sketch.cu.
#pragma once
#include "tqb_common.cuh"

namespace tqb {

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

// Projections of nq queries of `dtype`, eight to a warp: bit for bit those of projections_kernel.
int launch_projections_tile(int dim, const void* q, int dtype, long long nq, const uint32_t* rbits, float* rq, float inv_sqrt_d,
                            cudaStream_t s);

}  // namespace tqb
