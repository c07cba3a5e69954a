// QJL sign sketch on the tensor cores.
//
// Sign r of a residual e is the sign of a sum over d elements, s_r = sum_c (+-1)_rc e_c, and the reference adds left to
// right in f32 (src/qjl.rs:196-208).  Only the sign is kept, so the order matters for the few sums that rounding could
// carry across zero: the sums of 16 vectors are taken as one contraction with a +-1 operand (mma.sync bf16, f32
// accumulators; e as two bf16 terms), and every sum that is not clearly further from zero than both roundings can reach
// is added again, left to right in f32, by one lane.  The stored bits are those of the sequential sums, always.
//
// The bound: two bf16 terms (round to nearest) hold e to 2^-18, the tensor cores' f32 accumulation of 2 d products adds at
// most 2 d 2^-23 sum|e|, the reference's own d - 1 roundings d 2^-24 sum|e|: together below d 2^-21 sum|e| = tau for every
// d >= 32.  |s| > tau decides; about 5 sums of a 128-dim vector in 100 vectors do not, and cost one lane 128 additions.
//
// What bounds it: the MMAs (256 of m16n8k16 for 16 vectors of 128 dims, about 9 cycles each and SM sub-core) and as many
// other instructions.  tcgen05 would want 128 vectors a tile and the +-1 matrix staged in shared memory; the SIMT part
// (dequantize, residual, sequential norm) is as long as the MMAs already.
// Measured (whole calls, B200, before = sequential sums, three instructions an addition, one vector after the other in a
// warp): quantize with sketch of 65,536 vectors of 128 dims 197 -> 64 us, of 256 dims 1297 -> 183 us, 64 vectors of 128 dims
// 76 -> 21 us; residual sketch of 65,536 keys of 128 dims 131 -> 33 us, 4,096 keys 17.2 -> 14.3 us.
#include <type_traits>

#include "tqb_common.cuh"
#include "tqb_pqo_quant.cuh"
#include "tqb_sketch.cuh"

namespace tqb {
namespace {

constexpr int kTileVec = 16;   // vectors of a warp tile: one MMA row block

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// (lo, hi) -> leading bf16 terms, and what they leave as a second pair of terms
__device__ __forceinline__ void split2(float lo, float hi, uint32_t& lead, uint32_t& rest) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(lead) : "f"(hi), "f"(lo));
    const float rl = lo - __uint_as_float(lead << 16), rh = hi - __uint_as_float(lead & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(rest) : "f"(rh), "f"(rl));
}

// Signs and norms of the 16 residuals in `tile` (rows of D + 4 floats: lanes (n, j) read 4 n + j + const, all banks).
// s_rb: Rademacher words, row r at r * (W + 1).  rows: storage row of vector lane & 15.
template <int W>
__device__ __forceinline__ void sketch_tile(const float* tile, const uint32_t* s_rb, int nv, long long row, uint8_t* signs,
                                            uint16_t* norms, float inv_sqrt_d) {
    constexpr int D = 32 * W, P = D + 4, NT = W < 4 ? 4 * W : 16;
    const int lane = threadIdx.x & 31, n = lane >> 2, j = lane & 3;
    // lanes 0..15: the norm, a sequential sum of squares (quantize.rs:51-53); lanes 16..31: sum |e| of the same vector
    float sum = 0.0f;
    {
        const float* r = tile + (lane & 15) * P;
#pragma unroll 8
        for (int c = 0; c < D; c += 4) {
            const float4 v = *reinterpret_cast<const float4*>(r + c);
            sum = sum + fabsf(v.x * (lane < 16 ? v.x : 1.0f));
            sum = sum + fabsf(v.y * (lane < 16 ? v.y : 1.0f));
            sum = sum + fabsf(v.z * (lane < 16 ? v.z : 1.0f));
            sum = sum + fabsf(v.w * (lane < 16 ? v.w : 1.0f));
        }
        if (lane < nv) norms[row] = f32_to_f16_bits(__fsqrt_rn(sum));
    }
    float sa[2];   // sum |e| of vectors n, n + 8
    sa[0] = __shfl_sync(0xffffffffu, sum, 16 + n);
    sa[1] = __shfl_sync(0xffffffffu, sum, 24 + n);
    const long long orow0 = __shfl_sync(0xffffffffu, row, n), orow1 = __shfl_sync(0xffffffffu, row, n + 8);
#pragma unroll 1
    for (int pass = 0; pass < 4 * W / NT; ++pass) {   // NT * 8 sign rows a pass
        float acc[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[t][e] = 0.0f;
#pragma unroll 1
        for (int w = 0; w < W; ++w) {
            // k-slots of MMA half h, quad position j: dims 32 w + 8 h + j and + 16 (slots 2j, 2j + 1), + 4 and + 20 (2j + 8, 2j + 9)
            uint32_t a[2][2][4];   // [half][term][fragment register]
            const float* e0 = tile + n * P + 32 * w + j;
            const float* e1 = e0 + 8 * P;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                split2(e0[8 * h], e0[8 * h + 16], a[h][0][0], a[h][1][0]);
                split2(e1[8 * h], e1[8 * h + 16], a[h][0][1], a[h][1][1]);
                split2(e0[8 * h + 4], e0[8 * h + 20], a[h][0][2], a[h][1][2]);
                split2(e1[8 * h + 4], e1[8 * h + 20], a[h][0][3], a[h][1][3]);
            }
            const uint32_t* rb = s_rb + (pass * NT * 8 + n) * (W + 1) + w;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const uint32_t u = rb[t * 8 * (W + 1)] << (3 - j);   // bits j + 4 c, j + 4 c + 16 -> 3 + 4 c, 19 + 4 c
                uint32_t b[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) b[c] = ((u << (12 - 4 * c)) & 0x80008000u) | 0x3F803F80u;   // bit set: -1
#pragma unroll
                for (int term = 0; term < 2; ++term) {
                    mma_bf16(acc[t], a[0][term], b[0], b[1]);
                    mma_bf16(acc[t], a[1][term], b[2], b[3]);
                }
            }
        }
        // rows n (e = 0, 1) and n + 8 (e = 2, 3), sign rows 8 t + 2 j + (e & 1)
        uint32_t pos[2] = {0u, 0u}, open[2] = {0u, 0u};
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            // below 1e-25 the second terms may be flushed: every sum is taken again; all-zero residuals: 0 >= 0
            const float tau = sa[v] < 1e-25f ? (sa[v] == 0.0f ? -1.0f : INFINITY) : sa[v] * (D * 4.76837158203125e-7f);
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float s = acc[t][2 * v + e];
                    pos[v] |= (s >= 0.0f ? 1u : 0u) << (2 * t + e);
                    open[v] |= (fabsf(s) > tau ? 0u : 1u) << (2 * t + e);   // NaN stays open
                }
        }
        while (__any_sync(0xffffffffu, (open[0] | open[1]) != 0u)) {
            if ((open[0] | open[1]) != 0u) {
                const int v = open[0] != 0u ? 0 : 1;
                const uint32_t m = v == 0 ? open[0] : open[1];
                const int bit = __ffs(m) - 1;
                const int r = pass * NT * 8 + (bit >> 1) * 8 + 2 * j + (bit & 1);
                const float* e = tile + (n + 8 * v) * P;
                float s = 0.0f;
#pragma unroll 1
                for (int w = 0; w < W; ++w) {
                    const uint32_t word = s_rb[r * (W + 1) + w];
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        s = s + __uint_as_float(__float_as_uint(e[32 * w + c]) ^ ((word << (31 - c)) & 0x80000000u));
                }
                const uint32_t p = (s * inv_sqrt_d >= 0.0f ? 1u : 0u) << bit;   // qjl.rs:315
                if (v == 0) { pos[0] = (pos[0] & ~(1u << bit)) | p; open[0] &= open[0] - 1u; }
                else { pos[1] = (pos[1] & ~(1u << bit)) | p; open[1] &= open[1] - 1u; }
            }
        }
        // four sign rows tiles make one 32-bit word; quad lane k & 3 stores word k
#pragma unroll
        for (int k = 0; k < NT / 4; ++k) {
            uint32_t w0 = 0u, w1 = 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                w0 |= ((pos[0] >> (8 * k + 2 * i)) & 3u) << (8 * i + 2 * j);
                w1 |= ((pos[1] >> (8 * k + 2 * i)) & 3u) << (8 * i + 2 * j);
            }
#pragma unroll
            for (int m = 1; m <= 2; m <<= 1) {
                w0 |= __shfl_xor_sync(0xffffffffu, w0, m);
                w1 |= __shfl_xor_sync(0xffffffffu, w1, m);
            }
            if (j == (k & 3)) {
                const int word = pass * (NT / 4) + k;
                if (n < nv) reinterpret_cast<uint32_t*>(signs)[orow0 * W + word] = w0;
                if (n + 8 < nv) reinterpret_cast<uint32_t*>(signs)[orow1 * W + word] = w1;
            }
        }
    }
}

template <int W>
__device__ __forceinline__ void load_rbits(uint32_t* s_rb, const uint32_t* rbits) {
    for (int i = threadIdx.x; i < 32 * W * W; i += blockDim.x) s_rb[(i / W) * (W + 1) + (i % W)] = rbits[i];
}

template <int W>
constexpr int kSketchWarps = W >= 8 ? 4 : 8;
template <int W>
size_t sketch_smem(int table_floats) {
    return sizeof(uint32_t) * 32 * W * (W + 1) + sizeof(float) * table_floats + sizeof(float) * kSketchWarps<W> * kTileVec * (32 * W + 4);
}

// Core-crate vectors: residual = x - dequantize(packed, scale) (src/qjl.rs:355-377), EPL = W lanes per vector as in
// whole_dequantize_lane_kernel (same operations in the same order, so the residual has the same bits).
template <int W, int BITS>
__global__ void __launch_bounds__(kSketchWarps<W> * 32)
whole_sketch_kernel(const float* __restrict__ x, const uint8_t* __restrict__ packed, const uint16_t* __restrict__ scales,
                    long long n, const uint32_t* __restrict__ rbits, uint8_t* __restrict__ signs, uint16_t* __restrict__ norms,
                    Codebook cb, int seed_odd, float inv_sqrt_d) {
    constexpr int D = 32 * W, P = D + 4, KPW = 32 / W, NW = kSketchWarps<W>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* s_rb = reinterpret_cast<uint32_t*>(smem_raw);
    float* s_tab = reinterpret_cast<float*>(s_rb + D * (W + 1));   // [code][lane]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* tile = s_tab + (1 << BITS) * 32 + warp * kTileVec * P;
    load_rbits<W>(s_rb, rbits);
    for (int i = threadIdx.x; i < (1 << BITS) * 32; i += NW * 32) s_tab[i] = cb.c[i >> 5];
    __syncthreads();
    const float* tab = s_tab + lane;
    const int sub = lane % W, kin = lane / W;
    const float m_even = seed_odd ? -inv_sqrt_d : inv_sqrt_d, m_odd = -m_even;
    const uint32_t tile_s = (uint32_t)__cvta_generic_to_shared(tile);
    const long long tiles = (n + kTileVec - 1) / kTileVec;
    for (long long t = (long long)blockIdx.x * NW + warp; t < tiles; t += (long long)gridDim.x * NW) {
        const long long v0 = t * kTileVec;
        const int nv = (int)min((long long)kTileVec, n - v0);
#pragma unroll 8
        for (int i = lane; i < kTileVec * D / 4; i += 32) {
            const int r = i / (D / 4), c = i % (D / 4);
            const float* src = x + (v0 + min(r, nv - 1)) * D + 4 * c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tile_s + (r * P + 4 * c) * 4), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll 1
        for (int v = kin; v < (kTileVec > KPW ? kTileVec : KPW); v += KPW) {
            const long long vc = v0 + min(v & (kTileVec - 1), nv - 1);
            uint32_t w[BITS];
            const uint32_t* p = reinterpret_cast<const uint32_t*>(packed + vc * (D * BITS / 8)) + sub * BITS;
#pragma unroll
            for (int k = 0; k < BITS; ++k) w[k] = __ldg(p + k);
            const float sc = f16_bits_to_f32(__ldg(scales + vc));
            float y[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const int bit = BITS * i, k = bit >> 5, sh = bit & 31;
                const uint32_t code = (sh + BITS <= 32 ? (w[k] >> sh) : __funnelshift_r(w[k], w[k + 1 < BITS ? k + 1 : k], sh)) &
                                      ((1u << BITS) - 1u);
                y[i] = tab[code * 32];
            }
            butterfly32_regs(y);
#pragma unroll
            for (int hs = 1; hs < W; hs <<= 1) {
                const uint32_t flip = (sub & hs) ? 0x80000000u : 0u;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float other = __shfl_xor_sync(0xffffffffu, y[i], hs);
                    y[i] = other + __uint_as_float(__float_as_uint(y[i]) ^ flip);
                }
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
            if (v < kTileVec) {
                float4* row = reinterpret_cast<float4*>(tile + v * P + sub * 32);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    float4 f = row[k];
                    f.x -= (y[4 * k] * m_even) * sc;
                    f.y -= (y[4 * k + 1] * m_odd) * sc;
                    f.z -= (y[4 * k + 2] * m_even) * sc;
                    f.w -= (y[4 * k + 3] * m_odd) * sc;
                    row[k] = f;
                }
            }
        }
        __syncwarp();
        sketch_tile<W>(tile, s_rb, nv, v0 + min(lane & 15, nv - 1), signs, norms, inv_sqrt_d);
        __syncwarp();
    }
}

// Block-32 TQ cache: residual = original - dequantized (src/cache/tq.rs:380-411), rows mapped like the storage.
template <int W, typename T>
__global__ void __launch_bounds__(kSketchWarps<W> * 32)
residual_sketch_mma_kernel(const T* __restrict__ x, const float* __restrict__ xhat, long long n, const uint32_t* __restrict__ rbits,
                           uint8_t* __restrict__ signs, uint16_t* __restrict__ norms, long long rows_per_group,
                           long long group_stride, long long row_offset, float inv_sqrt_d) {
    constexpr int D = 32 * W, P = D + 4, NW = kSketchWarps<W>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* s_rb = reinterpret_cast<uint32_t*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* tile = reinterpret_cast<float*>(s_rb + D * (W + 1)) + warp * kTileVec * P;
    load_rbits<W>(s_rb, rbits);
    __syncthreads();
    const long long tiles = (n + kTileVec - 1) / kTileVec;
    for (long long t = (long long)blockIdx.x * NW + warp; t < tiles; t += (long long)gridDim.x * NW) {
        const long long v0 = t * kTileVec;
        const int nv = (int)min((long long)kTileVec, n - v0);
#pragma unroll 4
        for (int i = lane; i < kTileVec * D / 4; i += 32) {
            const int r = i / (D / 4), c = i % (D / 4);
            const long long e = (v0 + min(r, nv - 1)) * D + 4 * c;
            const float4 h = __ldg(reinterpret_cast<const float4*>(xhat + e));
            float4 f;
            if constexpr (sizeof(T) == 4) {
                f = __ldg(reinterpret_cast<const float4*>(x + e));
            } else {
                const uint2 u = __ldg(reinterpret_cast<const uint2*>(x + e));
                T q[4];
                *reinterpret_cast<uint2*>(q) = u;
                f = make_float4(to_f32<T>(q[0]), to_f32<T>(q[1]), to_f32<T>(q[2]), to_f32<T>(q[3]));
            }
            *reinterpret_cast<float4*>(tile + r * P + 4 * c) = make_float4(f.x - h.x, f.y - h.y, f.z - h.z, f.w - h.w);
        }
        __syncwarp();
        const long long i = v0 + min(lane & 15, nv - 1);
        long long row = i;
        if (rows_per_group != 0) {
            const long long g = i / rows_per_group;
            row = g * group_stride + row_offset + (i - g * rows_per_group);
        }
        sketch_tile<W>(tile, s_rb, nv, row, signs, norms, inv_sqrt_d);
        __syncwarp();
    }
}

// precompute_query_projections (src/qjl.rs:488-492) of many queries: a lane owns sign rows lane, lane + 32, ... and adds,
// left to right, for eight queries at a time, so a +-1 made from a bit (two instructions) serves eight additions
// (fma(q, +-1, s) rounds once, like s +- q).  One query per warp spends three instructions on every addition:
// 65,536 queries of 128 dims 117 -> 65 us (77 us with one query an instruction), 4,096 queries 13.1 -> 12.3 us.
constexpr int kProjQ = 8, kProjWarps = 4;
template <int W, typename T>
__global__ void __launch_bounds__(kProjWarps * 32)
projections_tile_kernel(const T* __restrict__ q, long long nq, const uint32_t* __restrict__ rbits, float* __restrict__ rq,
                        float inv_sqrt_d) {
    constexpr int D = 32 * W;
    __shared__ uint32_t s_rb[D * (W + 1)];
    __shared__ __align__(16) float s_q[kProjWarps][D * kProjQ];   // [element][query]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    load_rbits<W>(s_rb, rbits);
    __syncthreads();
    float* vec = s_q[warp];
    const long long tiles = (nq + kProjQ - 1) / kProjQ;
    for (long long t = (long long)blockIdx.x * kProjWarps + warp; t < tiles; t += (long long)gridDim.x * kProjWarps) {
        const long long q0 = t * kProjQ;
        const int nv = (int)min((long long)kProjQ, nq - q0);
        // lane: query lane & 7, elements lane >> 3 + 4 k: the 32 stores of an instruction are consecutive words
        const T* src = q + (q0 + min(lane & 7, nv - 1)) * D + (lane >> 3);
#pragma unroll 8
        for (int k = 0; k < D / 4; ++k) vec[32 * k + 8 * (lane >> 3) + (lane & 7)] = to_f32<T>(src[4 * k]);
        __syncwarp();
        F2 s[W][kProjQ / 2];   // two queries an instruction
#pragma unroll
        for (int k = 0; k < W; ++k)
#pragma unroll
            for (int i = 0; i < kProjQ / 2; ++i) s[k][i] = f2(0.0f);
#pragma unroll 1
        for (int cw = 0; cw < W; ++cw) {
            uint32_t rb[W];
#pragma unroll
            for (int k = 0; k < W; ++k) rb[k] = s_rb[(lane + 32 * k) * (W + 1) + cw];
#pragma unroll 8
            for (int c = 0; c < 32; ++c) {
                const float4 lo = *reinterpret_cast<const float4*>(vec + (cw * 32 + c) * kProjQ);
                const float4 hi = *reinterpret_cast<const float4*>(vec + (cw * 32 + c) * kProjQ + 4);
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const F2 m = f2(__uint_as_float((rb[k] << 31) | 0x3F800000u));
                    rb[k] >>= 1;
                    s[k][0] = fma2(f2(lo.x, lo.y), m, s[k][0]);
                    s[k][1] = fma2(f2(lo.z, lo.w), m, s[k][1]);
                    s[k][2] = fma2(f2(hi.x, hi.y), m, s[k][2]);
                    s[k][3] = fma2(f2(hi.z, hi.w), m, s[k][3]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kProjQ; ++i)
            if (i < nv)
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const float2 t = halves(s[k][i >> 1]);
                    rq[(q0 + i) * D + lane + 32 * k] = ((i & 1) ? t.y : t.x) * inv_sqrt_d;
                }
        __syncwarp();
    }
}

// A decode step's input of the TQ cache.  The same work as block_quantize_pqo_kernel, block_dequantize_lane_kernel,
// residual_sketch_kernel, a conversion and projections_kernel one after the other - the same operations in the same order, the
// same bytes - for the few vectors of one token: a warp takes a head's K and V rows (a lane per 32-block quantizes, then the
// warp dequantizes the key, sketches its residual), another warp takes a query.  What bounds it is the latency of
// one chain: about 4 us, where the five launches took 17 us and as much again in the gaps between them.
// Measured: 16 sequences x 4,001 tokens, 32 q / 8 KV heads, a layer's decode_fused call 76.6 -> 62 us.
constexpr int kAppendWarps = 4;
constexpr long long kAppendMax = 4096;   // keys and queries; about two rounds of the chip's warps, beyond which the separate kernels amortise their tables
template <int W, typename T, int BITS>
__global__ void __launch_bounds__(kAppendWarps * 32)
tq_append_kernel(TqAppend a, const __grid_constant__ Codebook cb, float outer_centroid, float sign_mag, float inv_sqrt_d) {
    constexpr int D = 32 * W;
    __shared__ uint32_t s_rb[D * (W + 1)];
    __shared__ float2 s_lut[kCells * 32];
    __shared__ float s_vec[kAppendWarps][D];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    load_rbits<W>(s_rb, a.rbits);
    build_cell_table(cb, cb.n - 1, s_lut, threadIdx.x, kAppendWarps * 32);
    __syncthreads();
    float* vec = s_vec[warp];
    const long long item = (long long)blockIdx.x * kAppendWarps + warp;
    if (item >= a.heads + a.nq) return;   // no block-wide barrier follows
    if (item >= a.heads) {
        const long long i = item - a.heads;
#pragma unroll
        for (int k = 0; k < W; ++k) vec[lane + 32 * k] = to_f32<T>(reinterpret_cast<const T*>(a.q)[i * D + lane + 32 * k]);
        __syncwarp();
        float proj[W];
        rademacher_rows<W>(vec, s_rb, lane, inv_sqrt_d, proj);
#pragma unroll
        for (int k = 0; k < W; ++k) a.rq[i * D + lane + 32 * k] = proj[k];
        return;
    }
    const T* key = reinterpret_cast<const T*>(a.k) + item * D;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    uint16_t sc = 0;
    if ((lane & 15) < W) {   // lanes 0 .. W-1: the key's blocks, 16 .. : the value's
        const int b = lane & 15;
        const T* src = (lane < 16 ? key : reinterpret_cast<const T*>(a.v) + item * D) + 32 * b;
        sc = f32_to_f16_bits(pqo_quantize_block<T, BITS, true>(src, cb, outer_centroid, w, s_lut + lane));
        const size_t blk = ((size_t)item * a.cap + a.row) * W + b;
        uint32_t* out = reinterpret_cast<uint32_t*>((lane < 16 ? a.ki : a.vi) + blk * (4 * BITS));
        out[0] = w[0]; out[1] = w[1]; out[2] = w[2];
        if (BITS == 4) out[3] = w[3];
        (lane < 16 ? a.ks : a.vs)[blk] = sc;
    }
    __syncwarp();
    const float sgn = ((kSignMask >> lane) & 1u) ? -sign_mag : sign_mag, inv_sqrt = 1.0f / sqrtf((float)kBlock);
    const int bit = BITS * lane, wi = bit >> 5;
#pragma unroll
    for (int b = 0; b < W; ++b) {
        uint32_t kw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) kw[i] = __shfl_sync(0xffffffffu, w[i], b);
        const uint32_t lo = wi == 0 ? kw[0] : wi == 1 ? kw[1] : wi == 2 ? kw[2] : kw[3];
        const uint32_t hi = wi == 0 ? kw[1] : wi == 1 ? kw[2] : kw[3];
        const int code = min((int)(__funnelshift_r(lo, hi, bit & 31) & ((1u << BITS) - 1u)), cb.n - 1);
        float y = cb.c[code] * sgn;
#pragma unroll
        for (int h = 1; h < 32; h <<= 1) {
            const float other = __shfl_xor_sync(0xffffffffu, y, h);
            y = (lane & h) ? (other - y) : (y + other);
        }
        y = (y * inv_sqrt) * fabsf(f16_bits_to_f32((uint16_t)__shfl_sync(0xffffffffu, (uint32_t)sc, b)));
        vec[lane + 32 * b] = to_f32<T>(key[lane + 32 * b]) - y;
    }
    __syncwarp();
    float s = 0.0f;   // left to right, every lane the same sum
#pragma unroll 8
    for (int c = 0; c < D; ++c) s = s + vec[c] * vec[c];
    const size_t dst = (size_t)item * a.sketch_cap + a.row;
    if (lane == 0) a.norms[dst] = f32_to_f16_bits(__fsqrt_rn(s));
    float proj[W];
    rademacher_rows<W>(vec, s_rb, lane, inv_sqrt_d, proj);
#pragma unroll
    for (int k = 0; k < W; ++k) {
        const uint32_t word = __ballot_sync(0xffffffffu, proj[k] >= 0.0f);
        if (lane == 0) reinterpret_cast<uint32_t*>(a.signs)[dst * W + k] = word;
    }
}

template <int W, typename T>
int launch_append(const TqAppend& a, const Codebook& cb, float outer, float sign_mag, float inv, cudaStream_t s) {
    const long long grid = (a.heads + a.nq + kAppendWarps - 1) / kAppendWarps;
    if (a.bits == 3) tq_append_kernel<W, T, 3><<<(unsigned)grid, kAppendWarps * 32, 0, s>>>(a, cb, outer, sign_mag, inv);
    else tq_append_kernel<W, T, 4><<<(unsigned)grid, kAppendWarps * 32, 0, s>>>(a, cb, outer, sign_mag, inv);
    return check_launch(s);
}

// The same for 16-bit queries on the tensor cores, 16 to a warp: a bf16 value is one bf16 term and an f16 value two, so every
// product with +-1 is exact and only the f32 accumulation rounds - over fewer steps than the sum element by element.
// Measured (24,576 queries of 128 dims, bf16): 27 -> 14 us; relative error against 64 bits 2.58e-8 (element by element 2.59e-8),
// at a log-normal spread of 2 over the elements 6.8e-8 (9.3e-8).
template <int W, typename T>
__global__ void __launch_bounds__(kSketchWarps<W> * 32)
projections_mma_kernel(const T* __restrict__ q, long long nq, const uint32_t* __restrict__ rbits, float* __restrict__ rq, float inv_sqrt_d) {
    static_assert(sizeof(T) == 2, "f32 queries: projections_tile_kernel");
    constexpr int D = 32 * W, P = D + 4, NW = kSketchWarps<W>, NT = W < 4 ? 4 * W : 16;
    constexpr int kTerms = std::is_same<T, __nv_bfloat16>::value ? 1 : 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* s_rb = reinterpret_cast<uint32_t*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = lane >> 2, j = lane & 3;
    float* tile = reinterpret_cast<float*>(s_rb + D * (W + 1)) + warp * kTileVec * P;
    load_rbits<W>(s_rb, rbits);
    __syncthreads();
    const long long tiles = (nq + kTileVec - 1) / kTileVec;
    for (long long t0 = (long long)blockIdx.x * NW + warp; t0 < tiles; t0 += (long long)gridDim.x * NW) {
        const long long q0 = t0 * kTileVec;
        const int nv = (int)min((long long)kTileVec, nq - q0);
#pragma unroll 4
        for (int i = lane; i < kTileVec * D / 4; i += 32) {
            const int r = i / (D / 4), c = i % (D / 4);
            T e[4];
            *reinterpret_cast<uint2*>(e) = __ldg(reinterpret_cast<const uint2*>(q + (q0 + min(r, nv - 1)) * D + 4 * c));
            *reinterpret_cast<float4*>(tile + r * P + 4 * c) = make_float4(to_f32<T>(e[0]), to_f32<T>(e[1]), to_f32<T>(e[2]), to_f32<T>(e[3]));
        }
        __syncwarp();
#pragma unroll 1
        for (int pass = 0; pass < 4 * W / NT; ++pass) {
            float acc[NT][4];
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[t][e] = 0.0f;
#pragma unroll 1
            for (int w = 0; w < W; ++w) {
                uint32_t a[2][2][4];   // [half][term][fragment register], k-slots as in sketch_tile
                const float* e0 = tile + n * P + 32 * w + j;
                const float* e1 = e0 + 8 * P;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    split2(e0[8 * h], e0[8 * h + 16], a[h][0][0], a[h][1][0]);
                    split2(e1[8 * h], e1[8 * h + 16], a[h][0][1], a[h][1][1]);
                    split2(e0[8 * h + 4], e0[8 * h + 20], a[h][0][2], a[h][1][2]);
                    split2(e1[8 * h + 4], e1[8 * h + 20], a[h][0][3], a[h][1][3]);
                    if (kTerms == 2) {   // an infinity leaves no second term (Inf - Inf)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if ((a[h][0][e] & 0x7F80u) == 0x7F80u) a[h][1][e] &= 0xFFFF0000u;
                            if ((a[h][0][e] & 0x7F800000u) == 0x7F800000u) a[h][1][e] &= 0x0000FFFFu;
                        }
                    }
                }
                const uint32_t* rb = s_rb + (pass * NT * 8 + n) * (W + 1) + w;
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const uint32_t u = rb[t * 8 * (W + 1)] << (3 - j);
                    uint32_t b[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) b[c] = ((u << (12 - 4 * c)) & 0x80008000u) | 0x3F803F80u;
                    // 32 dims at a time: the tensor cores' own accumulation truncates, the additions of the parts round
                    float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int term = kTerms - 1; term >= 0; --term) {   // the small terms first
                        mma_bf16(part, a[0][term], b[0], b[1]);
                        mma_bf16(part, a[1][term], b[2], b[3]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[t][e] += part[e];
                }
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                float* o = rq + (q0 + n) * D + (pass * NT + t) * 8 + 2 * j;
                if (n < nv) *reinterpret_cast<float2*>(o) = make_float2(acc[t][0] * inv_sqrt_d, acc[t][1] * inv_sqrt_d);
                if (n + 8 < nv) *reinterpret_cast<float2*>(o + 8 * D) = make_float2(acc[t][2] * inv_sqrt_d, acc[t][3] * inv_sqrt_d);
            }
        }
        __syncwarp();
    }
}

template <typename K>
int opt_in(K kernel, size_t smem) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_cuda_error(e); return TQB_ERR_CUDA; }
    return TQB_OK;
}

template <int W, int BITS>
int launch_whole(const float* x, const uint8_t* packed, const uint16_t* scales, long long n, const uint32_t* rbits, uint8_t* signs,
                 uint16_t* norms, const Codebook& cb, int seed_odd, float inv, cudaStream_t s) {
    constexpr int NW = kSketchWarps<W>;
    const size_t smem = sketch_smem<W>((1 << BITS) * 32);
    const int st = opt_in(whole_sketch_kernel<W, BITS>, smem);
    if (st != TQB_OK) return st;
    long long grid = (n + NW * kTileVec - 1) / (NW * kTileVec);
    if (grid > 148 * 2) grid = 148 * 2;
    whole_sketch_kernel<W, BITS><<<(int)grid, NW * 32, smem, s>>>(x, packed, scales, n, rbits, signs, norms, cb, seed_odd, inv);
    return check_launch(s);
}

template <int W, typename T>
int launch_residual(const T* x, const float* xhat, long long n, const uint32_t* rbits, uint8_t* signs, uint16_t* norms,
                    long long rpg, long long gs, long long off, float inv, cudaStream_t s) {
    constexpr int NW = kSketchWarps<W>;
    const size_t smem = sketch_smem<W>(0);
    const int st = opt_in(residual_sketch_mma_kernel<W, T>, smem);
    if (st != TQB_OK) return st;
    long long grid = (n + NW * kTileVec - 1) / (NW * kTileVec);
    if (grid > 148 * 2) grid = 148 * 2;
    residual_sketch_mma_kernel<W, T><<<(int)grid, NW * 32, smem, s>>>(x, xhat, n, rbits, signs, norms, rpg, gs, off, inv);
    return check_launch(s);
}

template <int W, typename T>
int launch_projections(const T* q, long long nq, const uint32_t* rbits, float* rq, float inv, cudaStream_t s) {
    // (32 dims are one part: there the sum element by element is the closer one, 4.6e-8 against 5.7e-8 at a wide spread)
    if constexpr (sizeof(T) == 2 && W > 1) {
        if (((uintptr_t)q % 8) == 0 && ((uintptr_t)rq % 8) == 0) {
            constexpr int NW = kSketchWarps<W>;
            const size_t smem = sketch_smem<W>(0);
            const int st = opt_in(projections_mma_kernel<W, T>, smem);
            if (st != TQB_OK) return st;
            long long tiles = (nq + NW * kTileVec - 1) / (NW * kTileVec);
            if (tiles > 148 * 2) tiles = 148 * 2;
            projections_mma_kernel<W, T><<<(int)tiles, NW * 32, smem, s>>>(q, nq, rbits, rq, inv);
            return check_launch(s);
        }
    }
    long long grid = (nq + kProjQ * kProjWarps - 1) / (kProjQ * kProjWarps);
    if (grid > 148 * 8) grid = 148 * 8;
    projections_tile_kernel<W, T><<<(int)grid, kProjWarps * 32, 0, s>>>(q, nq, rbits, rq, inv);
    return check_launch(s);
}

#define TQB_BY_DIM(dim, CALL)                        \
    switch (dim) {                                   \
        case 32: { constexpr int W = 1; return CALL; }   \
        case 64: { constexpr int W = 2; return CALL; }   \
        case 128: { constexpr int W = 4; return CALL; }  \
        case 256: { constexpr int W = 8; return CALL; }  \
        default: return TQB_ERR_UNSUPPORTED;         \
    }

}  // namespace

int launch_whole_sketch(int dim, int bits, const float* x, const uint8_t* packed, const uint16_t* scales, long long n,
                        const uint32_t* rbits, uint8_t* signs, uint16_t* norms, const Codebook& cb, int seed_odd, float inv_sqrt_d,
                        cudaStream_t s) {
    if (bits == 2) { TQB_BY_DIM(dim, (launch_whole<W, 2>(x, packed, scales, n, rbits, signs, norms, cb, seed_odd, inv_sqrt_d, s))) }
    if (bits == 3) { TQB_BY_DIM(dim, (launch_whole<W, 3>(x, packed, scales, n, rbits, signs, norms, cb, seed_odd, inv_sqrt_d, s))) }
    return TQB_ERR_UNSUPPORTED;
}

int launch_residual_sketch(int dim, const void* x, int dtype, const float* xhat, long long n, const uint32_t* rbits, uint8_t* signs,
                           uint16_t* norms, long long rows_per_group, long long group_stride, long long row_offset, float inv_sqrt_d,
                           cudaStream_t s) {
#define TQB_RES(T) TQB_BY_DIM(dim, (launch_residual<W, T>((const T*)x, xhat, n, rbits, signs, norms, rows_per_group, group_stride, row_offset, inv_sqrt_d, s)))
    if (dtype == TQB_F32) { TQB_RES(float) }
    if (dtype == TQB_F16) { TQB_RES(__half) }
    TQB_RES(__nv_bfloat16)
#undef TQB_RES
}

int launch_projections_tile(int dim, const void* q, int dtype, long long nq, const uint32_t* rbits, float* rq, float inv_sqrt_d,
                            cudaStream_t s) {
#define TQB_PROJ(T) TQB_BY_DIM(dim, (launch_projections<W, T>((const T*)q, nq, rbits, rq, inv_sqrt_d, s)))
    if (dtype == TQB_F32) { TQB_PROJ(float) }
    if (dtype == TQB_F16) { TQB_PROJ(__half) }
    TQB_PROJ(__nv_bfloat16)
#undef TQB_PROJ
}

int launch_tq_append(const TqAppend& a, cudaStream_t s) {
    Codebook normal, outlier;
    if ((a.bits != 3 && a.bits != 4) || !block_codebook(a.bits - 1, TQB_MAXNORM, normal) || !block_codebook(a.bits, TQB_MAXNORM, outlier))
        return TQB_ERR_UNSUPPORTED;
    const uintptr_t all = (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.q | (uintptr_t)a.ki | (uintptr_t)a.vi;
    if ((all % 16) != 0 || ((uintptr_t)a.signs % 4) != 0 || a.heads + a.nq > kAppendMax) return TQB_ERR_UNSUPPORTED;
    const float outer = outlier.c[outlier.n - 1];   // precomputed/mod.rs:78
    volatile float inv32 = 1.0f / sqrtf(32.0f), s32 = sqrtf(32.0f);
    const float sign_mag = inv32 * s32;             // src/cache/wht_tensor.rs:29-35: the sign pattern's magnitude in f32
    const float inv = 1.0f / sqrtf((float)a.dim);
    if (a.dtype == TQB_F32) { TQB_BY_DIM(a.dim, (launch_append<W, float>(a, normal, outer, sign_mag, inv, s))) }
    if (a.dtype == TQB_F16) { TQB_BY_DIM(a.dim, (launch_append<W, __half>(a, normal, outer, sign_mag, inv, s))) }
    TQB_BY_DIM(a.dim, (launch_append<W, __nv_bfloat16>(a, normal, outer, sign_mag, inv, s)))
}

}  // namespace tqb
