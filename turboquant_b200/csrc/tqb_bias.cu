// QJL logit bias of the TQ cache (compute_logit_bias, src/cache/tq.rs:185-253):
//   bias[h, i, t] = c_t * sum_d rq[h, i, d] * (+-1 by bit d of the token's sign sketch),  c_t = norm_t sqrt(pi/2) / sqrt(D)
// rq: [hq, q_len, D]; signs: [hkv, stride, D/8]; norms: [hkv, stride]; bias: [hq, q_len, kv_len] of type OT.
//
// The sum is a dense contraction [g * q_len rows x D] x [D x tokens] with a +-1 operand, so it runs on the tensor cores
// (mma.sync m16n8k16 bf16, f32 accumulate).  The projected query is split into three bf16 terms, which hold its 24
// significant bits exactly; +-1 is exact in bf16, so every product is exact and only the f32 accumulation loses anything.  The tensor
// cores truncate there, so the leading terms are added up in rounded parts of 16 dims: relative error against 64 bits, normal
// queries of 128 dims, 4.5e-8 (element by element 2.1e-7, all terms in one accumulator 4.2e-7); wide spreads likewise.
// A sign bit becomes a bf16 +-1 by one shift and one three-input logic operation per TWO of them (bits p and p + 16 of a
// sketch word land in the sign positions of the two halves), and the warp keeps the expanded signs of its tokens in
// registers for all query rows.  What bounds it: the latency of the prologue's loads and of few, short row tiles (stalls on
// loads 4.4 to 5.4 per issue, tensor pipe 19 to 26 % at 96 query tokens on 192 and 384).  tcgen05 would have to stage the expanded signs (16 x their stored size) in shared
// memory for 128 query rows at most; the register-fed MMA never leaves the register file.
// Measured (32 q / 8 KV heads x 8 sequences, 96 query tokens on 96..384 stored, bf16, mean of four lengths): one thread
// per token with an f32 FMA per sign 510 us, this kernel 32.8 us launch after launch (30.6 us with one
// accumulator).
#include "tqb_common.cuh"

namespace tqb {
namespace {

constexpr int kBiasWarps = 4;
constexpr int kBiasRows = 64;      // query rows per CTA: their operand fragments (48 KB at D = 128) live in shared memory
constexpr int kBiasPitch = 40;     // staging row pitch in floats: float2 stores of a half-warp hit 32 distinct banks

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// x = hi + mid + lo, each a bf16 (the leading 8 bits of what is left, truncated, so nothing overflows): exact for every
// finite f32 whose low term stays in the normal range.  A NaN stays one, whichever of its bits is set.
__device__ __forceinline__ void split3(float x, uint32_t (&t)[3]) {
    x = x == x ? x : __uint_as_float(0x7FFFFFFFu);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint32_t h = __float_as_uint(x) & 0xFFFF0000u;
        t[i] = h >> 16;
        x = fabsf(x) < INFINITY ? x - __uint_as_float(h) : 0.0f;
    }
}

// W = D / 32 sketch words per token; NT = 8-token column tiles per warp (their signs take 4 W NT registers).
// k-slots: MMA (w, half) contracts, in quad position j, the dims 32w + p and 32w + p + 16 for p = 4j + 2 half (slots 2j,
// 2j + 1) and p + 1 (slots 2j + 8, 2j + 9).
template <typename OT, int W, int NT>
__global__ void __launch_bounds__(kBiasWarps * 32)
logit_bias_mma_kernel(const float* __restrict__ rq, const uint8_t* __restrict__ signs, const uint16_t* __restrict__ norms,
                      OT* __restrict__ bias, int rows, int kv_len, int kv_stride, float scale_factor) {
    constexpr int D = 32 * W, KS = 2 * W;
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint4* s_a = reinterpret_cast<uint4*>(s_raw);                                   // [row tile][KS][3 terms][32 lanes]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = lane >> 2, j = lane & 3;
    const int kvh = blockIdx.y;
    const int r0 = blockIdx.z * kBiasRows;
    const int tiles = (min(kBiasRows, rows - r0) + 15) / 16;
    const int tok0 = (blockIdx.x * kBiasWarps + warp) * (8 * NT);
    const size_t row0 = (size_t)kvh * kv_stride;

    // signs of the warp's tokens: lane (n, j) holds, for column n of tile i, what its quad position contributes
    uint32_t b[NT][KS][2];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const int t = min(tok0 + 8 * i + n, kv_len - 1);
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(signs + (row0 + t) * (D / 8));
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t u = __ldg(sw + w) << (12 - 4 * j);    // bit 4j + c now sits at position 12 + c
#pragma unroll
            for (int c = 0; c < 4; ++c) b[i][2 * w + (c >> 1)][c & 1] = ((u << (3 - c)) & 0x80008000u) ^ 0xBF80BF80u;
        }
    }
    const int tw = min(tok0 + lane, kv_len - 1);                 // lane = token of the output rows (8 NT <= 32)
    const float c_t = f16_bits_to_f32(__ldg(norms + row0 + tw)) * scale_factor;

    // operand fragments of the CTA's query rows
    const float* q = rq + (size_t)kvh * rows * D;
    for (int u = threadIdx.x; u < tiles * KS * 32; u += kBiasWarps * 32) {
        const int l = u & 31, ks = (u >> 5) % KS, mt = (u >> 5) / KS;
        const int p = 32 * (ks >> 1) + 4 * (l & 3) + 2 * (ks & 1);
        uint32_t f[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {                            // a0: (row n, p), a1: (row n + 8, p), a2, a3: p + 1
            const int row = r0 + 16 * mt + (l >> 2) + 8 * (e & 1);
            uint32_t lo[3] = {0u, 0u, 0u}, hi[3] = {0u, 0u, 0u};
            if (row < rows) {
                split3(__ldg(q + (size_t)row * D + p + (e >> 1)), lo);
                split3(__ldg(q + (size_t)row * D + p + 16 + (e >> 1)), hi);
            }
#pragma unroll
            for (int t = 0; t < 3; ++t) f[t][e] = lo[t] | (hi[t] << 16);
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) s_a[((mt * KS + ks) * 3 + t) * 32 + l] = make_uint4(f[t][0], f[t][1], f[t][2], f[t][3]);
    }
    __syncthreads();
    if (tok0 >= kv_len) return;                                  // no barrier follows

    float* stage = reinterpret_cast<float*>(s_a + (min(kBiasRows, rows) + 15) / 16 * (KS * 3 * 32)) + warp * 16 * kBiasPitch;
    const int ntok = min(8 * NT, kv_len - tok0);
    for (int mt = 0; mt < tiles; ++mt) {
        // The tensor cores' accumulation truncates.  So the leading terms (8 bits each) are summed 16 dims at a time into a zero
        // accumulator, and the parts are added in f32, which rounds; the other two terms, 2^-8 of the sum, stay in one accumulator.
        float acc[NT][4], small[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] = small[i][e] = 0.0f;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            const uint4* f = s_a + (mt * KS + ks) * 3 * 32 + lane;
            const uint4 a0 = f[0], a1 = f[32], a2 = f[64];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                mma_bf16(small[i], a2, b[i][ks][0], b[i][ks][1]);
                mma_bf16(small[i], a1, b[i][ks][0], b[i][ks][1]);
                float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma_bf16(part, a0, b[i][ks][0], b[i][ks][1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][e] += part[e];
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] += small[i][e];
        // rows n / n + 8 (queries), columns 2j, 2j + 1 (tokens) -> one row of consecutive tokens per store
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            *reinterpret_cast<float2*>(stage + n * kBiasPitch + 8 * i + 2 * j) = make_float2(acc[i][0], acc[i][1]);
            *reinterpret_cast<float2*>(stage + (n + 8) * kBiasPitch + 8 * i + 2 * j) = make_float2(acc[i][2], acc[i][3]);
        }
        __syncwarp();
        const int nr = min(16, rows - r0 - 16 * mt);
        OT* dst = bias + ((size_t)kvh * rows + r0 + 16 * mt) * kv_len + tok0;
        if (lane < ntok)
            for (int r = 0; r < nr; ++r) dst[(size_t)r * kv_len + lane] = from_f32<OT>(stage[r * kBiasPitch + lane] * c_t);
        __syncwarp();
    }
}

// Few query rows, and head dims that are not 32 times a power of two: one thread per token, the group's projected queries in
// shared memory.
template <typename OT>
__global__ void logit_bias_kernel(const float* __restrict__ rq, const uint8_t* __restrict__ signs,
                                  const uint16_t* __restrict__ norms, OT* __restrict__ bias, int hq, int hkv, int q_len,
                                  int D, int kv_len, int kv_stride, float scale_factor) {
    extern __shared__ float s_rq[];   // [g * q_len][D]
    const int kvh = blockIdx.y, g = hq / hkv;
    const int rows = g * q_len;
    for (int i = threadIdx.x; i < rows * D; i += blockDim.x) s_rq[i] = rq[(size_t)kvh * rows * D + i];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kv_len) return;
    const size_t row = (size_t)kvh * kv_stride + t;
    const uint32_t* sw = reinterpret_cast<const uint32_t*>(signs + row * (D / 8));
    const float c = f16_bits_to_f32(norms[row]) * scale_factor;
    for (int r = 0; r < rows; ++r) {
        float acc = 0.0f;
        for (int w = 0; w < D / 32; ++w) {
            const uint32_t bits = sw[w];
#pragma unroll 8
            for (int b = 0; b < 32; ++b) acc = fmaf(s_rq[r * D + w * 32 + b], ((bits >> b) & 1u) ? 1.0f : -1.0f, acc);
        }
        const int head = kvh * g + r / q_len, qi = r % q_len;
        bias[((size_t)head * q_len + qi) * kv_len + t] = from_f32<OT>(acc * c);
    }
}


// Query rows per call are limited by what the general kernel keeps in shared memory (all of them): the same for every shape.
constexpr size_t kBiasMaxQueryBytes = 200 * 1024;

template <typename OT, int W>
int launch_bias_mma(const float* rq, const uint8_t* signs, const uint16_t* norms, OT* bias, int rows, int hkv, int kv_len,
                    int kv_stride, float scale_factor, cudaStream_t s) {
    constexpr int NT = W <= 4 ? 4 : 2;   // 64 registers of signs at D = 128 and 256
    const int tiles = ((rows < kBiasRows ? rows : kBiasRows) + 15) / 16;
    const size_t smem = (size_t)tiles * (2 * W) * 3 * 32 * sizeof(uint4) + kBiasWarps * 16 * kBiasPitch * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(logit_bias_mma_kernel<OT, W, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_cuda_error(e); return TQB_ERR_CUDA; }
    const int per_cta = kBiasWarps * 8 * NT;
    dim3 grid((kv_len + per_cta - 1) / per_cta, hkv, (rows + kBiasRows - 1) / kBiasRows);
    logit_bias_mma_kernel<OT, W, NT><<<grid, kBiasWarps * 32, smem, s>>>(rq, signs, norms, bias, rows, kv_len, kv_stride, scale_factor);
    return check_launch(s);
}

template <typename OT>
int launch_bias(const float* rq, const uint8_t* signs, const uint16_t* norms, OT* bias, int hq, int hkv, int q_len, int D,
                int kv_len, int kv_stride, float scale_factor, cudaStream_t s) {
    const int rows = hq / hkv * q_len;
    // The MMAs pay for 16 rows and for expanding every sign.  One row: a thread per token is ahead at every dim (64 KV heads x 8,000
    // tokens: 32 dims 6.7 against 9.8 us, 128 dims 14.7 against 28 us, 256 dims 25 against 59 us); two rows: from 128 dims on
    // (26 against 29 us, 48 against 60 us); three: nowhere.
    const bool few = rows == 1 || (rows == 2 && D >= 128);
    switch (few ? 0 : D) {
        case 32: return launch_bias_mma<OT, 1>(rq, signs, norms, bias, rows, hkv, kv_len, kv_stride, scale_factor, s);
        case 64: return launch_bias_mma<OT, 2>(rq, signs, norms, bias, rows, hkv, kv_len, kv_stride, scale_factor, s);
        case 128: return launch_bias_mma<OT, 4>(rq, signs, norms, bias, rows, hkv, kv_len, kv_stride, scale_factor, s);
        case 256: return launch_bias_mma<OT, 8>(rq, signs, norms, bias, rows, hkv, kv_len, kv_stride, scale_factor, s);
        default: break;
    }
    const size_t smem = sizeof(float) * (size_t)rows * D;
    cudaError_t e = cudaFuncSetAttribute(logit_bias_kernel<OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_cuda_error(e); return TQB_ERR_CUDA; }
    logit_bias_kernel<OT><<<dim3((kv_len + 127) / 128, hkv), 128, smem, s>>>(rq, signs, norms, bias, hq, hkv, q_len, D, kv_len,
                                                                             kv_stride, scale_factor);
    return check_launch(s);
}

}  // namespace
}  // namespace tqb

using namespace tqb;

extern "C" int tqb_qjl_logit_bias(int32_t head_dim, const float* rq, const uint8_t* signs, const uint16_t* norms, void* bias,
                                  int32_t bias_dtype, int32_t num_q_heads, int32_t num_kv_heads, int32_t q_len, int32_t kv_len,
                                  int32_t kv_stride, tqb_stream_t stream) {
    TQB_NVTX_RANGE();
    if (head_dim <= 0 || head_dim % 32 != 0) return TQB_ERR_INVALID_DIMENSION;
    if (num_q_heads <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads != 0 || q_len <= 0) return TQB_ERR_INVALID_ARGUMENT;
    if (kv_len < 0 || kv_len > kv_stride) return TQB_ERR_RANGE_OUT_OF_BOUNDS;
    if (kv_len == 0) return TQB_OK;
    if (!rq || !signs || !norms || !bias) return TQB_ERR_NULL_POINTER;
    if ((uintptr_t)signs % 4) return TQB_ERR_MISALIGNED;
    const int g = num_q_heads / num_kv_heads;
    if (sizeof(float) * (size_t)g * q_len * head_dim > kBiasMaxQueryBytes) return TQB_ERR_TOO_LARGE;
    // src/cache/tq.rs:215-216: sqrt(pi/2) as f32 divided by sqrt(head_dim) in f32
    const float scale_factor = (float)sqrt(1.5707963267948966) / sqrtf((float)head_dim);
    cudaStream_t s = as_stream(stream);
#define TQB_BIAS(OT) launch_bias<OT>(rq, signs, norms, (OT*)bias, num_q_heads, num_kv_heads, q_len, head_dim, kv_len, kv_stride, scale_factor, s)
    if (bias_dtype == TQB_F32) return TQB_BIAS(float);
    if (bias_dtype == TQB_F16) return TQB_BIAS(__half);
    if (bias_dtype == TQB_BF16) return TQB_BIAS(__nv_bfloat16);
#undef TQB_BIAS
    return TQB_ERR_INVALID_ARGUMENT;
}
