// One 32-block of the all-outlier MaxNorm cache format quantized by ONE thread (in-register butterfly):
// the body of block_quantize_pqo_kernel, shared with the decode kernel, which appends the new token's K and
// V rows itself.  polar_quantize (src/cache/quantize_tensor.rs:40-176) with the scalar arithmetic of
// src/cache/cuda/kernels/tq_quant_kernel.cu:216-259; results are bit-identical to the general kernel.
#pragma once
#include "tqb_common.cuh"
#include "tqb_f32x2.cuh"

namespace tqb {

template <typename T>
__device__ __forceinline__ void load32(const T* p, float (&v)[32]);
template <>
__device__ __forceinline__ void load32<float>(const float* p, float (&v)[32]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float4 a = __ldg(reinterpret_cast<const float4*>(p) + k);
        v[4 * k] = a.x; v[4 * k + 1] = a.y; v[4 * k + 2] = a.z; v[4 * k + 3] = a.w;
    }
}
template <>
__device__ __forceinline__ void load32<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[32]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint4 r = __ldg(reinterpret_cast<const uint4*>(p) + k);
        uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[8 * k + 2 * i] = __uint_as_float(w[i] << 16);
            v[8 * k + 2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
}
template <>
__device__ __forceinline__ void load32<__half>(const __half* p, float (&v)[32]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint4 r = __ldg(reinterpret_cast<const uint4*>(p) + k);
        const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 f = __half22float2(h[i]);
            v[8 * k + 2 * i] = f.x;
            v[8 * k + 2 * i + 1] = f.y;
        }
    }
}

// 32 f32 values from 16-byte pieces in shared memory
__device__ __forceinline__ void unpack32(const unsigned char* p, float (&v)[32]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float4 r = *reinterpret_cast<const float4*>(p + 16 * k);
        v[4 * k] = r.x;
        v[4 * k + 1] = r.y;
        v[4 * k + 2] = r.z;
        v[4 * k + 3] = r.w;
    }
}

__device__ __forceinline__ void butterfly32_regs(float (&v)[32]) {
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if ((i & h) == 0) {
                float x = v[i], y = v[i + h];
                v[i] = x + y;
                v[i + h] = x - y;
            }
        }
    }
}

constexpr uint32_t kSignMask = 0xB1A6D4B2u;   // bit j set <=> sign j is -1 (precomputed/rotation.rs:16-20)


// Cell table for the boundary search of the small codebooks: cell k >> 8 of k = round(t * kCellScale + kCellHalf), 32
// cells of 0.138 - narrower than any gap between two boundaries (0.49), so a cell (widened by kCellSlop on both sides to
// absorb the rounding of k) holds at most one boundary:  code = below + (t > bnd), exactly the count of
// boundaries below t.  .x = that boundary (3e38 when the cell has none), .y = the number of boundaries under the cell.
// Stored [cell][lane]: the 32 look-ups of a warp instruction touch 32 different bank pairs (256 unreplicated cells met
// ~6 wavefronts a look-up).  |t| <= outer centroid (2.1573) < 2.2 by construction of the MaxNorm scale, so k stays inside.
constexpr int kCells = 32, kMaxCellBounds = 7;   // codebooks of up to eight entries
constexpr float kCellScale = 1856.0f;
constexpr float kCellHalf = 4096.0f;   // an integer, so that kCellHalf + 1.5 * 2^23 is exact
constexpr float kCellSlop = 1e-3f;
__device__ __forceinline__ void build_cell_table(const Codebook& cb, int n_bnd, float2* lut, int tid, int nthreads) {
    // (no division and no loop of unknown length: a launch of a few blocks is mostly this table, 3.0 -> 2.4 us for one row)
    constexpr float kStep = 256.0f / kCellScale, kLo = (-0.5f - kCellHalf) / kCellScale - kCellSlop, kHi = (255.5f - kCellHalf) / kCellScale + kCellSlop;
#pragma unroll 4
    for (int i = tid; i < kCells * 32; i += nthreads) {
        const float at = kStep * (float)(i >> 5), lo = at + kLo, hi = at + kHi;
        float bnd = 3.0e38f;
        float below = 0.0f;
#pragma unroll
        for (int k = 0; k < kMaxCellBounds; ++k) {
            const float b = k < n_bnd ? cb.b[k] : 3.0e38f;
            below += b < lo ? 1.0f : 0.0f;
            bnd = (b >= lo && b <= hi) ? b : bnd;
        }
        lut[i] = make_float2(bnd, below);
    }
}

// v (x, 16-byte aligned): the block's 32 input values.  w: packed codes (4 * BITS bytes, LSB-first), returns the
// f32 scale (before the outlier sign).  cb: the codebook.  lut: the caller's lane of the cell table in
// shared memory (build_cell_table, + lane), or nullptr for the register bisection.  TABLE: the codebook is not the
// 4-bit uniform grid even when BITS = 4 (codes of a narrower codebook stored at BITS width); needs lut.
// Two values per instruction throughout (elements i and i + 16); the codes are whole f32 numbers that are packed by
// multiply-adds (16 or 24 bits of them are exact) instead of a mask, a shift and an add each.
template <int BITS, bool TABLE = false>
__device__ __forceinline__ float pqo_quantize_values(const float (&v)[32], const Codebook& cb, float outer_centroid, uint32_t (&w)[4],
                                                     const float2* lut = nullptr) {
    const float inv_sqrt = 1.0f / sqrtf((float)kBlock);
    const float R = cb.c[(1 << BITS) - 1];
    const float inv_step = 15.0f / (2.0f * R);
    const float kMagic = 12582912.0f;          // 1.5 * 2^23
    F2 p[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) p[i] = f2(v[i], v[i + 16]);
    butterfly32_pairs(p);
    float amax_w = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 t = halves(p[i]);
        amax_w = fmaxf(amax_w, fmaxf(fabsf(t.x), fabsf(t.y)));
    }
    const float amax = amax_w * inv_sqrt;          // rounding is monotone: equals max_i |W_i * inv_sqrt|
    const float raw = __fdiv_rn(amax, outer_centroid);
    const float scale = raw > kMinNorm ? raw : kMinNorm;
    const float r = __frcp_rn(scale);
    // (mag, mag) with the signs of elements i and i + 16
    auto signed2 = [](F2 pp, F2 pn, F2 np, F2 nn, int i) {
        return ((kSignMask >> i) & 1u) ? (((kSignMask >> (i + 16)) & 1u) ? nn : np) : (((kSignMask >> (i + 16)) & 1u) ? pn : pp);
    };
    F2 c[16];   // the codes
    if (BITS == 4 && !TABLE) {
        const float cpos = (inv_sqrt * r) * inv_step, cneg = -cpos;
        const F2 pp = f2(cpos, cpos), pn = f2(cpos, cneg), np = f2(cneg, cpos), nn = f2(cneg, cneg);
        float far = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const F2 u = fma2(p[i], signed2(pp, pn, np, nn, i), f2(7.5f));
            c[i] = add2(add2(u, f2(kMagic)), f2(-kMagic));
            const float2 d = halves(sub2(u, c[i]));
            far = fmaxf(far, fmaxf(fabsf(d.x), fabsf(d.y)));
        }
        if (far > 0.49998f) {   // rare: exact division and the f32 boundary table
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 v2 = halves(p[i]);
                const float t0 = __fdiv_rn((v2.x * inv_sqrt) * (((kSignMask >> i) & 1u) ? -1.0f : 1.0f), scale);
                const float t1 = __fdiv_rn((v2.y * inv_sqrt) * (((kSignMask >> (i + 16)) & 1u) ? -1.0f : 1.0f), scale);
                float c0 = 0.0f, c1 = 0.0f;
#pragma unroll
                for (int k = 0; k < 15; ++k) {
                    c0 += (t0 > cb.b[k]) ? 1.0f : 0.0f;
                    c1 += (t1 > cb.b[k]) ? 1.0f : 0.0f;
                }
                c[i] = f2(c0, c1);
            }
        }
    } else {
        const F2 pp = f2(inv_sqrt, inv_sqrt), pn = f2(inv_sqrt, -inv_sqrt), np = f2(-inv_sqrt, inv_sqrt), nn = f2(-inv_sqrt, -inv_sqrt);
        const F2 r2 = f2(r), ns2 = f2(-scale);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const F2 rot = mul2(p[i], signed2(pp, pn, np, nn, i));
            const F2 q = mul2(rot, r2);
            const F2 rem = fma2(q, ns2, rot);
            // rot / scale, correctly rounded: Markstein's correction of a quotient by its remainder (IBM J. Res. Dev. 34, 1990),
            // r being the correctly rounded reciprocal
            const float2 t = halves(fma2(rem, r2, q));
            if (lut != nullptr) {
                const float2 y = halves(fma2(q, f2(kCellScale), f2(kCellHalf + kMagic)));   // k in the low mantissa bits
                // byte offset of [k >> 8][lane]: a cell row is 256 bytes
                const unsigned char* l = reinterpret_cast<const unsigned char*>(lut);
                const float2 e0 = *reinterpret_cast<const float2*>(l + (__float_as_uint(y.x) & ((kCells - 1) << 8)));
                const float2 e1 = *reinterpret_cast<const float2*>(l + (__float_as_uint(y.y) & ((kCells - 1) << 8)));
                c[i] = add2(f2(e0.y, e1.y), f2(t.x > e0.x ? 1.0f : 0.0f, t.y > e1.x ? 1.0f : 0.0f));
            } else {
                // bisection over the 7 boundaries (constant bank operands)
                float code[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float th = h == 0 ? t.x : t.y;
                    const bool p1 = th > cb.b[3];
                    const bool p2 = th > (p1 ? cb.b[5] : cb.b[1]);
                    const float t3 = p1 ? (p2 ? cb.b[6] : cb.b[4]) : (p2 ? cb.b[2] : cb.b[0]);
                    code[h] = (p1 ? 4.0f : 0.0f) + (p2 ? 2.0f : 0.0f) + (th > t3 ? 1.0f : 0.0f);
                }
                c[i] = f2(code[0], code[1]);
            }
        }
    }
    if (BITS == 4) {
        uint32_t h[2][4];   // [codes 0..15 | 16..31][four codes in the low 16 bits]
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            F2 a = fma2(c[4 * m + 3], f2(16.0f), c[4 * m + 2]);
            a = fma2(a, f2(16.0f), c[4 * m + 1]);
            a = add2(fma2(a, f2(16.0f), c[4 * m]), f2(8388608.0f));
            const float2 t = halves(a);
            h[0][m] = __float_as_uint(t.x);
            h[1][m] = __float_as_uint(t.y);
        }
        w[0] = __byte_perm(h[0][0], h[0][1], 0x5410);
        w[1] = __byte_perm(h[0][2], h[0][3], 0x5410);
        w[2] = __byte_perm(h[1][0], h[1][1], 0x5410);
        w[3] = __byte_perm(h[1][2], h[1][3], 0x5410);
    } else {
        F2 a = c[7], b = c[15];   // eight codes, 24 bits: below 2^24, exact
#pragma unroll
        for (int i = 6; i >= 0; --i) {
            a = fma2(a, f2(8.0f), c[i]);
            b = fma2(b, f2(8.0f), c[i + 8]);
        }
        const float2 ta = halves(a), tb = halves(b);
        const uint32_t c0 = __float2uint_rz(ta.x), c1 = __float2uint_rz(tb.x), c2 = __float2uint_rz(ta.y), c3 = __float2uint_rz(tb.y);
        w[0] = c0 | (c1 << 24);
        w[1] = (c1 >> 8) | (c2 << 16);
        w[2] = (c2 >> 16) | (c3 << 8);
        w[3] = 0u;
    }
    return scale;
}

template <typename T, int BITS, bool TABLE = false>
__device__ __forceinline__ float pqo_quantize_block(const T* x, const Codebook& cb, float outer_centroid, uint32_t (&w)[4],
                                                    const float2* lut = nullptr) {
    float v[32];
    load32<T>(x, v);
    return pqo_quantize_values<BITS, TABLE>(v, cb, outer_centroid, w, lut);
}

}  // namespace tqb
