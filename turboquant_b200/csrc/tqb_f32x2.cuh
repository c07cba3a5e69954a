// Two f32 operations per instruction (add / mul / fma.rn.f32x2, sm_100): each half rounds like its scalar twin, so the
// bit-exact paths may use them.  x - y is fma(y, -1, x): one rounding, the same bits.
#pragma once
#include <stdint.h>

namespace tqb {

struct F2 {
    unsigned long long u;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ float2 halves(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.u));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, f2(-1.0f), a); }

// 32-point Walsh-Hadamard butterfly over p[i] = (v[i], v[i + 16]), stages in the order h = 1, 2, 4, 8, 16
// (src/cache/wht_tensor.rs:44-59): the same operand pairs as the scalar loop.
__device__ __forceinline__ void butterfly32_pairs(F2 (&p)[16]) {
#pragma unroll
    for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if ((i & h) == 0) {
                const F2 x = p[i], y = p[i + h];
                p[i] = add2(x, y);
                p[i + h] = sub2(x, y);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 t = halves(p[i]);
        p[i] = f2(t.x + t.y, t.x - t.y);
    }
}

}  // namespace tqb
