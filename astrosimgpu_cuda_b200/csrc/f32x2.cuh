// f32x2.cuh -- sm_100a's two-float instructions: one issue slot, each half rounded to
// nearest as the scalar instruction rounds it (denormals kept).
#pragma once

#include "model.cuh"

namespace astrosim {

struct f32x2 {
    unsigned long long v;
};
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ float lo2(f32x2 a) { return __uint_as_float(static_cast<u32>(a.v)); }
__device__ __forceinline__ float hi2(f32x2 a) { return __uint_as_float(static_cast<u32>(a.v >> 32)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// h6 (k1 + 2 k2 + 2 k3 + k4); the products by 2 are exact
__device__ __forceinline__ f32x2 rk4_sum(f32x2 h6, f32x2 k1, f32x2 k2, f32x2 k3, f32x2 k4) {
    const f32x2 two = both(2.0f);
    return mul2(h6, add2(fma2(two, k3, fma2(two, k2, k1)), k4));
}

}  // namespace astrosim
