// pairs.cuh — arithmetic on pairs of floats.
//
// fma / mul / add.rn.f32x2 (sm_100) do two single-precision operations in one
// instruction, each rounded as the scalar one is. The particle kernels were
// bound by instruction issue (63 % of the issue slots; 49 % with pairs), so the
// stencil sums carry a vector's x and y as one pair.
#pragma once
#include "mat3.cuh"

namespace empm {

// ---- pairs of floats: one instruction for two multiply-adds (sm_100) ------
struct F2 { unsigned long long v; };

__device__ __forceinline__ F2 f2_make(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 f2_both(float x) { return f2_make(x, x); }
__device__ __forceinline__ void f2_split(F2 a, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ float f2_x(F2 a) { float x, y; f2_split(a, x, y); return x; }
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// A 3-vector as an (x, y) pair and z.
struct P3 { F2 xy; float z; };
__device__ __forceinline__ P3 p3(F2 xy, float z) { P3 r; r.xy = xy; r.z = z; return r; }
__device__ __forceinline__ P3 p3_zero() { return p3(f2_make(0.f, 0.f), 0.f); }
// scalars that multiply a P3: the pair (s, s); its low half serves z
__device__ __forceinline__ P3 p3_mul(F2 s, const P3& a) { return p3(f2_mul(s, a.xy), f2_x(s) * a.z); }
__device__ __forceinline__ P3 p3_fma(F2 s, const P3& a, const P3& b) {
    return p3(f2_fma(s, a.xy, b.xy), fmaf(f2_x(s), a.z, b.z));
}
__device__ __forceinline__ P3 p3_add(const P3& a, const P3& b) { return p3(f2_add(a.xy, b.xy), a.z + b.z); }

}  // namespace empm
