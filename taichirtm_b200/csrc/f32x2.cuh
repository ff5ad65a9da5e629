// Packed FP32 arithmetic (two IEEE operations per instruction) that keeps the
// operation order of the scalar kernels bit for bit.
#pragma once
#include <cuda_runtime.h>

namespace rtm {

// ---- packed FP32 pairs.  add / sub are the packed IEEE operations.  A product
// is fma(a, b, -0.0) with the -0.0 opaque to the compiler (a kernel argument):
// exactly the rounded product, sign of zero included, and unlike mul.f32x2 it
// cannot be fused with a following addition (ptxas 12.9 does fuse those, even
// with -fmad=false: 68,271 of 524,288 random chains f + (d b)(a + b) then
// differ from the IEEE sequence; 0 with this form).
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float f2_lo(f2 a) {
    return __uint_as_float((unsigned)a);
}
__device__ __forceinline__ float f2_hi(f2 a) {
    return __uint_as_float((unsigned)(a >> 32));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b, f2 neg_zero) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(neg_zero));
    return d;
}

// Two lanes of arithmetic on an f2: packed instructions, or two scalar ones (for
// kernels that lose more to the even register pairs than packing saves).
template <bool PACKED>
struct Pairs {
    static __device__ __forceinline__ f2 pack(float lo, float hi) { return f2_pack(lo, hi); }
    static __device__ __forceinline__ f2 add(f2 a, f2 b) { return f2_add(a, b); }
    static __device__ __forceinline__ f2 sub(f2 a, f2 b) { return f2_sub(a, b); }
    static __device__ __forceinline__ f2 mul(f2 a, f2 b, f2 neg_zero) { return f2_mul(a, b, neg_zero); }
};
template <>
struct Pairs<false> {
    static __device__ __forceinline__ f2 pack(float lo, float hi) { return (f2)__float_as_uint(hi) << 32 | __float_as_uint(lo); }
    static __device__ __forceinline__ f2 add(f2 a, f2 b) { return pack(f2_lo(a) + f2_lo(b), f2_hi(a) + f2_hi(b)); }
    static __device__ __forceinline__ f2 sub(f2 a, f2 b) { return pack(f2_lo(a) - f2_lo(b), f2_hi(a) - f2_hi(b)); }
    static __device__ __forceinline__ f2 mul(f2 a, f2 b, f2) { return pack(f2_lo(a) * f2_lo(b), f2_hi(a) * f2_hi(b)); }
};

}  // namespace rtm
