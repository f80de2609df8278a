// Correctly rounded float arithmetic on two values at a time.
//
// sm_103a's packed f32x2 instructions do two float operations per issue slot
// and thread, which is what the neighbour passes are bound by.  Each lane of
// a pair rounds like the scalar operation.  Two rules keep it that way:
//  * ptxas fuses a packed multiply whose result goes into a packed add, so
//    sums of products are written as add2 below, a packed fma with a factor
//    of one that the compiler cannot see (`one`, from the step constants);
//  * the square root and the quotient are the textbook fma sequences
//    (P. Markstein, "Computation of elementary functions on the IBM RISC
//    System/6000 processor", IBM J. R&D 34, 1990): an approximation, its
//    exact residual by fma, and one correction, which rounds correctly.
//    They share one reciprocal square root.  tests/test_gpu_exact_pair.py
//    checks the root against sqrtf for every float in [1e-14, 1.1e4], and the
//    quotient against IEEE division for every significand of the dividend, at
//    three exponents, with 4,096 roots and with each of the 449 of that range
//    whose inverse is not the correctly rounded one.  (With the correctly
//    rounded inverse the last correction rounds correctly: Markstein's theorem.)
#pragma once

#include <cuda_runtime.h>

namespace pbf {

__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }

// a b and a + b, two at a time (`one`: 1.0f that the compiler cannot see).
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b, float one) {
    return __ffma2_rn(a, both(one), b);
}
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
// a - b, where b is no product.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// root = sqrt(x), correctly rounded, and inv = 1 / root to within an ulp, such
// that quotient(a, root, inv) rounds correctly, for x in [1e-14, 1e4].
__device__ __forceinline__ void root_and_inverse(float2 x, float2& root, float2& inv) {
    const float2 y = make_float2(rsqrt_approx(x.x), rsqrt_approx(x.y));
    const float2 s = mul2(x, y);
    const float2 d = __ffma2_rn(neg2(s), s, x);  // x - s s, exact
    root = __ffma2_rn(d, mul2(y, both(0.5f)), s);
    // 1 / root = u (1 + e + e^2 + ...) with e = 1 - root u.  u lies above the
    // approximation, so that the one root whose inverse is all but halfway
    // between two floats (its significand all ones) rounds to the upper one;
    // with e alone, two other significands get an inverse one ulp off.
    const float2 u = mul2(y, both(1.0000002384185791f));
    const float2 e = __ffma2_rn(neg2(root), u, both(1.0f));
    inv = __ffma2_rn(__ffma2_rn(e, e, e), u, u);
}

// a / b, correctly rounded, with inv = 1 / b correctly rounded or from
// root_and_inverse; a and the quotient far from the ends of the exponent range
// (or a = 0).
__device__ __forceinline__ float2 quotient(float2 a, float2 b, float2 inv) {
    const float2 q = mul2(a, inv);
    const float2 r = __ffma2_rn(neg2(b), q, a);  // a - b q, exact
    return __ffma2_rn(r, inv, q);
}

}  // namespace pbf
