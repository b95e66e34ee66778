// Packed pairs of floats for the FP32 pipe's two-wide instructions (fma / mul / add .f32x2: two
// independent IEEE operations per issued instruction), and the polynomial arctangent that the
// brute-force kernels evaluate on them.
//
// The brute-force loops (every query against every triangle or boundary row) are bound by instruction
// issue: their arithmetic is a third or less of what the FP32 pipe could take, the rest of the issue
// slots going to the arctangent's range reduction and division and to comparisons. Two records per
// instruction halve the slots of the arithmetic.
#pragma once

#include "gwnb_internal.cuh"

namespace gwnb {
namespace x2 {

struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 pack(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2 both(float x) { return pack(x, x); }
__device__ __forceinline__ void unpack(f2 a, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ f2 add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// Two packed values by one 128-bit read-only load.
__device__ __forceinline__ void load(float4 const *p, f2 &a, f2 &b) {
    ulonglong2 const v = __ldg(reinterpret_cast<ulonglong2 const *>(p));
    a.v = v.x;
    b.v = v.y;
}

// Reciprocal square root and reciprocal by the hardware's approximation alone (relative error below
// 2^-22; denormals count as zero, so their results are infinite and what they reach becomes NaN).
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f2 rsqrt(f2 a) {
    float lo, hi;
    unpack(a, lo, hi);
    return pack(rsqrt_ftz(lo), rsqrt_ftz(hi));
}

// a / b from the approximate reciprocal and one correction: the arctangent's arguments of far triangles
// all have the same denominator (4), so an uncorrected reciprocal's error would be common to all of
// them instead of averaging out.
__device__ __forceinline__ f2 divide(f2 a, f2 b) {
    float lo, hi;
    unpack(b, lo, hi);
    f2 const r = pack(rcp_ftz(lo), rcp_ftz(hi));
    f2 const t = mul(a, r);
    return fma(t, fma(mul(b, both(-1.0f)), r, both(1.0f)), t);
}
// 1 / sqrt(x), the approximation with one Newton step.
__device__ __forceinline__ f2 rsqrt_newton(f2 x) {
    f2 const y = rsqrt(x);
    f2 const e = fma(mul(mul(x, y), both(-0.5f)), y, both(0.5f)); // (1 - x y^2) / 2
    return fma(y, e, y);
}

__device__ __forceinline__ f2 dot(f2 ax, f2 ay, f2 az, f2 bx, f2 by, f2 bz) {
    return fma(az, bz, fma(ay, by, mul(ax, bx)));
}

// atan(t) = t + t u q(u), u = t^2, on |t| <= 1/2: q of degree 4 by weighted least squares iterated
// towards equal ripple (relative error 5.4e-9; evaluated in float 6.5e-8 at most, 2.5e-8 rms, as a
// correctly rounded result has).
__device__ __forceinline__ f2 atan_half(f2 t) {
    f2 const u = mul(t, t);
    f2 q = fma(both(-0.05132567882537842f), u, both(0.10159996896982193f));
    q = fma(q, u, both(-0.14175006747245789f));
    q = fma(q, u, both(0.19994226098060608f));
    q = fma(q, u, both(-0.3333323299884796f));
    return fma(mul(t, u), q, t);
}

// The same on |t| <= 1: q of degree 7 (relative error 1.7e-8; in float 8.3e-8 at most, 2.9e-8 rms).
__device__ __forceinline__ f2 atan_one(f2 t) {
    f2 const u = mul(t, t);
    f2 q = fma(both(0.002920565428212285f), u, both(-0.01636742241680622f));
    q = fma(q, u, both(0.04321104288101196f));
    q = fma(q, u, both(-0.07552145421504974f));
    q = fma(q, u, both(0.10665972530841827f));
    q = fma(q, u, both(-0.14211046695709229f));
    q = fma(q, u, both(0.19993771612644196f));
    q = fma(q, u, both(-0.33333152532577515f));
    return fma(mul(t, u), q, t);
}

} // namespace x2
} // namespace gwnb
