// Near-field (exact solid angle) and far-field (Taylor) terms of the winding number, shared by the
// query and adjoint translation units.
//
// Solid angle of a triangle seen from q: the Van Oosterom-Strackee formula in unnormalised form,
// tan(Omega/2) = a.(e1 x e2) / (|a||b||c| + (a.b)|c| + (a.c)|b| + (b.c)|a|) with a = v0 - q,
// b = a + e1, c = a + e2; it equals smallgwn's unit-vector form
// (detail/gwn_query_geometry_impl.cuh:16-45) and keeps its conventions: zero when the query sits on
// a vertex or the numerator vanishes.
//
// Far field of one child slot: smallgwn's expansion (detail/gwn_query_winding_impl.cuh:193-327)
// about the slot's area-weighted centre P with r = q - P: order 0 -(r.N)/|r|^3, order 1
// (tr M - 3 r^T M r / |r|^2) / |r|^3 with M_ij = sum n_i (c - P)_j, order 2 the third-moment terms.
#pragma once

#include "gwnb_f32x2.cuh"
#include "gwnb_internal.cuh"

namespace gwnb {
namespace field {

constexpr float k_pi_f = 3.14159265358979323846f;

// The head of a sidecar pair and the acceptance test of its two children. |q - P|^2 has one fixed
// rounding pattern (rx * rx rounded, then two fused multiply-adds, r = q - P rounded per component), so
// that every traversal (value, gradient, statistics, adjoint, batched) and the oracle's C restatement
// take identical accept / descend decisions for identical inputs. The rule is smallgwn's
// (detail/gwn_query_winding_impl.cuh:186-189): descend iff !(|q - P|^2 > 0) or |q - P|^2 <= r^2 beta^2
// (the product rounded on its own); a NaN bound therefore accepts, as there.
struct pair_head {
    x2::f2 rx, ry, rz, q2; // r = q - P and |r|^2
    bool valid0, valid1;   // slots that hold a child
    bool far0, far1;       // ... and pass the acceptance test
};
__device__ __forceinline__ pair_head load_head(float4 const *w, x2::f2 qx, x2::f2 qy, x2::f2 qz, float beta2) {
    using namespace x2;
    pair_head h;
    f2 px, py, pz, r2;
    load(w, px, py);
    load(w + 1, pz, r2);
    h.rx = add(qx, px);
    h.ry = add(qy, py);
    h.rz = add(qz, pz);
    h.q2 = dot(h.rx, h.ry, h.rz, h.rx, h.ry, h.rz);
    float q0, q1, b0, b1, v0, v1;
    unpack(h.q2, q0, q1);
    unpack(mul(r2, both(beta2)), b0, b1);
    unpack(r2, v0, v1);
    h.valid0 = !(v0 < 0.0f);
    h.valid1 = !(v1 < 0.0f);
    h.far0 = h.valid0 && q0 > 0.0f && !(q0 <= b0);
    h.far1 = h.valid1 && q1 > 0.0f && !(q1 <= b1);
    return h;
}

// a = v0 - q, e1, e2 edges, n = e1 x e2.
__device__ __forceinline__ float solid_angle_plain(float ax, float ay, float az, float e1x, float e1y,
                                                   float e1z, float e2x, float e2y, float e2z,
                                                   float nx, float ny, float nz) {
    float const bx = ax + e1x, by = ay + e1y, bz = az + e1z;
    float const cx = ax + e2x, cy = ay + e2y, cz = az + e2z;
    float const a2 = ax * ax + ay * ay + az * az;
    float const b2 = bx * bx + by * by + bz * bz;
    float const c2 = cx * cx + cy * cy + cz * cz;
    float const la = sqrtf(a2), lb = sqrtf(b2), lc = sqrtf(c2);
    if (la == 0.0f || lb == 0.0f || lc == 0.0f)
        return 0.0f;
    float const num = ax * nx + ay * ny + az * nz;
    if (num == 0.0f)
        return 0.0f;
    float const ab = ax * bx + ay * by + az * bz;
    float const ac = ax * cx + ay * cy + az * cz;
    float const bc = bx * cx + by * cy + bz * cz;
    float const den = la * lb * lc + ab * lc + ac * lb + bc * la;
    return 2.0f * atan2f(num, den);
}

// Error-free transformations (Dekker / Ogita-Rump-Oishi "Accurate sum and dot product", 2005).
__device__ __forceinline__ void two_prod(float a, float b, float &p, float &e) {
    p = a * b;
    e = fmaf(a, b, -p);
}
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = a + b;
    float const z = s - a;
    e = (a - (s - z)) + (b - z);
}
// Compensated dot product of length 3 (Dot2).
__device__ __forceinline__ float dot3_comp(float a0, float a1, float a2, float b0, float b1, float b2) {
    float p, s, h, r, q;
    two_prod(a0, b0, p, s);
    two_prod(a1, b1, h, r);
    two_sum(p, h, p, q);
    s += q + r;
    two_prod(a2, b2, h, r);
    two_sum(p, h, p, q);
    s += q + r;
    return p + s;
}

// FP64 evaluation of one (query, triangle) pair over the same float record (b = a + e1 and
// c = a + e2 are exact in double), for pairs whose numerator and denominator both cancel.
__device__ __forceinline__ float solid_angle_f64_fallback(float ax, float ay, float az, float e1x,
                                                          float e1y, float e1z, float e2x, float e2y,
                                                          float e2z, unsigned long long *fp64_count) {
    if (fp64_count != nullptr)
        atomicAdd(fp64_count, 1ull);
    double const dax = ax, day = ay, daz = az;
    double const dbx = dax + e1x, dby = day + e1y, dbz = daz + e1z;
    double const dcx = dax + e2x, dcy = day + e2y, dcz = daz + e2z;
    double const dla = sqrt(dax * dax + day * day + daz * daz);
    double const dlb = sqrt(dbx * dbx + dby * dby + dbz * dbz);
    double const dlc = sqrt(dcx * dcx + dcy * dcy + dcz * dcz);
    double const dnx = static_cast<double>(e1y) * e2z - static_cast<double>(e1z) * e2y;
    double const dny = static_cast<double>(e1z) * e2x - static_cast<double>(e1x) * e2z;
    double const dnz = static_cast<double>(e1x) * e2y - static_cast<double>(e1y) * e2x;
    double const dnum = dax * dnx + day * dny + daz * dnz;
    if (dnum == 0.0)
        return 0.0f;
    double const dden = dla * dlb * dlc + (dax * dbx + day * dby + daz * dbz) * dlc +
                        (dax * dcx + day * dcy + daz * dcz) * dlb +
                        (dbx * dcx + dby * dcy + dbz * dcz) * dla;
    return static_cast<float>(2.0 * atan2(dnum, dden));
}

// Exact-batch form: the plain FP32 evaluation, except that pairs with both |num| and |den| below
// |a||b||c| / 16 -- a query within a small angle of an edge's line or at a vertex, where FP32
// cancellation leaves errors up to ~1e-3 -- are evaluated in FP64. On near-surface query sets
// about 0.1 pairs per query take that branch.
constexpr float k_exact_guard = 1.0f / 16.0f;

__device__ __forceinline__ float solid_angle_guarded(float ax, float ay, float az, float e1x, float e1y,
                                                     float e1z, float e2x, float e2y, float e2z,
                                                     float nx, float ny, float nz) {
    float const bx = ax + e1x, by = ay + e1y, bz = az + e1z;
    float const cx = ax + e2x, cy = ay + e2y, cz = az + e2z;
    float const a2 = ax * ax + ay * ay + az * az;
    float const b2 = bx * bx + by * by + bz * bz;
    float const c2 = cx * cx + cy * cy + cz * cz;
    if (a2 == 0.0f || b2 == 0.0f || c2 == 0.0f)
        return 0.0f;
    // lengths as x * rsqrt(x) (within 2 ulp of the rounded square root): the brute-force batch
    // evaluates every pair, and the pairs it cannot take in float go to the FP64 branch below
    float const la = a2 * rsqrtf(a2), lb = b2 * rsqrtf(b2), lc = c2 * rsqrtf(c2);
    float const num = ax * nx + ay * ny + az * nz;
    float const labc = la * lb * lc;
    float const den = labc + (ax * bx + ay * by + az * bz) * lc + (ax * cx + ay * cy + az * cz) * lb +
                      (bx * cx + by * cy + bz * cz) * la;
    float const lim = k_exact_guard * labc;
    if (fabsf(num) < lim && fabsf(den) < lim)
        return solid_angle_f64_fallback(ax, ay, az, e1x, e1y, e1z, e2x, e2y, e2z, nullptr);
    if (num == 0.0f)
        return 0.0f;
    return 2.0f * atan2f(num, den);
}

// Compensated near field (Taylor traversal): the two atan2 arguments -- the triple product
// a.(e1 x e2) and the denominator's sum |a||b||c| + (a.b)|c| + (a.c)|b| + (b.c)|a| -- as compensated
// (Dot2) sums; pairs whose numerator and denominator are both below threshold * |a||b||c| take the
// FP64 evaluation. The rounding of b = a + e1 and c = a + e2 themselves bounds what compensation can
// recover (the FP64 branch removes it), so the three inner dot products stay plain FP32.
__device__ __forceinline__ float solid_angle_comp(float ax, float ay, float az, float e1x, float e1y,
                                                  float e1z, float e2x, float e2y, float e2z, float nx,
                                                  float ny, float nz, float threshold,
                                                  unsigned long long *fp64_count) {
    // Lengths are sums of squares (no cancellation): plain FP32. n = e1 x e2 is the record's.
    float const bx = ax + e1x, by = ay + e1y, bz = az + e1z;
    float const cx = ax + e2x, cy = ay + e2y, cz = az + e2z;
    float const la = sqrtf(ax * ax + ay * ay + az * az);
    float const lb = sqrtf(bx * bx + by * by + bz * bz);
    float const lc = sqrtf(cx * cx + cy * cy + cz * cz);
    if (la == 0.0f || lb == 0.0f || lc == 0.0f)
        return 0.0f;
    float const num = dot3_comp(ax, ay, az, nx, ny, nz);
    float const ab = ax * bx + ay * by + az * bz;
    float const ac = ax * cx + ay * cy + az * cz;
    float const bc = bx * cx + by * cy + bz * cz;
    float const labc = la * lb * lc;
    float const den = labc + dot3_comp(ab, ac, bc, lc, lb, la);
    float const scale = labc;
    if (fabsf(den) < threshold * scale && fabsf(num) < threshold * scale)
        return solid_angle_f64_fallback(ax, ay, az, e1x, e1y, e1z, e2x, e2y, e2z, fp64_count);
    if (num == 0.0f)
        return 0.0f;
    return 2.0f * atan2f(num, den);
}

// Gradient of the solid angle w.r.t. the query (Biot-Savart form), as smallgwn's
// gwn_gradient_solid_angle_triangle_impl (detail/gwn_query_winding_impl.cuh:21-60).
__device__ __forceinline__ float3 solid_angle_grad(float ax, float ay, float az, float e1x, float e1y,
                                                   float e1z, float e2x, float e2y, float e2z) {
    float3 const g[3] = {make_float3(ax, ay, az), make_float3(ax + e1x, ay + e1y, az + e1z),
                         make_float3(ax + e2x, ay + e2y, az + e2z)};
    float l[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        l[i] = sqrtf(g[i].x * g[i].x + g[i].y * g[i].y + g[i].z * g[i].z);
    if (l[0] == 0.0f || l[1] == 0.0f || l[2] == 0.0f)
        return make_float3(0.0f, 0.0f, 0.0f);
    float3 h[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        h[i] = make_float3(g[i].x / l[i], g[i].y / l[i], g[i].z / l[i]);
    float3 r = make_float3(0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        int const i = e, j = (e + 1) % 3;
        float3 const cr = make_float3(g[i].y * g[j].z - g[i].z * g[j].y, g[i].z * g[j].x - g[i].x * g[j].z,
                                      g[i].x * g[j].y - g[i].y * g[j].x);
        float const cs = cr.x * cr.x + cr.y * cr.y + cr.z * cr.z;
        if (cs == 0.0f)
            continue;
        float const sc = ((g[i].x - g[j].x) * (h[i].x - h[j].x) + (g[i].y - g[j].y) * (h[i].y - h[j].y) +
                          (g[i].z - g[j].z) * (h[i].z - h[j].z)) /
                         cs;
        r.x += sc * cr.x;
        r.y += sc * cr.y;
        r.z += sc * cr.z;
    }
    return r;
}

// Derivatives of the solid angle with respect to the three vertex offsets a = v0 - q, b = v1 - q,
// c = v2 - q. With Omega = 2 atan2(N, D), N = a.(b x c) and D = |a||b||c| + (a.b)|c| + (a.c)|b| +
// (b.c)|a|: dOmega = 2 (D dN - N dD) / (N^2 + D^2), where
//   dN/da = b x c,  dN/db = c x a,  dN/dc = a x b,
//   dD/da = a^ (|b||c| + b.c) + b|c| + c|b|  (and cyclically for b, c).
// The derivative with respect to the query is -(d/da + d/db + d/dc). Zero when the query sits on a
// vertex or N = D = 0.
struct vertex_grad {
    float3 a, b, c;
};

__device__ __forceinline__ vertex_grad solid_angle_vertex_grad(float ax, float ay, float az, float e1x,
                                                               float e1y, float e1z, float e2x, float e2y,
                                                               float e2z) {
    vertex_grad r{};
    float const bx = ax + e1x, by = ay + e1y, bz = az + e1z;
    float const cx = ax + e2x, cy = ay + e2y, cz = az + e2z;
    float const la = sqrtf(ax * ax + ay * ay + az * az);
    float const lb = sqrtf(bx * bx + by * by + bz * bz);
    float const lc = sqrtf(cx * cx + cy * cy + cz * cz);
    if (la == 0.0f || lb == 0.0f || lc == 0.0f)
        return r;
    // cross products b x c, c x a, a x b
    float const bcx = by * cz - bz * cy, bcy = bz * cx - bx * cz, bcz = bx * cy - by * cx;
    float const cax = cy * az - cz * ay, cay = cz * ax - cx * az, caz = cx * ay - cy * ax;
    float const abx = ay * bz - az * by, aby = az * bx - ax * bz, abz = ax * by - ay * bx;
    float const N = ax * bcx + ay * bcy + az * bcz;
    float const dab = ax * bx + ay * by + az * bz;
    float const dac = ax * cx + ay * cy + az * cz;
    float const dbc = bx * cx + by * cy + bz * cz;
    float const D = la * lb * lc + dab * lc + dac * lb + dbc * la;
    float const s = N * N + D * D;
    if (!(s > 0.0f))
        return r;
    float const kD = 2.0f * D / s;
    float const kN = 2.0f * N / s;
    float const fa = (lb * lc + dbc) / la, fb = (la * lc + dac) / lb, fc = (la * lb + dab) / lc;
    r.a.x = kD * bcx - kN * (fa * ax + bx * lc + cx * lb);
    r.a.y = kD * bcy - kN * (fa * ay + by * lc + cy * lb);
    r.a.z = kD * bcz - kN * (fa * az + bz * lc + cz * lb);
    r.b.x = kD * cax - kN * (fb * bx + ax * lc + cx * la);
    r.b.y = kD * cay - kN * (fb * by + ay * lc + cy * la);
    r.b.z = kD * caz - kN * (fb * bz + az * lc + cz * la);
    r.c.x = kD * abx - kN * (fc * cx + ax * lb + bx * la);
    r.c.y = kD * aby - kN * (fc * cy + ay * lb + by * la);
    r.c.z = kD * abz - kN * (fc * cz + az * lb + bz * la);
    return r;
}

// Far-field Taylor terms of the two children of a sidecar pair: smallgwn's expansion
// (gwn_query_winding_impl.cuh:193-327) on the folded coefficients the moment refit writes. r = q - P,
// n = r / |r|; the quadratic form M' over xx yy zz xy yz zx, the cubic form K over xxx yyy zzz xxy xxz yyx
// yyz zzx zzy xyz:
//   w = -(n.N) / |r|^2 + n^T M' n / |r|^3 + K(n,n,n) / |r|^4.
// With Grad, g is the derivative with respect to the query: the terms are P(r) / |r|^(2p+1) for
// homogeneous P of degree p = 1, 2, 3, whose gradient is (grad P(n) - (2p+1) P(n) n) / |r|^(p+2), and
// P(n) = n . grad P(n) / p. One child's |r|^2 may be anything (its result is then not used); one that
// underflows to the denormals gives a result that is not finite, and its child is entered.
template <int Order, bool Grad>
__device__ __forceinline__ x2::f2 far_pair(pair_head const &h, float4 const *w, x2::f2 &g0, x2::f2 &g1, x2::f2 &g2) {
    using namespace x2;
    f2 const m1 = rsqrt(h.q2);
    f2 const m2 = mul(m1, m1);
    f2 const x = mul(h.rx, m1), y = mul(h.ry, m1), z = mul(h.rz, m1);
    f2 Nx, Ny, Nz, ref; // -N
    load(w + 2, Nx, Ny);
    load(w + 3, Nz, ref);
    f2 const t0 = dot(x, y, z, Nx, Ny, Nz); // -(n.N)
    if constexpr (!Grad) {
        if constexpr (Order == 0) {
            return mul(m2, t0);
        } else {
            // the forms factored by components: M' in 7 and K in 13 operations on the shared squares
            f2 cxx, cyy, czz, cxy, cyz, czx;
            load(w + 4, cxx, cyy);
            load(w + 5, czz, cxy);
            load(w + 6, cyz, czx);
            f2 const xx = mul(x, x), yy = mul(y, y), zz = mul(z, z), yz = mul(y, z);
            f2 t = fma(cyz, yz, fma(czz, zz, fma(cyy, yy, mul(cxx, xx))));
            t = fma(x, fma(czx, z, mul(cxy, y)), t);
            if constexpr (Order >= 2) {
                f2 kxxx, kyyy, kzzz, kxxy, kxxz, kyyx, kyyz, kzzx, kzzy, kxyz;
                load(w + 7, kxxx, kyyy);
                load(w + 8, kzzz, kxxy);
                load(w + 9, kxxz, kyyx);
                load(w + 10, kyyz, kzzx);
                load(w + 11, kzzy, kxyz);
                f2 q = mul(x, fma(kxyz, yz, fma(kzzx, zz, fma(kyyx, yy, mul(kxxx, xx)))));
                q = fma(y, fma(kzzy, zz, fma(kxxy, xx, mul(kyyy, yy))), q);
                q = fma(z, fma(kyyz, yy, fma(kxxz, xx, mul(kzzz, zz))), q);
                t = fma(m1, q, t);
            }
            return mul(m2, fma(m1, t, t0));
        }
    } else {
        f2 const m3 = mul(m2, m1);
        f2 gx = Nx, gy = Ny, gz = Nz;       // grad P(n) / |r|^(p-1), summed
        f2 s = mul(t0, both(-3.0f));        // sum of -(2p+1) P(n) / |r|^(p-1)
        f2 value = t0;                      // sum of P(n) / |r|^(p-1)
        if constexpr (Order >= 1) {
            f2 cxx, cyy, czz, cxy, cyz, czx;
            load(w + 4, cxx, cyy);
            load(w + 5, czz, cxy);
            load(w + 6, cyz, czx);
            f2 const two = both(2.0f);
            f2 const dx = fma(mul(cxx, two), x, fma(cxy, y, mul(czx, z)));
            f2 const dy = fma(mul(cyy, two), y, fma(cxy, x, mul(cyz, z)));
            f2 const dz = fma(mul(czz, two), z, fma(cyz, y, mul(czx, x)));
            f2 const q1 = mul(m1, dot(x, y, z, dx, dy, dz)); // 2 P / |r|
            gx = fma(m1, dx, gx);
            gy = fma(m1, dy, gy);
            gz = fma(m1, dz, gz);
            s = fma(q1, both(-2.5f), s);
            value = fma(q1, both(0.5f), value);
            if constexpr (Order >= 2) {
                f2 kxxx, kyyy, kzzz, kxxy, kxxz, kyyx, kyyz, kzzx, kzzy, kxyz;
                load(w + 7, kxxx, kyyy);
                load(w + 8, kzzz, kxxy);
                load(w + 9, kxxz, kyyx);
                load(w + 10, kyyz, kzzx);
                load(w + 11, kzzy, kxyz);
                f2 const xx = mul(x, x), yy = mul(y, y), zz = mul(z, z);
                f2 const x2_ = mul(x, two), y2_ = mul(y, two), xy = mul(x2_, y), yz = mul(y2_, z), zx = mul(x2_, z);
                f2 const three = both(3.0f), half = both(0.5f);
                f2 const ex = fma(mul(kxxx, three), xx,
                                  fma(kxxy, xy, fma(kxxz, zx, fma(kyyx, yy, fma(kzzx, zz, mul(mul(kxyz, half), yz))))));
                f2 const ey = fma(mul(kyyy, three), yy,
                                  fma(kyyx, xy, fma(kyyz, yz, fma(kxxy, xx, fma(kzzy, zz, mul(mul(kxyz, half), zx))))));
                f2 const ez = fma(mul(kzzz, three), zz,
                                  fma(kzzx, zx, fma(kzzy, yz, fma(kxxz, xx, fma(kyyz, yy, mul(mul(kxyz, half), xy))))));
                f2 const q2 = mul(m2, dot(x, y, z, ex, ey, ez)); // 3 P / |r|^2
                gx = fma(m2, ex, gx);
                gy = fma(m2, ey, gy);
                gz = fma(m2, ez, gz);
                s = fma(q2, both(-7.0f / 3.0f), s);
                value = fma(q2, both(1.0f / 3.0f), value);
            }
        }
        g0 = mul(m3, fma(s, x, gx));
        g1 = mul(m3, fma(s, y, gy));
        g2 = mul(m3, fma(s, z, gz));
        return mul(m2, value);
    }
}

// Child references of a pair.
__device__ __forceinline__ void pair_refs(float4 const *w, std::uint32_t &r0, std::uint32_t &r1) {
    x2::f2 nz, ref;
    x2::load(w + 3, nz, ref);
    r0 = static_cast<std::uint32_t>(ref.v);
    r1 = static_cast<std::uint32_t>(ref.v >> 32);
}

} // namespace field
} // namespace gwnb
