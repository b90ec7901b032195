// Arithmetic of one step shared by the step kernels (sm_100a): every
// operation rounds once, in a fixed order, so that all layouts give the
// bits of the CPU restatement in the oracle.
#pragma once
#include "mb_internal.h"

namespace mb {

constexpr float kEps = 1e-12f;  // sim_kernel.cu:6

// Force modes, per mass, after the spring forces (fx, fy, fz) are gathered:
// environment forces, then x' = x + v dt + (F/m) dt^2, v' = damping (x' - x)/dt.
//   land : gravity -m g along z; below z = 0 a penalty normal force
//          fn = k_floor (-z) and Coulomb friction on the horizontal velocity
//          h = v + (F_h/m) dt the step would reach: static (the friction force
//          cancels the horizontal motion, F_h = -m v_h/dt) when |h| <= mu_s fn
//          dt/m, else kinetic, mu_k fn against h.
//   water: gravity balanced by buoyancy; quadratic drag -drag |v| v.
// Divisions by m and dt are multiplications by the correctly rounded
// reciprocals (inv_dt = RN(1/dt) per launch, RN(1/m) per mass and step);
// only the kinetic friction divides.
template <int MODE>
__device__ __forceinline__ void force_integrate(const StepParams& p, float3& x, float3& v, float m,
                                                float inv_dt, float fx, float fy, float fz) {
    const float dt = p.dt;
    const float inv_m = __frcp_rn(m);
    if (MODE == kModeForceLand) {
        fz = __fsub_rn(fz, __fmul_rn(m, p.g));
        if (x.z < 0.0f) {
            const float fn = __fmul_rn(p.floor_stiffness, -x.z);
            fz = __fadd_rn(fz, fn);
            const float hx = __fadd_rn(v.x, __fmul_rn(__fmul_rn(fx, inv_m), dt));
            const float hy = __fadd_rn(v.y, __fmul_rn(__fmul_rn(fy, inv_m), dt));
            const float hs = __fsqrt_rn(__fmaf_rn(hx, hx, __fmul_rn(hy, hy)));
            const float budget = __fmul_rn(__fmul_rn(fn, inv_m), dt);
            if (hs <= __fmul_rn(p.mu_s, budget)) {
                fx = __fmul_rn(__fmul_rn(-m, v.x), inv_dt);
                fy = __fmul_rn(__fmul_rn(-m, v.y), inv_dt);
            } else {
                const float s = __fdiv_rn(__fmul_rn(p.mu_k, fn), hs);
                fx = __fsub_rn(fx, __fmul_rn(s, hx));
                fy = __fsub_rn(fy, __fmul_rn(s, hy));
            }
        }
    } else {
        const float sp = __fsqrt_rn(__fmaf_rn(v.x, v.x, __fmaf_rn(v.y, v.y, __fmul_rn(v.z, v.z))));
        const float c = __fmul_rn(p.drag, sp);
        fx = __fsub_rn(fx, __fmul_rn(c, v.x));
        fy = __fsub_rn(fy, __fmul_rn(c, v.y));
        fz = __fsub_rn(fz, __fmul_rn(c, v.z));
    }
    const float dt2 = __fmul_rn(dt, dt);
    const float nx = __fadd_rn(__fadd_rn(x.x, __fmul_rn(v.x, dt)), __fmul_rn(__fmul_rn(fx, inv_m), dt2));
    const float ny = __fadd_rn(__fadd_rn(x.y, __fmul_rn(v.y, dt)), __fmul_rn(__fmul_rn(fy, inv_m), dt2));
    const float nz = __fadd_rn(__fadd_rn(x.z, __fmul_rn(v.z, dt)), __fmul_rn(__fmul_rn(fz, inv_m), dt2));
    v.x = __fmul_rn(p.damping, __fmul_rn(__fsub_rn(nx, x.x), inv_dt));
    v.y = __fmul_rn(p.damping, __fmul_rn(__fsub_rn(ny, x.y), inv_dt));
    v.z = __fmul_rn(p.damping, __fmul_rn(__fsub_rn(nz, x.z), inv_dt));
    x = make_float3(nx, ny, nz);
}

// Velocity of the reference step, v = (float)(0.99 * (double)delta / (double)dt)
// (sim_kernel.cu:265-267): the double product, the correctly rounded double
// quotient, then rounding to float -- without a double division in the
// common case.  q = RN(a * inv_dt), with inv_dt = RN(1/dt), differs from
// the exact a/dt by at most 2u + u^2 relative (u = 2^-53), so from the
// correctly rounded quotient by less than 3.01 units in the last place of
// q.  Rounding to float can only differ between q and that quotient if a
// float rounding boundary -- the midpoint between two floats, whose low 29
// significand bits are 1 << 28 in double -- lies between them.  So when
// q's low 29 bits are more than 4 units from 1 << 28 and q lies in the
// normal float range, (float)q is the result (Ziv's rounding test: Ziv,
// "Fast evaluation of elementary mathematical functions with correctly
// rounded last bit", ACM TOMS 17(3), 1991); otherwise -- about 9 inputs in
// 2^29, zeros excepted -- the division itself is done.
__device__ __forceinline__ float velocity_of(float delta, double dt, double inv_dt) {
    const double a = __dmul_rn(0.99, (double)delta);
    const double q = __dmul_rn(a, inv_dt);
    const unsigned long long bits = (unsigned long long)__double_as_longlong(q);
    const uint32_t e = (uint32_t)(bits >> 52) & 0x7FFu;
    const uint32_t low29 = (uint32_t)bits & 0x1FFFFFFFu;
    // normal float range 2^-126 <= |q| < 2^127 (biased double exponents 897..1149)
    const bool clear = (e - 897u) < 253u && (low29 - (0x10000000u - 4u)) > 8u;
    if (clear || (bits << 1) == 0) return __double2float_rn(q);
    return __double2float_rn(__ddiv_rn(a, dt));
}

// Length d = RN(sqrt(s)) and q = RN(1 / RN(d + eps)) of a spring from the
// squared length s, without the branches of the general square root and
// reciprocal: one approximate reciprocal square root y, then
//   d: g = s y, one residual step g + (s - g g) y/2
//   q: e = 1 - d y, second-order step y + y (e + e e)
// (Newton steps whose residuals an FMA gives with one rounding: Markstein,
// "IA-64 and Elementary Functions", 2000, ch. 8-9).  For d >= 2^-14,
// RN(d + eps) is d, and both results equal __fsqrt_rn and __frcp_rn on every
// float s there, except q where d's mantissa is all ones: then y is a power
// of two and e exactly 2^-24 (mb_check_spring_math compares all inputs on
// the device).  Where length_is_fast does not hold -- NaN and an infinite s,
// whose d is NaN here, among them -- the intrinsics are taken.  All values
// carry their sign: ns = -s, nd = -d, because a packed operation has no
// operand negation.
__device__ __forceinline__ float rsqrt_approx(float s) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    return y;
}
__device__ __forceinline__ bool length_is_fast(float nd, float e) {
    return nd <= -0x1p-14f && e != 0x1p-24f;
}
__device__ __forceinline__ void length_and_reciprocal_fast(float ns, float& nd, float& e, float& q) {
    const float y = rsqrt_approx(-ns);
    const float ng = __fmul_rn(ns, y), h = __fmul_rn(0.5f, y);
    nd = __fmaf_rn(__fmaf_rn(ng, ng, ns), h, ng);
    e = __fmaf_rn(nd, y, 1.0f);
    q = __fmaf_rn(y, __fmaf_rn(e, e, e), y);
}
__device__ __forceinline__ void length_and_reciprocal_exact(float ns, float& nd, float& q) {
    nd = -__fsqrt_rn(-ns);
    q = __frcp_rn(__fadd_rn(-nd, kEps));
}
__device__ __forceinline__ void length_and_reciprocal(float s, float& nd, float& q) {
    float e;
    length_and_reciprocal_fast(-s, nd, e, q);
    if (!length_is_fast(nd, e)) length_and_reciprocal_exact(-s, nd, q);
}

// RN(1 / x) from an approximation of one unit in the last place and one Newton step
// (Markstein, as above) for ordinary x.  Where it matters the caller compares
// the result with __frcp_rn once.
__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}

// Face drag of one surface triangle (water), the share of each corner:
// mean corner velocity v = (v0 + v1 + v2) * RN(1/3), N = (x1 - x0) x (x2 - x0), A = |N|, unit normal
// n = N * RN(1/(A + eps)) turned so that v.n > 0 (sim_kernel.cu:106-109),
// force coef * A * ((v.n) v + 0.2 |v|^2 n) with coef = -rho/6, i.e.
// -rho/2 A (...) / 3 (sim_kernel.cu:110-111).  Every operation rounds once,
// in this order.
__device__ __forceinline__ float4 face_force(const float4 x0, const float4 x1, const float4 x2, const float4 v0,
                                             const float4 v1, const float4 v2, const float coef) {
    constexpr float kThird = 0x1.555556p-2f;  // 1/3 rounded to nearest
    const float vx = __fmul_rn(__fadd_rn(__fadd_rn(v0.x, v1.x), v2.x), kThird);
    const float vy = __fmul_rn(__fadd_rn(__fadd_rn(v0.y, v1.y), v2.y), kThird);
    const float vz = __fmul_rn(__fadd_rn(__fadd_rn(v0.z, v1.z), v2.z), kThird);
    const float ax = __fsub_rn(x1.x, x0.x), ay = __fsub_rn(x1.y, x0.y), az = __fsub_rn(x1.z, x0.z);
    const float bx = __fsub_rn(x2.x, x0.x), by = __fsub_rn(x2.y, x0.y), bz = __fsub_rn(x2.z, x0.z);
    const float nx = __fsub_rn(__fmul_rn(ay, bz), __fmul_rn(az, by));
    const float ny = __fsub_rn(__fmul_rn(az, bx), __fmul_rn(ax, bz));
    const float nz = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
    float n_area, r;  // -A and RN(1/(A + eps))
    length_and_reciprocal(__fmaf_rn(nx, nx, __fmaf_rn(ny, ny, __fmul_rn(nz, nz))), n_area, r);
    float ux = __fmul_rn(nx, r), uy = __fmul_rn(ny, r), uz = __fmul_rn(nz, r);
    float vn = __fmaf_rn(ux, vx, __fmaf_rn(uy, vy, __fmul_rn(uz, vz)));
    if (!(vn > 0.0f)) {  // negating n negates the rounded dot product exactly
        ux = -ux;
        uy = -uy;
        uz = -uz;
        vn = -vn;
    }
    const float lift = __fmul_rn(0.2f, __fmaf_rn(vx, vx, __fmaf_rn(vy, vy, __fmul_rn(vz, vz))));
    const float c = __fmul_rn(coef, -n_area);
    return make_float4(__fmul_rn(c, __fmaf_rn(lift, ux, __fmul_rn(vn, vx))),
                       __fmul_rn(c, __fmaf_rn(lift, uy, __fmul_rn(vn, vy))),
                       __fmul_rn(c, __fmaf_rn(lift, uz, __fmul_rn(vn, vz))), 0.0f);
}

// Two floats in one 64-bit register pair: each half rounds like the scalar
// operation.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Both lengths of a pair of springs.
__device__ __forceinline__ void lengths_and_reciprocals_fast(f32x2 ns, f32x2& nd, f32x2& e, f32x2& q) {
    float n0, n1;
    unpack2(ns, n0, n1);
    const f32x2 y = pack2(rsqrt_approx(-n0), rsqrt_approx(-n1));
    const f32x2 ng = mul2(ns, y), h = mul2(y, pack2(0.5f, 0.5f));
    nd = fma2(fma2(ng, ng, ns), h, ng);
    e = fma2(nd, y, pack2(1.0f, 1.0f));
    q = fma2(y, fma2(e, e, e), y);
}

}  // namespace mb
