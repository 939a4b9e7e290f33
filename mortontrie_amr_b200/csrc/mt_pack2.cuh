// The reduced-precision collisions, written once for one cell (V = float) and
// for two cells in lockstep (V = float2, cell A in .x, cell B in .y, on the
// packed f32x2 instructions of sm_100: one issue slot does both cells'
// arithmetic, which halves the instruction count of the part of the fused
// brick pass that bounds it).  Every operation is an explicit
// round-to-nearest add, multiply or fused multiply-add in a fixed order, so
// that both forms, and every kernel that collides a cell, give the same bits.
#pragma once

#include <cuda_runtime.h>

#include "mt_lattice.cuh"

namespace mt {
namespace p2 {

template <class V> __device__ __forceinline__ V bc(float s);
template <> __device__ __forceinline__ float bc<float>(float s) { return s; }
template <> __device__ __forceinline__ float2 bc<float2>(float s) { return make_float2(s, s); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float neg(float a) { return -a; }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// (as PTX with an explicit rounding: never contracted into one another)
__device__ __forceinline__ float2 add(float2 a, float2 b)
{
    float2 r;
    asm("{.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 c, a, b;\n\t"
        "mov.b64 {%0, %1}, c;}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 mul(float2 a, float2 b)
{
    float2 r;
    asm("{.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 c, a, b;\n\t"
        "mov.b64 {%0, %1}, c;}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c)
{
    float2 r;
    asm("{.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }
// a - b in one rounding without negating a pair
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return fma(b, bc<float2>(-1.f), a); }
// a constant-bank operand c: two scalar instructions rather than a packed one
// that first needs the pair in registers
__device__ __forceinline__ float addc(float a, float c) { return __fadd_rn(a, c); }
__device__ __forceinline__ float2 addc(float2 a, float c) { return make_float2(__fadd_rn(a.x, c), __fadd_rn(a.y, c)); }
__device__ __forceinline__ float fmac(float w, float a, float c) { return __fmaf_rn(w, a, c); }
__device__ __forceinline__ float2 fmac(float w, float2 a, float c)
{
    return make_float2(__fmaf_rn(w, a.x, c), __fmaf_rn(w, a.y, c));
}
// 1 / rho with the reference's floor |rho| >= 1e-6 (SAFE_IRHO, Collision_Cumulant.cpp:17-20)
__device__ __forceinline__ float safe_inv(float r)
{
    return 1.f / ((r > -1e-6f && r < 1e-6f) ? ((r < 0.f) ? -1e-6f : 1e-6f) : r);
}
__device__ __forceinline__ float inv(float r) { return 1.f / r; }
__device__ __forceinline__ float2 inv(float2 r) { return make_float2(1.f / r.x, 1.f / r.y); }
__device__ __forceinline__ float2 safe_inv(float2 r) { return make_float2(safe_inv(r.x), safe_inv(r.y)); }

// e_k . u with the lattice constants folded
template <int Q, class V> __device__ __forceinline__ V eu(int k, V x, V y, V z)
{
    V s = bc<V>(0.f);
    bool any = false;
    auto acc = [&](int e, V v) {
        if (e == 0) return;
        if (!any) {
            s = e > 0 ? v : neg(v);
            any = true;
        } else {
            s = e > 0 ? add(s, v) : sub(s, v);
        }
    };
    acc(ex(k), x);
    acc(ey(k), y);
    acc(ez(k), z);
    return s;
}

// Macros and Collision_LBGK::collide (Collision_Manager.cpp:13-53) in place on
// stored deviations s_k = f_k - shift_k.  The moments are those of the full
// populations summed in direction order; out_k = s_k + omega (feq_k - shift_k -
// s_k).  q and inv(q) (listed as q, q + 1 for every odd q) share 4.5 (e.u)^2.
template <int Q, class V>
__device__ __forceinline__ void lbgk(V *s, V &rho, V &ux, V &uy, V &uz, float om, const Shift &sh)
{
#pragma unroll
    for (int k = 0; k < Q; ++k) s[k] = addc(s[k], sh.v[k]);
    V r = s[0], jx = bc<V>(0.f), jy = bc<V>(0.f), jz = bc<V>(0.f);
#pragma unroll
    for (int k = 1; k < Q; ++k) {
        r = add(r, s[k]);
        if (ex(k) > 0) jx = add(jx, s[k]);
        if (ex(k) < 0) jx = sub(jx, s[k]);
        if (ey(k) > 0) jy = add(jy, s[k]);
        if (ey(k) < 0) jy = sub(jy, s[k]);
        if (ez(k) > 0) jz = add(jz, s[k]);
        if (ez(k) < 0) jz = sub(jz, s[k]);
    }
    const V is = safe_inv(r);
    rho = r;
    ux = mul(jx, is);
    uy = mul(jy, is);
    uz = mul(jz, is);
    const V u2 = fma(uz, uz, fma(ux, ux, mul(uy, uy)));
    const V rm1 = add(r, bc<V>(-1.f));
    auto relax = [&](V &f, V poly, int k) {
        const V dfeq = fmac((float)w<Q>(k), fma(r, poly, rm1), -sh.dw[k]);
        const V d = addc(f, -sh.v[k]);
        f = fma(bc<V>(om), sub(dfeq, d), d);
    };
    relax(s[0], mul(bc<V>(-1.5f), u2), 0);
#pragma unroll
    for (int k = 1; k < Q; k += 2) {
        const V e = eu<Q, V>(k, ux, uy, uz);
        const V q = mul(mul(bc<V>(4.5f), e), e);
        relax(s[k], fma(bc<V>(-1.5f), u2, fma(bc<V>(3.f), e, q)), k);
        relax(s[k + 1], fma(bc<V>(-1.5f), u2, fma(bc<V>(-3.f), e, q)), k + 1);
    }
    // an infinite population leaves no component of the macros finite (the sums
    // leave its zero components out; the collision has NaN from u2)
    const V z = mul(add(add(ux, uy), uz), bc<V>(0.f));
    ux = add(ux, z);
    uy = add(uy, z);
    uz = add(uz, z);
}

// a direction's storage shift in FP32; NoShift (u_s = 0) the weight, which takes
// no kernel parameter (the table made a launch of a 16^3 cube 0.4 us longer)
struct NoShift {};
__device__ __forceinline__ float shift_at(const Shift &sh, int k) { return sh.v[k]; }
__device__ __forceinline__ constexpr float shift_at(const NoShift &, int k) { return (float)w<27>(k); }

// backward chimera step of one line (chim_back's FP32 polynomials); Z0, Z1,
// Z2 mark inputs known to be zero
template <bool Z0, bool Z1, bool Z2, class V>
__device__ __forceinline__ void chim_back(V a0, V a1, V a2, V v, V tv, V v2, V &pn, V &pz, V &pp)
{
    V t, hh;
    if (Z0) {
        t = Z2 ? mul(tv, a1) : fma(tv, a1, a2);
        hh = a1;
    } else {
        const V inner = Z1 ? a2 : (Z2 ? mul(tv, a1) : fma(tv, a1, a2));
        t = fma(a0, v2, inner);
        hh = Z1 ? mul(a0, v) : fma(a0, v, a1);
    }
    pz = Z0 ? neg(t) : sub(a0, t);
    const V ht = mul(t, bc<V>(0.5f));
    pp = fma(hh, bc<V>(0.5f), ht);
    pn = fma(hh, bc<V>(-0.5f), ht);
}

// Macros and D3Q27 cumulant collision in place on stored deviations s_k = f_k -
// shift_k (Collision_Cumulant.cpp:320-652): forward central moments by x, y, z
// chimera passes, second-order cumulants relaxed with omega1 and bulk rate 1, higher cumulants
// zero, backward transform (the moments the relaxation zeroes left out).  The
// (2,1,0), (1,0,2), (0,2,1) moments keep their forward values
// (Collision_Cumulant.cpp:451-454).
// shift_k = w_k (NoShift, the dense cube): rho - 1 and the momentum are sums of
// the deviations in direction order, without cancellation; else they come from
// the x pass's line sums of the full populations.  (Line sums of the deviations,
// the shift's own added once, would serve both and spare 60 packed additions of
// about 600 a pair, 256^3 FP16 414 -> 402 us, but round otherwise: results of
// this path do not change with the kernel that computes them.)
template <class V, class SH>
__device__ __forceinline__ void cumulant(V *s, V &rho, V &ux, V &uy, V &uz, float om1, const SH &sh)
{
    constexpr bool DEV = std::is_same<SH, NoShift>::value;
    V g[27];
    if constexpr (DEV) {
        V r = s[0], jx = bc<V>(0.f), jy = bc<V>(0.f), jz = bc<V>(0.f);
#pragma unroll
        for (int i = 1; i < 27; ++i) {
            r = add(r, s[i]);
            if (ex(i)) jx = ex(i) > 0 ? add(jx, s[i]) : sub(jx, s[i]);
            if (ey(i)) jy = ey(i) > 0 ? add(jy, s[i]) : sub(jy, s[i]);
            if (ez(i)) jz = ez(i) > 0 ? add(jz, s[i]) : sub(jz, s[i]);
        }
        rho = add(r, bc<V>(1.f));
        const V is = inv(rho);
        ux = mul(jx, is);
        uy = mul(jy, is);
        uz = mul(jz, is);
    }
#pragma unroll
    for (int i = 0; i < 27; ++i) g[(ex(i) + 1) + 3 * (ey(i) + 1) + 9 * (ez(i) + 1)] = addc(s[i], shift_at(sh, i));
    {
        // x lines: slot 0 line total k0, slot 1 difference d1, slot 2 sum of the ends s1
        V r, jx, jy, jz;
#pragma unroll
        for (int line = 0; line < 9; ++line) {
            const int b = 3 * line, ly = line % 3, lz = line / 3;
            const V fm = g[b], f0 = g[b + 1], fp = g[b + 2];
            const V s1 = add(fp, fm), d1 = sub(fp, fm), k0 = DEV ? add(add(fm, f0), fp) : add(s1, f0);
            g[b] = k0;
            g[b + 1] = d1;
            g[b + 2] = s1;
            if constexpr (DEV) continue;
            r = line ? add(r, k0) : k0;
            jx = line ? add(jx, d1) : d1;
            // (line 0 is the first of both, with the sign -1)
            if (ly == 2) jy = add(jy, k0);
            if (ly == 0) jy = line ? sub(jy, k0) : neg(k0);
            if (lz == 2) jz = add(jz, k0);
            if (lz == 0) jz = line ? sub(jz, k0) : neg(k0);
        }
        if constexpr (!DEV) {
            rho = r;
            const V is = safe_inv(rho);
            ux = mul(jx, is);
            uy = mul(jy, is);
            uz = mul(jz, is);
        }
        const V u2 = mul(ux, ux), mu = neg(ux), m2u = mul(ux, bc<V>(-2.f));
#pragma unroll
        for (int line = 0; line < 9; ++line) {
            const int b = 3 * line;
            const V k0 = g[b], d1 = g[b + 1], s1 = g[b + 2];
            g[b + 1] = fma(mu, k0, d1);
            g[b + 2] = fma(u2, k0, fma(m2u, d1, s1));
        }
    }
    const V vel[3] = {ux, uy, uz};
#pragma unroll
    for (int ax = 1; ax < 3; ++ax) {
        const int st = ax == 1 ? 3 : 9;
        const V u = vel[ax], u2 = mul(u, u), mu = neg(u), m2u = mul(u, bc<V>(-2.f));
#pragma unroll
        for (int line = 0; line < 9; ++line) {
            const int o1 = line % 3, o2 = line / 3;
            const int b = ax == 1 ? o1 + 9 * o2 : o1 + 3 * o2;
            const V fm = g[b], f0 = g[b + st], fp = g[b + 2 * st];
            const V k0 = add(add(fm, f0), fp), d1 = sub(fp, fm), s1 = add(fp, fm);
            g[b] = k0;
            g[b + st] = fma(mu, k0, d1);
            g[b + 2 * st] = fma(u2, k0, fma(m2u, d1, s1));
        }
    }
#define G(a, b, c) g[(a) + 3 * (b) + 9 * (c)]
    const V k000 = G(0, 0, 0), two = bc<V>(2.f), half = bc<V>(0.5f);
    V c200 = G(2, 0, 0), c020 = G(0, 2, 0), c002 = G(0, 0, 2);
    const V ir = safe_inv(rho);
    const V om = bc<V>(om1), omc = bc<V>(1.f - om1);
    const V d20 = sub(c200, c020), d02 = sub(c200, c002);
    // dxu = -(om1 (2 c200 - c020 - c002) + (c200 + c020 + c002 - k000)) ir / 2
    const V x = fma(om, sub(fma(two, c200, neg(c020)), c002), sub(add(add(c200, c020), c002), k000));
    const V dxu = mul(x, mul(ir, bc<V>(-0.5f)));
    const V o3 = bc<V>(3.f * om1);
    const V dyv = fma(mul(mul(o3, d20), half), ir, dxu);
    const V dzw = fma(mul(mul(o3, d02), half), ir, dxu);
    const V c110 = mul(G(1, 1, 0), omc), c101 = mul(G(1, 0, 1), omc), c011 = mul(G(0, 1, 1), omc);
    const V ux2 = mul(ux, ux), uy2 = mul(uy, uy), uz2 = mul(uz, uz);
    const V ax_ = mul(ux2, dxu);
    const V r3 = mul(rho, bc<V>(-3.f));
    const V r3o = mul(r3, bc<V>(1.f - 0.5f * om1));
    const V x1 = fma(omc, d20, mul(r3o, fma(neg(uy2), dyv, ax_)));
    const V x2 = fma(omc, d02, mul(r3o, fma(neg(uz2), dzw, ax_)));
    const V x3 = fma(mul(r3, half), fma(uz2, dzw, fma(uy2, dyv, ax_)), k000);
    c200 = mul(add(add(x1, x2), x3), bc<V>(1.f / 3.f));
    c020 = sub(c200, x1);
    c002 = sub(c200, x2);
    const V m210 = G(2, 1, 0), m102 = G(1, 0, 2), m021 = G(0, 2, 1);
    const V t110 = mul(two, c110), t101 = mul(two, c101), t011 = mul(two, c011);
    const V m211 = mul(fma(c200, c011, mul(t110, c101)), ir);
    const V m121 = mul(fma(c020, c101, mul(t011, c110)), ir);
    const V m112 = mul(fma(c002, c110, mul(t101, c011)), ir);
    const V m220 = mul(fma(c200, c020, mul(t110, c110)), ir);
    const V m022 = mul(fma(c020, c002, mul(t011, c011)), ir);
    const V m202 = mul(fma(c002, c200, mul(t101, c101)), ir);
    const V m122 = mul(fma(two, mul(c101, m021), mul(c020, m102)), ir);
    const V m212 = mul(fma(two, mul(c110, m102), mul(c002, m210)), ir);
    const V m221 = mul(fma(two, mul(c011, m210), mul(c200, m021)), ir);
    const V four = bc<V>(4.f);
    const V a = mul(fma(four, fma(c110, m112, fma(c011, m211, mul(c101, m121))),
                        fma(c002, m220, fma(c020, m202, mul(c200, m022)))), ir);
    const V b4 = mul(four, fma(mul(c110, c110), c002, fma(mul(c101, c101), c020, mul(mul(c011, c011), c200))));
    const V b = fma(mul(mul(two, c200), c020), c002, fma(mul(mul(bc<V>(16.f), c110), c101), c011, b4));
    const V m222 = fma(neg(mul(b, ir)), ir, a);
    // backward chimera, x lines (b, c) with (a0, a1, a2) = moments (0|1|2, b, c)
    V p1[27], p2[27];
    const V tvx = add(ux, ux);
    const V zero = bc<V>(0.f);
    chim_back<false, false, false>(k000, G(1, 0, 0), c200, ux, tvx, ux2, p1[0], p1[1], p1[2]);
    chim_back<false, false, false>(G(0, 1, 0), c110, m210, ux, tvx, ux2, p1[3], p1[4], p1[5]);
    chim_back<false, true, false>(c020, zero, m220, ux, tvx, ux2, p1[6], p1[7], p1[8]);        // (1,2,0) = 0
    chim_back<false, false, true>(G(0, 0, 1), c101, zero, ux, tvx, ux2, p1[9], p1[10], p1[11]); // (2,0,1) = 0
    chim_back<false, true, false>(c011, zero, m211, ux, tvx, ux2, p1[12], p1[13], p1[14]);     // (1,1,1) = 0
    chim_back<false, false, false>(m021, m121, m221, ux, tvx, ux2, p1[15], p1[16], p1[17]);
    chim_back<false, false, false>(c002, m102, m202, ux, tvx, ux2, p1[18], p1[19], p1[20]);
    chim_back<true, false, false>(zero, m112, m212, ux, tvx, ux2, p1[21], p1[22], p1[23]);     // (0,1,2) = 0
    chim_back<false, false, false>(m022, m122, m222, ux, tvx, ux2, p1[24], p1[25], p1[26]);
    const V tvy = add(uy, uy), tvz = add(uz, uz);
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
            chim_back<false, false, false>(p1[ix + 9 * cc], p1[ix + 3 + 9 * cc], p1[ix + 6 + 9 * cc], uy, tvy, uy2,
                                           p2[ix + 9 * cc], p2[ix + 3 + 9 * cc], p2[ix + 6 + 9 * cc]);
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
        for (int iy = 0; iy < 3; ++iy)
            chim_back<false, false, false>(p2[ix + 3 * iy], p2[ix + 3 * iy + 9], p2[ix + 3 * iy + 18], uz, tvz, uz2,
                                           g[ix + 3 * iy], g[ix + 3 * iy + 9], g[ix + 3 * iy + 18]);
#undef G
#pragma unroll
    for (int i = 0; i < 27; ++i) s[i] = addc(g[(ex(i) + 1) + 3 * (ey(i) + 1) + 9 * (ez(i) + 1)], -shift_at(sh, i));
}

}  // namespace p2
}  // namespace mt
