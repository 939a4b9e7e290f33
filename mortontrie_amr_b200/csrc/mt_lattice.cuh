// Lattice tables, Morton neighbour arithmetic and per-cell collision physics
// shared by every kernel of the library.
//
// Direction order, weights and inverse table: header/Constants.h:492-538 and
// LBM_Manager.cpp:137-169 of the reference.  The FP64 functions keep the
// reference's expression order so that, compiled without FMA contraction,
// they reproduce its results bit-for-bit; the FP32 variants are written for
// throughput (FMA, reciprocal of tau) and are compared against the FP64 path
// within stated tolerances.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#ifndef MT_HD
#define MT_HD __host__ __device__ __forceinline__
#endif

namespace mt {

MT_HD constexpr int ex(int k)
{
    constexpr int t[27] = {0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, -1, 1, -1, 1};
    return t[k];
}
MT_HD constexpr int ey(int k)
{
    constexpr int t[27] = {0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1, -1, 1, 1, -1};
    return t[k];
}
MT_HD constexpr int ez(int k)
{
    constexpr int t[27] = {0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1};
    return t[k];
}
MT_HD constexpr int inv(int k)
{
    constexpr int t[27] = {0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 14, 13, 16, 15, 18, 17, 20, 19, 22, 21, 24, 23, 26, 25};
    return t[k];
}
template <int Q> MT_HD constexpr double w(int k)
{
    return Q == 19 ? (k == 0 ? 1. / 3. : (k <= 6 ? 1. / 18. : 1. / 36.))
                   : (k == 0 ? 8. / 27. : (k <= 6 ? 2. / 27. : (k <= 18 ? 1. / 54. : 1. / 216.)));
}
// Storage shift of the reduced storages (FP32, FP16, BF16): they keep
// f_k - s_k with s_k = feq_k(1, u_s) = w_k (1 + 3 e.u_s + 4.5 (e.u_s)^2 -
// 1.5 u_s^2), so the stored deviations are small where the flow is near u_s
// (u_s = 0: s_k = w_k).  v: s_k rounded to FP32 (the compute type), dw: s_k -
// w_k rounded to FP32, d: s_k in FP64 (conversions from FP64 values), u: u_s.
// Kernels take it by value: with the direction loops unrolled its entries are
// constant-bank operands, as the literal weights were.
struct Shift {
    float v[27];
    float dw[27];
    float u[3];
    double d[27];
};
inline Shift make_shift(int q, const double *us)
{
    Shift s{};
    const double uu = us[0] * us[0] + us[1] * us[1] + us[2] * us[2];
    for (int k = 0; k < q; ++k) {
        const double wk = q == 19 ? w<19>(k) : w<27>(k);
        const double eu = ex(k) * us[0] + ey(k) * us[1] + ez(k) * us[2];
        const double dw = wk * (3.0 * eu + 4.5 * eu * eu - 1.5 * uu);
        s.d[k] = wk + dw;
        s.v[k] = (float)s.d[k];
        s.dw[k] = (float)dw;
    }
    for (int a = 0; a < 3; ++a) s.u[a] = (float)us[a];
    return s;
}

// A level's relaxation as kernels take it: the time, its reciprocal and the
// FP32 rate, formed once on the host (an FP64 division costs a thread as much
// as ten moments).
struct Relax {
    double tau = 1.0, inv = 1.0;
    float om = 1.f;
    Relax() = default;
    Relax(double t) : tau(t), inv(1.0 / t), om((float)(1.0 / t)) {}
};

// D3Q19 weights used by the solid-boundary treatment for every Q; entries
// 19..26 are zero (ComplexBoundary_Manager.cpp:102-107,184-189).
MT_HD constexpr double w19z(int k) { return k >= 19 ? 0.0 : w<19>(k); }

// ---------------------------------------------------------------------------
// Morton keys.  A level-l cell at (x, y, z) in level-l units has the key
// interleave(x << (L-l), y << (L-l), z << (L-l)), x at bit 3i (Morton_Assist.cpp
// :185-193).  Neighbour steps are the reference's masked increment/decrement
// (Morton_Assist.h:229-289); a periodic axis wraps instead.
// ---------------------------------------------------------------------------
struct MortonGeom {
    int L;
    int periodic[3];
    int64_t extent0[3];
};

MT_HD uint64_t axis_mask(int L, int level, int axis)
{
    uint64_t m = 0;
    for (int k = L - level; k < 21; ++k) m |= (uint64_t)1 << (3 * k + axis);
    return m;
}
MT_HD uint64_t compact3(uint64_t v)
{
    v &= 0x1249249249249249ULL;
    v = (v ^ (v >> 2)) & 0x10C30C30C30C30C3ULL;
    v = (v ^ (v >> 4)) & 0x100F00F00F00F00FULL;
    v = (v ^ (v >> 8)) & 0x1F0000FF0000FFULL;
    v = (v ^ (v >> 16)) & 0x1F00000000FFFFULL;
    v = (v ^ (v >> 32)) & 0x1FFFFFULL;
    return v;
}
MT_HD uint64_t dilate3(uint64_t v)
{
    v &= 0x1FFFFFULL;
    v = (v | (v << 32)) & 0x1F00000000FFFFULL;
    v = (v | (v << 16)) & 0x1F0000FF0000FFULL;
    v = (v | (v << 8)) & 0x100F00F00F00F00FULL;
    v = (v | (v << 4)) & 0x10C30C30C30C30C3ULL;
    v = (v | (v << 2)) & 0x1249249249249249ULL;
    return v;
}
MT_HD uint64_t axis_step(const MortonGeom &g, uint64_t key, int level, int axis, int dir)
{
    const int L = g.L;
    const uint64_t m1 = axis_mask(L, level, axis);
    uint64_t others = 0;
    for (int a = 0; a < 3; ++a)
        if (a != axis) others |= key & axis_mask(L, level, a);
    if (g.periodic[axis]) {
        const int64_t ext = g.extent0[axis] << level;
        const int sh = L - level;
        int64_t c = (int64_t)(compact3(key >> axis) >> sh) + dir;
        if (c < 0) c += ext;
        if (c >= ext) c -= ext;
        return ((dilate3((uint64_t)c << sh) << axis) & m1) | others;
    }
    const int low = 3 * (L - level);
    const uint64_t one = (uint64_t)1 << (low + axis);
    uint64_t t;
    if (dir > 0) {
        uint64_t fill = ~m1;
        if (low > 0) fill &= ~(((uint64_t)1 << low) - 1);
        t = (key | fill) + one;
    } else {
        t = (key & m1) - one;
    }
    return (t & m1) | others;
}
MT_HD uint64_t find_neighbor(const MortonGeom &g, uint64_t key, int level, int dx, int dy, int dz)
{
    uint64_t r = key;
    if (dx) r = axis_step(g, r, level, 0, dx);
    if (dy) r = axis_step(g, r, level, 1, dy);
    if (dz) r = axis_step(g, r, level, 2, dz);
    return r;
}
MT_HD int64_t lower_bound_u64(const uint64_t *k, int64_t n, uint64_t key)
{
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t mid = lo + ((hi - lo) >> 1);
        if (k[mid] < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}
MT_HD int64_t find_key(const uint64_t *k, int64_t n, uint64_t key)
{
    int64_t i = lower_bound_u64(k, n, key);
    return (i < n && k[i] == key) ? i : -1;
}


// Position of population k of slot i in a level's arrays.  A level is stored in
// bricks of 4x4x4 cells, 64 slots each in Morton order whether or not every
// cell exists, and a brick's Q x 64 populations are contiguous ([brick][Q][64]):
// one brick's values of a direction fill whole 128-byte lines (one line at 16
// bits), an x-adjacent pair of cells is an aligned word, and the Q accesses of
// a cell differ by constant offsets.
template <int Q> MT_HD constexpr int64_t at(int k, int64_t i) { return ((i >> 6) * Q + k) * 64 + (i & 63); }
template <int Q> MT_HD constexpr int64_t at(int k, int32_t i) { return at<Q>(k, (int64_t)i); }
template <int Q> MT_HD constexpr uint32_t at(int k, uint32_t i) { return ((i >> 6) * Q + k) * 64 + (i & 63); }

// The stored cells of one level: brick keys in ascending order and each
// brick's occupancy mask.  A cell's slot is 64 * brick + its local Morton index.
struct LevelMap {
    const uint64_t *bkey = nullptr;
    const unsigned long long *bmask = nullptr;
    int64_t nb = 0;
    int low = 0;  // key bits below this level's cells
    MT_HD uint64_t key(int64_t i) const { return (bkey[i >> 6] << (low + 6)) | ((uint64_t)(i & 63) << low); }
    // the slot of a key, -1 where the level stores no such cell
    MT_HD int64_t find(uint64_t k) const
    {
        if (k & (((uint64_t)1 << low) - 1)) return -1;
        const int64_t b = find_key(bkey, nb, k >> (low + 6));
        if (b < 0) return -1;
        const int m = (int)((k >> low) & 63);
        return ((bmask[b] >> m) & 1) ? 64 * b + m : -1;
    }
};

// ---------------------------------------------------------------------------
// FP64 physics in the reference's operation order
// ---------------------------------------------------------------------------
// In the FP64 forms a direction's zero components are left out (x + 0 y is x:
// the compiler has to keep such terms, a fifth of the operations), and
// quotients by a divisor that several values share come from its reciprocal:
// with rb = RN(1 / b), q = RN(x rb), r = x - q b (exact, one FMA), RN(q + r rb) is
// RN(x / b) (Markstein, IBM J. Res. Dev. 34, 1990; Brisebarre, Muller & Raina,
// IEEE Trans. Comput. 53, 2004), three operations where a division takes
// about ten.  That holds while nothing over- or underflows: b within
// 2^+-100, |x| below 2^900 and zero or above 2^-960 (differences and sums of
// populations are); other cells divide.
MT_HD double quot(double x, double b, double rb)
{
    const double q = x * rb;
    return fma(fma(-q, b, x), rb, q);
}
// |x| < 2^e (false for infinities and NaN)
template <int E> MT_HD bool below(double x)
{
    uint64_t bits;
    memcpy(&bits, &x, 8);
    return (uint32_t)((bits >> 32) & 0x7fffffffu) < (uint32_t)(E + 1023) << 20;
}
// LBM_Manager::calculateMacros(ddf, rho, v) (LBM_Manager.cpp:983-1001)
template <int Q> MT_HD void macros_ref(const double *d, double &rho, double &ux, double &uy, double &uz)
{
    double r = d[0], vx = 0., vy = 0., vz = 0.;
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        r += d[i];
        if (ex(i)) vx += d[i] * ex(i);
        if (ey(i)) vy += d[i] * ey(i);
        if (ez(i)) vz += d[i] * ez(i);
    }
    const double s = (r > -1e-6 && r < 1e-6) ? ((r < 0.0) ? -1e-6 : 1e-6) : r;
    rho = r;
    if (below<100>(s) && below<900>(vx) && below<900>(vy) && below<900>(vz)) {
        const double rs = 1.0 / s;
        ux = quot(vx, s, rs);
        uy = quot(vy, s, rs);
        uz = quot(vz, s, rs);
    } else {
        // an infinite population makes every component NaN: the products with
        // its zero components that the sums leave out do
        const double z = 0. * vx + 0. * vy + 0. * vz;
        ux = vx / s + z;
        uy = vy / s + z;
        uz = vz / s + z;
    }
}
// e_i . u, zero components left out
MT_HD double edot_ref(int i, double ux, double uy, double uz)
{
    if (ex(i) && ey(i) && ez(i)) return ex(i) * ux + ey(i) * uy + ez(i) * uz;
    if (ex(i) && ey(i)) return ex(i) * ux + ey(i) * uy;
    if (ex(i) && ez(i)) return ex(i) * ux + ez(i) * uz;
    if (ey(i) && ez(i)) return ey(i) * uy + ez(i) * uz;
    return ex(i) ? ex(i) * ux : (ey(i) ? ey(i) * uy : (ez(i) ? ez(i) * uz : 0.));
}
// LBM_Manager::calculateFeq (BGK), one direction (LBM_Manager.cpp:205-233)
template <int Q> MT_HD double feq_ref(int i, double rho, double ux, double uy, double uz)
{
    const double uu = ux * ux + uy * uy + uz * uz;
    const double euv = edot_ref(i, ux, uy, uz);
    return rho * w<Q>(i) * (1. + 3. * euv + 4.5 * euv * euv - 1.5 * uu);
}
// Collision_LBGK::collide on one cell in place (Collision_Manager.cpp:13-53):
// f - (f - feq) / tau, rtau = RN(1 / tau)
template <int Q>
MT_HD void lbgk_ref(double *f, double rho, double ux, double uy, double uz, double tau, double rtau)
{
    if (below<500>(rho) && below<200>(ux) && below<200>(uy) && below<200>(uz) && below<100>(tau) && below<100>(rtau)) {
#pragma unroll
        for (int k = 0; k < Q; ++k) f[k] = f[k] - quot(f[k] - feq_ref<Q>(k, rho, ux, uy, uz), tau, rtau);
    } else {
        // (a copy the compiler cannot see through: it would otherwise form the
        // equilibria both branches need ahead of them and hold all Q)
        double r = rho;
#ifdef __CUDA_ARCH__
        asm volatile("" : "+d"(r));
#endif
#pragma unroll
        for (int k = 0; k < Q; ++k) f[k] = f[k] - (f[k] - feq_ref<Q>(k, r, ux, uy, uz)) / tau;
    }
}
// LBM_Manager::calculateFeq_HeLuo, one direction (LBM_Manager.cpp:235-263)
template <int Q> MT_HD double feq_heluo_ref(int i, double rho, double ux, double uy, double uz)
{
    const double uu = ux * ux + uy * uy + uz * uz;
    const double euv = edot_ref(i, ux, uy, uz);
    return w<Q>(i) * (rho + 1.0 * (3. * euv + 4.5 * euv * euv - 1.5 * uu));
}

// The same three functions for any real type R: with R = double they are
// the reference-order versions above, with R = float the reduced-precision
// path's arithmetic.
template <int Q, class R> MT_HD void macros_g(const R *d, R &rho, R &ux, R &uy, R &uz)
{
    if constexpr (std::is_same<R, double>::value) {
        macros_ref<Q>(d, rho, ux, uy, uz);
        return;
    }
    R r = d[0], vx = 0, vy = 0, vz = 0;
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        r += d[i];
        vx += d[i] * ex(i);
        vy += d[i] * ey(i);
        vz += d[i] * ez(i);
    }
    const R s = (r > R(-1e-6) && r < R(1e-6)) ? ((r < R(0)) ? R(-1e-6) : R(1e-6)) : r;
    rho = r;
    const R is = R(1) / s;
    ux = vx * is;
    uy = vy * is;
    uz = vz * is;
}
// For a direction known at run time only: the whole product e . u (edot_ref asks
// for the components one by one, for which the compiler lays the direction
// table out in every thread's local memory: the boundary sweep of a 96^3 FP64
// cavity 172 us, 19 us this way).
template <int Q, class R> MT_HD R feq_dir(int i, R rho, R ux, R uy, R uz)
{
    const R uu = ux * ux + uy * uy + uz * uz;
    const R euv = ex(i) * ux + ey(i) * uy + ez(i) * uz;
    return rho * (R)w<Q>(i) * (R(1) + R(3) * euv + R(4.5) * euv * euv - R(1.5) * uu);
}
template <int Q, class R> MT_HD R feq_g(int i, R rho, R ux, R uy, R uz)
{
    if constexpr (std::is_same<R, double>::value) return feq_ref<Q>(i, rho, ux, uy, uz);
    return feq_dir<Q, R>(i, rho, ux, uy, uz);
}
template <int Q, class R> MT_HD R feq_heluo_g(int i, R rho, R ux, R uy, R uz)
{
    if constexpr (std::is_same<R, double>::value) return feq_heluo_ref<Q>(i, rho, ux, uy, uz);
    const R uu = ux * ux + uy * uy + uz * uz;
    const R euv = ex(i) * ux + ey(i) * uy + ez(i) * uz;
    return (R)w<Q>(i) * (rho + R(1) * (R(3) * euv + R(4.5) * euv * euv - R(1.5) * uu));
}

// backward chimera step of one line (Collision_Cumulant.cpp:486-651); Z0, Z1, Z2
// mark moments the relaxation set to zero, whose terms are left out
template <bool Z0 = false, bool Z1 = false, bool Z2 = false>
MT_HD void chim_back(double a0, double a1, double a2, double v, double v2, double &pn, double &pz, double &pp)
{
    const double t = Z1 ? 0. : a1 * 2 * v, n1 = Z1 ? 0. : a1 * (2 * v - 1), p1 = Z1 ? 0. : a1 * (2 * v + 1);
    pz = Z0 ? -t : (Z1 ? a0 * (1 - v2) : a0 * (1 - v2) - t);
    pn = Z0 ? n1 : (Z1 ? a0 * (v2 - v) : a0 * (v2 - v) + n1);
    pp = Z0 ? p1 : (Z1 ? a0 * (v2 + v) : a0 * (v2 + v) + p1);
    if (!Z2) {
        pz = pz - a2;
        pn = pn + a2;
        pp = pp + a2;
    }
    pn = pn * 0.5;
    pp = pp * 0.5;
}

// D3Q27 cumulant collision (Collision_Cumulant.cpp:320-652): central moments
// about u, second-order cumulants relaxed with omega1 = 1/tau and bulk rate 1,
// all cumulants of order >= 3 reset to zero, backward cumulant and chimera
// transforms.  Slot (a,b,c) of the moment arrays is a + 3b + 9c.  The
// (2,1,0), (1,0,2) and (0,2,1) moments keep their forward values in the
// backward pass, as in the reference (Collision_Cumulant.cpp:451-454).  FP64 in
// the reference's expression order: bit-for-bit without FMA contraction
// (terms with a moment that was set to zero left out).
MT_HD void cumulant_collide(const double *f, double rho, double ux, double uy, double uz, double omega1, double *out)
{
    double m[27];
#define MM(a, b, c) m[(a) + 3 * (b) + 9 * (c)]
#pragma unroll
    for (int i = 0; i < 27; ++i) m[i] = 0;
#pragma unroll
    for (int i = 0; i < 27; ++i) {
        const double cx = ex(i) - ux, cy = ey(i) - uy, cz = ez(i) - uz, fi = f[i];
        MM(0, 0, 0) += fi;
        MM(1, 0, 0) += cx * fi;
        MM(0, 1, 0) += cy * fi;
        MM(0, 0, 1) += cz * fi;
        MM(2, 0, 0) += cx * cx * fi;
        MM(0, 2, 0) += cy * cy * fi;
        MM(0, 0, 2) += cz * cz * fi;
        MM(1, 1, 0) += cx * cy * fi;
        MM(1, 0, 1) += cx * cz * fi;
        MM(0, 1, 1) += cy * cz * fi;
        MM(2, 1, 0) += cx * cx * cy * fi;
        MM(0, 2, 1) += cy * cy * cz * fi;
        MM(1, 0, 2) += cx * cz * cz * fi;
    }
    double c200 = MM(2, 0, 0), c020 = MM(0, 2, 0), c002 = MM(0, 0, 2);
    double c110 = MM(1, 1, 0), c101 = MM(1, 0, 1), c011 = MM(0, 1, 1);
    const double k000 = MM(0, 0, 0);
    const double om1 = omega1;
    const double ir = 1. / ((rho > -1e-6 && rho < 1e-6) ? ((rho < 0.) ? -1e-6 : 1e-6) : rho);
    // bulk rate 1: om2 = 1, and the terms with 1 - om2 vanish
    const double dxu = -(om1 * (2 * c200 - c020 - c002) + (c200 + c020 + c002 - k000)) * ir * 0.5;
    const double dyv = dxu + 3 * om1 * (c200 - c020) * 0.5 * ir;
    const double dzw = dxu + 3 * om1 * (c200 - c002) * 0.5 * ir;
    c110 *= (1 - om1);
    c101 *= (1 - om1);
    c011 *= (1 - om1);
    const double ux2 = ux * ux, uy2 = uy * uy, uz2 = uz * uz;
    const double x1 = (1 - om1) * (c200 - c020) - 3 * rho * (1 - om1 * 0.5) * (ux2 * dxu - uy2 * dyv);
    const double x2 = (1 - om1) * (c200 - c002) - 3 * rho * (1 - om1 * 0.5) * (ux2 * dxu - uz2 * dzw);
    const double x3 = k000 - 3 * rho * (1 - 0.5) * (ux2 * dxu + uy2 * dyv + uz2 * dzw);
    c200 = (x1 + x2 + x3) / 3;
    c020 = c200 - x1;
    c002 = c200 - x2;

    MM(1, 1, 0) = c110; MM(0, 1, 1) = c011; MM(1, 0, 1) = c101;
    MM(2, 0, 0) = c200; MM(0, 2, 0) = c020; MM(0, 0, 2) = c002;
    // (1,2,0), (0,1,2), (2,0,1) and (1,1,1) are zero
    MM(2, 1, 1) = (MM(2, 0, 0) * MM(0, 1, 1) + 2 * MM(1, 1, 0) * MM(1, 0, 1)) * ir;
    MM(1, 2, 1) = (MM(0, 2, 0) * MM(1, 0, 1) + 2 * MM(0, 1, 1) * MM(1, 1, 0)) * ir;
    MM(1, 1, 2) = (MM(0, 0, 2) * MM(1, 1, 0) + 2 * MM(1, 0, 1) * MM(0, 1, 1)) * ir;
    MM(2, 2, 0) = (MM(2, 0, 0) * MM(0, 2, 0) + 2 * MM(1, 1, 0) * MM(1, 1, 0)) * ir;
    MM(0, 2, 2) = (MM(0, 2, 0) * MM(0, 0, 2) + 2 * MM(0, 1, 1) * MM(0, 1, 1)) * ir;
    MM(2, 0, 2) = (MM(0, 0, 2) * MM(2, 0, 0) + 2 * MM(1, 0, 1) * MM(1, 0, 1)) * ir;
    MM(1, 2, 2) = (MM(0, 2, 0) * MM(1, 0, 2) + 2 * (MM(1, 0, 1) * MM(0, 2, 1))) * ir;
    MM(2, 1, 2) = (MM(0, 0, 2) * MM(2, 1, 0) + 2 * (MM(1, 1, 0) * MM(1, 0, 2))) * ir;
    MM(2, 2, 1) = (MM(2, 0, 0) * MM(0, 2, 1) + 2 * (MM(0, 1, 1) * MM(2, 1, 0))) * ir;
    {
        const double a = (MM(2, 0, 0) * MM(0, 2, 2) + MM(0, 2, 0) * MM(2, 0, 2) + MM(0, 0, 2) * MM(2, 2, 0) +
                          4 * (MM(0, 1, 1) * MM(2, 1, 1) + MM(1, 0, 1) * MM(1, 2, 1) + MM(1, 1, 0) * MM(1, 1, 2))) * ir;
        const double b = (16 * MM(1, 1, 0) * MM(1, 0, 1) * MM(0, 1, 1) +
                          4 * (MM(1, 0, 1) * MM(1, 0, 1) * MM(0, 2, 0) + MM(0, 1, 1) * MM(0, 1, 1) * MM(2, 0, 0) +
                               MM(1, 1, 0) * MM(1, 1, 0) * MM(0, 0, 2)) +
                          2 * MM(2, 0, 0) * MM(0, 2, 0) * MM(0, 0, 2)) * ir * ir;
        MM(2, 2, 2) = a - b;
    }
    double p1[27], p2[27];
    const double vx2 = ux * ux, vy2 = uy * uy, vz2 = uz * uz;
#define XLINE(b, c) MM(0, b, c), MM(1, b, c), MM(2, b, c), ux, vx2, p1[3 * (b) + 9 * (c)], p1[1 + 3 * (b) + 9 * (c)], \
                    p1[2 + 3 * (b) + 9 * (c)]
    chim_back<>(XLINE(0, 0));
    chim_back<>(XLINE(1, 0));
    chim_back<false, true, false>(XLINE(2, 0));  // (1,2,0) = 0
    chim_back<false, false, true>(XLINE(0, 1));  // (2,0,1) = 0
    chim_back<false, true, false>(XLINE(1, 1));  // (1,1,1) = 0
    chim_back<>(XLINE(2, 1));
    chim_back<>(XLINE(0, 2));
    chim_back<true, false, false>(XLINE(1, 2));  // (0,1,2) = 0
    chim_back<>(XLINE(2, 2));
#undef XLINE
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
            chim_back<>(p1[ix + 0 + 9 * cc], p1[ix + 3 + 9 * cc], p1[ix + 6 + 9 * cc], uy, vy2, p2[ix + 0 + 9 * cc],
                        p2[ix + 3 + 9 * cc], p2[ix + 6 + 9 * cc]);
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
        for (int iy = 0; iy < 3; ++iy)
            chim_back<>(p2[ix + 3 * iy + 0], p2[ix + 3 * iy + 9], p2[ix + 3 * iy + 18], uz, vz2, m[ix + 3 * iy + 0],
                        m[ix + 3 * iy + 9], m[ix + 3 * iy + 18]);
#pragma unroll
    for (int i = 0; i < 27; ++i) out[i] = m[(ex(i) + 1) + 3 * (ey(i) + 1) + 9 * (ez(i) + 1)];
#undef MM
}

}  // namespace mt
