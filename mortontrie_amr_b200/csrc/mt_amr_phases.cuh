// Per-phase kernels of the multi-level time step, templated on the
// population storage type S (mt_store.cuh).  With S = double every
// expression keeps the reference's operation order and, compiled without
// FMA contraction (mt_amr_f64.cu), reproduces its results bit-for-bit; the
// float / half / bfloat16 instantiations (mt_amr_lp.cu) store f - s_q, s_q
// the level's storage shift (the weights unless set), and compute in FP32.
//
// Macros are computed inside the collision kernel from the same f the
// reference's calculateMacros(level) reads just before collide(level)
// (LBM_Simulator.cpp:26-28), and written out for the solid boundary and the
// domain boundary that read them later in the substep.
#pragma once

#include <algorithm>

#include "mt_internal.hpp"
#include "mt_pack2.cuh"
#include "mt_store.cuh"

namespace mt {


// reserved boundary directions; one copy per translation unit, uploaded by
// AmrOps<S>::upload_tables when a case of that storage type is built
static __constant__ int8_t c_bdry19[26][14];
static __constant__ int8_t c_bdry27[26][18];

template <int Q, class S>
__global__ void k_init_eq(int64_t n, const uint32_t *tag, double rho0, double ux, double uy, double uz, S *f, S *fcol,
                          typename Store<S>::C *rho, typename Store<S>::C *u, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t t = tag[i];
    const bool solid = (t & TAG_SF) && !(t & (TAG_LATF | TAG_F2C | TAG_C2F | TAG_GC2F | TAG_BC));
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double v = solid ? 0. : feq_ref<Q>(k, rho0, ux, uy, uz);
        const C s = stored_f64<S>(sh, v, k);
        T::st(f, at<Q>(k, i), s);
        T::st(fcol, at<Q>(k, i), s);
    }
    rho[i] = (C)(solid ? 1. : rho0);
    u[i] = (C)(solid ? 0. : ux);
    u[n + i] = (C)(solid ? 0. : uy);
    u[2 * n + i] = (C)(solid ? 0. : uz);
}

// LBM_Manager::calculateMacros(level), LBM_Manager.cpp:1003-1050
template <int Q, class S>
__global__ void k_macros(const int32_t *list, int64_t nl, int64_t n, const S *f, typename Store<S>::C *rho,
                         typename Store<S>::C *u, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    C d[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = full_sh<S>(sh, T::ld(f, at<Q>(k, i)), k);
    C r, x, y, z;
    macros_g<Q, C>(d, r, x, y, z);
    rho[i] = r;
    u[i] = x;
    u[n + i] = y;
    u[2 * n + i] = z;
}

// the same for every level in one launch (the end of a coarse step): level l's
// blocks are [block[l], block[l + 1])
template <class S> struct MacroLevels {
    int nlev = 0;
    unsigned block[kMaxLevels + 1] = {};
    const int32_t *list[kMaxLevels] = {};
    int64_t nl[kMaxLevels] = {}, n[kMaxLevels] = {};
    const S *f[kMaxLevels] = {};
    typename Store<S>::C *rho[kMaxLevels] = {}, *u[kMaxLevels] = {};
    float shift[kMaxLevels][27] = {};
};
template <int Q, class S>
__global__ void k_macros_all(const __grid_constant__ MacroLevels<S> m)
{
    using T = Store<S>;
    using C = typename T::C;
    int l = 0;
    while (l + 1 < m.nlev && blockIdx.x >= m.block[l + 1]) ++l;
    const int64_t j = (blockIdx.x - m.block[l]) * (int64_t)blockDim.x + threadIdx.x;
    if (j >= m.nl[l]) return;
    const int64_t i = m.list[l][j], n = m.n[l];
    const S *__restrict__ f = m.f[l];
    C d[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = full_v<S>(m.shift[l], T::ld(f, at<Q>(k, i)), k);
    C r, x, y, z;
    macros_g<Q, C>(d, r, x, y, z);
    m.rho[l][i] = r;
    m.u[l][i] = x;
    m.u[l][n + i] = y;
    m.u[l][2 * n + i] = z;
}

// The macros (rho, u into r, x, y, z) of one cell from its stored values d (in
// the compute type; overwritten) and its post-collision populations into
// out[at(k, i)]: LBM_Manager::calculateMacros with Collision_LBGK::collide
// (Collision_Manager.cpp:13-53) or Collision_Cumulant::collide
// (Collision_Cumulant.cpp:22-159).  Shared by every kernel that collides one
// cell; the reduced storages run the arithmetic of the packed pairs
// (mt_pack2.cuh), so a cell's result does not depend on the kernel.
// (a kernel that shares a cell among several threads stores directions K0 to K1)
template <int Q, class S, int COLL, int K0 = 0, int K1 = Q, class I>
__device__ __forceinline__ void macros_collide_store(typename Store<S>::C *d, typename Store<S>::C &r,
                                                     typename Store<S>::C &x, typename Store<S>::C &y,
                                                     typename Store<S>::C &z, const Relax tau, S *out, I i,
                                                     const Shift &sh)
{
    using T = Store<S>;
    if constexpr (T::shifted) {
        const float om = tau.om;
        if constexpr (COLL == MT_COLL_LBGK) {
            p2::lbgk<Q, float>(d, r, x, y, z, om, sh);
        } else {
            p2::cumulant(d, r, x, y, z, om, sh);
        }
#pragma unroll
        for (int k = K0; k < K1; ++k) T::st(out, at<Q>(k, i), d[k]);
    } else {
        macros_g<Q, double>(d, r, x, y, z);
        if constexpr (COLL == MT_COLL_LBGK) {
            lbgk_ref<Q>(d, r, x, y, z, tau.tau, tau.inv);
#pragma unroll
            for (int k = K0; k < K1; ++k) out[at<Q>(k, i)] = d[k];
        } else if constexpr (Q == 27) {
            double o[27];
            cumulant_collide(d, r, x, y, z, tau.inv, o);
#pragma unroll
            for (int k = K0; k < K1; ++k) out[at<Q>(k, i)] = o[k];
        }
    }
}

// fcol = f of one overlap_C2F cell (Collision_Manager.cpp:45-52)
template <int Q, class S>
__device__ __forceinline__ void copy_fcol(int64_t i, const S *__restrict__ f, S *__restrict__ fcol)
{
    S v[Q];  // every load before the first store
#pragma unroll
    for (int k = 0; k < Q; ++k) v[k] = f[at<Q>(k, i)];
#pragma unroll
    for (int k = 0; k < Q; ++k) fcol[at<Q>(k, i)] = v[k];
}

// calculateMacros(level) + Collision_LBGK::collide / Collision_Cumulant::collide
// on lat_f then overlap_F2C (Collision_Manager.cpp:13-53, Collision_Cumulant.cpp:22-159),
// and the copy on overlap_C2F by the blocks behind them (other cells, nothing
// shared: one launch less per substep, 3-5 us of a small level's 15)
template <int Q, class S, int COLL>
__global__ void k_collide(const int32_t *__restrict__ list, int64_t nl, const int32_t *__restrict__ copy, int64_t ncopy,
                          int64_t n, const Relax tau, const S *__restrict__ f, typename Store<S>::C *__restrict__ rho,
                          typename Store<S>::C *__restrict__ u, S *__restrict__ fcol, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t nb = (nl + blockDim.x - 1) / blockDim.x;
    if (blockIdx.x >= nb) {
        const int64_t c = (blockIdx.x - nb) * (int64_t)blockDim.x + threadIdx.x;
        if (c < ncopy) copy_fcol<Q, S>(copy[c], f, fcol);
        return;
    }
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    C d[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = T::ld(f, at<Q>(k, i));
    C r, x, y, z;
    macros_collide_store<Q, S, COLL>(d, r, x, y, z, tau, fcol, i, sh);
    rho[i] = r;
    u[i] = x;
    u[n + i] = y;
    u[2 * n + i] = z;
}

// The eight children of a coarse cell are eight consecutive slots (base a
// multiple of 8): per direction 16 bytes at 16-bit storage, 32 at FP32, 64 at
// FP64, aligned, moved by accesses of up to 32 bytes (of 16, half a sector each: a
// D3Q27 FP32 explosion of 21,000 sources 21.4 us with warm caches against 11.0).
template <class S> __device__ __forceinline__ void store8(S *p, typename Store<S>::C v)
{
    if constexpr (sizeof(S) == 8) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            asm volatile("st.global.v4.f64 [%0], {%1, %1, %1, %1};" ::"l"(p + 4 * h), "d"(v) : "memory");
    } else if constexpr (sizeof(S) == 4) {
        asm volatile("st.global.v8.f32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"l"(p), "f"(v) : "memory");
    } else {
        alignas(16) S w[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) Store<S>::st(w, h, v);
        *(uint4 *)p = *(const uint4 *)w;
    }
}
template <class S> struct Eight {
    alignas(16) S w[8];
    __device__ __forceinline__ void load(const S *p)
    {
        if constexpr (sizeof(S) == 8) {
#pragma unroll
            for (int h = 0; h < 8; h += 4)
                asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                    : "=d"(w[h]), "=d"(w[h + 1]), "=d"(w[h + 2]), "=d"(w[h + 3])
                    : "l"(p + h));
        } else if constexpr (sizeof(S) == 4) {
            asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
                : "l"(p));
        } else {
            *(uint4 *)w = __ldg((const uint4 *)p);
        }
    }
    __device__ __forceinline__ typename Store<S>::C get(int m) const { return Store<S>::cv(w[m]); }
};

// AMR_transDDF_explosion (LBM_Manager.cpp:1059-1129) per coarse source cell:
// the rescaled populations are the same for its children, written
// by one vector store per direction (where a child is left out, by one store
// per child).  child[j] the first child's slot, mask[j] the children written.
// 4-level D3Q27 FP16 sphere, per launch up to 40 us with a thread per child,
// which loaded and rescaled the same source eight times, 25 us so; the
// coalescence, whose eight 2-byte loads per direction are one of 16 bytes,
// 20 -> 13 us.
// Most levels have a few thousand sources, a fraction of what the GPU holds, and
// one thread's instructions are the time: three warps share 32 sources, each
// with all of the loads and the moments and a third of the directions'
// equilibria and stores.
// With a second post-collision buffer (fused schedule) the children of sources
// from nf2c on are written to both: those of ghost F2C cells, since nothing
// else writes them and the reference keeps them over the second substep, and
// all of them where one explosion serves both substeps (k_brick_exploded).
// cprev (MT_ITIME_EXTRAP, second substep): the sources' parent values at the
// parent's previous step, [Q][ns]; the explosion then starts from
// 1.5 fcol - 0.5 prev, the parent state extrapolated to the half step.
// (4 blocks per SM: left to itself the compiler takes 48 registers and has a
// few of the loads in flight.)
constexpr int kParts = 3;
// f(0), f(1) or f(2), the argument a constant
template <class F> __device__ __forceinline__ void by_part(int part, F &&f)
{
    if (part == 0)
        f(std::integral_constant<int, 0>{});
    else if (part == 1)
        f(std::integral_constant<int, 1>{});
    else
        f(std::integral_constant<int, 2>{});
}
// the directions of part P of kParts
template <int Q, int P> struct PartOf {
    static constexpr int K0 = P * Q / kParts, K1 = (P + 1) * Q / kParts;
};
template <int Q, class S>
__global__ void __launch_bounds__(32 * kParts, 4) k_explosion(
    const int32_t *__restrict__ src, const int32_t *__restrict__ child, const uint8_t *__restrict__ mask, int64_t ns,
    const S *__restrict__ cfcol, S *__restrict__ ffcol, double scale, S *__restrict__ ffcol2, int64_t nf2c,
    const Shift csh, const Shift fsh, const S *__restrict__ cprev = nullptr)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)32 + (threadIdx.x & 31);
    const int part = threadIdx.x >> 5;
    if (j >= ns) return;
    const unsigned mk = mask[j];
    if (!mk) return;
    const int64_t i = src[j], ch = child[j];
    C d[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = full_sh<S>(csh, T::ld(cfcol, at<Q>(k, i)), k);
    if (cprev) {
#pragma unroll
        for (int k = 0; k < Q; ++k) d[k] = C(1.5) * d[k] - C(0.5) * full_sh<S>(csh, T::ld(cprev, k * ns + j), k);
    }
    C r, x, y, z;
    macros_g<Q, C>(d, r, x, y, z);
    const int nw = ffcol2 && j >= nf2c ? 2 : 1;
    by_part(part, [&](auto p) {
        constexpr int K0 = PartOf<Q, decltype(p)::value>::K0, K1 = PartOf<Q, decltype(p)::value>::K1;
#pragma unroll
        for (int k = K0; k < K1; ++k) {
            const C fe = feq_heluo_g<Q, C>(k, r, x, y, z);
            d[k] = stored_sh<S>(fsh, fe + (C)scale * (d[k] - fe), k);
        }
#pragma unroll 1
        for (int w = 0; w < nw; ++w) {
            S *out = w ? ffcol2 : ffcol;
            if (mk == 255u) {
#pragma unroll
                for (int k = K0; k < K1; ++k) store8<S>(out + at<Q>(k, ch), d[k]);
            } else {
#pragma unroll 1
                for (int m = 0; m < 8; ++m)
                    if ((mk >> m) & 1u) {
#pragma unroll
                        for (int k = K0; k < K1; ++k) T::st(out, at<Q>(k, ch + m), d[k]);
                    }
            }
        }
    });
}

// the explosion sources' parent values into prev [Q][ns] (MT_ITIME_EXTRAP)
template <int Q, class S>
__global__ void k_expl_save(const int32_t *__restrict__ src, int64_t ns, const S *__restrict__ cfcol, int64_t nc,
                            S *__restrict__ prev)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= ns) return;
    const int64_t i = src[j];
#pragma unroll
    for (int k = 0; k < Q; ++k) prev[k * ns + j] = cfcol[at<Q>(k, i)];
}

// The mean of a coarse cell's eight children at directions K0 to K1
// (LBM_Manager.cpp:1141-1152).
template <int Q, int K0, int K1, class S>
__device__ __forceinline__ void children_mean(const S *__restrict__ ff, int64_t ch, const Shift &fsh,
                                              typename Store<S>::C *a)
{
    using C = typename Store<S>::C;
    Eight<S> e[K1 - K0];
#pragma unroll
    for (int k = K0; k < K1; ++k) e[k - K0].load(ff + at<Q>(k, ch));
#pragma unroll
    for (int k = K0; k < K1; ++k) {
        C s = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m) s += full_sh<S>(fsh, e[k - K0].get(m), k);
        a[k] = s / (C)8.0;
    }
}

// AMR_transDDF_coalescence (LBM_Manager.cpp:1131-1169) of 32 cells by kParts
// warps: each takes the means of a third of the directions, all need the
// moments of the whole, so the means go through shared memory, and each stores
// its third of the rescaled populations (val: as stored, for a collision).
// A level's few thousand cells leave most of the GPU idle and one thread's
// instructions are the time, as in the explosion.  Per coarse step, against a
// thread with all of a cell: 4-level D3Q27 FP32 sphere 425 -> 393 us, FP32 cavity
// over three levels 116 -> 107 us, 3-level D3Q27 FP64 sphere 153 -> 144 us.
template <int Q, class S>
__device__ __forceinline__ void coalesce(typename Store<S>::C (*mean)[32], typename Store<S>::C (*val)[32], int part,
                                         int lane, bool on, int64_t i, int64_t ch, S *__restrict__ cf,
                                         const S *__restrict__ ff, double scale, const Shift &csh, const Shift &fsh)
{
    using T = Store<S>;
    using C = typename T::C;
    by_part(part, [&](auto p) {
        constexpr int K0 = PartOf<Q, decltype(p)::value>::K0, K1 = PartOf<Q, decltype(p)::value>::K1;
        C a[Q];
        children_mean<Q, K0, K1>(ff, ch, fsh, a);
#pragma unroll
        for (int k = K0; k < K1; ++k) mean[k][lane] = a[k];
    });
    __syncthreads();
    C a[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) a[k] = mean[k][lane];
    C r, x, y, z;
    macros_g<Q, C>(a, r, x, y, z);
    by_part(part, [&](auto p) {
        constexpr int K0 = PartOf<Q, decltype(p)::value>::K0, K1 = PartOf<Q, decltype(p)::value>::K1;
#pragma unroll
        for (int k = K0; k < K1; ++k) {
            const C fe = feq_heluo_g<Q, C>(k, r, x, y, z);
            const C st = stored_sh<S>(csh, fe + (C)scale * (a[k] - fe), k);
            if (on) T::st(cf, at<Q>(k, i), st);
            if (val) {
                S sv;
                T::st(&sv, 0, st);
                val[k][lane] = T::cv(sv);
            }
        }
    });
}
template <int Q, class S>
__global__ void __launch_bounds__(32 * kParts, 4) k_coalescence(const int32_t *__restrict__ list,
                                                             const int32_t *__restrict__ child, int64_t nl,
                                                             S *__restrict__ cf, const S *__restrict__ ff, double scale,
                                                             const Shift csh, const Shift fsh)
{
    using C = typename Store<S>::C;
    __shared__ C mean[Q][32];
    const int lane = threadIdx.x & 31;
    const int64_t j0 = blockIdx.x * (int64_t)32 + lane, j = j0 < nl ? j0 : nl - 1;
    coalesce<Q, S>(mean, nullptr, threadIdx.x >> 5, lane, j0 < nl, list[j], child[j], cf, ff, scale, csh, fsh);
}

// Fused schedule: coalescence onto the F2C cells, then (the cells' f being
// untouched until the next substep's collide) their next collision into
// fnext, from the stored f as the reference's collide would read it; the
// macros of that f are written when `macros` is set (the level's last
// substep of the coarse step: calculateMacros of every level follows).
template <int Q, class S, int COLL>
__global__ void __launch_bounds__(32 * kParts, 4) k_coal_collide(
    const int32_t *__restrict__ list, const int32_t *__restrict__ child, int64_t nl, int64_t nc, S *__restrict__ cf,
    const S *__restrict__ ff, double scale, const Relax tau, S *__restrict__ cfnext,
    typename Store<S>::C *__restrict__ rho, typename Store<S>::C *__restrict__ u, int macros, const Shift csh,
    const Shift fsh)
{
    using C = typename Store<S>::C;
    __shared__ C mean[Q][32], val[Q][32];
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int64_t j0 = blockIdx.x * (int64_t)32 + lane, j = j0 < nl ? j0 : nl - 1;
    const bool on = j0 < nl;
    const int64_t i = list[j];
    coalesce<Q, S>(mean, val, part, lane, on, i, child[j], cf, ff, scale, csh, fsh);
    __syncthreads();
    if (!on) return;
    auto collide = [&](auto k0, auto k1) {
        C a[Q], r, x, y, z;
#pragma unroll
        for (int k = 0; k < Q; ++k) a[k] = val[k][lane];
        macros_collide_store<Q, S, COLL, decltype(k0)::value, decltype(k1)::value>(a, r, x, y, z, tau, cfnext, i, csh);
        if (macros && part == 0) {
            rho[i] = r;
            u[i] = x;
            u[nc + i] = y;
            u[2 * nc + i] = z;
        }
    };
    if constexpr (COLL == MT_COLL_LBGK) {
        by_part(part, [&](auto p) {
            using D = PartOf<Q, decltype(p)::value>;
            collide(std::integral_constant<int, D::K0>{}, std::integral_constant<int, D::K1>{});
        });
    } else if (part == 0) {
        // a third of its outputs costs as much as all of them (done by each part,
        // the FP64 sphere's step was 160 us)
        collide(std::integral_constant<int, 0>{}, std::integral_constant<int, Q>{});
    }
}

// Non-equilibrium extrapolation ("eflow stable" form) on one boundary set:
// f_k(b) = feq_k(rho_b, u_bc) + f_k(b + e_k) - feq_k(rho_n, u_n) over the
// reserved directions (NonEquilibrumExtrapolation.cpp:33-71).  Boundary f
// is read by nothing but this update: a Jacobi sweep (values first, then
// writes) keeps it deterministic.
template <int Q, class S>
__global__ void k_bc_neq(const int32_t *list, int64_t nl, int b, int64_t n, const int32_t *nbr,
                         const typename Store<S>::C *rho, const typename Store<S>::C *u, S *f, double ubx,
                         double uby, double ubz, double *tmp, int phase, int *err, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    constexpr int W = Q == 19 ? 14 : 18;
    for (int t = 0; t < W; ++t) {
        const int k = Q == 19 ? c_bdry19[b][t] : c_bdry27[b][t];
        if (k < 0) break;
        if (phase == 0) {
            const int32_t nb = k == 0 ? (int32_t)i : nbr[(int64_t)(k - 1) * n + i];
            if (nb < 0) {
                atomicOr(err, DEVERR_MISSING_BC_NBR);
                tmp[t * nl + j] = (double)full_sh<S>(sh, T::ld(f, at<Q>(k, i)), k);
                continue;
            }
            const C fw = feq_dir<Q, C>(k, rho[i], (C)ubx, (C)uby, (C)ubz);
            const C fn = feq_dir<Q, C>(k, rho[nb], u[nb], u[n + nb], u[2 * n + nb]);
            tmp[t * nl + j] = (double)(fw + full_sh<S>(sh, T::ld(f, at<Q>(k, nb)), k) - fn);
        } else {
            T::st(f, at<Q>(k, i), stored_sh<S>(sh, (C)tmp[t * nl + j], k));
        }
    }
}

// the same sweep over every boundary set at once (one Jacobi pass: all values,
// then all writes); setb gives each cell's set, ub its face's velocity.  One
// thread per cell and reserved direction (t = blockIdx.y): a direction costs
// three dependent loads, and with the directions in one thread's loop their
// latencies came one after the other (a 45x37x41 cavity's 9,700 boundary
// cells, caches cold: 19.5 and 11 us for the two launches, 4.8 us each so).
struct BcVel {
    double u[26][3];
};
template <int Q> constexpr int kBcRows = Q == 19 ? 14 : 18;
template <int Q, class S>
__global__ void __launch_bounds__(128) k_bc_neq_all(const int32_t *__restrict__ list, const int8_t *__restrict__ setb,
                                                    int64_t nl, int64_t n, const int32_t *__restrict__ nbr,
                                                    const typename Store<S>::C *__restrict__ rho,
                                                    const typename Store<S>::C *__restrict__ u, S *__restrict__ f,
                                                    const BcVel ub, double *__restrict__ tmp, int phase, int *err,
                                                    const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (j >= nl) return;
    const int64_t i = list[j];
    const int b = setb[j];
    const int k = Q == 19 ? c_bdry19[b][t] : c_bdry27[b][t];
    if (k < 0) return;
    if (phase == 0) {
        const int32_t nb = k == 0 ? (int32_t)i : nbr[(int64_t)(k - 1) * n + i];
        if (nb < 0) {
            atomicOr(err, DEVERR_MISSING_BC_NBR);
            tmp[t * nl + j] = (double)full_sh<S>(sh, T::cv(f[at<Q>(k, i)]), k);
            return;
        }
        const C fw = feq_dir<Q, C>(k, rho[i], (C)ub.u[b][0], (C)ub.u[b][1], (C)ub.u[b][2]);
        const C fn = feq_dir<Q, C>(k, rho[nb], u[nb], u[n + nb], u[2 * n + nb]);
        tmp[t * nl + j] = (double)(fw + full_sh<S>(sh, T::cv(f[at<Q>(k, nb)]), k) - fn);
    } else {
        T::st(f, at<Q>(k, i), stored_sh<S>(sh, (C)tmp[t * nl + j], k));
    }
}

// Restated inlet/outflow on the x faces: West wall cells hold
// fcol = feq(rho0, u_bc) (BC/ZouHe_Velocity.cpp:62-115 writes the
// equilibrium at the boundary cell's own, never-updated density), East wall
// cells copy the inner cell's fcol (BC/Outflow.cpp:39-52).
template <int Q, class S>
__global__ void __launch_bounds__(64) k_bc_inout(const int32_t *__restrict__ west, int64_t nw,
                                                 const int32_t *__restrict__ east, int64_t ne, int64_t n,
                                                 const int32_t *__restrict__ nbr, double rho0, S *__restrict__ f,
                                                 S *__restrict__ fcol, double ubx, double uby, double ubz, int *err,
                                                 const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nw + ne) return;
    const bool out = j >= nw;
    const int64_t i = out ? east[j - nw] : west[j];
    const int32_t nb = nbr[(int64_t)((out ? 2 : 1) - 1) * n + i];
    if (nb < 0) {
        atomicOr(err, DEVERR_MISSING_BC_NBR);
        return;
    }
    S v[Q];
    if (out) {
#pragma unroll
        for (int k = 0; k < Q; ++k) v[k] = fcol[at<Q>(k, nb)];
    } else {
#pragma unroll
        for (int k = 0; k < Q; ++k) T::st(v, k, stored_sh<S>(sh, feq_g<Q, C>(k, (C)rho0, (C)ubx, (C)uby, (C)ubz), k));
    }
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        fcol[at<Q>(k, i)] = v[k];
        f[at<Q>(k, i)] = v[k];
    }
}

// Restated wet-node boundaries on the x faces (MT_BC_ZOUHE_HH, D3Q19):
// after the level-0 stream the West / East shell cells pull from their
// neighbours like fluid cells (a missing source keeps f) and complete the
// populations that come from outside the box -- West: the Zou-He velocity
// inlet with the Hecht-Harting transverse corrections (the formula family of
// BC/ZouHe_Velocity.cpp:81-93,170-199); East: the five incoming populations
// copied from the inner neighbour's streamed ones (BC/Outflow.cpp:39-52).
// The formulas are those of a textbook stream; under the reference's
// reversed pull they act on g_k = f_inv(k) with the velocity -u_bc.
// k_bc_wall_collide then collides the completed cells (LBGK, level-0 tau).
template <class S>
__global__ void k_bc_hh(const int32_t *list, int64_t nl, int east, int64_t n, int textbook,
                        const int32_t *__restrict__ nbr, const S *__restrict__ fcol, S *__restrict__ f, double ux,
                        double uy, double uz, int *err, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    C g[19];
#pragma unroll
    for (int k = 0; k < 19; ++k) {
        const int m = textbook ? k : inv(k);
        const int32_t src = m == 0 ? (int32_t)i : nbr[(int64_t)((textbook ? inv(m) : m) - 1) * n + i];
        g[k] = full_sh<S>(sh, src >= 0 ? T::ld(fcol, at<19>(m, src)) : T::ld(f, at<19>(m, i)), m);
    }
    const C sgn = textbook ? C(1) : C(-1);
    if (!east) {
        const C Ux = sgn * (C)ux, Uy = sgn * (C)uy, Uz = sgn * (C)uz;
        const C rho = (g[0] + g[3] + g[4] + g[5] + g[6] + g[15] + g[16] + g[17] + g[18] +
                       C(2) * (g[2] + g[8] + g[10] + g[12] + g[14])) / (C(1) - Ux);
        const C ny = C(0.5) * (g[3] + g[15] + g[17] - g[4] - g[16] - g[18]) - rho * Uy / C(3);
        const C nz = C(0.5) * (g[5] + g[15] + g[18] - g[6] - g[16] - g[17]) - rho * Uz / C(3);
        g[1] = g[2] + rho * Ux / C(3);
        g[7] = g[8] + rho * (Ux + Uy) / C(6) - ny;
        g[9] = g[10] + rho * (Ux - Uy) / C(6) + ny;
        g[11] = g[12] + rho * (Ux + Uz) / C(6) - nz;
        g[13] = g[14] + rho * (Ux - Uz) / C(6) + nz;
    } else {
        const int32_t nb = nbr[(int64_t)(2 - 1) * n + i];  // the cell at -x
        if (nb < 0) {
            atomicOr(err, DEVERR_MISSING_BC_NBR);
            return;
        }
        const int in_e[5] = {2, 8, 10, 12, 14};
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            const int k = in_e[t], m = textbook ? k : inv(k);
            g[k] = full_sh<S>(sh, T::ld(f, at<19>(m, nb)), m);
        }
    }
#pragma unroll
    for (int k = 0; k < 19; ++k) {
        const int m = textbook ? k : inv(k);
        T::st(f, at<19>(m, i), stored_sh<S>(sh, g[k], m));
    }
}

template <class S>
__global__ void k_bc_wall_collide(const int32_t *list, int64_t nl, int64_t n, const Relax tau, const S *__restrict__ f,
                                  S *__restrict__ fcol, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    C d[19];
#pragma unroll
    for (int k = 0; k < 19; ++k) d[k] = T::ld(f, at<19>(k, i));
    C r, x, y, z;
    macros_collide_store<19, S, MT_COLL_LBGK>(d, r, x, y, z, tau, fcol, i, sh);
}

// D3Q19_BC_Strategy::initial_Feq (D3Q19_BC_Manager.hpp:157-167) on one
// boundary set: f = fcol = feq(rho0, u) with the face's velocity
template <int Q, class S>
__global__ void k_bc_set_eq(const int32_t *list, int64_t nl, int64_t n, double rho0, double ux, double uy, double uz,
                            S *f, S *fcol, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double v = feq_ref<Q>(k, rho0, ux, uy, uz);
        const C st = stored_f64<S>(sh, v, k);
        T::st(f, at<Q>(k, i), st);
        T::st(fcol, at<Q>(k, i), st);
    }
}

// SinglePointInterpolation::treat (ComplexBoundary_Manager.cpp:43-225) on
// one cell: wall links by Filippova-Haenel or distance-weighted
// interpolation, free links by plain pull, density clamp, eight
// multi-direct-forcing sweeps (each cell only touches its own populations:
// the sweeps run in registers).  g receives the new f, (fx, fy, fz) the
// cell's momentum-exchange force.
// The cell count is small (a sphere's skin), so the time is one thread's
// chain of dependent loads.  What does not change is laid out once per case,
// by cell of the IB list (IbTab, k_ib_tables): a mask of the wall links, each
// link's interpolation factor and its source slot.  A cell then loads its tables
// in one round and every population in a second, with addresses and operands
// selected instead of branches taken (a link without a source reads the cell's
// own opposite population, which is its value).  One warp per SM has only its
// own instructions to issue, 6 cycles each: a wall link costs no division, a
// sweep one (quot) instead of three and a root.
// One launch, caches cold, D3Q19 FP16 / D3Q27 FP16 / D3Q27 FP64: 35 / 50 / 49 us
// with the links' loads behind branches, 16 / 28 / 23 us from the neighbour
// table and the distance rows in three rounds; two launches of 4 us each that
// summed the force are gone (ib_force_add).  Caches warm, D3Q19 FP16 / FP64 in
// phase order / D3Q27 FP64: 11.4 / 14.1 / 22.7 us with divisions per link and the
// force finished in every launch, 7.5 / 9.0 / 19.7 us so.
template <class C> struct IbTab {
    const uint2 *__restrict__ wall;  // [nib] x bit k: link k meets the wall, y bit k: closer than half a link
    const int32_t *__restrict__ src; // [(Q - 1) nib] link k's source slot, -1 none
    // [(Q - 1) nib] of wall links the distance d (distance-weighted); or 2 d where
    // closer than half a link, else 1 / (2 d) (Filippova-Haenel)
    const C *__restrict__ factor;
    int64_t nib;
};
template <int Q, class C>
__global__ void k_ib_tables(const int32_t *__restrict__ list, int64_t nl, int64_t n, const int32_t *__restrict__ disrow,
                            const double *__restrict__ dis, const int32_t *__restrict__ nbr, int fh, uint2 *wall,
                            int32_t *src, C *factor)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    const double *dr = dis + (int64_t)disrow[i] * (Q - 1);
    uint2 m = make_uint2(0, 0);
    for (int k = 1; k < Q; ++k) {
        const double v = dr[inv(k) - 1];
        const bool hit = v != -1.;
        const C d = (C)v;
        if (hit) m.x |= 1u << k;
        if (hit && d < (C)0.5) m.y |= 1u << k;
        // a wall link interpolates with the population arriving from the far side
        src[(int64_t)(k - 1) * nl + j] = nbr[(int64_t)((hit ? inv(k) : k) - 1) * n + i];
        factor[(int64_t)(k - 1) * nl + j] = !fh ? d : d < (C)0.5 ? (C)2.0 * d : (C)1.0 / ((C)2.0 * d);
    }
    wall[j] = m;
}
// FP32 multiplications and additions are paired into FMAs as written here
// (pm_*), whatever surrounds them; in FP64 pm_fma is a multiplication and an
// addition.
__device__ __forceinline__ float pm_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float pm_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float pm_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double pm_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double pm_add(double a, double b) { return a + b; }
__device__ __forceinline__ double pm_fma(double a, double b, double c) { return a * b + c; }
// x / b from rb = 1 / b: one correction gives the rounded quotient (FP64: mt_lattice's
// quot; FP32: all 2^23 mantissas of b with 100 x each, no difference)
__device__ __forceinline__ float pm_quot(float x, float b, float rb)
{
    const float q = __fmul_rn(x, rb);
    return __fmaf_rn(__fmaf_rn(-q, b, x), rb, q);
}
__device__ __forceinline__ double pm_quot(double x, double b, double rb) { return quot(x, b, rb); }
template <class C> __device__ constexpr C pm_tiny() { return sizeof(C) == 8 ? (C)0x1p-100 : (C)0x1p-40f; }
template <class C> __device__ constexpr C pm_huge() { return sizeof(C) == 8 ? (C)0x1p100 : (C)0x1p40f; }
// the smallest s with sqrt(s) >= 1e-10
template <class C> __device__ constexpr C pm_still()
{
    return sizeof(C) == 8 ? (C)0x1.79ca10c924223p-67 : (C)0x1.79ca1p-67f;
}
template <int Q, int FH, class S>
__device__ __forceinline__ void ib_cell(int64_t i, int64_t j, const IbTab<typename Store<S>::C> &t,
                                        const S *__restrict__ fcol, typename Store<S>::C rho_b,
                                        typename Store<S>::C *g, typename Store<S>::C &fx, typename Store<S>::C &fy,
                                        typename Store<S>::C &fz, const Shift &sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const uint2 masks = __ldg(t.wall + j);
    const uint32_t wall = masks.x;
    C fac[Q], own[Q], src[Q];
    int32_t si[Q];
#pragma unroll
    for (int k = 1; k < Q; ++k) si[k] = __ldg(t.src + (int64_t)(k - 1) * t.nib + j);
#pragma unroll
    for (int k = 1; k < Q; ++k) fac[k] = __ldg(t.factor + (int64_t)(k - 1) * t.nib + j);
#pragma unroll
    for (int k = 0; k < Q; ++k) own[k] = T::ld(fcol, at<Q>(k, i));
#pragma unroll
    for (int k = 1; k < Q; ++k) src[k] = T::ld(fcol, si[k] >= 0 ? at<Q>(k, si[k]) : at<Q>(inv(k), i));
    g[0] = full_sh<S>(sh, own[0], 0);
    fx = 0;
    fy = 0;
    fz = 0;
#pragma unroll
    for (int k = 1; k < Q; ++k) {
        // the value of a missing source is the cell's own opposite one
        const C from = si[k] >= 0 ? full_sh<S>(sh, src[k], k) : full_sh<S>(sh, src[k], inv(k));
        g[k] = from;
        if ((wall >> k) & 1) {
            const C finc = full_sh<S>(sh, own[inv(k)], inv(k));
            const C fstr = from;
            // FH: near (1 - 2 d) finc + 2 d fstr, else 1 / (2 d) fstr + (1 - 1 / (2 d)) feq
            const C a = fac[k], b = (C)1.0 - a;
            const bool near = !FH || ((masks.y >> k) & 1);
            const C fnew = near ? pm_fma(b, finc, pm_mul(a, fstr))
                                : pm_fma(a, fstr, pm_mul(b, pm_mul((C)w19z(inv(k)), rho_b)));
            g[k] = fnew;
            const C mt = pm_add(finc, fnew);
            fx = pm_add(fx, -mt * ex(k));
            fy = pm_add(fy, -mt * ey(k));
            fz = pm_add(fz, -mt * ez(k));
        }
    }
    C ra = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k) ra = pm_add(ra, g[k]);
    if (ra < (C)0.3)
        g[0] += (C)1.0 * ((C)0.3 - ra);
    else if (ra < (C)0.5)
        g[0] += (C)0.5 * ((C)0.5 - ra);
    else if (ra > (C)3.0)
        g[0] += (C)1.0 * ((C)3.0 - ra);
    else if (ra > (C)2.0)
        g[0] += (C)0.5 * ((C)2.0 - ra);
#pragma unroll 1
    for (int it = 0; it < 8; ++it) {
        C r = 0, ux = 0, uy = 0, uz = 0;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            r = pm_add(r, g[k]);
            if (ex(k)) ux = pm_add(ux, ex(k) > 0 ? g[k] : -g[k]);
            if (ey(k)) uy = pm_add(uy, ey(k) > 0 ? g[k] : -g[k]);
            if (ez(k)) uz = pm_add(uz, ez(k) > 0 ? g[k] : -g[k]);
        }
        if (r <= (C)0.) continue;
        if (r > pm_tiny<C>() && r < pm_huge<C>()) {
            const C rr = (C)1.0 / r;
            ux = pm_quot(ux, r, rr);
            uy = pm_quot(uy, r, rr);
            uz = pm_quot(uz, r, rr);
        } else {
            ux = ux / r;
            uy = uy / r;
            uz = uz / r;
        }
        // |u| < 1e-10, the root taken on the bound
        if (ux * ux + uy * uy + uz * uz < pm_still<C>()) continue;
        const C hr = pm_mul((C)-0.5, r);
        const C mx = pm_mul(hr, ux), my = pm_mul(hr, uy), mz = pm_mul(hr, uz);
        C adj = 0;
#pragma unroll
        for (int k = 1; k < Q; ++k) {
            if (!((wall >> k) & 1)) continue;
            C m = 0;
            bool any = false;
            auto part = [&](int e, C v) {
                if (!e) return;
                const C t = e > 0 ? v : -v;
                m = any ? pm_add(m, t) : t;
                any = true;
            };
            part(ex(k), mx);
            part(ey(k), my);
            part(ez(k), mz);
            const C w3 = (C)w19z(k) * (C)3.0;
            g[k] = pm_fma(w3, m, g[k]);
            adj = pm_fma(-w3, m, adj);
        }
        g[0] = pm_add(g[0], adj);
    }
}

// The force of treat() (LBM_Manager::accumIBForce): the kernel that computed it
// adds each 32-cell block's sum (a fixed tree) to the block's own partial, and
// once per coarse step k_ib_force_sum adds the partials in block order
// (strided over the warp, then the same tree) to the accumulator.  (Finished
// in every launch by the last block, behind a fence and a counter, the sum
// was 2 us at the end of the substep's longest kernel.)
// part: [3 * blocks] partials, then the number of calls.
constexpr int kIbBlock = 32;
__device__ __forceinline__ void ib_force_tree(double &x, double &y, double &z)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        x += __shfl_down_sync(0xffffffffu, x, o);
        y += __shfl_down_sync(0xffffffffu, y, o);
        z += __shfl_down_sync(0xffffffffu, z, o);
    }
}
__device__ __forceinline__ void ib_force_add(double fx, double fy, double fz, double *part)
{
    ib_force_tree(fx, fy, fz);
    if (threadIdx.x != 0) return;
    double *p = part + 3 * (int64_t)blockIdx.x;
    p[0] += fx;
    p[1] += fy;
    p[2] += fz;
    if (blockIdx.x == 0) part[3 * (int64_t)gridDim.x] += 1.0;
}
static __global__ void __launch_bounds__(32) k_ib_force_sum(double *part, int64_t nb, double *acc)
{
    double x = 0., y = 0., z = 0.;
    for (int64_t b = threadIdx.x; b < nb; b += 32) {
        x += part[3 * b];
        y += part[3 * b + 1];
        z += part[3 * b + 2];
        part[3 * b] = part[3 * b + 1] = part[3 * b + 2] = 0.;
    }
    ib_force_tree(x, y, z);
    if (threadIdx.x == 0) {
        acc[0] += x;
        acc[1] += y;
        acc[2] += z;
        acc[3] += part[3 * nb];
        part[3 * nb] = 0.;
    }
}

template <int Q, int FH, class S>
__global__ void __launch_bounds__(kIbBlock) k_ib_treat(const int32_t *__restrict__ list, int64_t nl,
                                                       const IbTab<typename Store<S>::C> t,
                                                       const S *__restrict__ fcol,
                                                       const typename Store<S>::C *__restrict__ rho, S *__restrict__ f,
                                                       double *part, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)kIbBlock + threadIdx.x;
    C fx = 0, fy = 0, fz = 0;
    if (j < nl) {
        const int64_t i = list[j];
        C g[Q];
        ib_cell<Q, FH, S>(i, j, t, fcol, rho[i], g, fx, fy, fz, sh);
#pragma unroll
        for (int k = 0; k < Q; ++k) T::st(f, at<Q>(k, i), stored_sh<S>(sh, g[k], k));
    }
    ib_force_add((double)fx, (double)fy, (double)fz, part);
}

// ---- fused schedule ---------------------------------------------------------
// The level keeps two post-collision buffers.  A substep streams from the
// current one (fcol) and, in the same pass, runs the next substep's
// calculateMacros + collide on the streamed f, writing fnext.  Between the
// stream of one substep and the collision of the next the reference touches a
// lat_f cell's f only through treat() (IB cells, fused below) and a C2F
// cell's fcol only through the copy fcol = f, so the lookahead collision sees
// the same f as the reference's and gives the same populations.

// gather of one cell's streamed populations from the source indices src[k]
// (k >= 1; -1 = no neighbour): every load is issued before any store (f and
// fcol are distinct buffers), so the Q - 1 gathers overlap.  A missing
// neighbour keeps f (read back from f, not written).
template <int Q, class S>
__device__ __forceinline__ void pull_src(int64_t i, int64_t n, const int32_t *src, const S *__restrict__ fcol,
                                         S *__restrict__ f, S *v)
{
    v[0] = fcol[at<Q>(0, i)];
#pragma unroll
    for (int k = 1; k < Q; ++k) v[k] = src[k] >= 0 ? fcol[at<Q>(k, src[k])] : f[at<Q>(k, i)];
    f[at<Q>(0, i)] = v[0];
#pragma unroll
    for (int k = 1; k < Q; ++k)
        if (src[k] >= 0) f[at<Q>(k, i)] = v[k];
}

template <int Q, class S>
__device__ __forceinline__ void pull_cell(int64_t i, int64_t n, int textbook, const int32_t *__restrict__ nbr,
                                          const S *__restrict__ fcol, S *__restrict__ f, S *v)
{
    int32_t src[Q];
#pragma unroll
    for (int k = 1; k < Q; ++k) src[k] = __ldg(nbr + (int64_t)((textbook ? inv(k) : k) - 1) * n + i);
    pull_src<Q, S>(i, n, src, fcol, f, v);
}

// ABPatternPull::stream (Stream_Manager.cpp:43-76): a missing neighbour keeps f
template <int Q, class S>
__global__ void k_stream(const int32_t *__restrict__ list, int64_t nl, int64_t n, int textbook,
                         const int32_t *__restrict__ nbr, const S *__restrict__ fcol, S *__restrict__ f)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    S v[Q];
    pull_cell<Q, S>(list[j], n, textbook, nbr, fcol, f, v);
}

// ABPatternPull::stream then the next collide, on lat_f cells that are not IB
// cells.
template <int Q, class S, int COLL>
__global__ void k_pull_collide(const int32_t *__restrict__ list, int64_t nl, int64_t n, int textbook,
                               const int32_t *__restrict__ nbr, const S *__restrict__ fcol, S *__restrict__ f,
                               S *__restrict__ fnext, const Relax tau, typename Store<S>::C *__restrict__ rho,
                               typename Store<S>::C *__restrict__ u, int macros, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    C d[Q];
    {
        S v[Q];
        pull_cell<Q, S>(i, n, textbook, nbr, fcol, f, v);
#pragma unroll
        for (int k = 0; k < Q; ++k) d[k] = T::cv(v[k]);
    }
    C r, x, y, z;
    macros_collide_store<Q, S, COLL>(d, r, x, y, z, tau, fnext, i, sh);
    if (macros) {
        rho[i] = r;
        u[i] = x;
        u[n + i] = y;
        u[2 * n + i] = z;
    }
}

// stream on overlap_C2F cells and their next collision, fcol = f
// (Collision_Manager.cpp:45-52)
template <int Q, class S>
__global__ void k_pull_copy(const int32_t *__restrict__ list, int64_t nl, int64_t n, int textbook,
                            const int32_t *__restrict__ nbr, const S *__restrict__ fcol, S *__restrict__ f,
                            S *__restrict__ fnext)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nl) return;
    const int64_t i = list[j];
    S v[Q];
    pull_cell<Q, S>(i, n, textbook, nbr, fcol, f, v);
#pragma unroll
    for (int k = 0; k < Q; ++k) fnext[at<Q>(k, i)] = v[k];
}

// The fused pass over a level's 4x4x4 bricks, one warp per brick that has work.
// A cell's sources lie in its own brick and the 26 around it: the warp reads
// those 27 brick numbers once (108 B per brick; a table of every cell's
// sources would be 4 (Q - 1) B per cell) and each source slot follows from
// the cell's local coordinates.  The brick neighbours come from
// Morton_Assist::find_neighbor on a corner cell, so each source is the cell the
// reference's find() returns.
// Classes (bcls): 1 stream + collide, 3 the same with the streamed f stored, 2
// stream (f stored) + copy, 4 a direct-forcing band cell (stream; collided
// after the forcing), 6 stream (f stored; the explosion wrote the next
// collision).  The streamed f of class-1 cells is read by nothing in
// the coarse step (their next collision is computed here, a missing link's
// f never changes), so it is stored only when `fall` is set or when the
// state leaves the fused schedule (k_brick_pull).
// When `macros` is set (the level's last substep of the coarse step) the
// macros of the streamed f are written too: they are what the all-level
// calculateMacros at the end of the coarse step computes.
struct BrickTab {
    const int32_t *__restrict__ list, *__restrict__ nbr;
    const unsigned long long *__restrict__ mask;
    const uint8_t *__restrict__ cls, *__restrict__ flag;
};

// a warp's neighbourhood in shared memory: where each neighbour brick's
// populations start (an absent one: the brick's own, never used as a source)
// and, for bricks with a missing source, its occupancy
struct BrickHood {
    uint32_t off[27];
    unsigned long long mask[27];
};
template <int Q>
__device__ __forceinline__ void brick_hood(int32_t b, int lane, const BrickTab &t, bool complete, BrickHood &h)
{
    if (lane < 27) {
        const int32_t e = __ldg(t.nbr + 27 * (int64_t)b + lane);
        h.off[lane] = (uint32_t)(e >= 0 ? e : b) * (64u * Q);
        if (!complete) h.mask[lane] = e >= 0 ? __ldg(t.mask + e) : 0ull;
    }
    __syncwarp();
}

// one axis of a source position, v = local coordinate + offset in -1..4: bits
// 0-5 its share of the local Morton index, bits 6 and up of the neighbour's
// number; the three axes' shares add
template <int A> __device__ __forceinline__ int axis_pos(int v)
{
    constexpr int step = A == 0 ? 1 : (A == 1 ? 3 : 9);
    return ((((v >> 2) + 1) * step) << 6) | ((v & 1) << A) | ((v & 2) << (A + 2));
}

// the streamed populations of one cell (local Morton index m)
template <int Q, class S>
__device__ __forceinline__ void brick_gather(uint32_t i, int textbook, bool complete, const BrickHood &h,
                                             const S *__restrict__ fcol, const S *__restrict__ f, S *v)
{
    const int m = (int)(i & 63u);
    const int x = (m & 1) | ((m >> 2) & 2), y = ((m >> 1) & 1) | ((m >> 3) & 2), z = ((m >> 2) & 1) | ((m >> 4) & 2);
    int px[3], py[3], pz[3];
#pragma unroll
    for (int d = -1; d <= 1; ++d) {
        const int s = textbook ? -d : d;
        px[1 + d] = axis_pos<0>(x + s);
        py[1 + d] = axis_pos<1>(y + s);
        pz[1 + d] = axis_pos<2>(z + s);
    }
    v[0] = fcol[at<Q>(0, i)];
#pragma unroll
    for (int k = 1; k < Q; ++k) {
        const int p = px[1 + ex(k)] + py[1 + ey(k)] + pz[1 + ez(k)];
        const S *src = fcol + (h.off[p >> 6] + (uint32_t)(p & 63)) + 64 * k;
        if (complete)
            v[k] = *src;
        else
            v[k] = ((h.mask[p >> 6] >> (p & 63)) & 1) ? *src : f[at<Q>(k, i)];
    }
}

// one cell of the pass (i its slot): FP64, and form 1 of the reduced storages
template <int Q, class S, int COLL>
__device__ __forceinline__ void brick_cell(uint32_t i, int cls, bool complete, const BrickHood &h, uint32_t n,
                                           int textbook, const S *__restrict__ fcol, S *__restrict__ f,
                                           S *__restrict__ fnext, const Relax tau, typename Store<S>::C *__restrict__ rho,
                                           typename Store<S>::C *__restrict__ u, int macros, int fall,
                                           long long *__restrict__ acc, const Shift &sh)
{
    using T = Store<S>;
    using C = typename T::C;
    if (!cls) return;
    S v[Q];
    brick_gather<Q, S>(i, textbook, complete, h, fcol, f, v);
    if (cls != 1 || fall) {
        // a missing link's value is f's own: storing it again changes nothing
#pragma unroll
        for (int k = 0; k < Q; ++k) f[at<Q>(k, i)] = v[k];
    }
    if (cls == 2) {
#pragma unroll
        for (int k = 0; k < Q; ++k) fnext[at<Q>(k, i)] = v[k];
        return;
    }
    if (cls == 6) return;
    C d[Q];
    if (cls == 4) {
        // direct-forcing band: collided after the forcing; with acc the
        // band's rho, unforced velocity and cleared accumulator are
        // written here (what k_band_macros computes from the stored f)
        if constexpr (COLL == MT_COLL_LBGK) {
            if (acc) {
                C r, x, y, z;
#pragma unroll
                for (int k = 0; k < Q; ++k) d[k] = full_sh<S>(sh, T::cv(v[k]), k);
                macros_g<Q, C>(d, r, x, y, z);
                rho[i] = r;
                u[i] = x;
                u[n + i] = y;
                u[2 * n + i] = z;
                acc[i] = 0;
                acc[n + i] = 0;
                acc[2 * n + i] = 0;
            }
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = T::cv(v[k]);
    C r, x, y, z;
    macros_collide_store<Q, S, COLL>(d, r, x, y, z, tau, fnext, i, sh);
    if (macros) {
        rho[i] = r;
        u[i] = x;
        u[n + i] = y;
        u[2 * n + i] = z;
    }
}

// The gather of a pair, lane = its y, z, x coordinates' bits (y0 z0 x1 y1 z1).
// For each (y, z) offset the sources are the pair at the same x and, for
// e_x = +-1, also the next pair on that side, whose near cell completes the
// word.  All 9 + 2 x 18 loads are issued before the first is used.
template <int Q, class S, bool TB>
__device__ __forceinline__ void pair_gather(int lane, const BrickHood &h, const S *__restrict__ fcol,
                                            typename CellPair<S>::W *v)
{
    using CP = CellPair<S>;
    constexpr int sg = TB ? -1 : 1;
    const int x1 = (lane >> 2) & 1;
    const int y = (lane & 1) | ((lane >> 2) & 2), z = ((lane >> 1) & 1) | ((lane >> 3) & 2);
    const int xm = 64 + 8 * x1, xl = x1 ? 64 : 8, xr = x1 ? 128 : 72;
    typename CP::W e[Q];
#pragma unroll
    for (int g = 0; g < 9; ++g) {
        const int dy = g % 3 - 1, dz = g / 3 - 1;
        const int pyz = axis_pos<1>(y + dy) + axis_pos<2>(z + dz);
        const int pm = xm + pyz, pl = xl + pyz, pr = xr + pyz;
        const S *sm = fcol + (h.off[pm >> 6] + (uint32_t)(pm & 63));
        const S *sl = fcol + (h.off[pl >> 6] + (uint32_t)(pl & 63));
        const S *sr = fcol + (h.off[pr >> 6] + (uint32_t)(pr & 63));
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            if (ey(k) != sg * dy || ez(k) != sg * dz) continue;
            v[k] = CP::ld(sm + 64 * k);
            if (sg * ex(k) < 0) e[k] = CP::ld(sl + 64 * k);
            if (sg * ex(k) > 0) e[k] = CP::ld(sr + 64 * k);
        }
    }
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        if (sg * ex(k) < 0) v[k] = CP::straddle(e[k], v[k]);
        if (sg * ex(k) > 0) v[k] = CP::straddle(v[k], e[k]);
    }
}

// a missing link keeps f (bricks without BRICK_COMPLETE)
template <int Q, class S>
__device__ __forceinline__ void pair_missing(int lane, int textbook, const BrickHood &h, const S *own,
                                             typename CellPair<S>::W *v)
{
    const int x1 = (lane >> 2) & 1;
    const int y = (lane & 1) | ((lane >> 2) & 2), z = ((lane >> 1) & 1) | ((lane >> 3) & 2);
    const int s = textbook ? -1 : 1;
#pragma unroll
    for (int k = 1; k < Q; ++k) {
        const int pyz = axis_pos<1>(y + s * ey(k)) + axis_pos<2>(z + s * ez(k));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int p = axis_pos<0>(2 * x1 + c + s * ex(k)) + pyz;
            if (!((h.mask[p >> 6] >> (p & 63)) & 1)) CellPair<S>::put(v[k], c, own + 64 * k);
        }
    }
}

// One warp's brick for the reduced storages: a lane gathers, collides and
// stores a pair of cells, the collision in packed FP32 (mt_pack2.cuh).
// Against one cell per lane step (form 1) a pair has 45 loads of a word for
// D3Q27 where the cells have 54 of a value, 27 addresses (the Q accesses of a
// source pair are constant offsets) for 54, half the stores and conversions
// and half the arithmetic's issue slots: 79 M instructions for the finest
// level of the 4-level cumulant sphere where the cell-by-cell pass over a
// [Q][n] array had 133 M, 124 us for 215 us (108 B of populations per cell:
// 72 us at the measured copy rate), FP32 168 us for 310 us.  What bounds it
// now: the FP32 pipe (65 % active) and the gathers' latency at 28 warps per SM
// side by side, DRAM at 46 % of its peak (both of a capture at 24).
template <int Q, class S, int COLL>
__device__ __forceinline__ void brick_warp_pair(int32_t b, int lane, BrickHood &h, const BrickTab &t, uint32_t n,
                                                int textbook, const S *__restrict__ fcol, S *__restrict__ f,
                                                S *__restrict__ fnext, const Relax tau, float *__restrict__ rho,
                                                float *__restrict__ u, int macros, int fall,
                                                long long *__restrict__ acc, const Shift &sh)
{
    using CP = CellPair<S>;
    const int flag = __ldg(t.flag + b);
    const bool complete = flag & BRICK_COMPLETE, uniform = flag & BRICK_UNIFORM;
    brick_hood<Q>(b, lane, t, complete, h);
    const uint32_t i = 64u * (uint32_t)b + 2u * lane;
    int c0 = 1, c1 = 1;
    if (!uniform) {
        const unsigned short cc = __ldg((const unsigned short *)(t.cls + i));
        c0 = cc & 255;
        c1 = cc >> 8;
        if (!cc) return;
    }
    const uint32_t o = at<Q>(0, i);
    typename CP::W v[Q];
    if (textbook)
        pair_gather<Q, S, true>(lane, h, fcol, v);
    else
        pair_gather<Q, S, false>(lane, h, fcol, v);
    if (!complete) pair_missing<Q, S>(lane, textbook, h, f + o, v);
    auto store = [&](S *p, bool s0, bool s1) {
        if (s0 && s1) {
#pragma unroll
            for (int k = 0; k < Q; ++k) CP::st(p + 64 * k, v[k]);
        } else if (s0 || s1) {
            const int w = s1;
#pragma unroll
            for (int k = 0; k < Q; ++k) CP::st_one(p + 64 * k, v[k], w);
        }
    };
    if (fall || !uniform) {
        store(f + o, c0 && (c0 != 1 || fall), c1 && (c1 != 1 || fall));
        store(fnext + o, c0 == 2, c1 == 2);
    }
    const bool k0 = c0 & 1, k1 = c1 & 1;  // classes 1 and 3
    const bool b0 = c0 == 4 && acc, b1 = c1 == 4 && acc;
    if (!(k0 || k1 || b0 || b1)) return;
    float2 d[Q], r, x, y, z;
    const float om = tau.om;
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = CP::f2(v[k]);
    if constexpr (COLL == MT_COLL_LBGK)
        p2::lbgk<Q, float2>(d, r, x, y, z, om, sh);
    else
        p2::cumulant(d, r, x, y, z, om, sh);
#pragma unroll
    for (int k = 0; k < Q; ++k) v[k] = CP::word(d[k]);
    store(fnext + o, k0, k1);
    const bool m0 = (macros && k0) || b0, m1 = (macros && k1) || b1;
    if (m0 && m1) {
        *(float2 *)(rho + i) = r;
        *(float2 *)(u + i) = x;
        *(float2 *)(u + n + i) = y;
        *(float2 *)(u + 2 * n + i) = z;
    } else if (m0 || m1) {
        const uint32_t j = i + (m1 ? 1u : 0u);
        rho[j] = m1 ? r.y : r.x;
        u[j] = m1 ? x.y : x.x;
        u[n + j] = m1 ? y.y : y.x;
        u[2 * n + j] = m1 ? z.y : z.x;
    }
    if constexpr (COLL == MT_COLL_LBGK) {
        // the band's accumulator restarts from zero
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (c ? b1 : b0) {
                acc[i + c] = 0;
                acc[n + i + c] = 0;
                acc[2 * n + i + c] = 0;
            }
    }
}

// a brick in form V: the reduced storages' forms 0, 2, 3 are the pair form at
// different numbers of resident blocks, 1 goes cell by cell; FP64 goes cell by
// cell (3: the lane's two cells in one unrolled sequence)
template <int Q, class S, int COLL, int V>
__device__ __forceinline__ void brick_warp(int32_t b, int lane, BrickHood &h, const BrickTab &t, uint32_t n,
                                           int textbook, const S *__restrict__ fcol, S *__restrict__ f,
                                           S *__restrict__ fnext, const Relax tau, typename Store<S>::C *__restrict__ rho,
                                           typename Store<S>::C *__restrict__ u, int macros, int fall,
                                           long long *__restrict__ acc, const Shift &sh)
{
    if constexpr (Store<S>::shifted && V != 1) {
        brick_warp_pair<Q, S, COLL>(b, lane, h, t, n, textbook, fcol, f, fnext, tau, rho, u, macros, fall, acc, sh);
    } else {
        const bool complete = __ldg(t.flag + b) & BRICK_COMPLETE;
        brick_hood<Q>(b, lane, t, complete, h);
        const uint32_t i = 64u * (uint32_t)b + (uint32_t)lane;
        const int c0 = __ldg(t.cls + i), c1 = __ldg(t.cls + i + 32);
        if constexpr (V == 3) {
            brick_cell<Q, S, COLL>(i, c0, complete, h, n, textbook, fcol, f, fnext, tau, rho, u, macros, fall, acc, sh);
            brick_cell<Q, S, COLL>(i + 32, c1, complete, h, n, textbook, fcol, f, fnext, tau, rho, u, macros, fall, acc,
                                   sh);
        } else {
#pragma unroll 1
            for (int part = 0; part < 2; ++part)
                brick_cell<Q, S, COLL>(i + 32 * part, part ? c1 : c0, complete, h, n, textbook, fcol, f, fnext, tau, rho,
                                       u, macros, fall, acc, sh);
        }
    }
}

// Resident 128-thread blocks per SM asked of a brick pass.  Measured per launch
// (finest level of the 4-level D3Q27 cumulant sphere, 4.28 M cells; direct-
// forcing sphere R 8, D3Q19 LBGK, 8.9 M cells), pair form:
//   D3Q27 FP16: 4 blocks 143.7 us, 5 136.2, 6 128.0, 7 124.6, 8 (spills) 144.4
//   D3Q27 FP32: 4 blocks 191.5 us, 5 175.1, 6 (40 B of spills) 166.9, 7 183.3
//   D3Q19 FP16: 5 blocks 216.1 us, 6 194.2, 7 183.3, 8 177.2, 9 175.1
//   D3Q19 FP32: 5 blocks 283.0 us, 6 263.2, 7 250.9
// Form 0 is what a level runs untuned: the fastest number, but 7 for D3Q19 at 16
// bits, where 9 (56 registers, 52 B of spills) lose on levels of less than a
// wave (a 537,000-cell sphere's coarse step 141 us with 7, 146 with 9).
template <int Q, class S, int COLL, int V> constexpr int brick_min_blocks()
{
    if (!Store<S>::shifted) return 1;
    if (V == 1) return Store<S>::bytes == 2 ? ((COLL == MT_COLL_LBGK && Q == 19) ? 10 : 8) : 7;
    if (Store<S>::bytes == 2) return Q == 19 ? (V == 0 ? 7 : (V == 2 ? 8 : 9)) : (V == 0 ? 7 : (V == 2 ? 6 : 8));
    return Q == 19 ? (V == 0 ? 7 : (V == 2 ? 6 : 5)) : (V == 0 ? 6 : (V == 2 ? 5 : 7));
}
// the form a level runs until mt_case_tune_bricks times them
template <class S> constexpr int brick_default_variant() { return 0; }

template <int Q, class S, int COLL, int V>
__global__ void __launch_bounds__(128, brick_min_blocks<Q, S, COLL, V>()) k_brick_step(
    int64_t nb, const BrickTab t, uint32_t n, int textbook, const S *__restrict__ fcol, S *__restrict__ f,
    S *__restrict__ fnext, const Relax tau, typename Store<S>::C *__restrict__ rho, typename Store<S>::C *__restrict__ u,
    int macros, int fall, long long *__restrict__ acc, const Shift sh)
{
    __shared__ BrickHood hood[4];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t j = 4 * (int64_t)blockIdx.x + w;
    if (j >= nb) return;
    brick_warp<Q, S, COLL, V>(__ldg(t.list + j), lane, hood[w], t, n, textbook, fcol, f, fnext, tau, rho, u, macros,
                              fall, acc, sh);
}

// ABPatternPull::stream (Stream_Manager.cpp:43-76) over bricks: the lat_f and
// overlap_C2F cells pull from sources found as in the fused pass, without the
// neighbour table's 4 (Q - 1) B per cell (D3Q19 FP64: 304 B of populations).
// skip_ib: without the IB cells, which treat() writes whole (amr_lbm_kernel).
template <int Q, class S>
__global__ void __launch_bounds__(128) k_stream_bricks(int64_t nb, const int32_t *__restrict__ nbr,
                                                       const unsigned long long *__restrict__ mask,
                                                       const uint32_t *__restrict__ tag, int skip_ib, int textbook,
                                                       const S *__restrict__ fcol, S *__restrict__ f)
{
    __shared__ BrickHood hood[4];
    auto streamed = [skip_ib](uint32_t t) {
        return (t & (TAG_LATF | TAG_C2F)) && !(skip_ib && (t & TAG_LATF) && (t & TAG_IB));
    };
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t b = 4 * (int64_t)blockIdx.x + w;
    if (b >= nb) return;
    const uint32_t i0 = 64u * (uint32_t)b + (uint32_t)lane;
    const uint32_t t0 = __ldg(tag + i0), t1 = __ldg(tag + i0 + 32);
    if (!__any_sync(0xffffffffu, streamed(t0) || streamed(t1))) return;
    brick_hood<Q>((int32_t)b, lane, BrickTab{nullptr, nbr, mask, nullptr, nullptr}, false, hood[w]);
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        if (!streamed(part ? t1 : t0)) continue;
        const uint32_t i = i0 + 32u * part;
        S v[Q];
        brick_gather<Q, S>(i, textbook, false, hood[w], fcol, f, v);
        // a missing link's value is f's own: storing it again changes nothing
#pragma unroll
        for (int k = 0; k < Q; ++k) f[at<Q>(k, i)] = v[k];
    }
}

// The streamed f of the class-1 cells, from the buffer the last fused pass
// read (the values that pass would have stored).
template <int Q, class S>
__global__ void __launch_bounds__(128) k_brick_pull(int64_t nb, const BrickTab t, int textbook,
                                                    const S *__restrict__ fcol, S *__restrict__ f)
{
    __shared__ BrickHood hood[4];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t j = 4 * (int64_t)blockIdx.x + w;
    if (j >= nb) return;
    const int32_t b = __ldg(t.list + j);
    const bool complete = __ldg(t.flag + b) & BRICK_COMPLETE;
    brick_hood<Q>(b, lane, t, complete, hood[w]);
    for (int part = 0; part < 2; ++part) {
        const uint32_t i = 64u * (uint32_t)b + (uint32_t)lane + 32u * part;
        if (__ldg(t.cls + i) != 1) continue;
        S v[Q];
        brick_gather<Q, S>(i, textbook, complete, hood[w], fcol, f, v);
#pragma unroll
        for (int k = 0; k < Q; ++k) f[at<Q>(k, i)] = v[k];
    }
}

// treat() on the IB cells of the finest level, then their next collision.
// rho_b is the density calculateMacros(level) gives at the start of the
// substep: the macros of the cell's f before this treat.
template <int Q, int FH, class S, int COLL>
__global__ void __launch_bounds__(kIbBlock) k_ib_collide(
    const int32_t *__restrict__ list, int64_t nl, int64_t n, const IbTab<typename Store<S>::C> t,
    const S *__restrict__ fcol, S *__restrict__ f,
    S *__restrict__ fnext, const Relax tau, double *part, typename Store<S>::C *__restrict__ rho,
    typename Store<S>::C *__restrict__ u, int macros, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)kIbBlock + threadIdx.x;
    C fx = 0, fy = 0, fz = 0;
    if (j < nl) {
        const int64_t i = list[j];
        C g[Q];
        C r, x, y, z;
#pragma unroll
        for (int k = 0; k < Q; ++k) g[k] = full_sh<S>(sh, T::cv(f[at<Q>(k, i)]), k);
        macros_g<Q, C>(g, r, x, y, z);
        ib_cell<Q, FH, S>(i, j, t, fcol, r, g, fx, fy, fz, sh);
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const C st = stored_sh<S>(sh, g[k], k);
            T::st(f, at<Q>(k, i), st);
            // the next collision reads the stored value
            S sv;
            T::st(&sv, 0, st);
            g[k] = T::cv(sv);
        }
        macros_collide_store<Q, S, COLL>(g, r, x, y, z, tau, fnext, i, sh);
        if (macros) {
            rho[i] = r;
            u[i] = x;
            u[n + i] = y;
            u[2 * n + i] = z;
        }
    }
    ib_force_add((double)fx, (double)fy, (double)fz, part);
}

// ---- direct-forcing immersed boundary (Lagrangian markers) --------------------
// No reference counterpart: a rigid sphere represented by surface markers on
// the finest level, explicit direct forcing (Uhlmann 2005) with the 3-point
// kernel of Roma, Peskin & Berger (1999) and Guo forcing in the collision.
// The Eulerian force of a substep is spread into int64 fixed point (2^-32),
// so the atomic sums are exact and independent of the order of arrival.
constexpr double kForceScale = 4294967296.0;  // 2^32
constexpr double kForceInv = 1.0 / 4294967296.0;

__host__ __device__ __forceinline__ double roma3(double r)
{
    r = fabs(r);
    if (r <= 0.5) return (1.0 + sqrt(1.0 - 3.0 * r * r)) / 3.0;
    if (r <= 1.5) {
        const double a = 1.0 - r;
        return (5.0 - 3.0 * r - sqrt(1.0 - 3.0 * a * a)) / 6.0;
    }
    return 0.0;
}

// rho and the unforced velocity of the band cells from their streamed f; the
// band's force accumulator restarts from zero
template <int Q, class S>
__global__ void k_band_macros(const int32_t *band, int64_t nb, int64_t n, const S *f, typename Store<S>::C *rho,
                              typename Store<S>::C *u, long long *acc, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nb) return;
    const int64_t i = band[j];
    C d[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) d[k] = full_sh<S>(sh, T::ld(f, at<Q>(k, i)), k);
    C r, x, y, z;
    macros_g<Q, C>(d, r, x, y, z);
    rho[i] = r;
    u[i] = x;
    u[n + i] = y;
    u[2 * n + i] = z;
    acc[i] = 0;
    acc[n + i] = 0;
    acc[2 * n + i] = 0;
}

// one marker: interpolate rho and u at X(t), force F = 2 rho (U - u), spread
// F dv phi into the band cells; fk receives -F dv (the force on the body)
// grid[(x - lo) + dx ((y - lo) + dy (z - lo))] = index of band cell (x, y, z) or -1
static __global__ void k_band_grid(const int32_t *band, int64_t nb, const LevelMap map, int64_t lx, int64_t ly,
                            int64_t lz, int64_t dx, int64_t dy, int64_t dz, int32_t *grid)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nb) return;
    const int32_t i = band[j];
    const uint64_t k = map.key(i);
    const int64_t x = (int64_t)compact3(k) - lx, y = (int64_t)compact3(k >> 1) - ly, z = (int64_t)compact3(k >> 2) - lz;
    if (x < 0 || y < 0 || z < 0 || x >= dx || y >= dy || z >= dz) return;
    grid[x + dx * (y + dy * z)] = i;
}

// One warp per marker, a lane per stencil cell: 27 lookups, 108 gathers and 81
// additions each go out as one instruction's worth of independent accesses,
// where a thread with all of them had a few dozen per marker in flight on one
// warp per SM.  Lanes 0 to 3 then add up rho and u over the cells in the order
// of the stencil (a cell outside the band, idx -1, adds nothing).  5,864 markers:
// 16.7 us per launch by a thread each, 8.4 us so, bound by the issue of address
// arithmetic and the additions at L2.
constexpr int kMarkerWarps = 4;
template <class C>
__global__ void __launch_bounds__(32 * kMarkerWarps) k_df_markers(
    int64_t nm, const double *__restrict__ ref, const double *__restrict__ dv, double cx, double cy, double cz,
    const double *__restrict__ path, int64_t period, const long long *__restrict__ tstep,
    const int32_t *__restrict__ grid, int64_t lx, int64_t ly, int64_t lz, int64_t dx, int64_t dy, int64_t dz, int64_t n,
    const C *__restrict__ rho, const C *__restrict__ u, long long *__restrict__ acc, double *__restrict__ fk)
{
    __shared__ C val[kMarkerWarps][4][27];
    __shared__ double wgt[kMarkerWarps][27];
    __shared__ bool has[kMarkerWarps][27];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t m = blockIdx.x * (int64_t)kMarkerWarps + w;
    if (m >= nm) return;  // the whole warp
    const int64_t ph = *tstep % period;
    const double *pp = path + 6 * ph;
    const double X = cx + pp[0] + ref[m], Y = cy + pp[1] + ref[nm + m], Z = cz + pp[2] + ref[2 * nm + m];
    const double d = dv[m];
    const int64_t ix = (int64_t)floor(X), iy = (int64_t)floor(Y), iz = (int64_t)floor(Z);
    const int c = lane < 27 ? lane : 26;
    const int ox = c % 3, oy = (c / 3) % 3, oz = c / 9;
    // only band cells take force; they all lie in the grid's box
    const int64_t gx = ix + ox - 1 - lx, gy = iy + oy - 1 - ly, gz = iz + oz - 1 - lz;
    const bool in = gx >= 0 && gy >= 0 && gz >= 0 && gx < dx && gy < dy && gz < dz;
    const int32_t idx = in ? __ldg(grid + gx + dx * (gy + dy * gz)) : -1;
    // the stencil weight wx wy wz, multiplied in that order
    const double wv = roma3((double)(ix + ox - 1) + 0.5 - X) * roma3((double)(iy + oy - 1) + 0.5 - Y) *
                      roma3((double)(iz + oz - 1) + 0.5 - Z);
    if (lane < 27) {
        const int64_t i = idx >= 0 ? idx : 0;
        val[w][0][lane] = rho[i];
        val[w][1][lane] = u[i];
        val[w][2][lane] = u[n + i];
        val[w][3][lane] = u[2 * n + i];
        wgt[w][lane] = wv;
        has[w][lane] = idx >= 0;
    }
    __syncwarp();
    double sum = 0.0;
    if (lane < 4) {
#pragma unroll
        for (int k = 0; k < 27; ++k)
            if (has[w][k]) sum += wgt[w][k] * (double)val[w][lane][k];
    }
    const double r = __shfl_sync(0xffffffffu, sum, 0), vx = __shfl_sync(0xffffffffu, sum, 1);
    const double vy = __shfl_sync(0xffffffffu, sum, 2), vz = __shfl_sync(0xffffffffu, sum, 3);
    const double fx = 2.0 * r * (pp[3] - vx), fy = 2.0 * r * (pp[4] - vy), fz = 2.0 * r * (pp[5] - vz);
    if (lane < 27 && idx >= 0) {
        const double s = wv * d;
        atomicAdd((unsigned long long *)(acc + idx), (unsigned long long)__double2ll_rn(fx * s * kForceScale));
        atomicAdd((unsigned long long *)(acc + n + idx), (unsigned long long)__double2ll_rn(fy * s * kForceScale));
        atomicAdd((unsigned long long *)(acc + 2 * n + idx), (unsigned long long)__double2ll_rn(fz * s * kForceScale));
    }
    if (lane == 0) {
        fk[m] = -fx * d;
        fk[nm + m] = -fy * d;
        fk[2 * nm + m] = -fz * d;
    }
}

// the body force of one forcing step: a fixed-order sum of the markers'
// forces into the accumulator (fx, fy, fz, count), then the substep count
static __global__ void __launch_bounds__(256) k_df_sum(const double *fk, int64_t nm, double *part, unsigned *done,
                                                        double *acc, long long *tstep)
{
    // body force: a fixed-order tree over each block of 256 markers, then the
    // last block to finish sums the partials in block order (deterministic)
    __shared__ double s[3][256];
    __shared__ bool last;
    const int t = threadIdx.x;
    const int64_t j = blockIdx.x * (int64_t)256 + t;
    for (int c = 0; c < 3; ++c) s[c][t] = j < nm ? fk[c * nm + j] : 0.0;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (t < w)
            for (int c = 0; c < 3; ++c) s[c][t] += s[c][t + w];
        __syncthreads();
    }
    if (t == 0) {
        for (int c = 0; c < 3; ++c) part[3 * blockIdx.x + c] = s[c][0];
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a[3] = {0., 0., 0.};
    for (int64_t b = t; b < gridDim.x; b += 256)
        for (int c = 0; c < 3; ++c) a[c] += __ldcg(part + 3 * b + c);
    for (int c = 0; c < 3; ++c) s[c][t] = a[c];
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (t < w)
            for (int c = 0; c < 3; ++c) s[c][t] += s[c][t + w];
        __syncthreads();
    }
    if (t == 0) {
        for (int c = 0; c < 3; ++c) acc[c] += s[c][0];
        acc[3] += 1.0;
        *tstep += 1;
        *done = 0u;
    }
}

// LBGK collision with Guo forcing on the band cells: u = (j + g / 2) / rho,
// fcol = f - (f - feq(rho, u)) / tau + (1 - 1 / (2 tau)) w [3 (e - u) + 9 (e.u) e].g
// (the band's rho and unforced velocity are written by k_band_macros)
template <int Q, class S>
__global__ void k_band_collide(const int32_t *band, int64_t nb, int64_t n, const Relax tau, const S *f,
                               const long long *acc, S *fcol, const Shift sh)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nb) return;
    const int64_t i = band[j];
    if constexpr (T::shifted) {
        // reduced precision: the stored deviations s = f - s_k throughout
        // (the shift sums to 1 and its first moment is u_s), the forcing term
        // as 3 (e.g - u.g) + 9 (e.u)(e.g)
        float sd[Q];
        float rd = 0.f, jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            sd[k] = T::ld(f, at<Q>(k, i));
            rd += sd[k];
            jx += sd[k] * ex(k);
            jy += sd[k] * ey(k);
            jz += sd[k] * ez(k);
        }
        const float gx = (float)((double)acc[i] * kForceInv), gy = (float)((double)acc[n + i] * kForceInv),
                    gz = (float)((double)acc[2 * n + i] * kForceInv);
        const float r = 1.f + rd;
        jx += sh.u[0];
        jy += sh.u[1];
        jz += sh.u[2];
        const float rs = (r > -1e-6f && r < 1e-6f) ? ((r < 0.f) ? -1e-6f : 1e-6f) : r;
        const float ir = 1.f / rs;
        const float x = (jx + 0.5f * gx) * ir, y = (jy + 0.5f * gy) * ir, z = (jz + 0.5f * gz) * ir;
        const float om = tau.om;
        const float fpre = 1.f - 0.5f * om;
        const float uu = 1.5f * (x * x + y * y + z * z);
        const float ug = x * gx + y * gy + z * gz;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const float eu = ex(k) * x + ey(k) * y + ez(k) * z;
            const float eg = ex(k) * gx + ey(k) * gy + ez(k) * gz;
            const float wk = (float)w<Q>(k);
            const float dfeq = wk * ((r - 1.f) + r * (3.f * eu + 4.5f * eu * eu - uu)) - sh.dw[k];
            const float ge = 3.f * (eg - ug) + 9.f * eu * eg;
            T::st(fcol, at<Q>(k, i), fmaf(om, dfeq - sd[k], sd[k]) + fpre * wk * ge);
        }
        return;
    }
    C d[Q];
    C r = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        d[k] = full_sh<S>(sh, T::ld(f, at<Q>(k, i)), k);
        r += d[k];
        jx += d[k] * ex(k);
        jy += d[k] * ey(k);
        jz += d[k] * ez(k);
    }
    // times 2^-32: exactly the division by the power-of-two scale
    const C gx = (C)((double)acc[i] * kForceInv), gy = (C)((double)acc[n + i] * kForceInv),
            gz = (C)((double)acc[2 * n + i] * kForceInv);
    const C rs = (r > C(-1e-6) && r < C(1e-6)) ? ((r < C(0)) ? C(-1e-6) : C(1e-6)) : r;
    const C x = (jx + gx * C(0.5)) / rs, y = (jy + gy * C(0.5)) / rs, z = (jz + gz * C(0.5)) / rs;
    const C om = (C)tau.inv;
    const C fpre = C(1) - C(0.5) * om;
    const C uu = x * x + y * y + z * z;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const C eu = ex(k) * x + ey(k) * y + ez(k) * z;
        const C feq = r * (C)w<Q>(k) * (C(1) + C(3) * eu + C(4.5) * eu * eu - C(1.5) * uu);
        const C ge = (C(3) * (ex(k) - x) + C(9) * eu * ex(k)) * gx + (C(3) * (ey(k) - y) + C(9) * eu * ey(k)) * gy +
                     (C(3) * (ez(k) - z) + C(9) * eu * ez(k)) * gz;
        const C out = d[k] - (d[k] - feq) * om + fpre * (C)w<Q>(k) * ge;
        T::st(fcol, at<Q>(k, i), stored_sh<S>(sh, out, k));
    }
}

static __global__ void k_force_tick(double *acc, double steps) { acc[3] += steps; }

// Host arrays hold a level's stored cells in key order ([Q][nc], [nc]); slot[r]
// is the slot of cell r.
template <int Q, class S>
__global__ void k_to_f64(const S *src, double *dst, const int32_t *__restrict__ slot, int64_t nc, const Shift sh)
{
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nc) return;
    const int64_t i = slot[r];
#pragma unroll
    for (int k = 0; k < Q; ++k) dst[k * nc + r] = (double)full_sh<S>(sh, Store<S>::ld(src, at<Q>(k, i)), k);
}
template <int Q, class S>
__global__ void k_from_f64(const double *src, S *dst, const int32_t *__restrict__ slot, int64_t nc, const Shift sh)
{
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nc) return;
    const int64_t i = slot[r];
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double v = src[k * nc + r];
        Store<S>::st(dst, at<Q>(k, i), stored_f64<S>(sh, v, k));
    }
}
// rho [nc] and u [3][nc] of the stored cells as FP64
template <class C>
__global__ void k_macro_to_f64(const C *rho, const C *u, int64_t n, const int32_t *__restrict__ slot, int64_t nc,
                               double *drho, double *du)
{
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nc) return;
    const int64_t i = slot[r];
    drho[r] = (double)rho[i];
    du[r] = (double)u[i];
    du[nc + r] = (double)u[n + i];
    du[2 * nc + r] = (double)u[2 * n + i];
}
// (slots without a cell hold anything)  A block per brick, whose Q x 64 values of
// each buffer are contiguous: 16-byte loads, a thread's slots and their share of
// the brick's occupancy from the position in the row.  (Value by value, each with
// a division for its brick and its cell's tag, a 96^3 D3Q19 cavity's check took
// 460 us; FP64 160, FP32 100, FP16 125 us so.)
template <class S>
__global__ void __launch_bounds__(128) k_guard(const S *__restrict__ f, const S *__restrict__ fcol,
                                               const unsigned long long *__restrict__ mask, int64_t nb, int q, int *err)
{
    constexpr int E = 16 / (int)sizeof(S), ROW = 64 / E;
    const bool both = f != fcol;
    bool bad = false;
    for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const unsigned long long m = mask[b];
        const int64_t base = b * q * ROW;
        auto check = [&](const uint4 &v, int o) {
            alignas(16) S w[E];
            *(uint4 *)w = v;
#pragma unroll
            for (int e = 0; e < E; ++e) bad |= ((m >> ((o % ROW) * E + e)) & 1) && !isfinite((double)Store<S>::cv(w[e]));
        };
#pragma unroll 4
        for (int o = threadIdx.x; o < q * ROW; o += blockDim.x) {
            const uint4 x = __ldg((const uint4 *)f + base + o);
            const uint4 y = both ? __ldg((const uint4 *)fcol + base + o) : x;
            check(x, o);
            if (both) check(y, o);
        }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(err, DEVERR_NONFINITE);
}

// ----------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------
template <class S> struct AmrTyped {
    using C = typename Store<S>::C;
    static S *f(Level &lv) { return (S *)lv.f; }
    static S *fcol(Level &lv) { return (S *)lv.fcol; }
    static C *rho(Level &lv) { return (C *)lv.rho; }
    static C *u(Level &lv) { return (C *)lv.u; }
    static IbTab<C> ib(const Case &c)
    {
        return IbTab<C>{c.ib_wall, c.ib_src, (const C *)c.ib_factor, c.lv[c.d.max_level].nib};
    }
};

inline int upload_bdry_tables(Ctx &ctx)
{
    static const int8_t b19[26][14] = {
        {0, 1, 3, 4, 5, 6, 7, 9, 11, 13, 15, 16, 17, 18}, {0, 2, 3, 4, 5, 6, 8, 10, 12, 14, 15, 16, 17, 18},
        {0, 1, 2, 3, 5, 6, 7, 10, 11, 12, 13, 14, 15, 17}, {0, 1, 2, 4, 5, 6, 8, 9, 11, 12, 13, 14, 16, 18},
        {0, 1, 2, 3, 4, 5, 7, 8, 9, 10, 11, 14, 15, 18}, {0, 1, 2, 3, 4, 6, 7, 8, 9, 10, 12, 13, 16, 17},
        {0, 2, 4, 5, 6, 8, 12, 14, 16, 18, -1, -1, -1, -1}, {0, 1, 4, 5, 6, 9, 11, 13, 16, 18, -1, -1, -1, -1},
        {0, 1, 3, 5, 6, 7, 11, 13, 15, 17, -1, -1, -1, -1}, {0, 2, 3, 5, 6, 10, 12, 14, 15, 17, -1, -1, -1, -1},
        {0, 1, 2, 4, 6, 8, 9, 12, 13, 16, -1, -1, -1, -1}, {0, 1, 2, 3, 6, 7, 10, 12, 13, 17, -1, -1, -1, -1},
        {0, 1, 2, 4, 5, 8, 9, 11, 14, 18, -1, -1, -1, -1}, {0, 1, 2, 3, 5, 7, 10, 11, 14, 15, -1, -1, -1, -1},
        {0, 2, 3, 4, 6, 8, 10, 12, 16, 17, -1, -1, -1, -1}, {0, 1, 3, 4, 6, 7, 9, 13, 16, 17, -1, -1, -1, -1},
        {0, 2, 3, 4, 5, 8, 10, 14, 15, 18, -1, -1, -1, -1}, {0, 1, 3, 4, 5, 7, 9, 11, 15, 18, -1, -1, -1, -1},
        {0, 2, 4, 6, 8, 12, 16, -1, -1, -1, -1, -1, -1, -1}, {0, 1, 4, 6, 9, 13, 16, -1, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 6, 7, 13, 17, -1, -1, -1, -1, -1, -1, -1}, {0, 2, 3, 6, 10, 12, 17, -1, -1, -1, -1, -1, -1, -1},
        {0, 2, 4, 5, 8, 14, 18, -1, -1, -1, -1, -1, -1, -1}, {0, 1, 4, 5, 9, 11, 18, -1, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 5, 7, 11, 15, -1, -1, -1, -1, -1, -1, -1}, {0, 2, 3, 5, 10, 14, 15, -1, -1, -1, -1, -1, -1, -1}};
    static const int8_t b27[26][18] = {
        {0, 1, 3, 4, 5, 6, 7, 9, 11, 13, 15, 16, 17, 18, 19, 21, 24, 26},
        {0, 2, 3, 4, 5, 6, 8, 10, 12, 14, 15, 16, 17, 18, 20, 22, 23, 25},
        {0, 1, 2, 3, 5, 6, 7, 10, 11, 12, 13, 14, 15, 17, 19, 22, 24, 25},
        {0, 1, 2, 4, 5, 6, 8, 9, 11, 12, 13, 14, 16, 18, 20, 21, 23, 26},
        {0, 1, 2, 3, 4, 5, 7, 8, 9, 10, 11, 14, 15, 18, 19, 21, 23, 25},
        {0, 1, 2, 3, 4, 6, 7, 8, 9, 10, 12, 13, 16, 17, 20, 22, 24, 26},
        {0, 2, 4, 5, 6, 8, 12, 14, 16, 18, 20, 23, -1, -1, -1, -1, -1, -1},
        {0, 1, 4, 5, 6, 9, 11, 13, 16, 18, 21, 26, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 5, 6, 7, 11, 13, 15, 17, 19, 24, -1, -1, -1, -1, -1, -1},
        {0, 2, 3, 5, 6, 10, 12, 14, 15, 17, 22, 25, -1, -1, -1, -1, -1, -1},
        {0, 1, 2, 4, 6, 8, 9, 12, 13, 16, 20, 26, -1, -1, -1, -1, -1, -1},
        {0, 1, 2, 3, 6, 7, 10, 12, 13, 17, 22, 24, -1, -1, -1, -1, -1, -1},
        {0, 1, 2, 4, 5, 8, 9, 11, 14, 18, 21, 23, -1, -1, -1, -1, -1, -1},
        {0, 1, 2, 3, 5, 7, 10, 11, 14, 15, 19, 25, -1, -1, -1, -1, -1, -1},
        {0, 2, 3, 4, 6, 8, 10, 12, 16, 17, 20, 22, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 4, 6, 7, 9, 13, 16, 17, 24, 26, -1, -1, -1, -1, -1, -1},
        {0, 2, 3, 4, 5, 8, 10, 14, 15, 18, 23, 25, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 4, 5, 7, 9, 11, 15, 18, 19, 21, -1, -1, -1, -1, -1, -1},
        {0, 2, 4, 6, 8, 12, 16, 20, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 1, 4, 6, 9, 13, 16, 26, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 6, 7, 13, 17, 24, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 2, 3, 6, 10, 12, 17, 22, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 2, 4, 5, 8, 14, 18, 23, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 1, 4, 5, 9, 11, 18, 21, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 1, 3, 5, 7, 11, 15, 19, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
        {0, 2, 3, 5, 10, 14, 15, 25, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1}};
    MT_CUDA(ctx, cudaMemcpyToSymbol(c_bdry19, b19, sizeof(b19)));
    MT_CUDA(ctx, cudaMemcpyToSymbol(c_bdry27, b27, sizeof(b27)));
    return MT_OK;
}

// boundary sets of each face strategy (West, East, South, North, Bot, Top):
// the face, its edges and corners as NonEquilibrumExtrapolation.hpp:24-110
// registers them
static const int kFaceSets[6][9] = {
    {0, 7, 8, 15, 17, 19, 20, 23, 24}, {1, 6, 9, 14, 16, 18, 21, 22, 25},
    {2, 11, 13, -1, -1, -1, -1, -1, -1}, {3, 10, 12, -1, -1, -1, -1, -1, -1},
    {4, -1, -1, -1, -1, -1, -1, -1, -1}, {5, -1, -1, -1, -1, -1, -1, -1, -1}};

// Rescaling of the non-equilibrium part across a level interface.  The
// reference's factors (LBM_Manager.cpp:1065, 1137): 2 tau_f / tau_c onto the
// fine post-collision populations and tau_c / (2 tau_f) onto the coarse
// post-stream ones.  MT_SCALE_STANDARD uses the rescaling that keeps the
// physical viscous stress continuous under 2:1 convective scaling (Dupuis &
// Chopard 2003): fneq_f = tau_f / (2 tau_c) fneq_c, written for post-collision
// populations as (tau_f - 1) / (2 (tau_c - 1)), and fneq_c = 2 tau_c / tau_f fneq_f.
inline double c2f_scale(const Case &c, int fine)
{
    const double tf = c.d.tau[fine], tc = c.d.tau[fine - 1];
    return c.scaling == MT_SCALE_STANDARD ? (tf - 1.0) / (2.0 * (tc - 1.0)) : (2.0 * tf) / tc;
}
inline double f2c_scale(const Case &c, int coarse)
{
    const double tc = c.d.tau[coarse], tf = c.d.tau[coarse + 1];
    return c.scaling == MT_SCALE_STANDARD ? (2.0 * tc) / tf : tc / (2.0 * tf);
}

// the direct-forcing step on level l (after its stream): band macros, the
// markers' interpolation and spreading, the body force
// (band_macros_done: the level's brick pass already wrote the band macros)
template <class S, int Q>
int df_force(Ctx &ctx, Case &c, int l, bool band_macros_done = false)
{
    using A = AmrTyped<S>;
    using C = typename Store<S>::C;
    cudaStream_t s = ctx.stream;
    Level &lv = c.lv[l];
    if (!lv.nband) return MT_OK;
    if (!band_macros_done) {
        k_band_macros<Q, S><<<grid_for(lv.nband, 128), 128, 0, s>>>(lv.band, lv.nband, lv.n, A::f(lv), A::rho(lv),
                                                                     A::u(lv), c.acc, c.shift[l]);
        MT_LAUNCHED(ctx);
    }
    if (!c.nm) {
        k_force_tick<<<1, 1, 0, s>>>(c.force_acc, 1.0);
        MT_LAUNCHED(ctx);
        return MT_OK;
    }
    k_df_markers<C><<<grid_for(c.nm, kMarkerWarps), 32 * kMarkerWarps, 0, s>>>(
        c.nm, c.mref, c.mdv, c.center[0], c.center[1], c.center[2], c.path, c.period, c.tstep, c.mgrid, c.mlo[0],
        c.mlo[1], c.mlo[2], c.mdim[0], c.mdim[1], c.mdim[2], lv.n, (const C *)A::rho(lv), (const C *)A::u(lv), c.acc,
        c.mforce);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

// the body force of df_force's markers, which nothing of the step reads
inline int df_sum(Ctx &ctx, Case &c, cudaStream_t s)
{
    const int64_t nbf = (c.nm + 255) / 256;
    k_df_sum<<<(unsigned)nbf, 256, 0, s>>>(c.mforce, c.nm, c.mforce + 3 * c.nm,
                                           (unsigned *)(c.mforce + 3 * (c.nm + nbf)), c.force_acc, c.tstep);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

template <class S, int Q>
int band_collide(Ctx &ctx, Case &c, int l, void *out)
{
    using A = AmrTyped<S>;
    Level &lv = c.lv[l];
    if (!lv.nband) return MT_OK;
    k_band_collide<Q, S><<<grid_for(lv.nband, 64), 64, 0, ctx.stream>>>(lv.band, lv.nband, lv.n, c.d.tau[l],
                                                                         A::f(lv), c.acc, (S *)out, c.shift[l]);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

// treat()'s forces since the last call into the accumulator
inline bool has_ib_cells(const Case &c) { return c.d.ib_method != MT_IB_DF && c.lv[c.d.max_level].nib; }
inline int ib_force_sum(Ctx &ctx, Case &c, cudaStream_t s)
{
    k_ib_force_sum<<<1, 32, 0, s>>>(c.ib_force, grid_for(c.lv[c.d.max_level].nib, kIbBlock), c.force_acc);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

// collide(level): macros and collision of lat_f and overlap_F2C with the copy on
// overlap_C2F, then the direct-forcing band with its force (band_collide)
template <class S, int Q>
int collide_level(Ctx &ctx, Case &c, int l, S *fcol)
{
    using A = AmrTyped<S>;
    Level &lv = c.lv[l];
    const int32_t *cl = lv.nband ? lv.collide_nb : lv.collide_list;
    const int64_t ncl = lv.nband ? lv.ncollide_nb : lv.ncollide, ncopy = lv.nlist[2];
    // one launch for both; where some cell is in both lists the copy comes last
    auto launch = [&](int64_t n0, int64_t n1) {
        if (n0 + n1 == 0) return MT_OK;
        // the cumulant model exists for D3Q27 only (checked at case creation)
        const int B = c.d.collision == MT_COLL_LBGK ? 128 : 64;
        const unsigned g = grid_for(n0, B) + grid_for(n1, B);
        if (c.d.collision == MT_COLL_LBGK) {
            k_collide<Q, S, MT_COLL_LBGK><<<g, B, 0, ctx.stream>>>(cl, n0, lv.list[2], n1, lv.n, c.d.tau[l], A::f(lv),
                                                                   A::rho(lv), A::u(lv), fcol, c.shift[l]);
        } else {
            if constexpr (Q == 27)
                k_collide<Q, S, MT_COLL_CUMULANT><<<g, B, 0, ctx.stream>>>(cl, n0, lv.list[2], n1, lv.n, c.d.tau[l],
                                                                           A::f(lv), A::rho(lv), A::u(lv), fcol,
                                                                           c.shift[l]);
        }
        MT_LAUNCHED(ctx);
        return MT_OK;
    };
    if (int rc = launch(ncl, lv.mixed ? 0 : ncopy)) return rc;
    if (int rc = band_collide<S, Q>(ctx, c, l, fcol)) return rc;
    return lv.mixed ? launch(0, ncopy) : MT_OK;
}

// One fused brick pass of level l in the form `variant` (brick_warp) on stream
// s, writing the next collision into fnext.
inline BrickTab brick_tab(const Level &lv)
{
    return BrickTab{lv.blist, lv.bnbr, (const unsigned long long *)lv.bmask, lv.bcls, lv.bflag};
}
template <int Q, class S>
void brick_launch(Case &c, int l, int variant, cudaStream_t s, S *fnext, int mac, int fall, long long *bacc)
{
    using A = AmrTyped<S>;
    Level &lv = c.lv[l];
    const unsigned g = grid_for(lv.nblist, 4);
    if (!g) return;
    const uint32_t n32 = (uint32_t)lv.n;
    const int tb = c.d.stream_convention;
    auto go = [&](auto coll, auto v) {
        constexpr int COLL = decltype(coll)::value, V = decltype(v)::value;
        k_brick_step<Q, S, COLL, V><<<g, 128, 0, s>>>(lv.nblist, brick_tab(lv), n32, tb, A::fcol(lv), A::f(lv), fnext, c.d.tau[l], A::rho(lv), A::u(lv), mac, fall,
                                                      COLL == MT_COLL_LBGK ? bacc : nullptr, c.shift[l]);
    };
    using LB = std::integral_constant<int, MT_COLL_LBGK>;
    using CU = std::integral_constant<int, MT_COLL_CUMULANT>;
    using V0 = std::integral_constant<int, 0>;
    using V1 = std::integral_constant<int, 1>;
    using V2 = std::integral_constant<int, 2>;
    using V3 = std::integral_constant<int, 3>;
    const int v = (Store<S>::shifted || variant == 3) ? variant : 0;
    if (c.d.collision == MT_COLL_LBGK) {
        if (v == 1) go(LB{}, V1{}); else if (v == 2) go(LB{}, V2{}); else if (v == 3) go(LB{}, V3{}); else go(LB{}, V0{});
    } else {
        if constexpr (Q == 27) {
            if (v == 1) go(CU{}, V1{}); else if (v == 2) go(CU{}, V2{}); else if (v == 3) go(CU{}, V3{}); else go(CU{}, V0{});
        }
    }
}

template <class S, int Q>
int amr_phase_q(Ctx &ctx, Case &c, int phase, int l)
{
    using A = AmrTyped<S>;
    const int B = 128;
    cudaStream_t s = ctx.stream;
    Level &lv = c.lv[l];
    const int64_t n = lv.n;
    switch (phase) {
    case PH_MACROS:
        if (lv.ncollide) {
            k_macros<Q, S><<<grid_for(lv.ncollide, B), B, 0, s>>>(lv.collide_list, lv.ncollide, n, A::f(lv),
                                                                   A::rho(lv), A::u(lv), c.shift[l]);
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    case PH_MACROS_ALL: {
        MacroLevels<S> m;
        unsigned blocks = 0;
        for (int k = 0; k <= c.d.max_level; ++k) {
            Level &x = c.lv[k];
            if (!x.ncollide) continue;
            const int j = m.nlev++;
            m.block[j] = blocks;
            m.list[j] = x.collide_list;
            m.nl[j] = x.ncollide;
            m.n[j] = x.n;
            m.f[j] = A::f(x);
            m.rho[j] = A::rho(x);
            m.u[j] = A::u(x);
            for (int q = 0; q < 27; ++q) m.shift[j][q] = c.shift[k].v[q];
            blocks += grid_for(x.ncollide, B);
        }
        m.block[m.nlev] = blocks;
        if (blocks) {
            k_macros_all<Q, S><<<blocks, B, 0, s>>>(m);
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    }
    case PH_COLLIDE:
        return collide_level<S, Q>(ctx, c, l, A::fcol(lv));
    case PH_STREAM:
        if (lv.nstream && lv.bnbr && n * Q < ((int64_t)1 << 32)) {
            k_stream_bricks<Q, S><<<grid_for(lv.nbrick, 4), 128, 0, s>>>(lv.nbrick, lv.bnbr,
                                                                        (const unsigned long long *)lv.bmask, lv.tag,
                                                                        c.skip_ib ? 1 : 0, c.d.stream_convention,
                                                                        A::fcol(lv), A::f(lv));
            MT_LAUNCHED(ctx);
        } else if (lv.nstream) {
            k_stream<Q, S><<<grid_for(lv.nstream, B), B, 0, s>>>(lv.stream_list, lv.nstream, n, c.d.stream_convention,
                                                                  lv.nbr, A::fcol(lv), A::f(lv));
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    case PH_EXPLOSION:
    case PH_EXPLOSION_B: {
        // PH_EXPLOSION_B: the second substep's explosion of MT_ITIME_HOLD /
        // MT_ITIME_EXTRAP (the latter from the extrapolated parent state, then
        // the sources' values are kept for the next one)
        if (l < 1 || !lv.nexpl) return MT_OK;
        Level &cl = c.lv[l - 1];
        const double scale = c2f_scale(c, l);
        const bool ex = phase == PH_EXPLOSION_B && c.itime == MT_ITIME_EXTRAP;
        // held parent state over bricks: once, into both buffers (k_brick_exploded)
        const bool once = c.fused_now && lv.bricks && c.itime == MT_ITIME_HOLD && lv.hold_once;
        if (once && phase == PH_EXPLOSION_B) return MT_OK;
        if (ex && !lv.expl_prev) return set_err(ctx, MT_ERR_STATE, "extrapolated explosion without saved sources");
        k_explosion<Q, S><<<grid_for(lv.nexpl, 32), 32 * kParts, 0, s>>>(lv.expl_src, lv.expl_child, lv.expl_mask, lv.nexpl,
                                                               A::fcol(cl), A::fcol(lv), scale, (S *)lv.fcol_alt,
                                                               once ? 0 : lv.nexpl_f2c, c.shift[l - 1], c.shift[l],
                                                               ex ? (const S *)lv.expl_prev : nullptr);
        MT_LAUNCHED(ctx);
        if (ex) {
            k_expl_save<Q, S><<<grid_for(lv.nexpl, B), B, 0, s>>>(lv.expl_src, lv.nexpl, A::fcol(cl), cl.n,
                                                                (S *)lv.expl_prev);
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    }
    case PH_EXPL_SAVE: {
        // the sources' current parent values (the state was set or the option turned on)
        if (l < 1 || !lv.nexpl || !lv.expl_prev) return MT_OK;
        Level &cl = c.lv[l - 1];
        k_expl_save<Q, S><<<grid_for(lv.nexpl, B), B, 0, s>>>(lv.expl_src, lv.nexpl, A::fcol(cl), cl.n,
                                                            (S *)lv.expl_prev);
        MT_LAUNCHED(ctx);
        return MT_OK;
    }
    case PH_COALESCENCE: {
        if (l >= c.d.max_level || !lv.nlist[1]) return MT_OK;
        Level &fl = c.lv[l + 1];
        const double scale = f2c_scale(c, l);
        k_coalescence<Q, S><<<grid_for(lv.nlist[1], 32), 32 * kParts, 0, s>>>(lv.list[1], lv.coal_child, lv.nlist[1], A::f(lv),
                                                                      A::f(fl), scale, c.shift[l], c.shift[l + 1]);
        MT_LAUNCHED(ctx);
        return MT_OK;
    }
    case PH_BC:
    case PH_BC_FACE0 + 0: case PH_BC_FACE0 + 1: case PH_BC_FACE0 + 2:
    case PH_BC_FACE0 + 3: case PH_BC_FACE0 + 4: case PH_BC_FACE0 + 5: {
        // all six face groups in the reference's order (LBM_Simulator.cpp:90-95), or one
        const int f0 = phase == PH_BC ? 0 : phase - PH_BC_FACE0, f1 = phase == PH_BC ? 6 : f0 + 1;
        Level &l0 = c.lv[0];
        if (phase == PH_BC && c.bc_all && c.nbc_all) {
            BcVel ub;
            for (int face = 0; face < 6; ++face)
                for (int g = 0; g < 9; ++g) {
                    const int b = kFaceSets[face][g];
                    if (b < 0) break;
                    for (int a = 0; a < 3; ++a) ub.u[b][a] = c.face_u[face][a];
                }
            for (int ph = 0; ph < 2; ++ph) {
                k_bc_neq_all<Q, S><<<dim3(grid_for(c.nbc_all, 128), kBcRows<Q>), 128, 0, s>>>(c.bc_all, c.bc_setb, c.nbc_all, l0.n, l0.nbr,
                                                                         A::rho(l0), A::u(l0), A::f(l0), ub,
                                                                         c.bc_tmp_all, ph, c.dev_err, c.shift[0]);
                MT_LAUNCHED(ctx);
            }
            return MT_OK;
        }
        double *tmp = c.bc_tmp;
        if (!tmp) return MT_OK;
        for (int face = f0; face < f1; ++face)
            for (int g = 0; g < 9; ++g) {
                const int b = kFaceSets[face][g];
                if (b < 0) break;
                if (!l0.nbc[b]) continue;
                for (int ph = 0; ph < 2; ++ph) {
                    k_bc_neq<Q, S><<<grid_for(l0.nbc[b], B), B, 0, s>>>(
                        l0.bclist[b], l0.nbc[b], b, l0.n, l0.nbr, A::rho(l0), A::u(l0), A::f(l0), c.face_u[face][0],
                        c.face_u[face][1], c.face_u[face][2], tmp, ph, c.dev_err, c.shift[0]);
                    MT_LAUNCHED(ctx);
                }
            }
        return MT_OK;
    }
    case PH_BC_HH: {
        if constexpr (Q == 19) {
            Level &l0 = c.lv[0];
            for (int face = 0; face < 2; ++face) {
                if (!l0.nbc[face]) continue;
                k_bc_hh<S><<<grid_for(l0.nbc[face], B), B, 0, s>>>(l0.bclist[face], l0.nbc[face], face, l0.n,
                                                                    c.d.stream_convention, l0.nbr, A::fcol(l0),
                                                                    A::f(l0), c.face_u[0][0], c.face_u[0][1],
                                                                    c.face_u[0][2], c.dev_err, c.shift[0]);
                MT_LAUNCHED(ctx);
            }
            for (int face = 0; face < 2; ++face) {
                if (!l0.nbc[face]) continue;
                k_bc_wall_collide<S><<<grid_for(l0.nbc[face], B), B, 0, s>>>(l0.bclist[face], l0.nbc[face], l0.n,
                                                                              c.d.tau[0], A::f(l0), A::fcol(l0),
                                                                              c.shift[0]);
                MT_LAUNCHED(ctx);
            }
            return MT_OK;
        } else {
            return set_err(ctx, MT_ERR_ARG, "the Zou-He / Hecht-Harting boundary is D3Q19");
        }
    }
    case PH_BC_INOUT: {
        Level &l0 = c.lv[0];
        // one launch for both faces, unless East's inner neighbours are West cells
        const int64_t nw = l0.nbc[0], ne = l0.nbc[1];
        const bool one = c.d.extent0[0] > 2;
        for (int part = 0; part < (one ? 1 : 2); ++part) {
            const int64_t mw = one || part == 0 ? nw : 0, me = one || part == 1 ? ne : 0;
            if (mw + me == 0) continue;
            k_bc_inout<Q, S><<<grid_for(mw + me, 64), 64, 0, s>>>(
                l0.bclist[0], mw, l0.bclist[1], me, l0.n, l0.nbr, c.d.rho0, A::f(l0), A::fcol(l0), c.face_u[0][0],
                c.face_u[0][1], c.face_u[0][2], c.dev_err, c.shift[0]);
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    }
    case PH_IB: {
        if (c.d.ib_method == MT_IB_DF) {
            if (int rc = df_force<S, Q>(ctx, c, c.d.max_level)) return rc;
            return c.lv[c.d.max_level].nband && c.nm ? df_sum(ctx, c, s) : MT_OK;
        }
        Level &fl = c.lv[c.d.max_level];
        if (!fl.nib) {
            k_force_tick<<<1, 1, 0, s>>>(c.force_acc, 1.0);
            MT_LAUNCHED(ctx);
            return MT_OK;
        }
        {
            const unsigned gi = grid_for(fl.nib, kIbBlock);
            const Shift &fsh = c.shift[c.d.max_level];
            if (c.d.ib_method == MT_IB_FH)
                k_ib_treat<Q, 1, S><<<gi, kIbBlock, 0, s>>>(fl.iblist, fl.nib, A::ib(c), A::fcol(fl), A::rho(fl),
                                                            A::f(fl), c.ib_force, fsh);
            else
                k_ib_treat<Q, 0, S><<<gi, kIbBlock, 0, s>>>(fl.iblist, fl.nib, A::ib(c), A::fcol(fl), A::rho(fl),
                                                            A::f(fl), c.ib_force, fsh);
        }
        MT_LAUNCHED(ctx);
        return MT_OK;
    }
    case PH_COAL_COLLIDE: {
        if (l >= c.d.max_level || !lv.nlist[1]) return MT_OK;
        Level &fl = c.lv[l + 1];
        const double scale = f2c_scale(c, l);
        if (c.d.collision == MT_COLL_LBGK) {
            k_coal_collide<Q, S, MT_COLL_LBGK><<<grid_for(lv.nlist[1], 32), 32 * kParts, 0, s>>>(
                lv.list[1], lv.coal_child, lv.nlist[1], n, A::f(lv), A::f(fl), scale, c.d.tau[l],
                (S *)lv.fcol_alt, A::rho(lv), A::u(lv), c.macros_now, c.shift[l], c.shift[l + 1]);
        } else {
            if constexpr (Q == 27)
                k_coal_collide<Q, S, MT_COLL_CUMULANT><<<grid_for(lv.nlist[1], 32), 32 * kParts, 0, s>>>(
                    lv.list[1], lv.coal_child, lv.nlist[1], n, A::f(lv), A::f(fl), scale, c.d.tau[l],
                    (S *)lv.fcol_alt, A::rho(lv), A::u(lv), c.macros_now, c.shift[l], c.shift[l + 1]);
        }
        MT_LAUNCHED(ctx);
        return MT_OK;
    }
    case PH_FACE_EQ0 + 0: case PH_FACE_EQ0 + 1: case PH_FACE_EQ0 + 2:
    case PH_FACE_EQ0 + 3: case PH_FACE_EQ0 + 4: case PH_FACE_EQ0 + 5: {
        const int face = phase - PH_FACE_EQ0;
        Level &l0 = c.lv[0];
        for (int g = 0; g < 9; ++g) {
            const int b = kFaceSets[face][g];
            if (b < 0) break;
            if (!l0.nbc[b]) continue;
            k_bc_set_eq<Q, S><<<grid_for(l0.nbc[b], B), B, 0, s>>>(l0.bclist[b], l0.nbc[b], l0.n, c.d.rho0,
                                                                    c.face_u[face][0], c.face_u[face][1],
                                                                    c.face_u[face][2], A::f(l0), A::fcol(l0), c.shift[0]);
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    }
    case PH_DF: {
        // after PH_PULL_COLLIDE: a brick level's pass wrote the band macros
        if (int rc = df_force<S, Q>(ctx, c, l, lv.bricks)) return rc;
        {
            // the body force beside the band's collision (6 us of a substep's chain)
            const bool sum = lv.nband && c.nm, fork = sum && c.side;
            if (fork) {
                MT_CUDA(ctx, cudaEventRecord(c.side->fork, s));
                MT_CUDA(ctx, cudaStreamWaitEvent(c.side->s, c.side->fork, 0));
            }
            int rc = sum ? df_sum(ctx, c, fork ? c.side->s : s) : MT_OK;
            if (!rc) rc = band_collide<S, Q>(ctx, c, l, lv.fcol_alt);
            if (fork) {
                MT_CUDA(ctx, cudaEventRecord(c.side->join, c.side->s));
                MT_CUDA(ctx, cudaStreamWaitEvent(s, c.side->join, 0));
            }
            return rc;
        }
    }
    case PH_BAND_GRID:
        if (lv.nband && c.mgrid) {
            k_band_grid<<<grid_for(lv.nband, 256), 256, 0, s>>>(lv.band, lv.nband, lv.map(), c.mlo[0], c.mlo[1], c.mlo[2],
                                                                c.mdim[0], c.mdim[1], c.mdim[2], c.mgrid);
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    case PH_SYNC_F:
        if (lv.bricks && lv.nblist) {
            k_brick_pull<Q, S><<<grid_for(lv.nblist, 4), 128, 0, s>>>(lv.nblist, brick_tab(lv), c.d.stream_convention,
                                                                       A::fcol(lv), A::f(lv));
            MT_LAUNCHED(ctx);
        }
        return MT_OK;
    case PH_PRIME:
        // lookahead of the fused schedule from the current f: the second
        // buffer gets every cell's fcol, then the collision of lat_f and F2C
        // and the copy of C2F (the first collide(level) of the next substep)
        if (!n) return MT_OK;
        MT_CUDA(ctx, cudaMemcpyAsync(lv.fcol_alt, lv.fcol, sizeof(S) * Q * n, cudaMemcpyDeviceToDevice, s));
        return collide_level<S, Q>(ctx, c, l, (S *)lv.fcol_alt);
    case PH_PULL_COLLIDE: {
        // stream(level) of this substep fused with collide(level) of the next,
        // reading fcol and writing f and fcol_alt; treat() on the finest level
        // (its cells are disjoint from the fused pass: on the side stream when
        // the case has one, overlapping the pass)
        const int L = c.d.max_level;
        const bool ib_level = l == L && l > 0 && c.d.ib_method != MT_IB_DF;
        const int tb = c.d.stream_convention;
        const int mac = c.macros_now;
        // level 0's boundary sweep reads the streamed f of inner cells
        const int fall = (l == 0 && c.d.bc_mode == MT_BC_NEQ) ? 1 : 0;
        cudaStream_t is = s;
        if (ib_level && lv.nib && c.side) {
            MT_CUDA(ctx, cudaEventRecord(c.side->fork, s));
            MT_CUDA(ctx, cudaStreamWaitEvent(c.side->s, c.side->fork, 0));
            is = c.side->s;
        }
        if (ib_level) {
            if (!lv.nib) {
                // the coarse step's 2^L counts at its last substep (3 us a launch)
                if (mac) {
                    k_force_tick<<<1, 1, 0, s>>>(c.force_acc, (double)(1 << L));
                    MT_LAUNCHED(ctx);
                }
            } else {
                const double tau = c.d.tau[l];
                auto ib = [&](auto fh, auto coll) {
                    constexpr int FH = decltype(fh)::value, COLL = decltype(coll)::value;
                    k_ib_collide<Q, FH, S, COLL><<<grid_for(lv.nib, kIbBlock), kIbBlock, 0, is>>>(
                        lv.iblist, lv.nib, n, A::ib(c), A::fcol(lv), A::f(lv), (S *)lv.fcol_alt, tau,
                        c.ib_force, A::rho(lv), A::u(lv), mac, c.shift[l]);
                };
                using I0 = std::integral_constant<int, 0>;
                using I1 = std::integral_constant<int, 1>;
                using LB = std::integral_constant<int, MT_COLL_LBGK>;
                using CU = std::integral_constant<int, MT_COLL_CUMULANT>;
                if (c.d.collision == MT_COLL_LBGK) {
                    if (c.d.ib_method == MT_IB_FH) ib(I1{}, LB{}); else ib(I0{}, LB{});
                } else {
                    if constexpr (Q == 27) {
                        if (c.d.ib_method == MT_IB_FH) ib(I1{}, CU{}); else ib(I0{}, CU{});
                    }
                }
                MT_LAUNCHED(ctx);
            }
        }
        if (lv.bricks) {
            // the band's macros come out of the pass (the direct-forcing step skips k_band_macros)
            long long *bacc = (l == L && lv.nband) ? c.acc : nullptr;
            brick_launch<Q, S>(c, l, lv.brick_variant, s, (S *)lv.fcol_alt, mac, fall, bacc);
            MT_LAUNCHED(ctx);
        } else {
            if (lv.nfused) {
                if (c.d.collision == MT_COLL_LBGK) {
                    k_pull_collide<Q, S, MT_COLL_LBGK><<<grid_for(lv.nfused, B), B, 0, s>>>(
                        lv.fused_list, lv.nfused, n, tb, lv.nbr, A::fcol(lv), A::f(lv), (S *)lv.fcol_alt,
                        c.d.tau[l], A::rho(lv), A::u(lv), mac, c.shift[l]);
                } else {
                    if constexpr (Q == 27)
                        k_pull_collide<Q, S, MT_COLL_CUMULANT><<<grid_for(lv.nfused, 64), 64, 0, s>>>(
                            lv.fused_list, lv.nfused, n, tb, lv.nbr, A::fcol(lv), A::f(lv), (S *)lv.fcol_alt,
                            c.d.tau[l], A::rho(lv), A::u(lv), mac, c.shift[l]);
                }
                MT_LAUNCHED(ctx);
            }
            if (lv.nlist[2]) {
                k_pull_copy<Q, S><<<grid_for(lv.nlist[2], B), B, 0, s>>>(lv.list[2], lv.nlist[2], n, tb, lv.nbr,
                                                                          A::fcol(lv), A::f(lv), (S *)lv.fcol_alt);
                MT_LAUNCHED(ctx);
            }
            if (lv.nband) {
                k_stream<Q, S><<<grid_for(lv.nband, B), B, 0, s>>>(lv.band, lv.nband, n, tb, lv.nbr, A::fcol(lv),
                                                                    A::f(lv));
                MT_LAUNCHED(ctx);
            }
        }
        if (is != s) {
            MT_CUDA(ctx, cudaEventRecord(c.side->join, is));
            MT_CUDA(ctx, cudaStreamWaitEvent(s, c.side->join, 0));
        }
        // the coarse step's last: its force, beside the coarser levels' work
        // (record_fused_step waits for it)
        if (ib_level && lv.nib && mac) {
            if (int rc = ib_force_sum(ctx, c, is)) return rc;
            c.side_open = is != s;
        }
        return MT_OK;
    }
    case PH_IB_SUM:
        return has_ib_cells(c) ? ib_force_sum(ctx, c, s) : MT_OK;
    }
    return set_err(ctx, MT_ERR_ARG, "unknown phase");
}

template <class S>
int AmrOps<S>::phase(Ctx &ctx, Case &c, int phase, int level)
{
    return c.d.q == 19 ? amr_phase_q<S, 19>(ctx, c, phase, level) : amr_phase_q<S, 27>(ctx, c, phase, level);
}

template <class S>
int AmrOps<S>::ib_tables(Ctx &ctx, Case &c)
{
    using C = typename Store<S>::C;
    Level &fl = c.lv[c.d.max_level];
    const int64_t nib = fl.nib, links = c.d.q - 1;
    const int fh = c.d.ib_method == MT_IB_FH;
    MT_CUDA(ctx, cudaMallocAsync(&c.ib_wall, sizeof(uint2) * nib, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&c.ib_src, sizeof(int32_t) * links * nib, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&c.ib_factor, sizeof(C) * links * nib, ctx.stream));
    if (c.d.q == 19)
        k_ib_tables<19, C><<<grid_for(nib, 128), 128, 0, ctx.stream>>>(fl.iblist, nib, fl.n, fl.disrow, c.dis, fl.nbr,
                                                                      fh, c.ib_wall, c.ib_src, (C *)c.ib_factor);
    else
        k_ib_tables<27, C><<<grid_for(nib, 128), 128, 0, ctx.stream>>>(fl.iblist, nib, fl.n, fl.disrow, c.dis, fl.nbr,
                                                                      fh, c.ib_wall, c.ib_src, (C *)c.ib_factor);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

template <class S>
int AmrOps<S>::upload_tables(Ctx &ctx)
{
    return upload_bdry_tables(ctx);
}

template <class S>
int AmrOps<S>::alloc(Ctx &ctx, Case &c, int l)
{
    using C = typename Store<S>::C;
    Level &lv = c.lv[l];
    const int64_t n = lv.n, Q = c.d.q;
    if (l == 0) {
        int rc = upload_bdry_tables(ctx);
        if (rc) return rc;
    }
    lv.brick_variant = brick_default_variant<S>();
    MT_CUDA(ctx, cudaMallocAsync(&lv.f, sizeof(S) * n * Q, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&lv.fcol, sizeof(S) * n * Q, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&lv.rho, sizeof(C) * n, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&lv.u, sizeof(C) * 3 * n, ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(lv.f, 0, sizeof(S) * n * Q, ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(lv.fcol, 0, sizeof(S) * n * Q, ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(lv.rho, 0, sizeof(C) * n, ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(lv.u, 0, sizeof(C) * 3 * n, ctx.stream));
    return MT_OK;
}

template <class S>
int AmrOps<S>::init_eq(Ctx &ctx, Case &c, double rho0, const double *u0)
{
    using A = AmrTyped<S>;
    for (int l = 0; l <= c.d.max_level; ++l) {
        Level &lv = c.lv[l];
        if (!lv.n) continue;
        if (c.d.q == 19)
            k_init_eq<19, S><<<grid_for(lv.n, 256), 256, 0, ctx.stream>>>(lv.n, lv.tag, rho0, u0[0], u0[1], u0[2],
                                                                           A::f(lv), A::fcol(lv), A::rho(lv), A::u(lv), c.shift[l]);
        else
            k_init_eq<27, S><<<grid_for(lv.n, 256), 256, 0, ctx.stream>>>(lv.n, lv.tag, rho0, u0[0], u0[1], u0[2],
                                                                           A::f(lv), A::fcol(lv), A::rho(lv), A::u(lv), c.shift[l]);
        MT_LAUNCHED(ctx);
    }
    return MT_OK;
}

template <class S>
int AmrOps<S>::get(Ctx &ctx, Case &c, int l, int which, double *d_out)
{
    Level &lv = c.lv[l];
    const S *src = (const S *)(which == 0 ? lv.f : lv.fcol);
    if (!lv.n) return MT_OK;
    if (c.d.q == 19)
        k_to_f64<19, S><<<grid_for(lv.ncell, 256), 256, 0, ctx.stream>>>(src, d_out, lv.slot, lv.ncell, c.shift[l]);
    else
        k_to_f64<27, S><<<grid_for(lv.ncell, 256), 256, 0, ctx.stream>>>(src, d_out, lv.slot, lv.ncell, c.shift[l]);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

template <class S>
int AmrOps<S>::set(Ctx &ctx, Case &c, int l, int which, const double *d_in)
{
    Level &lv = c.lv[l];
    S *dst = (S *)(which == 0 ? lv.f : lv.fcol);
    if (!lv.n) return MT_OK;
    if (c.d.q == 19)
        k_from_f64<19, S><<<grid_for(lv.ncell, 256), 256, 0, ctx.stream>>>(d_in, dst, lv.slot, lv.ncell, c.shift[l]);
    else
        k_from_f64<27, S><<<grid_for(lv.ncell, 256), 256, 0, ctx.stream>>>(d_in, dst, lv.slot, lv.ncell, c.shift[l]);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

template <class S>
int AmrOps<S>::macros_out(Ctx &ctx, Case &c, int l, double *d_rho, double *d_u)
{
    using C = typename Store<S>::C;
    Level &lv = c.lv[l];
    if (!lv.n) return MT_OK;
    k_macro_to_f64<C><<<grid_for(lv.ncell, 256), 256, 0, ctx.stream>>>((const C *)lv.rho, (const C *)lv.u, lv.n,
                                                                        lv.slot, lv.ncell, d_rho, d_u);
    MT_LAUNCHED(ctx);
    return MT_OK;
}

// ---- the brick pass autotuner (mt_case_tune_bricks) ----------------------
// Each brick level's fused pass is timed in each of its forms (brick_warp; FP64
// has forms 0 and 3) on the case's own bricks: one warm-up and three timed launches per form, CUDA
// events on the case's stream.  The passes read the current post-collision
// buffer and write the next collision into a scratch buffer; the f they
// store is what the last real pass stored, and no macros are written, so the
// state is untouched.  The faster form is kept for the level.
template <class S>
int AmrOps<S>::tune_bricks(Ctx &ctx, Case &c, int32_t *variant, float *ms)
{
    int64_t nmax = 0;
    for (int l = 0; l <= c.d.max_level; ++l)
        if (c.lv[l].bricks) nmax = std::max(nmax, c.lv[l].n);
    for (int l = 0; l <= c.d.max_level; ++l) {
        if (variant) variant[l] = -1;
        if (ms)
            for (int v = 0; v < MT_BRICK_FORMS; ++v) ms[MT_BRICK_FORMS * l + v] = -1.f;
    }
    if (!nmax) return MT_OK;
    S *scratch = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&scratch, sizeof(S) * (size_t)c.d.q * (size_t)nmax, ctx.stream));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int rc = MT_OK;
    for (int l = 0; l <= c.d.max_level && !rc; ++l) {
        Level &lv = c.lv[l];
        if (!lv.bricks || !lv.nblist) continue;
        float best = 0.f;
        int pick = lv.brick_variant;
        for (int v = 0; v < MT_BRICK_FORMS && !rc; ++v) {
            if (!Store<S>::shifted && v != 0 && v != 3) continue;  // FP64: forms 0 and 3
            auto launch = [&]() {
                if (c.d.q == 19)
                    brick_launch<19, S>(c, l, v, ctx.stream, scratch, 0, 0, nullptr);
                else
                    brick_launch<27, S>(c, l, v, ctx.stream, scratch, 0, 0, nullptr);
            };
            launch();
            cudaEventRecord(e0, ctx.stream);
            for (int r = 0; r < 3; ++r) launch();
            cudaEventRecord(e1, ctx.stream);
            cudaError_t e = cudaEventSynchronize(e1);
            if (e == cudaSuccess) e = cudaGetLastError();
            if (e != cudaSuccess) {
                rc = set_err(ctx, MT_ERR_CUDA, std::string("brick tuner: ") + cudaGetErrorString(e));
                break;
            }
            float t = 0.f;
            cudaEventElapsedTime(&t, e0, e1);
            t /= 3.f;
            ctx.launches += 4;
            if (ms) ms[MT_BRICK_FORMS * l + v] = t;
            if (v == 0 || t < best) {  // form 0 is always timed first
                best = t;
                pick = v;
            }
        }
        lv.brick_variant = pick;
        if (variant) variant[l] = pick;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFreeAsync(scratch, ctx.stream);
    return rc;
}

// ---- FP64 reductions of a multi-level case (mt_case_reduce_levels) -------
// Per-block partial sums over a level's stepped cells (the collide list,
// lat_f then overlap_F2C: the cells LBM_Manager::calculateMacros visits,
// LBM_Manager.cpp:1003-1050) of mass sum_q f_q, momentum sum_q f_q e_q and
// kinetic energy |j|^2 / (2 rho), every value widened to FP64 before the
// storage shift (FP64) is added back.  partial: [5][gridDim.x].
template <int Q, class S>
__global__ void k_level_reduce(const S *f, int64_t n, const int32_t *list, int64_t m, const Shift sh,
                               double *partial)
{
    __shared__ double red[5][256];
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double a[5] = {0, 0, 0, 0, 0};
    if (j < m) {
        const int64_t i = list[j];
        double r = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            double v = (double)Store<S>::ld(f, at<Q>(k, i));
            if (Store<S>::shifted) v += sh.d[k];
            r += v;
            jx += v * ex(k);
            jy += v * ey(k);
            jz += v * ez(k);
        }
        a[0] = r;
        a[1] = jx;
        a[2] = jy;
        a[3] = jz;
        a[4] = 0.5 * (jx * jx + jy * jy + jz * jz) / r;
    }
    for (int c = 0; c < 5; ++c) red[c][threadIdx.x] = a[c];
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st)
            for (int c = 0; c < 5; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 5; ++c) partial[(int64_t)c * gridDim.x + blockIdx.x] = red[c][0];
}

// where each level's partials start in the scratch and how many blocks it has
struct LevelPartials {
    int64_t off[kMaxLevels];
    int64_t nb[kMaxLevels];
    int nlev;
};

// one block: level rows in a fixed order (strided sums, then a tree), then
// the global row sum_l 8^-l row_l (a level-l cell is 8^-l coarse cells).
// out: [(nlev + 1) * 5]
static __global__ void k_level_totals(const double *partial, const LevelPartials P, double *out)
{
    __shared__ double red[256];
    for (int l = 0; l < P.nlev; ++l)
        for (int c = 0; c < 5; ++c) {
            const double *p = partial + P.off[l] + (int64_t)c * P.nb[l];
            double a = 0;
            for (int64_t j = threadIdx.x; j < P.nb[l]; j += blockDim.x) a += p[j];
            red[threadIdx.x] = a;
            __syncthreads();
            for (int st = blockDim.x / 2; st > 0; st >>= 1) {
                if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
                __syncthreads();
            }
            if (threadIdx.x == 0) out[l * 5 + c] = red[0];
            __syncthreads();
        }
    if (threadIdx.x < 5) {
        double g = 0, wl = 1.0;
        for (int l = 0; l < P.nlev; ++l) {
            g += wl * out[l * 5 + threadIdx.x];
            wl *= 0.125;
        }
        out[P.nlev * 5 + threadIdx.x] = g;
    }
}

template <class S>
int AmrOps<S>::reduce(Ctx &ctx, Case &c, double *d_out)
{
    LevelPartials P{};
    P.nlev = c.d.max_level + 1;
    int64_t total = 0;
    for (int l = 0; l < P.nlev; ++l) {
        P.off[l] = total;
        P.nb[l] = (c.lv[l].ncollide + 255) / 256;
        total += 5 * P.nb[l];
    }
    double *partial = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&partial, sizeof(double) * std::max<int64_t>(total, 1), ctx.stream));
    cudaError_t err = cudaSuccess;
    auto launched = [&]() {
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) err = e;
        else ctx.launches++;
        return e == cudaSuccess;
    };
    bool ok = true;
    for (int l = 0; l < P.nlev && ok; ++l) {
        Level &lv = c.lv[l];
        if (!P.nb[l]) continue;
        if (c.d.q == 19)
            k_level_reduce<19, S><<<(unsigned)P.nb[l], 256, 0, ctx.stream>>>(
                (const S *)lv.f, lv.n, lv.collide_list, lv.ncollide, c.shift[l], partial + P.off[l]);
        else
            k_level_reduce<27, S><<<(unsigned)P.nb[l], 256, 0, ctx.stream>>>(
                (const S *)lv.f, lv.n, lv.collide_list, lv.ncollide, c.shift[l], partial + P.off[l]);
        ok = launched();
    }
    if (ok) {
        k_level_totals<<<1, 256, 0, ctx.stream>>>(partial, P, d_out);
        ok = launched();
    }
    cudaFreeAsync(partial, ctx.stream);
    if (!ok) return set_err(ctx, MT_ERR_CUDA, std::string("reduction launch: ") + cudaGetErrorString(err));
    return MT_OK;
}

// ---- LBM_Manager::infoPrint's diagnostics (mt_case_info) ----------------
// Per block over a level's collide list (lat_f then overlap_F2C, the cells
// infoPrint visits, LBM_Manager.cpp:914-955): the largest |u| and the number
// of cells with |u| > 1 over both sets, and over the lat_f cells (the first
// nlatf entries) sum |u - u_prev|^2 and sum |u|^2, u_prev the velocity the
// previous call saw (prev [3][nlatf], FP64, rewritten here).  A NaN velocity
// never wins the maximum, as in the reference's comparisons.
// partial: [4][gridDim.x]
template <class C>
__global__ void k_level_info(const int32_t *__restrict__ list, int64_t m, int64_t nlatf, const C *__restrict__ u,
                             int64_t n, double *__restrict__ prev, int have_prev, double *__restrict__ partial)
{
    __shared__ double red[4][256];
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double a[4] = {0, 0, 0, 0};
    if (j < m) {
        const int64_t i = list[j];
        const double ux = (double)u[i], uy = (double)u[n + i], uz = (double)u[2 * n + i];
        const double v2 = ux * ux + uy * uy + uz * uz;
        const double vmag = sqrt(v2);
        a[0] = vmag > 0.0 ? vmag : 0.0;
        a[1] = vmag > 1.0 ? 1.0 : 0.0;
        if (j < nlatf) {
            if (have_prev) {
                const double dx = ux - prev[j], dy = uy - prev[nlatf + j], dz = uz - prev[2 * nlatf + j];
                a[2] = dx * dx + dy * dy + dz * dz;
            }
            a[3] = v2;
            prev[j] = ux;
            prev[nlatf + j] = uy;
            prev[2 * nlatf + j] = uz;
        }
    }
    for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = a[c];
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) {
            red[0][threadIdx.x] = fmax(red[0][threadIdx.x], red[0][threadIdx.x + st]);
            for (int c = 1; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + st];
        }
        __syncthreads();
    }
    if (threadIdx.x < 4) partial[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = red[threadIdx.x][0];
}

// one block: each level's row (column 0 the maximum, the others sums) in a
// fixed order.  out: [nlev * 4]
static __global__ void k_info_totals(const double *partial, const LevelPartials P, double *out)
{
    __shared__ double red[256];
    for (int l = 0; l < P.nlev; ++l)
        for (int c = 0; c < 4; ++c) {
            const double *p = partial + P.off[l] + (int64_t)c * P.nb[l];
            double a = 0;
            for (int64_t j = threadIdx.x; j < P.nb[l]; j += blockDim.x) a = c == 0 ? fmax(a, p[j]) : a + p[j];
            red[threadIdx.x] = a;
            __syncthreads();
            for (int st = blockDim.x / 2; st > 0; st >>= 1) {
                if (threadIdx.x < st)
                    red[threadIdx.x] = c == 0 ? fmax(red[threadIdx.x], red[threadIdx.x + st])
                                              : red[threadIdx.x] + red[threadIdx.x + st];
                __syncthreads();
            }
            if (threadIdx.x == 0) out[l * 4 + c] = red[0];
            __syncthreads();
        }
}

template <class S>
int AmrOps<S>::info(Ctx &ctx, Case &c, double *d_out)
{
    using C = typename Store<S>::C;
    LevelPartials P{};
    P.nlev = c.d.max_level + 1;
    int64_t total = 0;
    for (int l = 0; l < P.nlev; ++l) {
        P.off[l] = total;
        P.nb[l] = (c.lv[l].ncollide + 255) / 256;
        total += 4 * P.nb[l];
        Level &lv = c.lv[l];
        if (!lv.info_prev && lv.nlist[0])
            MT_CUDA(ctx, cudaMallocAsync(&lv.info_prev, sizeof(double) * 3 * (size_t)lv.nlist[0], ctx.stream));
    }
    double *partial = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&partial, sizeof(double) * std::max<int64_t>(total, 1), ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(d_out, 0, sizeof(double) * 4 * (size_t)P.nlev, ctx.stream));
    cudaError_t err = cudaSuccess;
    bool ok = true;
    for (int l = 0; l < P.nlev && ok; ++l) {
        Level &lv = c.lv[l];
        if (!P.nb[l]) continue;
        k_level_info<C><<<(unsigned)P.nb[l], 256, 0, ctx.stream>>>(lv.collide_list, lv.ncollide, lv.nlist[0],
                                                                 AmrTyped<S>::u(lv), lv.n, lv.info_prev,
                                                                 lv.info_have ? 1 : 0, partial + P.off[l]);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            err = e;
            ok = false;
        } else {
            ctx.launches++;
            lv.info_have = true;
        }
    }
    if (ok) {
        k_info_totals<<<1, 256, 0, ctx.stream>>>(partial, P, d_out);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            err = e;
            ok = false;
        } else {
            ctx.launches++;
        }
    }
    cudaFreeAsync(partial, ctx.stream);
    if (!ok) return set_err(ctx, MT_ERR_CUDA, std::string("info launch: ") + cudaGetErrorString(err));
    return MT_OK;
}


template <class S>
int AmrOps<S>::guard(Ctx &ctx, Case &c, bool current_only)
{
    for (int l = 0; l <= c.d.max_level; ++l) {
        Level &lv = c.lv[l];
        if (!lv.n) continue;
        k_guard<S><<<(unsigned)std::min<int64_t>(lv.nbrick, 148 * 16), 128, 0, ctx.stream>>>(
            (const S *)(current_only ? lv.fcol : lv.f), (const S *)lv.fcol, (const unsigned long long *)lv.bmask,
            lv.nbrick, c.d.q, c.dev_err);
        MT_LAUNCHED(ctx);
    }
    return MT_OK;
}

// ---- remap of a state onto another lattice (mt_case_remap) ---------------
// one population set of Q values rescaled about its own equilibrium:
// feq(rho, u) + s (in - feq(rho, u)), rho and u from the values themselves
template <int Q> __device__ void remap_rescale(double *v, double s)
{
    double r = 0.0, jx = 0.0, jy = 0.0, jz = 0.0;
    for (int k = 0; k < Q; ++k) {
        r += v[k];
        jx += v[k] * ex(k);
        jy += v[k] * ey(k);
        jz += v[k] * ez(k);
    }
    const double rs = (r > -1e-6 && r < 1e-6) ? ((r < 0.0) ? -1e-6 : 1e-6) : r;
    const double ux = jx / rs, uy = jy / rs, uz = jz / rs;
    const double uu = ux * ux + uy * uy + uz * uz;
    for (int k = 0; k < Q; ++k) {
        const double eu = ex(k) * ux + ey(k) * uy + ez(k) * uz;
        const double feq = r * w<Q>(k) * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu);
        v[k] = feq + s * (v[k] - feq);
    }
}

__host__ __device__ __forceinline__ uint64_t cell_key_at(int L, int l, int64_t x, int64_t y, int64_t z)
{
    const int sh = L - l;
    return dilate3((uint64_t)x << sh) | (dilate3((uint64_t)y << sh) << 1) | (dilate3((uint64_t)z << sh) << 2);
}

template <class S> struct RemapLevels {
    struct Src {
        LevelMap map;
        const uint32_t *tag = nullptr;
        int64_t n = 0;
        const S *f = nullptr, *fcol = nullptr;
        float shift[27] = {};  // the level's storage shift (reduced storages)
    } lv[kMaxLevels];
    // explosion factors from coarser source level m, coalescence factors
    // from finer source level m (products over the levels crossed)
    double up_f[kMaxLevels], up_c[kMaxLevels], down_f[kMaxLevels], down_c[kMaxLevels];
};

// Each cell of a destination level takes f and fcol from the source: the same
// key on the same level as they are (the stored values, bit for bit); else
// the nearest coarser source level holding its ancestor, rescaled as an
// explosion; else the mean of its descendants on the nearest finer source
// level holding any, rescaled as a coalescence; else the equilibrium
// (rho0, u0).  Solid cells hold zeros (the build's convention); a fluid cell
// that is solid in the source takes the equilibrium at rest.  kind[i]: 0..3.
template <int Q, class S>
__global__ void k_remap(const LevelMap dmap, const int32_t *__restrict__ dslot, int64_t ncell, const uint32_t *dtag, int L, int l, RemapLevels<S> src,
                        double rho0, double ux0, double uy0, double uz0, S *fo, S *co, uint8_t *kind, const Shift dsh,
                        int same_shift)
{
    using T = Store<S>;
    using C = typename T::C;
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= ncell) return;
    const int64_t i = dslot[r];
    const uint64_t k = dmap.key(i);
    double a[Q], b[Q];
    auto put = [&](const double *pf, const double *pc, int kd) {
        for (int q = 0; q < Q; ++q) {
            T::st(fo, at<Q>(q, i), stored_sh<S>(dsh, (C)pf[q], q));
            T::st(co, at<Q>(q, i), stored_sh<S>(dsh, (C)pc[q], q));
        }
        kind[r] = (uint8_t)kd;
    };
    if (dtag[i] & TAG_SF) {
        for (int q = 0; q < Q; ++q) a[q] = 0.0;
        put(a, a, 0);
        return;
    }
    const auto &same = src.lv[l];
    int64_t j = same.n ? same.map.find(k) : -1;
    bool uncovered = false;
    if (j >= 0 && (same.tag[j] & TAG_SF)) {
        uncovered = true;
        j = -1;
    }
    if (j >= 0) {
        if (same_shift) {
            for (int q = 0; q < Q; ++q) {
                fo[at<Q>(q, i)] = same.f[at<Q>(q, j)];
                co[at<Q>(q, i)] = same.fcol[at<Q>(q, j)];
            }
        } else {
            for (int q = 0; q < Q; ++q) {
                T::st(fo, at<Q>(q, i), stored_sh<S>(dsh, full_v<S>(same.shift, T::ld(same.f, at<Q>(q, j)), q), q));
                T::st(co, at<Q>(q, i), stored_sh<S>(dsh, full_v<S>(same.shift, T::ld(same.fcol, at<Q>(q, j)), q), q));
            }
        }
        kind[r] = 0;
        return;
    }
    const int sh = L - l;
    const int64_t x = (int64_t)(compact3(k) >> sh), y = (int64_t)(compact3(k >> 1) >> sh),
                  z = (int64_t)(compact3(k >> 2) >> sh);
    for (int m = l - 1; m >= 0 && !uncovered; --m) {
        const auto &cs = src.lv[m];
        if (!cs.n) continue;
        const int up = l - m;
        const int64_t jm = cs.map.find(cell_key_at(L, m, x >> up, y >> up, z >> up));
        if (jm < 0) continue;
        for (int q = 0; q < Q; ++q) {
            a[q] = (double)full_v<S>(cs.shift, T::ld(cs.f, at<Q>(q, jm)), q);
            b[q] = (double)full_v<S>(cs.shift, T::ld(cs.fcol, at<Q>(q, jm)), q);
        }
        remap_rescale<Q>(a, src.up_f[m]);
        remap_rescale<Q>(b, src.up_c[m]);
        put(a, b, 1);
        return;
    }
    for (int d = 1; l + d <= L && !uncovered; ++d) {
        const auto &fine = src.lv[l + d];
        if (!fine.n) continue;
        const int side = 1 << d;
        int nch = 0;
        for (int q = 0; q < Q; ++q) a[q] = b[q] = 0.0;
        for (int c = 0; c < side * side * side; ++c) {
            const int64_t cx = (x << d) + c % side, cy = (y << d) + (c / side) % side, cz = (z << d) + c / (side * side);
            const int64_t jc = fine.map.find(cell_key_at(L, l + d, cx, cy, cz));
            if (jc < 0 || (fine.tag[jc] & TAG_SF)) continue;
            for (int q = 0; q < Q; ++q) {
                a[q] += (double)full_v<S>(fine.shift, T::ld(fine.f, at<Q>(q, jc)), q);
                b[q] += (double)full_v<S>(fine.shift, T::ld(fine.fcol, at<Q>(q, jc)), q);
            }
            ++nch;
        }
        if (!nch) continue;
        for (int q = 0; q < Q; ++q) {
            a[q] /= nch;
            b[q] /= nch;
        }
        remap_rescale<Q>(a, src.down_f[l + d]);
        remap_rescale<Q>(b, src.down_c[l + d]);
        put(a, b, 2);
        return;
    }
    if (uncovered) ux0 = uy0 = uz0 = 0.0;
    const double uu = ux0 * ux0 + uy0 * uy0 + uz0 * uz0;
    for (int q = 0; q < Q; ++q) {
        const double eu = ex(q) * ux0 + ey(q) * uy0 + ez(q) * uz0;
        a[q] = rho0 * w<Q>(q) * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu);
    }
    put(a, a, 3);
}

template <class S>
int AmrOps<S>::remap(Ctx &ctx, Case &dst, Case &src, int64_t *counts)
{
    const int L = dst.d.max_level, Q = dst.d.q;
    RemapLevels<S> rl;
    for (int m = 0; m <= L && m <= src.d.max_level; ++m) {
        if (!src.lv[m].n) continue;
        rl.lv[m].map = src.lv[m].map();
        rl.lv[m].tag = src.lv[m].tag;
        rl.lv[m].n = src.lv[m].n;
        rl.lv[m].f = (const S *)src.lv[m].f;
        rl.lv[m].fcol = (const S *)src.lv[m].fcol;
        for (int k = 0; k < 27; ++k) rl.lv[m].shift[k] = src.shift[m].v[k];
    }
    // the interface factors of dst: the reference's (the same on f and
    // fcol), or the stress-continuous ones (tau on f, tau - 1 on fcol)
    const bool st = dst.scaling == MT_SCALE_STANDARD;
    auto c2f = [&](int fine, bool col) {
        const double tf = dst.d.tau[fine], tc = dst.d.tau[fine - 1];
        if (!st) return (2.0 * tf) / tc;
        return col ? (tf - 1.0) / (2.0 * (tc - 1.0)) : tf / (2.0 * tc);
    };
    uint8_t *kind = nullptr;
    int64_t maxn = 0;
    for (int l = 0; l <= L; ++l) maxn = std::max(maxn, dst.lv[l].ncell);
    MT_CUDA(ctx, cudaMallocAsync(&kind, std::max<int64_t>(maxn, 1), ctx.stream));
    int rc = MT_OK;
    for (int l = 0; l <= L && !rc; ++l) {
        Level &lv = dst.lv[l];
        if (counts)
            for (int k = 0; k < 4; ++k) counts[4 * l + k] = 0;
        if (!lv.n) continue;
        for (int m = 0; m < kMaxLevels; ++m) rl.up_f[m] = rl.up_c[m] = rl.down_f[m] = rl.down_c[m] = 1.0;
        for (int m = l - 1; m >= 0; --m)
            for (int j = m + 1; j <= l; ++j) {
                rl.up_f[m] *= c2f(j, false);
                rl.up_c[m] *= c2f(j, true);
            }
        for (int m = l + 1; m <= L; ++m)
            for (int j = l + 1; j <= m; ++j) {
                rl.down_f[m] /= c2f(j, false);
                rl.down_c[m] /= c2f(j, true);
            }
        const double r0 = dst.d.rho0, u0 = dst.d.u_bc[0], u1 = dst.d.u_bc[1], u2 = dst.d.u_bc[2];
        // equal storage shifts on level l: cells present on both lattices copy their stored values
        int same_shift = l <= src.d.max_level;
        for (int k = 0; k < 27; ++k) same_shift &= dst.shift[l].d[k] == src.shift[l].d[k];
        if (Q == 19)
            k_remap<19, S><<<grid_for(lv.ncell, 128), 128, 0, ctx.stream>>>(lv.map(), lv.slot, lv.ncell, lv.tag, L, l, rl, r0, u0, u1, u2,
                                                                       (S *)lv.f, (S *)lv.fcol, kind, dst.shift[l],
                                                                       same_shift);
        else
            k_remap<27, S><<<grid_for(lv.ncell, 128), 128, 0, ctx.stream>>>(lv.map(), lv.slot, lv.ncell, lv.tag, L, l, rl, r0, u0, u1, u2,
                                                                       (S *)lv.f, (S *)lv.fcol, kind, dst.shift[l],
                                                                       same_shift);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            rc = set_err(ctx, MT_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
            break;
        }
        ctx.launches++;
        if (counts) {
            std::vector<uint8_t> hk((size_t)lv.ncell);
            e = cudaMemcpyAsync(hk.data(), kind, lv.ncell, cudaMemcpyDeviceToHost, ctx.stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(ctx.stream);
            if (e != cudaSuccess) {
                rc = set_err(ctx, MT_ERR_CUDA, std::string("remap counts: ") + cudaGetErrorString(e));
                break;
            }
            for (uint8_t v : hk) counts[4 * l + (v & 3)] += 1;
        }
    }
    cudaFreeAsync(kind, ctx.stream);
    return rc;
}

}  // namespace mt
