// Multi-level path: device build of the Morton-sorted SoA levels and the
// driver of the reference's recursive time step (the phase kernels live in
// mt_amr_phases.cuh, one instantiation per storage type).
//
// Layout per level: 64 slots for each 4x4x4 Morton brick that holds a cell,
// bricks in key order (Level in mt_internal.hpp); populations f/fcol as
// [brick][Q][64] in the storage type; nbr as [(Q-1)][n] int32 (slot of the cell
// at key + e_k or -1); index lists (int32 slots) for each reference set in
// ascending key order.
#include <cub/cub.cuh>

#include <algorithm>
#include <utility>
#include <cstring>

#include "mt_internal.hpp"

namespace mt {

// ----------------------------------------------------------------------------
// build kernels
// ----------------------------------------------------------------------------
// sorted raw keys (with repeats): a cell starts where the key changes (low
// half), a brick where the key's brick part does (high half).  A key with bits
// below the level's cells names no slot.
__global__ void k_starts(const uint64_t *key, int64_t n, int low, unsigned long long *flag, int *err)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long v = 0;
    if (i == 0 || key[i] != key[i - 1]) v |= 1ull;
    if (i == 0 || (key[i] >> (low + 6)) != (key[i - 1] >> (low + 6))) v |= 1ull << 32;
    flag[i] = v;
    if (key[i] & ((1ull << low) - 1ull)) atomicOr(err, DEVERR_KEY_BITS);
}

// c = inclusive scan of the starts: cell rank and brick of sorted key i
__global__ void k_fill_bricks(const uint64_t *key, const unsigned long long *c, int64_t n, int low, uint64_t *bkey,
                              unsigned long long *bmask, int32_t *bstart, int32_t *slot)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i > 0 && c[i] == c[i - 1]) return;
    const int64_t r = (int64_t)(c[i] & 0xffffffffull) - 1, b = (int64_t)(c[i] >> 32) - 1;
    const int m = (int)((key[i] >> low) & 63);
    slot[r] = (int32_t)(64 * b + m);
    atomicOr(bmask + b, 1ull << m);
    if (i == 0 || (c[i] >> 32) != (c[i - 1] >> 32)) {
        bkey[b] = key[i] >> (low + 6);
        bstart[b] = (int32_t)r;
    }
}

__global__ void k_tag_cells(const uint64_t *raw, const uint8_t *set, int64_t nraw, const LevelMap map, uint32_t *tag,
                            int8_t *bcidx)
{
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nraw) return;
    int64_t i = map.find(raw[j]);
    if (i < 0) return;
    const uint8_t s = set[j];
    uint32_t bit;
    if (s >= 16) {
        bit = TAG_BC;
        bcidx[i] = (int8_t)(s - 16);
    } else if (s == MT_SET_IB_BAND) {
        bit = TAG_BAND;
    } else {
        const uint32_t bits[kNumSets] = {TAG_LATF, TAG_F2C, TAG_C2F, TAG_GC2F, TAG_GF2C, TAG_SF};
        bit = bits[s];
    }
    atomicOr(&tag[i], bit);
}

// slot of the cell at key + e_k, or -1 (also for slots without a cell): from
// the neighbour bricks where they are exact, else by the key of
// Morton_Assist::find_neighbor
template <int Q>
__global__ void k_neighbors(MortonGeom g, int level, const LevelMap map, const int32_t *__restrict__ bnbr, int64_t n,
                            int32_t *nbr)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t b = i >> 6;
    const int m = (int)(i & 63);
    const bool here = (map.bmask[b] >> m) & 1;
    const uint64_t k0 = map.key(i);
    const int x = (m & 1) | ((m >> 2) & 2), y = ((m >> 1) & 1) | ((m >> 3) & 2), z = ((m >> 2) & 1) | ((m >> 4) & 2);
#pragma unroll
    for (int k = 1; k < Q; ++k) {
        int32_t out = -1;
        if (here && bnbr) {
            const int nx = x + ex(k), ny = y + ey(k), nz = z + ez(k);
            const int s = ((nx >> 2) + 1) + 3 * ((ny >> 2) + 1) + 9 * ((nz >> 2) + 1);
            const int ax = nx & 3, ay = ny & 3, az = nz & 3;
            const int mm = (ax & 1) | ((ax & 2) << 2) | ((ay & 1) << 1) | ((ay & 2) << 3) | ((az & 1) << 2) | ((az & 2) << 4);
            const int32_t bb = __ldg(bnbr + 27 * b + s);
            if (bb >= 0 && ((map.bmask[bb] >> mm) & 1)) out = 64 * bb + mm;
        } else if (here) {
            out = (int32_t)map.find(find_neighbor(g, k0, level, ex(k), ey(k), ez(k)));
        }
        nbr[(int64_t)(k - 1) * n + i] = out;
    }
}

__global__ void k_dis_rows(const LevelMap map, const int32_t *slot, int64_t nc, const uint64_t *dkey, int64_t nd,
                           int32_t *disrow, uint32_t *tag)
{
    int64_t r0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r0 >= nc) return;
    const int64_t i = slot[r0];
    int64_t r = find_key(dkey, nd, map.key(i));
    disrow[i] = (int32_t)r;
    if (r >= 0) tag[i] |= TAG_IB;
}

__global__ void k_dis_check(const uint64_t *dkey, int64_t nd, const LevelMap map, int *err)
{
    int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nd) return;
    if (map.find(dkey[r]) < 0) atomicOr(err, DEVERR_DIS_NOT_FINEST);
}

// children of a coarse cell on the fine level, in the order of
// LBM_Manager.cpp:1074-1082: (0,0,0) (1,0,0) (0,1,0) (1,1,0) (0,0,1) (1,0,1) (0,1,1) (1,1,1)
MT_HD void children(const MortonGeom &g, uint64_t code, int fine, uint64_t *ch)
{
    const uint64_t x1 = find_neighbor(g, code, fine, 1, 0, 0);
    const uint64_t y1 = find_neighbor(g, code, fine, 0, 1, 0);
    const uint64_t xy1 = find_neighbor(g, x1, fine, 0, 1, 0);
    ch[0] = code;
    ch[1] = x1;
    ch[2] = y1;
    ch[3] = xy1;
    ch[4] = find_neighbor(g, code, fine, 0, 0, 1);
    ch[5] = find_neighbor(g, x1, fine, 0, 0, 1);
    ch[6] = find_neighbor(g, y1, fine, 0, 0, 1);
    ch[7] = find_neighbor(g, xy1, fine, 0, 0, 1);
}

// explosion children (AMR_transDDF_explosion, LBM_Manager.cpp:1072-1128):
// F2C sources need every child stored and skip children listed in dis;
// ghost sources write only children in ghost_overlap_C2F and not in dis.
// child[j]: the slot of the first child (the eight are consecutive), mask[j]
// the slots to write.  found: EXPL_*, what some written child is besides.
__global__ void k_expl_children(MortonGeom g, int fine, const int32_t *src, int64_t nsrc, int64_t nf2c,
                                const LevelMap cmap, const LevelMap fmap, const uint32_t *ftag, const uint64_t *dkey,
                                int64_t nd, int32_t *child, uint8_t *mask, int *err, int *found)
{
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nsrc) return;
    uint64_t ch[8];
    children(g, cmap.key(src[j]), fine, ch);
    const int64_t b = find_key(fmap.bkey, fmap.nb, ch[0] >> (fmap.low + 6));
    const int m0 = (int)((ch[0] >> fmap.low) & 63);
    const unsigned there = b >= 0 ? (unsigned)(fmap.bmask[b] >> m0) & 255u : 0u;
    unsigned out = 0;
    for (int m = 0; m < 8; ++m) {
        if (find_key(dkey, nd, ch[m]) >= 0) continue;
        const bool stored = (there >> m) & 1u;
        if (j < nf2c) {
            if (!stored)
                atomicOr(err, DEVERR_MISSING_CHILD);
            else
                out |= 1u << m;
        } else if (stored && (ftag[64 * b + m0 + m] & TAG_GC2F)) {
            out |= 1u << m;
        }
    }
    int is = 0;
    for (int m = 0; m < 8; ++m)
        if ((out >> m) & 1u) {
            const uint32_t t = ftag[64 * b + m0 + m];
            if (t & (TAG_F2C | TAG_GF2C)) is |= EXPL_SOURCE;
            if ((t & TAG_LATF) && !(t & TAG_C2F)) is |= EXPL_COLLIDED;
        }
    if (is) atomicOr(found, is);
    // slots without a cell may be written too: most sources (a ghost source has
    // only its children next to the interface) then take whole-vector stores
    if (out) out |= ~there & 255u;
    child[j] = b >= 0 ? (int32_t)(64 * b + m0) : 0;
    mask[j] = (uint8_t)out;
}

// child[j]: the slot of the first child; all eight are stored (else an error)
__global__ void k_coal_children(MortonGeom g, int fine, const int32_t *src, int64_t nsrc, const LevelMap cmap,
                                const LevelMap fmap, int32_t *child, int *err)
{
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nsrc) return;
    uint64_t ch[8];
    children(g, cmap.key(src[j]), fine, ch);
    const int64_t b = find_key(fmap.bkey, fmap.nb, ch[0] >> (fmap.low + 6));
    const int m0 = (int)((ch[0] >> fmap.low) & 63);
    if (b < 0 || ((fmap.bmask[b] >> m0) & 255u) != 255u) atomicOr(err, DEVERR_MISSING_CHILD);
    child[j] = b >= 0 ? (int32_t)(64 * b + m0) : 0;
}

// ---- the fused pass's tables over a level's bricks -----------------------------
__global__ void k_brick_cls(const uint32_t *tag, int64_t n, int ib_level, uint8_t *bcls)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t t = tag[i];
    // stream covers lat_f then overlap_C2F, and a C2F cell's fcol = f copy
    // comes after the collision (Collision_Manager.cpp:45-52)
    uint8_t cls = 0;
    if (t & TAG_C2F)
        cls = 2;
    else if ((t & TAG_LATF) && (t & TAG_BAND))
        cls = 4;  // direct-forcing band: stream only, collided after the forcing
    else if ((t & TAG_LATF) && !(ib_level && (t & TAG_IB)))
        cls = 1;
    bcls[i] = cls;
}

// cells whose streamed f a coarser level's coalescence reads: stream +
// collide with f stored (class 3)
__global__ void k_brick_mark(const int32_t *child, int64_t count, uint8_t *bcls)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= 8 * count) return;
    const int64_t ci = (int64_t)child[t >> 3] + (t & 7);
    if (bcls[ci] == 1) bcls[ci] = 3;
}

// MT_ITIME_HOLD: the C2F cells the explosion writes (class 6).  Its sources do not
// change between a fine level's two substeps, so the first substep's explosion
// writes both post-collision buffers, the second one is left out, and the
// pass leaves these cells' next collision alone.
__global__ void k_brick_exploded(const int32_t *child, const uint8_t *mask, int64_t count, uint8_t *bcls)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= 8 * count || !((mask[t >> 3] >> (t & 7)) & 1)) return;
    const int64_t ci = (int64_t)child[t >> 3] + (t & 7);
    if (bcls[ci] == 2) bcls[ci] = 6;
}

// one warp per brick, two cells per lane
template <int Q>
__global__ void k_brick_flag(int64_t nb, const uint8_t *__restrict__ bcls, const int32_t *__restrict__ nbr,
                             uint8_t *bflag)
{
    const int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (b >= nb) return;
    const int lane = threadIdx.x & 31;
    bool work = false, whole = true, one = true;
    for (int h = 0; h < 2; ++h) {
        const int64_t i = 64 * b + lane + 32 * h;
        const int cls = bcls[i];
        one &= cls == 1;
        if (!cls) continue;
        work = true;
        for (int k = 1; k < Q; ++k) whole &= nbr[(int64_t)(k - 1) * (64 * nb) + i] >= 0;
    }
    const unsigned all = 0xffffffffu;
    work = __any_sync(all, work);
    whole = __all_sync(all, whole);
    one = __all_sync(all, one);
    if (lane == 0)
        bflag[b] = (uint8_t)((work ? BRICK_WORK : 0) | (whole ? BRICK_COMPLETE : 0) | (one ? BRICK_UNIFORM : 0));
}

// neighbour bricks: Morton_Assist::find_neighbor applied to the corner cell
// of the brick that faces the offset, then a search of the brick keys
__global__ void k_brick_nbrs(MortonGeom g, int level, const uint64_t *bkey, int64_t nb, int shift, int low,
                             int32_t *bnbr)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= 27 * nb) return;
    const int64_t b = t / 27;
    const int s = (int)(t - 27 * b);
    const int dx = s % 3 - 1, dy = (s / 3) % 3 - 1, dz = s / 9 - 1;
    const int lx = dx > 0 ? 3 : 0, ly = dy > 0 ? 3 : 0, lz = dz > 0 ? 3 : 0;
    const uint64_t m = (uint64_t)((lx & 1) | ((lx & 2) << 2) | ((ly & 1) << 1) | ((ly & 2) << 3) | ((lz & 1) << 2) |
                                  ((lz & 2) << 4));
    const uint64_t rep = (bkey[b] << shift) | (m << low);
    const uint64_t nk = find_neighbor(g, rep, level, dx, dy, dz);
    bnbr[t] = (int32_t)find_key(bkey, nb, nk >> shift);
}

struct BrickHasWork {
    const uint8_t *flag;
    __host__ __device__ bool operator()(const int32_t &b) const { return (flag[b] & BRICK_WORK) != 0; }
};
struct TagHas {
    const uint32_t *tag;
    uint32_t bit;
    __host__ __device__ bool operator()(const int32_t &i) const { return (tag[i] & bit) != 0; }
};
struct BcIs {
    const int8_t *bc;
    int8_t b;
    __host__ __device__ bool operator()(const int32_t &i) const { return bc[i] == b; }
};
struct LatfNotBand {
    const uint32_t *tag;
    __host__ __device__ bool operator()(const int32_t &i) const
    {
        return (tag[i] & TAG_LATF) && !(tag[i] & TAG_BAND);
    }
};
struct LatfNotIb {
    const uint32_t *tag;
    __host__ __device__ bool operator()(const int32_t &i) const
    {
        return (tag[i] & TAG_LATF) && !(tag[i] & TAG_IB);
    }
};
struct IbLatf {
    const uint32_t *tag;
    __host__ __device__ bool operator()(const int32_t &i) const
    {
        return (tag[i] & TAG_LATF) && (tag[i] & TAG_IB);
    }
};

// indices satisfying pred, ascending; their number is known
template <class Pred>
static int select_known(Ctx &ctx, int64_t n, Pred pred, int64_t count, int32_t **out, int64_t *nout)
{
    *out = nullptr;
    *nout = count;
    if (!count) return MT_OK;
    cub::CountingInputIterator<int32_t> it(0);
    size_t tmp = 0;
    MT_CUDA(ctx, cub::DeviceSelect::If(nullptr, tmp, it, (int32_t *)nullptr, (int *)nullptr, (int)n, pred, ctx.stream));
    // one allocation for the selected count and the scratch
    char *buf = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(out, sizeof(int32_t) * count, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&buf, tmp + 256, ctx.stream));
    MT_CUDA(ctx, cub::DeviceSelect::If(buf + 256, tmp, it, *out, (int *)buf, (int)n, pred, ctx.stream));
    cudaFreeAsync(buf, ctx.stream);
    return MT_OK;
}

// how many slots carry each tag bit (0..8) and each boundary set (9..34): the
// sizes of a level's lists, read back once; and how many cells are both
// collided and copied (35)
constexpr int kTagBits = 9, kCounts = kTagBits + 27;
__global__ void k_count_sets(const uint32_t *__restrict__ tag, const int8_t *__restrict__ bc, int64_t n,
                             unsigned *__restrict__ count)
{
    __shared__ unsigned s[kCounts];
    for (int k = threadIdx.x; k < kCounts; k += blockDim.x) s[k] = 0;
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const uint32_t t = i < n ? tag[i] : 0u;
    for (int k = 0; k < kTagBits; ++k) {
        const unsigned m = __ballot_sync(0xffffffffu, (t >> k) & 1u);
        if (m && (threadIdx.x & 31) == 0) atomicAdd(s + k, __popc(m));
    }
    if (t & TAG_BC) atomicAdd(s + kTagBits + bc[i], 1u);
    if ((t & TAG_C2F) && (t & (TAG_LATF | TAG_F2C))) atomicAdd(s + kCounts - 1, 1u);
    __syncthreads();
    for (int k = threadIdx.x; k < kCounts; k += blockDim.x)
        if (s[k]) atomicAdd(count + k, s[k]);
}

template <class Pred>
static int select_indices(Ctx &ctx, int64_t n, Pred pred, int32_t **out, int64_t *nout)
{
    *out = nullptr;
    *nout = 0;
    if (n == 0) return MT_OK;
    int32_t *buf = nullptr;
    int *d_num = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&buf, sizeof(int32_t) * n, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&d_num, sizeof(int), ctx.stream));
    cub::CountingInputIterator<int32_t> it(0);
    size_t tmp = 0;
    MT_CUDA(ctx, cub::DeviceSelect::If(nullptr, tmp, it, buf, d_num, (int)n, pred, ctx.stream));
    void *dtmp = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&dtmp, tmp, ctx.stream));
    MT_CUDA(ctx, cub::DeviceSelect::If(dtmp, tmp, it, buf, d_num, (int)n, pred, ctx.stream));
    int h_num = 0;
    MT_CUDA(ctx, cudaMemcpyAsync(&h_num, d_num, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(dtmp, ctx.stream);
    cudaFreeAsync(d_num, ctx.stream);
    if (h_num == 0) {
        cudaFreeAsync(buf, ctx.stream);
        return MT_OK;
    }
    *out = buf;
    *nout = h_num;
    return MT_OK;
}

static int concat_lists(Ctx &ctx, const int32_t *a, int64_t na, const int32_t *b, int64_t nb, int32_t **out,
                        int64_t *nout)
{
    *nout = na + nb;
    *out = nullptr;
    if (*nout == 0) return MT_OK;
    MT_CUDA(ctx, cudaMallocAsync(out, sizeof(int32_t) * (*nout), ctx.stream));
    if (na) MT_CUDA(ctx, cudaMemcpyAsync(*out, a, sizeof(int32_t) * na, cudaMemcpyDeviceToDevice, ctx.stream));
    if (nb) MT_CUDA(ctx, cudaMemcpyAsync(*out + na, b, sizeof(int32_t) * nb, cudaMemcpyDeviceToDevice, ctx.stream));
    return MT_OK;
}

static int build_level(Ctx &ctx, Case &c, int l)
{
    Level &lv = c.lv[l];
    const int Q = c.d.q;
    const bool on_dev = lv.draw_keys != nullptr;
    const int64_t nraw = on_dev ? lv.ndraw : (int64_t)lv.raw_keys.size();
    lv.n = lv.ncell = lv.nbrick = 0;
    if (nraw > 0) {
        uint64_t *d_raw = nullptr, *d_sorted = nullptr;
        uint8_t *d_set = nullptr;
        unsigned long long *d_start = nullptr, *d_scan = nullptr;
        if (on_dev) {
            d_raw = lv.draw_keys;
            d_set = lv.draw_set;
            lv.draw_keys = nullptr;
            lv.draw_set = nullptr;
            lv.ndraw = 0;
        } else {
            MT_CUDA(ctx, cudaMallocAsync(&d_raw, 8 * nraw, ctx.stream));
            MT_CUDA(ctx, cudaMallocAsync(&d_set, nraw, ctx.stream));
            MT_CUDA(ctx, cudaMemcpyAsync(d_raw, lv.raw_keys.data(), 8 * nraw, cudaMemcpyHostToDevice, ctx.stream));
            MT_CUDA(ctx, cudaMemcpyAsync(d_set, lv.raw_set.data(), nraw, cudaMemcpyHostToDevice, ctx.stream));
        }
        lv.low = 3 * (c.d.max_level - l);
        MT_CUDA(ctx, cudaMallocAsync(&d_sorted, 8 * nraw, ctx.stream));
        MT_CUDA(ctx, cudaMallocAsync(&d_start, 8 * nraw, ctx.stream));
        MT_CUDA(ctx, cudaMallocAsync(&d_scan, 8 * nraw, ctx.stream));
        size_t t1 = 0, t2 = 0;
        MT_CUDA(ctx, cub::DeviceRadixSort::SortKeys(nullptr, t1, d_raw, d_sorted, (int)nraw, 0, 64, ctx.stream));
        MT_CUDA(ctx, cub::DeviceScan::InclusiveSum(nullptr, t2, d_start, d_scan, (int)nraw, ctx.stream));
        void *tmp = nullptr;
        MT_CUDA(ctx, cudaMallocAsync(&tmp, std::max(t1, t2), ctx.stream));
        MT_CUDA(ctx, cub::DeviceRadixSort::SortKeys(tmp, t1, d_raw, d_sorted, (int)nraw, 0, 64, ctx.stream));
        k_starts<<<grid_for(nraw, 256), 256, 0, ctx.stream>>>(d_sorted, nraw, lv.low, d_start, c.dev_err);
        MT_LAUNCHED(ctx);
        MT_CUDA(ctx, cub::DeviceScan::InclusiveSum(tmp, t2, d_start, d_scan, (int)nraw, ctx.stream));
        unsigned long long h_num = 0;
        MT_CUDA(ctx, cudaMemcpyAsync(&h_num, d_scan + (nraw - 1), 8, cudaMemcpyDeviceToHost, ctx.stream));
        MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
        const int64_t nc = (int64_t)(h_num & 0xffffffffull), nb = (int64_t)(h_num >> 32);
        if (64 * nb >= ((int64_t)1 << 31))
            return set_err(ctx, MT_ERR_MESH, "a level holds more than 2^31 cell slots (64 per 4x4x4 brick in use)");
        lv.ncell = nc;
        lv.nbrick = nb;
        lv.n = 64 * nb;
        const int64_t n = lv.n;
        MT_CUDA(ctx, cudaMallocAsync(&lv.slot, 4 * nc, ctx.stream));
        MT_CUDA(ctx, cudaMallocAsync(&lv.bkey, 8 * nb, ctx.stream));
        MT_CUDA(ctx, cudaMallocAsync(&lv.bmask, 8 * nb, ctx.stream));
        MT_CUDA(ctx, cudaMallocAsync(&lv.bstart, 4 * nb, ctx.stream));
        MT_CUDA(ctx, cudaMemsetAsync(lv.bmask, 0, 8 * nb, ctx.stream));
        k_fill_bricks<<<grid_for(nraw, 256), 256, 0, ctx.stream>>>(d_sorted, d_scan, nraw, lv.low, lv.bkey,
                                                                   (unsigned long long *)lv.bmask, lv.bstart, lv.slot);
        MT_LAUNCHED(ctx);
        MT_CUDA(ctx, cudaMallocAsync(&lv.tag, 4 * n, ctx.stream));
        MT_CUDA(ctx, cudaMemsetAsync(lv.tag, 0, 4 * n, ctx.stream));
        MT_CUDA(ctx, cudaMallocAsync(&lv.bcidx, n, ctx.stream));
        MT_CUDA(ctx, cudaMemsetAsync(lv.bcidx, 0xff, n, ctx.stream));
        k_tag_cells<<<grid_for(nraw, 256), 256, 0, ctx.stream>>>(d_raw, d_set, nraw, lv.map(), lv.tag, lv.bcidx);
        MT_LAUNCHED(ctx);
        // neighbour bricks, where the periodic wraps fall on brick boundaries
        bool exact = true;
        for (int a = 0; a < 3; ++a) exact &= !(c.d.periodic[a] && ((c.d.extent0[a] << l) % 4) != 0);
        if (exact) {
            MT_CUDA(ctx, cudaMallocAsync(&lv.bnbr, 4 * 27 * nb, ctx.stream));
            k_brick_nbrs<<<grid_for(27 * nb, 256), 256, 0, ctx.stream>>>(c.geom, l, lv.bkey, nb, lv.low + 6, lv.low,
                                                                         lv.bnbr);
            MT_LAUNCHED(ctx);
        }
        cudaFreeAsync(tmp, ctx.stream);
        cudaFreeAsync(d_raw, ctx.stream);
        cudaFreeAsync(d_sorted, ctx.stream);
        cudaFreeAsync(d_start, ctx.stream);
        cudaFreeAsync(d_scan, ctx.stream);
        cudaFreeAsync(d_set, ctx.stream);
    }
    const int64_t n = lv.n;
    if (n == 0) return MT_OK;
    MT_CUDA(ctx, cudaMallocAsync(&lv.disrow, 4 * n, ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(lv.disrow, 0xff, 4 * n, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&lv.nbr, 4 * n * (Q - 1), ctx.stream));
    if (Q == 19)
        k_neighbors<19><<<grid_for(n, 128), 128, 0, ctx.stream>>>(c.geom, l, lv.map(), lv.bnbr, n, lv.nbr);
    else
        k_neighbors<27><<<grid_for(n, 128), 128, 0, ctx.stream>>>(c.geom, l, lv.map(), lv.bnbr, n, lv.nbr);
    MT_LAUNCHED(ctx);
    {
        int rc = amr_dispatch(c, [&](auto *tag) {
            using S = std::remove_pointer_t<decltype(tag)>;
            return AmrOps<S>::alloc(ctx, c, l);
        });
        if (rc) return rc;
    }
    unsigned *d_count = nullptr, count[kCounts];
    MT_CUDA(ctx, cudaMallocAsync(&d_count, sizeof(count), ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(count), ctx.stream));
    k_count_sets<<<grid_for(n, 256), 256, 0, ctx.stream>>>(lv.tag, lv.bcidx, n, d_count);
    MT_LAUNCHED(ctx);
    MT_CUDA(ctx, cudaMemcpyAsync(count, d_count, sizeof(count), cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d_count, ctx.stream);
    lv.mixed = count[kCounts - 1] != 0;
    const uint32_t bits[kNumSets] = {TAG_LATF, TAG_F2C, TAG_C2F, TAG_GC2F, TAG_GF2C, TAG_SF};
    for (int s = 0; s < kNumSets; ++s) {
        int at = 0;
        while ((bits[s] >> at) != 1u) ++at;
        int rc = select_known(ctx, n, TagHas{lv.tag, bits[s]}, count[at], &lv.list[s], &lv.nlist[s]);
        if (rc) return rc;
    }
    if (l == 0)
        for (int b = 0; b < 26; ++b) {
            int rc = select_known(ctx, n, BcIs{lv.bcidx, (int8_t)b}, count[kTagBits + b], &lv.bclist[b], &lv.nbc[b]);
            if (rc) return rc;
        }
    int rc = concat_lists(ctx, lv.list[0], lv.nlist[0], lv.list[1], lv.nlist[1], &lv.collide_list, &lv.ncollide);
    if (rc) return rc;
    return concat_lists(ctx, lv.list[0], lv.nlist[0], lv.list[2], lv.nlist[2], &lv.stream_list, &lv.nstream);
}

int amr_build(Ctx &ctx, Case &c)
{
    for (int f = 0; f < 6; ++f)
        for (int a = 0; a < 3; ++a) c.face_u[f][a] = c.d.u_bc[a];
    const int L = c.d.max_level;
    c.geom.L = L;
    for (int a = 0; a < 3; ++a) {
        c.geom.periodic[a] = c.d.periodic[a];
        c.geom.extent0[a] = c.d.extent0[a];
    }
    // the error flags, then the levels' EXPL_* flags, read back together below
    int herr[1 + kMaxLevels];
    MT_CUDA(ctx, cudaMallocAsync(&c.dev_err, sizeof(herr), ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(c.dev_err, 0, sizeof(herr), ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&c.force_acc, 4 * sizeof(double), ctx.stream));
    MT_CUDA(ctx, cudaMemsetAsync(c.force_acc, 0, 4 * sizeof(double), ctx.stream));
    for (int l = 0; l <= L; ++l) {
        int rc = build_level(ctx, c, l);
        if (rc) return rc;
    }
    // dis rows and the IB cell list on the finest level
    if (!c.dis_on_device) c.ndis = (int64_t)c.h_dis_key.size();
    const int W = c.d.q - 1;
    if (c.ndis > 0) {
        if (!c.dis_on_device) {
            MT_CUDA(ctx, cudaMallocAsync(&c.dis_key, 8 * c.ndis, ctx.stream));
            MT_CUDA(ctx, cudaMallocAsync(&c.dis, 8 * c.ndis * W, ctx.stream));
            MT_CUDA(ctx, cudaMemcpyAsync(c.dis_key, c.h_dis_key.data(), 8 * c.ndis, cudaMemcpyHostToDevice,
                                         ctx.stream));
            MT_CUDA(ctx, cudaMemcpyAsync(c.dis, c.h_dis.data(), 8 * c.ndis * W, cudaMemcpyHostToDevice, ctx.stream));
        }
        Level &fl = c.lv[L];
        if (fl.n > 0) {
            k_dis_rows<<<grid_for(fl.ncell, 256), 256, 0, ctx.stream>>>(fl.map(), fl.slot, fl.ncell, c.dis_key, c.ndis,
                                                                        fl.disrow, fl.tag);
            MT_LAUNCHED(ctx);
        }
        k_dis_check<<<grid_for(c.ndis, 256), 256, 0, ctx.stream>>>(c.dis_key, c.ndis, fl.map(), c.dev_err);
        MT_LAUNCHED(ctx);
        int rc = select_indices(ctx, fl.n, IbLatf{fl.tag}, &fl.iblist, &fl.nib);
        if (rc) return rc;
        // the force partials of 32-cell blocks and the number of calls
        if (fl.nib) {
            const size_t bytes = 8 * (3 * (size_t)grid_for(fl.nib, 32) + 1);
            MT_CUDA(ctx, cudaMallocAsync(&c.ib_force, bytes, ctx.stream));
            MT_CUDA(ctx, cudaMemsetAsync(c.ib_force, 0, bytes, ctx.stream));
            if ((rc = amr_dispatch(c, [&](auto *tag) {
                     using S = std::remove_pointer_t<decltype(tag)>;
                     return AmrOps<S>::ib_tables(ctx, c);
                 })))
                return rc;
        }
    }
    {
        int64_t maxn = 0;
        for (int b = 0; b < 26; ++b) maxn = std::max(maxn, c.lv[0].nbc[b]);
        if (maxn) MT_CUDA(ctx, cudaMallocAsync(&c.bc_tmp, sizeof(double) * 18 * maxn, ctx.stream));
        // the concatenated list of all 26 sets for the one-pass sweep
        int64_t tot = 0;
        for (int b = 0; b < 26; ++b) tot += c.lv[0].nbc[b];
        if (tot) {
            c.nbc_all = tot;
            MT_CUDA(ctx, cudaMallocAsync(&c.bc_all, sizeof(int32_t) * tot, ctx.stream));
            MT_CUDA(ctx, cudaMallocAsync(&c.bc_setb, tot, ctx.stream));
            MT_CUDA(ctx, cudaMallocAsync(&c.bc_tmp_all, sizeof(double) * 18 * tot, ctx.stream));
            int64_t off = 0;
            for (int b = 0; b < 26; ++b) {
                const int64_t nb = c.lv[0].nbc[b];
                if (!nb) continue;
                MT_CUDA(ctx, cudaMemcpyAsync(c.bc_all + off, c.lv[0].bclist[b], sizeof(int32_t) * nb,
                                             cudaMemcpyDeviceToDevice, ctx.stream));
                MT_CUDA(ctx, cudaMemsetAsync(c.bc_setb + off, b, nb, ctx.stream));
                off += nb;
            }
        }
    }
    // direct-forcing band of the finest level and its collide list without the band
    {
        Level &fl = c.lv[L];
        if (fl.n) {
            int rc = select_indices(ctx, fl.n, TagHas{fl.tag, TAG_BAND}, &fl.band, &fl.nband);
            if (rc) return rc;
            if (fl.nband) {
                int32_t *lat = nullptr;
                int64_t nlat = 0;
                rc = select_indices(ctx, fl.n, LatfNotBand{fl.tag}, &lat, &nlat);
                if (rc) return rc;
                rc = concat_lists(ctx, lat, nlat, fl.list[1], fl.nlist[1], &fl.collide_nb, &fl.ncollide_nb);
                cudaFreeAsync(lat, ctx.stream);
                if (rc) return rc;
                MT_CUDA(ctx, cudaMallocAsync(&c.acc, sizeof(long long) * 3 * fl.n, ctx.stream));
                MT_CUDA(ctx, cudaMemsetAsync(c.acc, 0, sizeof(long long) * 3 * fl.n, ctx.stream));
                MT_CUDA(ctx, cudaMallocAsync(&c.tstep, sizeof(long long), ctx.stream));
                MT_CUDA(ctx, cudaMemsetAsync(c.tstep, 0, sizeof(long long), ctx.stream));
            }
        }
    }
    // cross-level child tables
    for (int l = 1; l <= L; ++l) {
        Level &cl = c.lv[l - 1], &fl = c.lv[l];
        int rc = concat_lists(ctx, cl.list[1], cl.nlist[1], cl.list[4], cl.nlist[4], &fl.expl_src, &fl.nexpl);
        if (rc) return rc;
        fl.nexpl_f2c = cl.nlist[1];
        if (fl.nexpl) {
            MT_CUDA(ctx, cudaMallocAsync(&fl.expl_child, 4 * fl.nexpl, ctx.stream));
            MT_CUDA(ctx, cudaMallocAsync(&fl.expl_mask, fl.nexpl, ctx.stream));
            k_expl_children<<<grid_for(fl.nexpl, 128), 128, 0, ctx.stream>>>(
                c.geom, l, fl.expl_src, fl.nexpl, fl.nexpl_f2c, cl.map(), fl.map(), fl.tag, c.dis_key, c.ndis,
                fl.expl_child, fl.expl_mask, c.dev_err, c.dev_err + 1 + l);
            MT_LAUNCHED(ctx);
        }
        if (cl.nlist[1]) {
            MT_CUDA(ctx, cudaMallocAsync(&cl.coal_child, 4 * cl.nlist[1], ctx.stream));
            k_coal_children<<<grid_for(cl.nlist[1], 128), 128, 0, ctx.stream>>>(
                c.geom, l, cl.list[1], cl.nlist[1], cl.map(), fl.map(), cl.coal_child, c.dev_err);
            MT_LAUNCHED(ctx);
        }
    }
    MT_CUDA(ctx, cudaMemcpyAsync(herr, c.dev_err, sizeof(herr), cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    if (herr[0] & DEVERR_KEY_BITS)
        return set_err(ctx, MT_ERR_MESH, "a key has bits set below the cells of its level");
    if (herr[0] & DEVERR_MISSING_CHILD)
        return set_err(ctx, MT_ERR_MESH, "a child of an overlap_F2C cell is not stored on the finer level");
    if (herr[0] & DEVERR_DIS_NOT_FINEST) return set_err(ctx, MT_ERR_MESH, "a dis key is not a finest-level cell");
    for (int l = 0; l <= L; ++l) {
        c.lv[l].chained = herr[1 + l] & EXPL_SOURCE;
        c.lv[l].hold_once = herr[1 + l] == 0;
        c.lv[l].raw_keys.clear();
        c.lv[l].raw_keys.shrink_to_fit();
        c.lv[l].raw_set.clear();
        c.lv[l].raw_set.shrink_to_fit();
    }
    c.built = true;
    return MT_OK;
}

void amr_drop_fused(Ctx &ctx, Case &c)
{
    for (int p = 0; p < 2; ++p) {
        if (c.fgraph[p]) cudaGraphExecDestroy(c.fgraph[p]);
        c.fgraph[p] = nullptr;
    }
    for (int l = 0; l < kMaxLevels; ++l) {
        Level &lv = c.lv[l];
        void *ptrs[] = {lv.fused_list, lv.bcls, lv.bflag, lv.blist};
        for (void *p : ptrs)
            if (p) cudaFreeAsync(p, ctx.stream);
        lv.fused_list = nullptr;
        lv.nfused = 0;
        lv.bcls = nullptr;
        lv.bflag = nullptr;
        lv.blist = nullptr;
        lv.nblist = 0;
        lv.bricks = false;
    }
}

void amr_free(Case &c)
{
    for (int l = 0; l < kMaxLevels; ++l) {
        Level &lv = c.lv[l];
        void *ptrs[] = {lv.slot, lv.bkey, lv.tag, lv.bcidx, lv.disrow, lv.nbr, lv.f, lv.fcol, lv.rho, lv.u,
                        lv.collide_list, lv.stream_list, lv.iblist, lv.expl_src, lv.expl_child, lv.expl_mask, lv.coal_child,
                        lv.fcol_alt, lv.fused_list, lv.bstart, lv.bmask, lv.bnbr, lv.bcls, lv.bflag, lv.blist,
                        lv.band, lv.collide_nb, lv.draw_keys, lv.draw_set, lv.expl_prev, lv.info_prev};
        for (void *p : ptrs)
            if (p) cudaFree(p);
        for (int s = 0; s < kNumSets; ++s)
            if (lv.list[s]) cudaFree(lv.list[s]);
        for (int b = 0; b < 26; ++b)
            if (lv.bclist[b]) cudaFree(lv.bclist[b]);
        lv = Level();
    }
    if (c.h_force) cudaFreeHost(c.h_force);
    c.h_force = nullptr;
    void *ptrs[] = {c.dis_key, c.dis, c.ib_wall, c.ib_src, c.ib_factor, c.ib_force, c.force_acc, c.dev_err, c.bc_tmp, c.bc_all, c.bc_setb, c.bc_tmp_all,
                    c.mref, c.mdv, c.path, c.mforce, c.tstep, c.acc, c.mgrid};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    c.bc_tmp = nullptr;
    c.bc_all = nullptr;
    c.bc_setb = nullptr;
    c.bc_tmp_all = nullptr;
    c.nbc_all = 0;
    c.dis_key = nullptr;
    c.dis = nullptr;
    c.ib_wall = nullptr;
    c.ib_src = nullptr;
    c.ib_factor = nullptr;
    c.ib_force = nullptr;
    c.force_acc = nullptr;
    c.dev_err = nullptr;
    c.mref = c.mdv = c.path = c.mforce = nullptr;
    c.tstep = nullptr;
    c.acc = nullptr;
    c.mgrid = nullptr;
    c.nm = 0;
    if (c.graph) cudaGraphExecDestroy(c.graph);
    c.graph = nullptr;
    for (int p = 0; p < 2; ++p) {
        if (c.fgraph[p]) cudaGraphExecDestroy(c.fgraph[p]);
        c.fgraph[p] = nullptr;
    }
    c.side = nullptr;
}

// ----------------------------------------------------------------------------
// driver: the reference's recursion issued as phase kernels of the case's
// storage type (mt_amr_phases.cuh, instantiated in mt_amr_f64.cu and
// mt_amr_lp.cu)
// ----------------------------------------------------------------------------

int amr_phase(Ctx &ctx, Case &c, int phase, int level)
{
    if (level < 0 || level > c.d.max_level) return set_err(ctx, MT_ERR_ARG, "level out of range");
    return amr_dispatch(c, [&](auto *tag) {
        using S = std::remove_pointer_t<decltype(tag)>;
        return AmrOps<S>::phase(ctx, c, phase, level);
    });
}

int amr_init_equilibrium(Ctx &ctx, Case &c, double rho0, const double *u0)
{
    c.prev_stale = true;
    return amr_dispatch(c, [&](auto *tag) {
        using S = std::remove_pointer_t<decltype(tag)>;
        return AmrOps<S>::init_eq(ctx, c, rho0, u0);
    });
}

// LBM_Manager::LBMkernel (LBM_Simulator.cpp:20-229).  The collision kernel
// computes the macros it needs from the same populations the reference's
// calculateMacros(level) reads just before collide(level), so the separate
// macros pass of each substep is folded into it.
int make_branch(Ctx &ctx, Branch &b)
{
    if (!b.s) MT_CUDA(ctx, cudaStreamCreateWithFlags(&b.s, cudaStreamNonBlocking));
    if (!b.fork) MT_CUDA(ctx, cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming));
    if (!b.join) MT_CUDA(ctx, cudaEventCreateWithFlags(&b.join, cudaEventDisableTiming));
    return MT_OK;
}
void free_branch(Branch &b)
{
    if (b.s) cudaStreamDestroy(b.s);
    if (b.fork) cudaEventDestroy(b.fork);
    if (b.join) cudaEventDestroy(b.join);
    b = Branch{};
}
void free_side(Side &side)
{
    for (Branch &b : side.level) free_branch(b);
    side.level.clear();
    free_branch(side);
}
static int open_side(Ctx &ctx, Side &side, int levels)
{
    if (int rc = make_branch(ctx, side)) return rc;
    if ((int)side.level.size() < levels) side.level.resize(levels);
    for (int l = 0; l < levels; ++l)
        if (int rc = make_branch(ctx, side.level[l])) return rc;
    return MT_OK;
}
static int make_side(Ctx &ctx, Case &c)
{
    if (!c.side) c.side = &ctx.side;
    return open_side(ctx, *c.side, c.d.max_level);
}
// A case holds its side streams only while its work is issued: it may move to
// another context between two calls (mt_case_transfer), and the one it leaves
// may be destroyed.
struct SideScope {
    Case &c;
    ~SideScope() { c.side = nullptr; }
};
// (the brick stream can leave cells out)
static bool ib_beside_stream(const Case &c)
{
    const Level &lv = c.lv[c.d.max_level];
    return c.d.ib_method != MT_IB_DF && lv.nib && lv.nstream && lv.bnbr && lv.n * c.d.q < ((int64_t)1 << 32);
}

static int phase_lbm_kernel(Ctx &ctx, Case &c, int l)
{
    const int L = c.d.max_level;
    int rc;
#define RUN(ph, lev)                               \
    do {                                           \
        if ((rc = amr_phase(ctx, c, (ph), (lev)))) \
            return rc;                             \
    } while (0)
    for (int sub = 0; sub < 2; ++sub) {
        RUN(PH_COLLIDE, l);
        if (l == 0 && c.d.bc_mode == MT_BC_ZOUHE_OUTFLOW) RUN(PH_BC_INOUT, 0);
        if (l < L)
            if ((rc = phase_lbm_kernel(ctx, c, l + 1))) return rc;
        if (l > 0 && sub == 0) RUN(PH_EXPLOSION, l);
        if (l > 0 && sub == 1 && c.itime != MT_ITIME_REFERENCE) RUN(PH_EXPLOSION_B, l);
        if (l > 0 && l == L && ib_beside_stream(c)) {
            // treat() reads fcol and writes every population of its cells, so
            // their stream would be overwritten: left out, the two run side by
            // side
            if ((rc = make_side(ctx, c))) return rc;
            cudaStream_t main = ctx.stream;
            MT_CUDA(ctx, cudaEventRecord(c.side->fork, main));
            MT_CUDA(ctx, cudaStreamWaitEvent(c.side->s, c.side->fork, 0));
            ctx.stream = c.side->s;
            rc = amr_phase(ctx, c, PH_IB, L);
            ctx.stream = main;
            c.skip_ib = true;
            if (!rc) rc = amr_phase(ctx, c, PH_STREAM, l);
            c.skip_ib = false;
            // (joined on an error too: the streams may be capturing)
            MT_CUDA(ctx, cudaEventRecord(c.side->join, c.side->s));
            MT_CUDA(ctx, cudaStreamWaitEvent(main, c.side->join, 0));
            if (rc) return rc;
        } else {
            RUN(PH_STREAM, l);
            if (l == 0) {
                if (c.d.bc_mode == MT_BC_NEQ) RUN(PH_BC, 0);
                if (c.d.bc_mode == MT_BC_ZOUHE_HH) RUN(PH_BC_HH, 0);
            } else if (l == L) {
                RUN(PH_IB, L);
            }
        }
        if (l < L) RUN(PH_COALESCENCE, l);
        if (l == 0) break;
    }
#undef RUN
    return MT_OK;
}

int amr_lbm_kernel(Ctx &ctx, Case &c, int l)
{
    SideScope scope{c};
    return phase_lbm_kernel(ctx, c, l);
}

static int record_step(Ctx &ctx, Case &c)
{
    int rc = phase_lbm_kernel(ctx, c, 0);
    if (rc) return rc;
    if (!c.side) {
        if ((rc = amr_phase(ctx, c, PH_IB_SUM, 0))) return rc;
        return amr_phase(ctx, c, PH_MACROS_ALL, 0);
    }
    cudaStream_t main = ctx.stream;
    MT_CUDA(ctx, cudaEventRecord(c.side->fork, main));
    MT_CUDA(ctx, cudaStreamWaitEvent(c.side->s, c.side->fork, 0));
    ctx.stream = c.side->s;
    rc = amr_phase(ctx, c, PH_IB_SUM, 0);
    ctx.stream = main;
    if (!rc) rc = amr_phase(ctx, c, PH_MACROS_ALL, 0);
    MT_CUDA(ctx, cudaEventRecord(c.side->join, c.side->s));
    MT_CUDA(ctx, cudaStreamWaitEvent(main, c.side->join, 0));
    return rc;
}

static int capture(Ctx &ctx, Case &c, int (*record)(Ctx &, Case &), cudaGraphExec_t *out, int64_t *launches)
{
    const int64_t before = ctx.launches;
    SideScope scope{c};
    MT_CUDA(ctx, cudaStreamBeginCapture(ctx.stream, cudaStreamCaptureModeThreadLocal));
    int rc = record(ctx, c);
    cudaGraph_t captured = nullptr;
    cudaError_t e = cudaStreamEndCapture(ctx.stream, &captured);
    if (rc) {
        if (captured) cudaGraphDestroy(captured);
        return rc;
    }
    if (e != cudaSuccess) return set_err(ctx, MT_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
    *launches = ctx.launches - before;
    ctx.launches = before;
    e = cudaGraphInstantiate(out, captured, 0);
    cudaGraphDestroy(captured);
    if (e != cudaSuccess) {
        *out = nullptr;
        return set_err(ctx, MT_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
    }
    return MT_OK;
}

// ---- fused schedule ---------------------------------------------------------
// Per substep of level l: swap the post-collision buffers (fcol now holds the
// collision computed one substep ahead, F2C cells included), the
// inlet/outflow wall cells, the finer levels, the explosion, then one pass
// that streams lat_f and C2F, treats the IB cells and collides all of them
// into the other buffer for the next substep; then the boundary sweep, and
// coalescence followed by the F2C cells' next collision, as in
// LBM_Simulator.cpp:20-229.  On each level's last substep of the coarse step
// the passes also write the macros of the f they leave (the all-level
// calculateMacros of LBM_Simulator.cpp:11-17), except on level 0 under the
// non-equilibrium boundary, whose sweep reads the substep's earlier macros.
static void swap_buffers(Case &c, int l)
{
    std::swap(c.lv[l].fcol, c.lv[l].fcol_alt);
    if (l == 0) c.par0 ^= 1;
}

static int fused_lbm_kernel(Ctx &ctx, Case &c, int l, bool last_parent)
{
    const int L = c.d.max_level;
    int rc;
#define RUN(ph, lev)                               \
    do {                                           \
        if ((rc = amr_phase(ctx, c, (ph), (lev)))) \
            return rc;                             \
    } while (0)
    for (int sub = 0; sub < 2; ++sub) {
        const bool last = last_parent && (l == 0 || sub == 1);
        const int mac = last && !(l == 0 && c.d.bc_mode == MT_BC_NEQ);
        swap_buffers(c, l);
        if (l == 0 && c.d.bc_mode == MT_BC_ZOUHE_OUTFLOW) RUN(PH_BC_INOUT, 0);
        auto own = [&]() -> int {
            if (l > 0 && sub == 0) RUN(PH_EXPLOSION, l);
            if (l > 0 && sub == 1 && c.itime != MT_ITIME_REFERENCE) RUN(PH_EXPLOSION_B, l);
            c.macros_now = mac;
            RUN(PH_PULL_COLLIDE, l);
            if (l == L && c.lv[l].nband) RUN(PH_DF, l);
            if (l == 0 && c.d.bc_mode == MT_BC_NEQ) RUN(PH_BC, 0);
            return MT_OK;
        };
        if (l < L && !c.lv[l].chained) {
            // the finer levels read this level's fcol, which its own work leaves
            // alone (its explosion writes none of their sources): side by side
            Branch &b = c.side->level[l];
            cudaStream_t main = ctx.stream;
            MT_CUDA(ctx, cudaEventRecord(b.fork, main));
            MT_CUDA(ctx, cudaStreamWaitEvent(b.s, b.fork, 0));
            ctx.stream = b.s;
            rc = own();
            ctx.stream = main;
            if (!rc) rc = fused_lbm_kernel(ctx, c, l + 1, last);
            // (joined on an error too: the streams may be capturing)
            MT_CUDA(ctx, cudaEventRecord(b.join, b.s));
            MT_CUDA(ctx, cudaStreamWaitEvent(main, b.join, 0));
            if (rc) return rc;
        } else {
            if (l < L)
                if ((rc = fused_lbm_kernel(ctx, c, l + 1, last))) return rc;
            if ((rc = own())) return rc;
        }
        if (l < L) {
            c.macros_now = mac;
            RUN(PH_COAL_COLLIDE, l);
        }
        c.macros_now = 0;
        if (l == 0) break;
    }
#undef RUN
    return MT_OK;
}

static int record_fused_step(Ctx &ctx, Case &c)
{
    if (c.d.max_level > 0)
        if (int rc = make_side(ctx, c)) return rc;
    c.fused_now = true;
    int rc = fused_lbm_kernel(ctx, c, 0, true);
    c.fused_now = false;
    if (c.side_open) {
        MT_CUDA(ctx, cudaEventRecord(c.side->join, c.side->s));
        MT_CUDA(ctx, cudaStreamWaitEvent(ctx.stream, c.side->join, 0));
        c.side_open = false;
    }
    if (rc) return rc;
    if (c.d.bc_mode == MT_BC_NEQ)
        if ((rc = amr_phase(ctx, c, PH_MACROS, 0))) return rc;
    return MT_OK;
}

// The fused pass's tables of level l, where the neighbour bricks are exact.
static int build_bricks(Ctx &ctx, Case &c, int l)
{
    Level &lv = c.lv[l];
    const int L = c.d.max_level;
    const int64_t n = lv.n, nb = lv.nbrick;
    if (!lv.bnbr) return MT_OK;
    if (n * c.d.q >= ((int64_t)1 << 32)) return MT_OK;  // the brick pass uses 32-bit element offsets
    MT_CUDA(ctx, cudaMallocAsync(&lv.bcls, n, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&lv.bflag, nb, ctx.stream));
    const int ib_level = (l == L && l > 0) ? 1 : 0;
    k_brick_cls<<<grid_for(n, 256), 256, 0, ctx.stream>>>(lv.tag, n, ib_level, lv.bcls);
    MT_LAUNCHED(ctx);
    if (l > 0 && c.lv[l - 1].coal_child && c.lv[l - 1].nlist[1]) {
        const int64_t cnt = c.lv[l - 1].nlist[1];
        k_brick_mark<<<grid_for(8 * cnt, 256), 256, 0, ctx.stream>>>(c.lv[l - 1].coal_child, cnt, lv.bcls);
        MT_LAUNCHED(ctx);
    }
    if (l > 0 && lv.nexpl && c.itime == MT_ITIME_HOLD && lv.hold_once) {
        k_brick_exploded<<<grid_for(8 * lv.nexpl, 256), 256, 0, ctx.stream>>>(lv.expl_child, lv.expl_mask, lv.nexpl,
                                                                             lv.bcls);
        MT_LAUNCHED(ctx);
    }
    if (c.d.q == 19)
        k_brick_flag<19><<<grid_for(32 * nb, 128), 128, 0, ctx.stream>>>(nb, lv.bcls, lv.nbr, lv.bflag);
    else
        k_brick_flag<27><<<grid_for(32 * nb, 128), 128, 0, ctx.stream>>>(nb, lv.bcls, lv.nbr, lv.bflag);
    MT_LAUNCHED(ctx);
    if (int rc = select_indices(ctx, nb, BrickHasWork{lv.bflag}, &lv.blist, &lv.nblist)) return rc;
    lv.bricks = true;
    return MT_OK;
}

// second buffers, the fused cell lists, and the lookahead collision of the
// current f on every level
static int prime_fused(Ctx &ctx, Case &c)
{
    const int L = c.d.max_level;
    if (L > 0)  // (made here, not while the step is captured)
        if (int rc = open_side(ctx, ctx.side, L)) return rc;
    for (int l = 0; l <= L; ++l) {
        Level &lv = c.lv[l];
        if (!lv.n) continue;
        if (!lv.fcol_alt) {
            const size_t bytes = (size_t)c.d.q * (size_t)lv.n *
                                 (c.d.storage == MT_STORE_F64 ? 8 : c.d.storage == MT_STORE_F32 ? 4 : 2);
            MT_CUDA(ctx, cudaMallocAsync(&lv.fcol_alt, bytes, ctx.stream));
        }
        if (!lv.bricks && c.use_bricks) {
            int rc = build_bricks(ctx, c, l);
            if (rc) return rc;
        }
        if (!lv.bricks && !lv.fused_list && lv.nlist[0]) {
            int rc = lv.nband ? select_indices(ctx, lv.n, LatfNotBand{lv.tag}, &lv.fused_list, &lv.nfused)
                     : (l == L && l > 0) ? select_indices(ctx, lv.n, LatfNotIb{lv.tag}, &lv.fused_list, &lv.nfused)
                                         : select_indices(ctx, lv.n, TagHas{lv.tag, TAG_LATF}, &lv.fused_list,
                                                          &lv.nfused);
            if (rc) return rc;
        }
        int rc = amr_phase(ctx, c, PH_PRIME, l);
        if (rc) return rc;
    }
    c.primed = true;
    return MT_OK;
}

// the streamed f the fused passes left unstored (class-1 brick cells), for
// every reader outside the fused schedule
int amr_sync_f(Ctx &ctx, Case &c)
{
    if (!c.f_stale) return MT_OK;
    for (int l = 0; l <= c.d.max_level; ++l) {
        int rc = amr_phase(ctx, c, PH_SYNC_F, l);
        if (rc) return rc;
    }
    c.f_stale = false;
    return MT_OK;
}

// a face strategy's velocity: its boundary cells restart from feq(rho0, u)
// and its non-equilibrium sweep (or the West inlet) uses u from now on
int amr_set_face(Ctx &ctx, Case &c, int face, const double *u)
{
    if (int rc = amr_sync_f(ctx, c)) return rc;
    for (int a = 0; a < 3; ++a) c.face_u[face][a] = u[a];
    if (c.graph) cudaGraphExecDestroy(c.graph);
    c.graph = nullptr;
    for (int p = 0; p < 2; ++p) {
        if (c.fgraph[p]) cudaGraphExecDestroy(c.fgraph[p]);
        c.fgraph[p] = nullptr;
    }
    c.primed = false;
    return amr_phase(ctx, c, PH_FACE_EQ0 + face, 0);
}

// n coarse steps replayed from one captured graph (fluidSimulate loop body)
int amr_prev_sync(Ctx &ctx, Case &c)
{
    if (c.itime != MT_ITIME_EXTRAP) return MT_OK;
    const size_t sb = c.d.storage == MT_STORE_F64 ? 8 : c.d.storage == MT_STORE_F32 ? 4 : 2;
    for (int l = 1; l <= c.d.max_level; ++l) {
        Level &lv = c.lv[l];
        if (!lv.nexpl || lv.expl_prev) continue;
        MT_CUDA(ctx, cudaMallocAsync(&lv.expl_prev, sb * (size_t)c.d.q * (size_t)lv.nexpl, ctx.stream));
        c.prev_stale = true;
    }
    if (!c.prev_stale) return MT_OK;
    for (int l = 1; l <= c.d.max_level; ++l)
        if (int rc = amr_phase(ctx, c, PH_EXPL_SAVE, l)) return rc;
    c.prev_stale = false;
    return MT_OK;
}

int amr_step(Ctx &ctx, Case &c, int n)
{
    int rc;
    if ((rc = amr_prev_sync(ctx, c))) return rc;
    if (c.schedule == MT_SCHED_FUSED) {
        if (!c.primed && (rc = prime_fused(ctx, c))) return rc;
        for (int s = 0; s < n; ++s) {
            const int p = c.par0;
            if (!c.fgraph[p]) {
                // recording swaps the host-side buffer pointers exactly as one
                // replay does, so after it the state matches a launched step
                if ((rc = capture(ctx, c, record_fused_step, &c.fgraph[p], &c.fgraph_launches[p]))) {
                    c.primed = false;
                    return rc;
                }
            } else {
                // the host-side effect of one replay: level 0 swaps once,
                // levels >= 1 an even number of times
                swap_buffers(c, 0);
            }
            MT_CUDA(ctx, cudaGraphLaunch(c.fgraph[p], ctx.stream));
            ctx.launches += c.fgraph_launches[p];
            for (int l = 0; l <= c.d.max_level; ++l) c.f_stale |= c.lv[l].bricks;
        }
        return MT_OK;
    }
    if ((rc = amr_sync_f(ctx, c))) return rc;
    c.primed = false;
    if (c.graph && c.graph_par0 != c.par0) {
        cudaGraphExecDestroy(c.graph);
        c.graph = nullptr;
    }
    if (!c.graph) {
        if ((rc = capture(ctx, c, record_step, &c.graph, &c.graph_launches))) return rc;
        c.graph_par0 = c.par0;
    }
    for (int s = 0; s < n; ++s) {
        MT_CUDA(ctx, cudaGraphLaunch(c.graph, ctx.stream));
        ctx.launches += c.graph_launches;
    }
    return MT_OK;
}

int amr_prime(Ctx &ctx, Case &c)
{
    return c.primed ? MT_OK : prime_fused(ctx, c);
}

// ---- batches ------------------------------------------------------------------
// The members never interact: each one's fused step is a branch of the
// captured graph of its own, from the step's fork to its end.  (Members in
// lockstep, joined after every phase, with one kernel over all members' bricks
// per level and model, waited for the slowest member at each phase: 8 mid-sized
// members 1.63 ms a coarse step against 1.38, 16 small ones 1.83 / 1.48, 4 of
// 32^3 0.217 / 0.125, 48 up to 128x64x64 16.4 / 16.2.)
namespace {

int record_batch_step(Ctx &ctx, Batch &B, const std::vector<Case *> &cases)
{
    cudaStream_t main = ctx.stream;
    const size_t P = std::min(B.pool.size(), cases.size());
    MT_CUDA(ctx, cudaEventRecord(B.ev_fork, main));
    for (size_t p = 0; p < P; ++p) MT_CUDA(ctx, cudaStreamWaitEvent(B.pool[p].s, B.ev_fork, 0));
    int rc = MT_OK;
    for (size_t i = 0; i < cases.size() && !rc; ++i) {
        Case &c = *cases[i];
        SideScope scope{c};
        ctx.stream = B.pool[i % P].s;
        c.side = B.side[i % P].get();
        // (a single-level member too: its forcing forks)
        rc = make_side(ctx, c);
        if (!rc) rc = record_fused_step(ctx, c);
    }
    ctx.stream = main;
    for (size_t p = 0; p < P; ++p) {
        MT_CUDA(ctx, cudaEventRecord(B.pool[p].join, B.pool[p].s));
        MT_CUDA(ctx, cudaStreamWaitEvent(main, B.pool[p].join, 0));
    }
    return rc;
}

}  // namespace

void batch_drop(Batch &b)
{
    for (int p = 0; p < 3; ++p) {
        if (b.graph[p]) cudaGraphExecDestroy(b.graph[p]);
        b.graph[p] = nullptr;
    }
    b.par = 0;
}

void batch_free(Batch &b)
{
    batch_drop(b);
    for (Branch &x : b.pool) free_branch(x);
    for (auto &x : b.side) free_side(*x);
    if (b.ev_fork) cudaEventDestroy(b.ev_fork);
    b.pool.clear();
    b.side.clear();
    b.ev_fork = nullptr;
}

int batch_step(Ctx &ctx, Batch &B, const std::vector<Case *> &cases, int n)
{
    if (cases.empty() || n <= 0) return MT_OK;
    int rc;
    for (Case *c : cases) {
        if ((rc = amr_prev_sync(ctx, *c))) return rc;
        if ((rc = amr_sync_f(ctx, *c))) return rc;
        if (!c->primed && (rc = prime_fused(ctx, *c))) return rc;
    }
    const size_t P = std::min<size_t>(kBatchStreams, cases.size());
    while (B.pool.size() < P) {
        Branch b;
        if ((rc = make_branch(ctx, b))) return rc;
        B.pool.push_back(b);
        B.side.emplace_back(new Side);
    }
    if (!B.ev_fork) MT_CUDA(ctx, cudaEventCreateWithFlags(&B.ev_fork, cudaEventDisableTiming));
    // capture graph g (0/1: one step from that parity, 2: two steps from parity 0)
    auto record = [&](int g) -> int {
        const int steps = g == 2 ? 2 : 1;
        const int64_t before = ctx.launches;
        cudaGraph_t captured = nullptr;
        cudaError_t e = cudaStreamBeginCapture(ctx.stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return set_err(ctx, MT_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
        int r = MT_OK;
        for (int k = 0; k < steps && !r; ++k) r = record_batch_step(ctx, B, cases);
        e = cudaStreamEndCapture(ctx.stream, &captured);
        if (r || e != cudaSuccess) {
            if (captured) cudaGraphDestroy(captured);
            batch_drop(B);
            return r ? r : set_err(ctx, MT_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
        }
        B.graph_launches[g] = ctx.launches - before;
        ctx.launches = before;
        e = cudaGraphInstantiate(&B.graph[g], captured, 0);
        cudaGraphDestroy(captured);
        if (e != cudaSuccess) {
            B.graph[g] = nullptr;
            return set_err(ctx, MT_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
        }
        // recording swapped the members' buffers as executing does; undo it
        // so that the caller applies one consistent host-side update per launch
        for (int k = 0; k < steps; ++k)
            for (Case *c : cases) swap_buffers(*c, 0);
        return MT_OK;
    };
    int s = 0;
    while (s < n) {
        // (from parity 1 a single step leads to where the two start: the buffers
        // a graph reads are those of the parity it was recorded from)
        const int g = (n - s >= 2 && B.par == 0) ? 2 : B.par;
        if (!B.graph[g] && (rc = record(g))) return rc;
        MT_CUDA(ctx, cudaGraphLaunch(B.graph[g], ctx.stream));
        ctx.launches += B.graph_launches[g];
        const int steps = g == 2 ? 2 : 1;
        for (int k = 0; k < steps; ++k) {
            for (Case *c : cases) swap_buffers(*c, 0);
            B.par ^= 1;
        }
        s += steps;
        for (Case *c : cases)
            for (int l = 0; l <= c->d.max_level; ++l) c->f_stale |= c->lv[l].bricks;
    }
    return MT_OK;
}

int amr_guard(Ctx &ctx, Case &c, int *flags)
{
    if (int rc = amr_sync_f(ctx, c)) return rc;
    MT_CUDA(ctx, cudaMemsetAsync(c.dev_err, 0, sizeof(int), ctx.stream));
    int rc = amr_dispatch(c, [&](auto *tag) {
        using S = std::remove_pointer_t<decltype(tag)>;
        return AmrOps<S>::guard(ctx, c);
    });
    if (rc) return rc;
    MT_CUDA(ctx, cudaMemcpyAsync(flags, c.dev_err, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    return MT_OK;
}

// FP64 per-level and volume-weighted sums of mass, momentum and kinetic
// energy (host out[(max_level + 2) * 5]); the streamed f is rebuilt first
// where the fused schedule does not store it
int amr_reduce(Ctx &ctx, Case &c, double *h_out)
{
    if (int rc = amr_sync_f(ctx, c)) return rc;
    const size_t nb = sizeof(double) * 5 * (size_t)(c.d.max_level + 2);
    double *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, nb, ctx.stream));
    int rc = amr_dispatch(c, [&](auto *tag) {
        using S = std::remove_pointer_t<decltype(tag)>;
        return AmrOps<S>::reduce(ctx, c, d);
    });
    if (!rc) MT_CUDA(ctx, cudaMemcpyAsync(h_out, d, nb, cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d, ctx.stream);
    return rc;
}

// LBM_Manager::infoPrint's per-level diagnostics (mt_case_info): the
// end-of-step macros are current after every coarse step under both
// schedules, so no population sync is needed
int amr_info(Ctx &ctx, Case &c, double *h_out)
{
    const size_t nb = sizeof(double) * 4 * (size_t)(c.d.max_level + 1);
    double *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, nb, ctx.stream));
    int rc = amr_dispatch(c, [&](auto *tag) {
        using S = std::remove_pointer_t<decltype(tag)>;
        return AmrOps<S>::info(ctx, c, d);
    });
    if (!rc) MT_CUDA(ctx, cudaMemcpyAsync(h_out, d, nb, cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d, ctx.stream);
    return rc;
}

// populations of one level as FP64 [Q][n] (host buffers), in either direction
int amr_get(Ctx &ctx, Case &c, int level, double *h_f, double *h_fcol)
{
    if (int rc = amr_sync_f(ctx, c)) return rc;
    Level &lv = c.lv[level];
    if (!lv.n) return MT_OK;
    const size_t nb = sizeof(double) * (size_t)c.d.q * (size_t)lv.ncell;
    double *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, nb, ctx.stream));
    int rc = MT_OK;
    for (int which = 0; which < 2 && !rc; ++which) {
        double *dst = which == 0 ? h_f : h_fcol;
        if (!dst) continue;
        rc = amr_dispatch(c, [&](auto *tag) {
            using S = std::remove_pointer_t<decltype(tag)>;
            return AmrOps<S>::get(ctx, c, level, which, d);
        });
        if (!rc) rc = copy_out(ctx, dst, d, nb);
    }
    cudaFreeAsync(d, ctx.stream);
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    return rc;
}

int amr_set(Ctx &ctx, Case &c, int level, const double *h_f, const double *h_fcol)
{
    if (int rc = amr_sync_f(ctx, c)) return rc;
    c.prev_stale = true;
    Level &lv = c.lv[level];
    if (!lv.n) return MT_OK;
    const size_t nb = sizeof(double) * (size_t)c.d.q * (size_t)lv.ncell;
    double *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, nb, ctx.stream));
    int rc = MT_OK;
    for (int which = 0; which < 2 && !rc; ++which) {
        const double *src = which == 0 ? h_f : h_fcol;
        if (!src) continue;
        MT_CUDA(ctx, cudaMemcpyAsync(d, src, nb, cudaMemcpyHostToDevice, ctx.stream));
        rc = amr_dispatch(c, [&](auto *tag) {
            using S = std::remove_pointer_t<decltype(tag)>;
            return AmrOps<S>::set(ctx, c, level, which, d);
        });
    }
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d, ctx.stream);
    return rc;
}

int amr_macros(Ctx &ctx, Case &c, int level, double *h_rho, double *h_u)
{
    Level &lv = c.lv[level];
    if (!lv.n) return MT_OK;
    double *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, sizeof(double) * 4 * lv.ncell, ctx.stream));
    int rc = amr_dispatch(c, [&](auto *tag) {
        using S = std::remove_pointer_t<decltype(tag)>;
        return AmrOps<S>::macros_out(ctx, c, level, d, d + lv.ncell);
    });
    if (!rc && h_rho) rc = copy_out(ctx, h_rho, d, sizeof(double) * lv.ncell);
    if (!rc && h_u) rc = copy_out(ctx, h_u, d + lv.ncell, sizeof(double) * 3 * lv.ncell);
    cudaFreeAsync(d, ctx.stream);
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    return rc;
}

// rank (position in key order) of a slot
__device__ __forceinline__ int64_t rank_of(const LevelMap &map, const int32_t *bstart, int64_t i)
{
    const unsigned long long m = map.bmask[i >> 6];
    return bstart[i >> 6] + __popcll(m & ((1ull << (i & 63)) - 1ull));
}

__global__ void k_find(const LevelMap map, const int32_t *bstart, const uint64_t *q, int64_t nq, int64_t *out)
{
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= nq) return;
    const int64_t i = map.find(q[j]);
    out[j] = i < 0 ? -1 : rank_of(map, bstart, i);
}

// keys and tags of a level's cells in key order
__global__ void k_cells_out(const LevelMap map, const int32_t *slot, const uint32_t *tag, int64_t nc, uint64_t *key,
                            uint32_t *tg)
{
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nc) return;
    const int64_t i = slot[r];
    key[r] = map.key(i);
    tg[r] = tag[i];
}

// the neighbour table by ranks
__global__ void k_nbr_out(const LevelMap map, const int32_t *bstart, const int32_t *slot, int64_t nc, const int32_t *nbr,
                          int links, int32_t *out)
{
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nc) return;
    const int64_t i = slot[r], n = 64 * map.nb;
    for (int k = 0; k < links; ++k) {
        const int32_t j = nbr[k * n + i];
        out[k * nc + r] = j < 0 ? -1 : (int32_t)rank_of(map, bstart, j);
    }
}

// rows of 64-bit values between slots and key order
__global__ void k_rows_move(const int32_t *slot, int64_t nc, int64_t n, int rows, long long *by_slot, long long *by_rank,
                            int to_rank)
{
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nc) return;
    const int64_t i = slot[r];
    for (int a = 0; a < rows; ++a) {
        if (to_rank)
            by_rank[a * nc + r] = by_slot[a * n + i];
        else
            by_slot[a * n + i] = by_rank[a * nc + r];
    }
}

int amr_get_keys(Ctx &ctx, Case &c, int level, uint64_t *h_keys, uint32_t *h_tags)
{
    Level &lv = c.lv[level];
    const int64_t nc = lv.ncell;
    if (!nc) return MT_OK;
    uint64_t *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, 12 * nc, ctx.stream));
    uint32_t *t = (uint32_t *)(d + nc);
    k_cells_out<<<grid_for(nc, 256), 256, 0, ctx.stream>>>(lv.map(), lv.slot, lv.tag, nc, d, t);
    MT_LAUNCHED(ctx);
    if (h_keys) MT_CUDA(ctx, cudaMemcpyAsync(h_keys, d, 8 * nc, cudaMemcpyDeviceToHost, ctx.stream));
    if (h_tags) MT_CUDA(ctx, cudaMemcpyAsync(h_tags, t, 4 * nc, cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d, ctx.stream);
    return MT_OK;
}

int amr_get_neighbors(Ctx &ctx, Case &c, int level, int32_t *h_nbr)
{
    Level &lv = c.lv[level];
    const int64_t nc = lv.ncell;
    const int links = c.d.q - 1;
    if (!nc) return MT_OK;
    int32_t *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, 4 * nc * links, ctx.stream));
    k_nbr_out<<<grid_for(nc, 256), 256, 0, ctx.stream>>>(lv.map(), lv.bstart, lv.slot, nc, lv.nbr, links, d);
    MT_LAUNCHED(ctx);
    MT_CUDA(ctx, cudaMemcpyAsync(h_nbr, d, 4 * nc * links, cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d, ctx.stream);
    return MT_OK;
}

int amr_df_force_field(Ctx &ctx, Case &c, int64_t *h, bool get)
{
    Level &lv = c.lv[c.d.max_level];
    const int64_t nc = lv.ncell;
    if (!nc) return MT_OK;
    const size_t bytes = sizeof(long long) * 3 * (size_t)nc;
    long long *d = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&d, bytes, ctx.stream));
    if (!get) MT_CUDA(ctx, cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, ctx.stream));
    k_rows_move<<<grid_for(nc, 256), 256, 0, ctx.stream>>>(lv.slot, nc, lv.n, 3, c.acc, d, get ? 1 : 0);
    MT_LAUNCHED(ctx);
    if (get) MT_CUDA(ctx, cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(d, ctx.stream);
    return MT_OK;
}

int amr_find(Ctx &ctx, Case &c, int level, const uint64_t *h_keys, int64_t nq, int64_t *h_idx)
{
    if (nq == 0) return MT_OK;
    Level &lv = c.lv[level];
    uint64_t *dq = nullptr;
    int64_t *dout = nullptr;
    MT_CUDA(ctx, cudaMallocAsync(&dq, 8 * nq, ctx.stream));
    MT_CUDA(ctx, cudaMallocAsync(&dout, 8 * nq, ctx.stream));
    MT_CUDA(ctx, cudaMemcpyAsync(dq, h_keys, 8 * nq, cudaMemcpyHostToDevice, ctx.stream));
    k_find<<<grid_for(nq, 256), 256, 0, ctx.stream>>>(lv.map(), lv.bstart, dq, nq, dout);
    MT_LAUNCHED(ctx);
    MT_CUDA(ctx, cudaMemcpyAsync(h_idx, dout, 8 * nq, cudaMemcpyDeviceToHost, ctx.stream));
    MT_CUDA(ctx, cudaStreamSynchronize(ctx.stream));
    cudaFreeAsync(dq, ctx.stream);
    cudaFreeAsync(dout, ctx.stream);
    return MT_OK;
}

}  // namespace mt
