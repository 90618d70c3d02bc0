/*
 * conncomp.cu -- connected-component labelling of the unwrapped phase (A16).
 *
 * Semantics of cuphu_conncomp_gpu (cuphu_conncomp.cu:83-93, 96-114, 178-286,
 * 290-428): a pixel is valid when corr >= 0.05 and mask != 0; two 4-neighbours
 * are joined when both are valid, |unw_a - unw_b| < pi (float) and, when MCF
 * incremental costs are given, min(poscost, negcost) >= conncompthresh.
 * Components of at least max(1, (int)(minconncompfrac * npix)) pixels get
 * labels 1..maxncomps in increasing order of their smallest pixel index;
 * everything else is 0.
 *
 * B200 design: union-find with atomicMin linking (roots are always component
 * minima, so the canonical order comes for free) in two levels: each work item
 * labels its own pixels in shared memory, then only the pairs across item borders
 * are linked through global memory.  The label map is built on the device by a
 * per-row ballot scan (the reference downloads all npix counts, builds the map on
 * the host and uploads it again, cuphu_conncomp.cu:401-424).  Every kernel takes a
 * list of tiles so all tiles of all scenes label in one launch per step.
 */
#include "kernels.cuh"

namespace cuphu {

constexpr uint32_t kInvalid = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t uf_find(uint32_t *P, uint32_t x)
{
    while (true) {
        uint32_t p = __ldcg(P + x);
        if (p == x) return x;
        uint32_t gp = __ldcg(P + p);
        if (gp != p) P[x] = gp;   /* path halving: gp is an ancestor of x */
        x = gp;
    }
}

__device__ __forceinline__ void uf_unite(uint32_t *P, uint32_t a, uint32_t b)
{
    while (true) {
        a = uf_find(P, a);
        b = uf_find(P, b);
        if (a == b) return;
        if (a < b) { uint32_t t = a; a = b; b = t; }
        uint32_t old = atomicMin(P + a, b);
        if (old == a) return;
        a = old;
    }
}

/* may arc's incremental costs join its two pixels */
__device__ __forceinline__ bool arc_joins(const CcArgs &a, size_t arc)
{
    if (!a.poscost) return true;
    short mc = min(a.poscost[arc], a.negcost[arc]);
    return (long)mc >= a.conncompthresh;
}
__device__ __forceinline__ bool arc_joins_right(const CcArgs &a, const TileDesc &T, int r, int c)
{
    return arc_joins(a, (size_t)(T.nr - 1) * T.nc + (size_t)r * (T.nc - 1) + c);
}
__device__ __forceinline__ bool arc_joins_below(const CcArgs &a, const TileDesc &T, int r, int c)
{
    return arc_joins(a, (size_t)r * T.nc + c);
}

constexpr int kCcPix = kItemBy * kItemBx;
constexpr int kCcRows = kItemThreads / kItemBx;   /* rows of an item that one sweep covers */
static_assert(kItemBx == 64 && kItemBy % kCcRows == 0, "two warps a row, whole sweeps");

/* roots of the item's own union-find, in shared memory */
__device__ __forceinline__ uint32_t lab_find(const volatile uint32_t *lab, uint32_t x)
{
    while (true) {
        const uint32_t p = lab[x];
        if (p == x) return x;
        x = p;
    }
}
__device__ __forceinline__ void lab_unite(uint32_t *lab, uint32_t a, uint32_t b)
{
    while (true) {
        a = lab_find(lab, a);
        b = lab_find(lab, b);
        if (a == b) return;
        if (a < b) { uint32_t t = a; a = b; b = t; }
        const uint32_t old = atomicMin(lab + a, b);
        if (old == a) return;
        a = old;
    }
}

/* Components of each item by itself: par = the tile index of the component's smallest pixel in the
 * item, aux = its size there (0 elsewhere).  Runs along a row come out of a ballot, so unions are
 * left only between rows, one per stretch of touching runs, and they run at shared-memory latency.
 * Before, every pixel linked to its right and lower neighbour through the L2 (0.62 ms at
 * 2048 x 2048) and counted itself with an atomic on its root, which one large component serialised
 * (2.3 ms); labelling a 2048 x 2048 map took 3.2 ms on the device and takes 0.26. */
__global__ void __launch_bounds__(kItemThreads) k_cc_local(const TileDesc *__restrict__ tiles,
                                                           const int *__restrict__ item_tile,
                                                           int nitems, SolverPlanes P, CcArgs a)
{
    __shared__ uint32_t lab[kCcPix], cnt[kCcPix];
    __shared__ unsigned joined[kItemBy][2];   /* bit l: pixel l of the half row joins its left one */
    constexpr int kSweeps = kItemBy / kCcRows;
    const int x = threadIdx.x % kItemBx, y0 = threadIdx.x / kItemBx;
    const int lane = threadIdx.x & 31, half = x >> 5;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const TileDesc &T = tiles[item_tile[item]];
        const int iby = (item - T.item0) / T.nbx, ibx = (item - T.item0) % T.nbx;
        const int c = ibx * kItemBx + x;
        const float *u = P.unw + T.pix;
        float uv[kSweeps];
#pragma unroll
        for (int k = 0; k < kSweeps; ++k) {
            const int y = y0 + kCcRows * k, r = iby * kItemBy + y, id = y * kItemBx + x;
            const bool in = r < T.nr && c < T.nc;
            bool valid = false;
            uv[k] = 0.0f;
            if (in) {
                const size_t gi = (size_t)r * T.ph_pitch + c;
                valid = !(sane(T.corr[gi]) < a.corr_thresh);
                if (T.mask) valid = valid && T.mask[gi] != 0;
                uv[k] = u[(size_t)r * T.pitch + c];
            }
            const unsigned live = __ballot_sync(0xffffffffu, valid);
            const float ul = __shfl_up_sync(0xffffffffu, uv[k], 1);
            const bool jl = valid && lane > 0 && ((live >> (lane - 1)) & 1u) &&
                            fabsf(ul - uv[k]) < kPiF && arc_joins_right(a, T, r, c - 1);
            const unsigned m = __ballot_sync(0xffffffffu, jl);
            const int start = 31 - __clz(~m & ((2u << lane) - 1u));   /* the run's first lane */
            lab[id] = valid ? (uint32_t)(id - lane + start) : kInvalid;
            cnt[id] = 0u;
            if (lane == 0) joined[y][half] = m;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSweeps; ++k) {
            const int y = y0 + kCcRows * k, r = iby * kItemBy + y, id = y * kItemBx + x;
            const bool valid = lab[id] != kInvalid;
            bool down = false;
            if (valid && y + 1 < kItemBy && r + 1 < T.nr && lab[id + kItemBx] != kInvalid)
                down = fabsf(uv[k] - u[(size_t)(r + 1) * T.pitch + c]) < kPiF &&
                       arc_joins_below(a, T, r, c);
            const unsigned d = __ballot_sync(0xffffffffu, down);
            if (down) {
                /* the pair on the left joins the same two runs already */
                const bool dup = lane > 0 && ((d >> (lane - 1)) & (joined[y][half] >> lane) &
                                              (joined[y + 1][half] >> lane) & 1u);
                if (!dup) lab_unite(lab, id, id + kItemBx);
            }
            if (x == 32 && valid && lab[id - 1] != kInvalid &&
                fabsf(u[(size_t)r * T.pitch + c - 1] - uv[k]) < kPiF &&
                arc_joins_right(a, T, r, c - 1))
                lab_unite(lab, id - 1, id);
        }
        __syncthreads();
        uint32_t root[kSweeps];
#pragma unroll
        for (int k = 0; k < kSweeps; ++k) {
            const int y = y0 + kCcRows * k, id = y * kItemBx + x;
            root[k] = lab[id] == kInvalid ? kInvalid : lab_find(lab, id);
            const unsigned m = joined[y][half];
            if (root[k] != kInvalid && !((m >> lane) & 1u)) {   /* the run's first lane counts it */
                const unsigned rest = lane == 31 ? 0u : ~(m >> (lane + 1));
                atomicAdd(cnt + root[k], (uint32_t)(lane == 31 ? 1 : __ffs(rest)));
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSweeps; ++k) {
            const int y = y0 + kCcRows * k, r = iby * kItemBy + y, id = y * kItemBx + x;
            if (r >= T.nr || c >= T.nc) continue;
            const size_t li = T.pix + (size_t)r * T.pitch + c;
            P.cc[li] = root[k] == kInvalid
                           ? kInvalid
                           : (uint32_t)((size_t)(iby * kItemBy + root[k] / kItemBx) * T.pitch +
                                        ibx * kItemBx + root[k] % kItemBx);
            P.aux[li] = cnt[id];
        }
        __syncthreads();
    }
}

/* links across the items' right and lower borders: 64 + 16 pairs per
 * item, in three warp jobs.  A pair whose left (or
 * upper) neighbour pair lies in the same two components and is joined leaves the link to it; parents
 * read here may be newer than the item's own, and equal parents always mean one component. */
__global__ void __launch_bounds__(kItemThreads) k_cc_border(const TileDesc *__restrict__ tiles,
                                                            const int *__restrict__ item_tile,
                                                            int nitems, SolverPlanes P, CcArgs a)
{
    const int warp = (blockIdx.x * kItemThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int nwarps = gridDim.x * (kItemThreads >> 5);
    for (int job = warp; job < 3 * nitems; job += nwarps) {
        const int item = job / 3, part = job - 3 * item;
        const TileDesc &T = tiles[item_tile[item]];
        const int iby = (item - T.item0) / T.nbx, ibx = (item - T.item0) % T.nbx;
        const bool right = part == 2;
        const int r = right ? iby * kItemBy + lane : iby * kItemBy + kItemBy - 1;
        const int c = right ? ibx * kItemBx + kItemBx - 1 : ibx * kItemBx + 32 * part + lane;
        bool in = right ? lane < kItemBy && r < T.nr && c + 1 < T.nc : r + 1 < T.nr && c < T.nc;
        uint32_t *par = P.cc + T.pix;
        const float *u = P.unw + T.pix;
        const uint32_t i = (uint32_t)((size_t)r * T.pitch + c);
        const uint32_t o = right ? i + 1u : i + (uint32_t)T.pitch;
        uint32_t pi = kInvalid, po = kInvalid;
        if (in) { pi = __ldcg(par + i); po = __ldcg(par + o); }
        const bool join = pi != kInvalid && po != kInvalid && fabsf(u[i] - u[o]) < kPiF &&
                          (right ? arc_joins_right(a, T, r, c) : arc_joins_below(a, T, r, c));
        const unsigned j = __ballot_sync(0xffffffffu, join);
        const uint32_t li = __shfl_up_sync(0xffffffffu, pi, 1);
        const uint32_t lo = __shfl_up_sync(0xffffffffu, po, 1);
        const bool dup = lane > 0 && ((j >> (lane - 1)) & 1u) && li == pi && lo == po;
        if (join && !dup) uf_unite(par, pi, po);
    }
}

/* the root of every valid pixel, and each item's share of a component onto the root's size.  No
 * link is made any more and a pixel's parent is written by its own thread only, so whatever a find
 * reads is an ancestor; sizes of item roots that are not component roots stay as they were. */
__global__ void __launch_bounds__(kItemThreads) k_cc_flatten(const TileDesc *__restrict__ tiles,
                                                             const int *__restrict__ item_tile,
                                                             int nitems, SolverPlanes P)
{
    const int x = threadIdx.x % kItemBx, y0 = threadIdx.x / kItemBx;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const TileDesc &T = tiles[item_tile[item]];
        const int iby = (item - T.item0) / T.nbx, ibx = (item - T.item0) % T.nbx;
        const int c = ibx * kItemBx + x;
        if (c >= T.nc) continue;
        uint32_t *par = P.cc + T.pix, *size = P.aux + T.pix;
#pragma unroll
        for (int k = 0; k < kItemBy / kCcRows; ++k) {
            const int r = iby * kItemBy + y0 + kCcRows * k;
            if (r >= T.nr) break;
            const uint32_t i = (uint32_t)((size_t)r * T.pitch + c);
            const uint32_t p = __ldcg(par + i);
            if (p == kInvalid || p == i) continue;
            uint32_t root = p, q;
            while ((q = __ldcg(par + root)) != root) root = q;
            if (root != p) par[i] = root;
            const uint32_t n = size[i];
            if (n) atomicAdd(size + root, n);
        }
    }
}

__device__ __forceinline__ int tile_min_size(const TileDesc &T, double minfrac)
{
    int m = (int)(minfrac * (double)((long long)T.nr * T.nc));
    return m < 1 ? 1 : m;
}

/* one warp per tile row: number of labelled roots in the row */
__global__ void k_cc_rowcount(const TileDesc *__restrict__ tiles, const int *__restrict__ row_tile,
                              int total_rows, SolverPlanes P, CcArgs a, int *rowcnt)
{
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= total_rows) return;
    const TileDesc &T = tiles[row_tile[warp]];
    int r = warp - T.row0;
    int ms = tile_min_size(T, a.minfrac);
    const uint32_t *par = P.cc + T.pix;
    const uint32_t *cnt = P.aux + T.pix;
    int n = 0;
    for (int c0 = 0; c0 < T.nc; c0 += 32) {
        int c = c0 + lane;
        bool qv = false;
        if (c < T.nc) {
            uint32_t i = (uint32_t)((size_t)r * T.pitch + c);
            qv = __ldcg(par + i) == i && __ldcg(cnt + i) >= (uint32_t)ms;
        }
        n += __popc(__ballot_sync(0xffffffffu, qv));
    }
    if (lane == 0) rowcnt[warp] = n;
}

/* one block per tile: exclusive scan of its row counts; labels in the tile */
__global__ void __launch_bounds__(1024) k_cc_rowscan(const TileDesc *__restrict__ tiles,
                                                     int ntiles, int *rowcnt, CcArgs a,
                                                     int *ntile_labels)
{
    __shared__ int swarp[32];
    __shared__ int s_carry;
    int t = blockIdx.x;
    if (t >= ntiles) return;
    const TileDesc &T = tiles[t];
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int base = 0; base < T.nr; base += blockDim.x) {
        int i = base + threadIdx.x;
        int v = i < T.nr ? rowcnt[T.row0 + i] : 0;
        int x = v;
        for (int off = 1; off < 32; off <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) swarp[w] = x;
        __syncthreads();
        if (w == 0) {
            int s = lane < (int)(blockDim.x >> 5) ? swarp[lane] : 0;
            for (int off = 1; off < 32; off <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, s, off);
                if (lane >= off) s += y;
            }
            swarp[lane] = s;
        }
        __syncthreads();
        int incl = x + (w > 0 ? swarp[w - 1] : 0);
        int carry = s_carry;
        if (i < T.nr) rowcnt[T.row0 + i] = carry + incl - v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) s_carry = carry + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) ntile_labels[t] = min(s_carry, a.maxncomps);
}

/* one warp per tile row: labels of the row's roots (rank < maxncomps) */
__global__ void k_cc_rowlabel(const TileDesc *__restrict__ tiles, const int *__restrict__ row_tile,
                              int total_rows, SolverPlanes P, CcArgs a, const int *rowoff)
{
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= total_rows) return;
    const TileDesc &T = tiles[row_tile[warp]];
    int r = warp - T.row0;
    int ms = tile_min_size(T, a.minfrac);
    const uint32_t *par = P.cc + T.pix;
    uint32_t *aux = P.aux + T.pix;
    int run = rowoff[warp];
    for (int c0 = 0; c0 < T.nc; c0 += 32) {
        int c = c0 + lane;
        bool root = false, qv = false;
        uint32_t i = 0;
        if (c < T.nc) {
            i = (uint32_t)((size_t)r * T.pitch + c);
            root = __ldcg(par + i) == i;
            qv = root && __ldcg(aux + i) >= (uint32_t)ms;
        }
        unsigned b = __ballot_sync(0xffffffffu, qv);
        if (root) {
            int rank = run + __popc(b & ((1u << lane) - 1u));
            aux[i] = (qv && rank < a.maxncomps) ? (uint32_t)(rank + 1) : 0u;
        }
        run += __popc(b);
    }
}

__global__ void __launch_bounds__(kItemThreads) k_cc_final(const TileDesc *__restrict__ tiles,
                                                           const int *__restrict__ item_tile,
                                                           int nitems, SolverPlanes P)
{
    const int x = threadIdx.x % kItemBx, y0 = threadIdx.x / kItemBx;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const TileDesc &T = tiles[item_tile[item]];
        const int iby = (item - T.item0) / T.nbx, ibx = (item - T.item0) % T.nbx;
        const int c = ibx * kItemBx + x;
        if (c >= T.nc) continue;
        uint32_t *par = P.cc + T.pix;
        const uint32_t *aux = P.aux + T.pix;
#pragma unroll
        for (int k = 0; k < kItemBy / kCcRows; ++k) {
            const int r = iby * kItemBy + y0 + kCcRows * k;
            if (r >= T.nr) break;
            const uint32_t i = (uint32_t)((size_t)r * T.pitch + c);
            const uint32_t p = par[i];
            par[i] = p == kInvalid ? 0u : __ldcg(aux + p);
        }
    }
}

int launch_conncomp(const TileDesc *tiles, int ntiles, int total_rows, const int *item_tile,
                    int nitems, const SolverPlanes &P, const CcArgs &a, int *rowcnt,
                    int *ntile_labels, cudaStream_t s)
{
    /* rowcnt: [total_rows] scratch followed by [total_rows] row->tile map */
    const int *row_tile = rowcnt + total_rows;
    int g = std::min(nitems, 148 * 16);
    int gw = (total_rows * 32 + 255) / 256;
    k_cc_local<<<g, kItemThreads, 0, s>>>(tiles, item_tile, nitems, P, a);
    k_cc_border<<<(3 * std::min(nitems, 148 * 16) + 7) / 8, kItemThreads, 0, s>>>(
        tiles, item_tile, nitems, P, a);
    k_cc_flatten<<<g, kItemThreads, 0, s>>>(tiles, item_tile, nitems, P);
    k_cc_rowcount<<<gw, 256, 0, s>>>(tiles, row_tile, total_rows, P, a, rowcnt);
    k_cc_rowscan<<<ntiles, 1024, 0, s>>>(tiles, ntiles, rowcnt, a, ntile_labels);
    k_cc_rowlabel<<<gw, 256, 0, s>>>(tiles, row_tile, total_rows, P, a, rowcnt);
    k_cc_final<<<g, kItemThreads, 0, s>>>(tiles, item_tile, nitems, P);
    return cuda_fail(cudaGetLastError(), "conncomp kernels");
}

}  // namespace cuphu
