/*
 * stitch.cu -- tile registration and merge (A19), all on the device.
 *
 * Reference (cuphu_solver.cpp:1846-2031): for every adjacent tile pair the
 * coherence-weighted median of (unw_A - unw_B) over the shared overlap
 * (pixels with corr >= 0.05 in both and valid in the confidence mask),
 * divided by 2*pi (left fractional for Laplace); a BFS from tile (0,0),
 * right neighbour before bottom neighbour, accumulates tile offsets; the
 * merge writes each tile's interior (overlap halves trimmed, later tiles
 * win on odd overlaps) plus its offset, and shifts conncomp labels by the
 * running maximum label of the preceding tiles.  The Python reference-pixel
 * shift (_unwrap.py:605-617) is applied in the same merge pass.
 *
 * B200 design: a cluster of eight CTAs per tile pair finds the weighted median
 * by a 3-pass radix select (11, 11 and 10 bits) over the order-preserving
 * 32-bit key of the float differences, with weights accumulated as exact 2^-28
 * fixed point (every coherence weight >= 0.05 is an exact multiple of 2^-28, so
 * the sums equal the reference's double accumulation exactly); no sort, no host
 * copy, no workspace: the histograms are added up over the cluster's shared memory.
 */
#include "kernels.cuh"

#include <cooperative_groups.h>

namespace cuphu {

__device__ __forceinline__ uint32_t fkey(float v)
{
    uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float fkey_inv(uint32_t k)
{
    uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(u);
}

constexpr int kMedCtas = 8;       /* CTAs per pair, one portable cluster */
constexpr int kMedThreads = 512;
constexpr int kMedBins = 2048;
constexpr int kMedVec = 4;        /* samples per thread and step, 32 columns apart */
constexpr int kMedSlice = kMedBins / kMedCtas;

/* the pair's overlap: sample (i, j) is A's pixel (ar0 + i, ac0 + j) and B's (i, j) */
struct PairOverlap {
    const float *ca, *cb, *ua, *ub;
    const unsigned char *fa, *fb;   /* confidence masks, or null */
    size_t pa, pb, qa, qb;          /* row pitches: inputs, unwrapped planes */
    int n1, n2;
};

/* hist[bin] += w modulo 2^64 from two native 32-bit shared atomics: the carry is read off the
 * value that the first one returns (a 64-bit shared atomic is a compare-and-swap loop, which the
 * narrow distribution of the differences makes long) */
__device__ __forceinline__ void hist_add(uint32_t *lo, uint32_t *hi, uint32_t bin,
                                         unsigned long long w)
{
    const uint32_t wl = (uint32_t)w, old = atomicAdd(lo + bin, wl);
    const uint32_t wh = (uint32_t)(w >> 32) + (old + wl < old ? 1u : 0u);
    if (wh) atomicAdd(hi + bin, wh);
}

/* one sample of every lane (all 32 are here).  The lanes that share the first counting lane's bin
 * are added up in registers first: in the upper digits that is nearly the whole warp. */
__device__ __forceinline__ void warp_hist(uint32_t *lo, uint32_t *hi, bool ok, uint32_t bin,
                                          unsigned long long w)
{
    const unsigned live = __ballot_sync(0xffffffffu, ok);
    if (live == 0u) return;
    const int first = __ffs(live) - 1;
    const uint32_t lead = __shfl_sync(0xffffffffu, bin, first);
    const bool same = ok && bin == lead;
    const unsigned long long ws = same ? w : 0ull;
    /* 24 + 24 + 16 bits: 32 lanes cannot overflow 32 bits, and the total is exact modulo 2^64 */
    const uint32_t s0 = __reduce_add_sync(0xffffffffu, (uint32_t)(ws & 0xFFFFFFull));
    const uint32_t s1 = __reduce_add_sync(0xffffffffu, (uint32_t)(ws >> 24) & 0xFFFFFFu);
    const uint32_t s2 = __reduce_add_sync(0xffffffffu, (uint32_t)(ws >> 48));
    if ((int)(threadIdx.x & 31u) == first)
        hist_add(lo, hi, bin, (unsigned long long)s0 + ((unsigned long long)s1 << 24) +
                                  ((unsigned long long)s2 << 48));
    else if (ok && !same)
        hist_add(lo, hi, bin, w);
}

/* the differences whose key agrees with `prefix` under `mask`, into the CTA's histogram */
__device__ __forceinline__ void pair_pass(const PairOverlap &o, uint32_t *lo, uint32_t *hi,
                                          uint32_t prefix, uint32_t mask, int shift, uint32_t digit,
                                          unsigned rank)
{
    const int lane = threadIdx.x & 31;
    const unsigned nwarps = kMedCtas * kMedThreads / 32;
    const unsigned nb = ((unsigned)o.n2 + 32u * kMedVec - 1u) / (32u * kMedVec);
    const unsigned units = nb * (unsigned)o.n1;
    for (unsigned u = rank * (kMedThreads / 32) + (threadIdx.x >> 5); u < units; u += nwarps) {
        const int i = (int)(u / nb), j0 = (int)(u % nb) * 32 * kMedVec + lane;
        float ca[kMedVec], cb[kMedVec], ua[kMedVec], ub[kMedVec];
        bool ok[kMedVec];
#pragma unroll
        for (int v = 0; v < kMedVec; ++v) {
            const int j = j0 + 32 * v;
            ca[v] = cb[v] = ua[v] = ub[v] = 0.0f;
            ok[v] = j < o.n2;
            if (!ok[v]) continue;
            ca[v] = o.ca[(size_t)i * o.pa + j];
            cb[v] = o.cb[(size_t)i * o.pb + j];
            ua[v] = o.ua[(size_t)i * o.qa + j];
            ub[v] = o.ub[(size_t)i * o.qb + j];
            if (o.fa) ok[v] = o.fa[(size_t)i * o.pa + j] != 0;
            if (o.fb) ok[v] = ok[v] && o.fb[(size_t)i * o.pb + j] != 0;
        }
#pragma unroll
        for (int v = 0; v < kMedVec; ++v) {
            const float a = sane(ca[v]), b = sane(cb[v]);
            const uint32_t key = fkey(ua[v] - ub[v]);
            const bool in = ok[v] && !(a < 0.05f || b < 0.05f) && (key & mask) == prefix;
            const float w = a < b ? a : b;
            /* a power of two: the product is exact, as in 64 bits */
            warp_hist(lo, hi, in, (key >> shift) & digit,
                      in ? (unsigned long long)(w * 268435456.0f) : 0ull);
        }
    }
}

/* Latency-bound at one CTA per pair: 16.25 ms for the one pair of a 2051 x 1537 scene, five passes
 * of 256 threads with one load chain each and a 64-bit compare-and-swap histogram that the narrow
 * distribution serialised.  Sixteen times the threads, four samples in flight each, three passes
 * (the total is the first histogram's sum) and register sums for the crowded bin: 0.050 ms. */
__global__ void __cluster_dims__(kMedCtas, 1, 1) __launch_bounds__(kMedThreads)
    k_pair_median(const PairDesc *__restrict__ pairs, const TileDesc *__restrict__ tiles,
                  SolverPlanes P, double *pair_k)
{
    namespace cg = cooperative_groups;
    __shared__ uint32_t s_lo[kMedBins], s_hi[kMedBins];
    __shared__ unsigned long long s_tot[kMedBins];     /* the pair's histogram, in every CTA */
    __shared__ unsigned long long s_warp[kMedThreads / 32];
    __shared__ unsigned long long s_below;
    __shared__ int s_sel;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const unsigned pair = blockIdx.x / kMedCtas;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const PairDesc pd = pairs[pair];
    const TileDesc &A = tiles[pd.a];
    const TileDesc &B = tiles[pd.b];
    bool valid = pd.ov > 0 && (pd.dir == 0 ? (pd.ov <= A.nc && pd.ov <= B.nc)
                                          : (pd.ov <= A.nr && pd.ov <= B.nr));
    if (!valid) {   /* the same in all CTAs of the cluster */
        if (rank == 0 && t == 0) pair_k[pair] = 0.0;
        return;
    }
    PairOverlap o;
    o.n1 = pd.dir == 0 ? min(A.nr, B.nr) : pd.ov;
    o.n2 = pd.dir == 0 ? pd.ov : min(A.nc, B.nc);
    const size_t ar0 = pd.dir == 0 ? 0 : A.nr - pd.ov, ac0 = pd.dir == 0 ? A.nc - pd.ov : 0;
    o.pa = A.ph_pitch; o.pb = B.ph_pitch; o.qa = A.pitch; o.qb = B.pitch;
    o.ca = A.corr + ar0 * o.pa + ac0; o.cb = B.corr;
    o.fa = A.conf ? A.conf + ar0 * o.pa + ac0 : nullptr; o.fb = B.conf;
    o.ua = P.unw + A.pix + ar0 * o.qa + ac0; o.ub = P.unw + B.pix;

    unsigned long long total = 0ull, below = 0ull;
    uint32_t prefix = 0u, mask = 0u;
    for (int pass = 0; pass < 3; ++pass) {
        const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
        const uint32_t digit = pass == 2 ? 1023u : 2047u;
        for (int b = t; b < kMedBins; b += kMedThreads) { s_lo[b] = 0u; s_hi[b] = 0u; }
        __syncthreads();
        pair_pass(o, s_lo, s_hi, prefix, mask, shift, digit, rank);
        cluster.sync();
        /* each CTA adds up its slice of the bins over the cluster and hands it to all */
        if (t < kMedSlice) {
            const int b = (int)rank * kMedSlice + t;
            unsigned long long sum = 0ull;
            for (int c = 0; c < kMedCtas; ++c)
                sum += cluster.map_shared_rank(s_lo, c)[b] +
                       ((unsigned long long)cluster.map_shared_rank(s_hi, c)[b] << 32);
            for (int c = 0; c < kMedCtas; ++c) cluster.map_shared_rank(s_tot, c)[b] = sum;
        }
        cluster.sync();   /* also the last access to another CTA's histogram in this pass */

        /* exclusive prefix of the thread's bins over the CTA */
        constexpr int kPer = kMedBins / kMedThreads;
        unsigned long long mine = 0ull;
        for (int k = 0; k < kPer; ++k) mine += s_tot[t * kPer + k];
        unsigned long long incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        if (lane == 31) s_warp[wp] = incl;
        if (t == 0) s_sel = (int)digit;   /* stays only if the weights overflow 63 bits */
        __syncthreads();
        unsigned long long before = below, all = 0ull;
        for (int k = 0; k < kMedThreads / 32; ++k) {
            if (k < wp) before += s_warp[k];
            all += s_warp[k];
        }
        before += incl - mine;
        if (pass == 0) {
            total = all;
            if (total == 0ull) {   /* the same in all CTAs */
                if (rank == 0 && t == 0) pair_k[pair] = 0.0;
                return;
            }
        }
        /* the first bin at which twice the weight up to it reaches the total */
        unsigned long long run = before;
        int sel = -1;
        for (int k = 0; k < kPer; ++k) {
            const unsigned long long next = run + s_tot[t * kPer + k];
            if (2ull * next >= total) { sel = t * kPer + k; break; }
            run = next;
        }
        if (sel >= 0) atomicMin(&s_sel, sel);
        if (t == 0) s_below = below + all;
        __syncthreads();
        if (sel >= 0 && s_sel == sel) s_below = run;
        __syncthreads();
        below = s_below;
        prefix |= (uint32_t)s_sel << shift;
        mask |= digit << shift;
    }
    if (rank == 0 && t == 0) pair_k[pair] = (double)fkey_inv(prefix) / kTwoPiD;
}

/* one thread per scene: BFS tile offsets, label offsets, reference shift */
__global__ void k_stitch_finalize(const ScenePlan *__restrict__ scenes, int nscenes,
                                  const TileDesc *__restrict__ tiles, SolverPlanes P,
                                  const int *__restrict__ ntile_labels,
                                  const double *__restrict__ pair_k, double *tile_k,
                                  unsigned *comp_off, SceneOut *sout, int *queue)
{
    int sidx = blockIdx.x * blockDim.x + threadIdx.x;
    if (sidx >= nscenes) return;
    const ScenePlan &S = scenes[sidx];
    int nt = S.ntr * S.ntc;
    double *tk = tile_k + S.tile0;
    for (int i = 0; i < nt; ++i) tk[i] = 0.0;
    if (nt > 1 && (S.rovl > 0 || S.covl > 0)) {
        int *q = queue + S.tile0;          /* BFS queue of local tile indices */
        int qh = 0, qt = 0;
        unsigned *seen = comp_off + S.tile0; /* visited marks; comp_off is filled below */
        for (int i = 0; i < nt; ++i) seen[i] = 0u;
        q[qt++] = 0;
        seen[0] = 1u;
        const int nh = S.ntr * (S.ntc - 1);
        while (qh < qt) {
            int idx = q[qh++];
            int br = idx / S.ntc, bc = idx % S.ntc;
            if (bc + 1 < S.ntc) {
                int nb = br * S.ntc + bc + 1;
                if (!seen[nb]) {
                    tk[nb] = tk[idx] + pair_k[S.pair0 + br * (S.ntc - 1) + bc];
                    seen[nb] = 1u;
                    q[qt++] = nb;
                }
            }
            if (br + 1 < S.ntr) {
                int nb = (br + 1) * S.ntc + bc;
                if (!seen[nb]) {
                    tk[nb] = tk[idx] + pair_k[S.pair0 + nh + br * S.ntc + bc];
                    seen[nb] = 1u;
                    q[qt++] = nb;
                }
            }
        }
    }
    unsigned run = 0u;
    for (int i = 0; i < nt; ++i) {
        comp_off[S.tile0 + i] = run;
        run += (unsigned)ntile_labels[S.tile0 + i];
    }
    SceneOut o;
    o.shift = 0.0f;
    o.do_shift = 0;
    if (S.ref_row >= 0 && S.ref_col >= 0 && S.ref_row < S.nrow && S.ref_col < S.ncol) {
        int tr = S.rowmap[S.ref_row], tc = S.colmap[S.ref_col];
        int t = S.tile0 + tr * S.ntc + tc;
        const TileDesc &T = tiles[t];
        float u = P.unw[T.pix + (size_t)(S.ref_row - T.r0) * T.pitch + (S.ref_col - T.c0)];
        if (!S.single) u = u + (float)(tk[tr * S.ntc + tc] * kTwoPiD);
        double ref = (double)S.ph[(size_t)S.ref_row * S.ncol + S.ref_col];
        double n = rint(((double)u - ref) / kTwoPiD);
        if (n != 0.0) {
            o.shift = (float)(n * kTwoPiD);
            o.do_shift = 1;
        }
    }
    sout[sidx] = o;
}

__global__ void __launch_bounds__(256) k_merge(const ScenePlan *__restrict__ scenes, int sidx,
                                               const TileDesc *__restrict__ tiles,
                                               SolverPlanes P, const double *__restrict__ tile_k,
                                               const unsigned *__restrict__ comp_off,
                                               const SceneOut *__restrict__ sout)
{
    const ScenePlan &S = scenes[sidx];
    const SceneOut o = sout[sidx];
    long long n = (long long)S.nrow * S.ncol;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        int R = (int)(i / S.ncol), Cc = (int)(i % S.ncol);
        int tr = S.rowmap[R], tc = S.colmap[Cc];
        int t = S.tile0 + tr * S.ntc + tc;
        const TileDesc &T = tiles[t];
        size_t pi = T.pix + (size_t)(R - T.r0) * T.pitch + (Cc - T.c0);
        float u = P.unw[pi];
        if (!S.single) u = u + (float)(tile_k[t] * kTwoPiD);
        if (o.do_shift) u = u - o.shift;
        S.unw_out[i] = u;
        if (S.cc_out) {
            uint32_t c = P.cc[pi];
            S.cc_out[i] = c == 0u ? 0u : c + comp_off[t];
        }
    }
}

/* the reference-pixel shift of a merged scene whose post-passes ran after
 * the merge: n = rint((unw[ref] - phi[ref]) / 2pi), then unw -= float(n 2pi)
 * (the merge kernel's rule, on the post-processed value) */
__global__ void k_ref_shift_n(const float *unw, const float *ph, int ncol, int ref_row,
                              int ref_col, SceneOut *o)
{
    size_t i = (size_t)ref_row * ncol + ref_col;
    double n = rint(((double)unw[i] - (double)ph[i]) / kTwoPiD);
    o->shift = (float)(n * kTwoPiD);
    o->do_shift = n != 0.0 ? 1 : 0;
}

__global__ void __launch_bounds__(256) k_ref_shift_apply(float *unw, long long n,
                                                         const SceneOut *o)
{
    if (!o->do_shift) return;
    const float sh = o->shift;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        unw[i] = unw[i] - sh;
}

int launch_ref_shift(float *unw, const float *ph, int nrow, int ncol, int ref_row, int ref_col,
                     SceneOut *tmp, cudaStream_t s)
{
    if (ref_row < 0 || ref_col < 0 || ref_row >= nrow || ref_col >= ncol) return 0;
    k_ref_shift_n<<<1, 1, 0, s>>>(unw, ph, ncol, ref_row, ref_col, tmp);
    long long n = (long long)nrow * ncol;
    int blocks = (int)std::min<long long>((n + 255) / 256, 148LL * 16);
    k_ref_shift_apply<<<blocks, 256, 0, s>>>(unw, n, tmp);
    return cuda_fail(cudaGetLastError(), "reference-pixel shift");
}

int launch_stitch(const ScenePlan *scenes, int nscenes, const TileDesc *tiles,
                  const PairDesc *pairs, int npairs, const SolverPlanes &P,
                  const int *ntile_labels, double *pair_k, double *tile_k,
                  unsigned *comp_off, SceneOut *sout, cudaStream_t s)
{
    if (npairs > 0)
        k_pair_median<<<npairs * kMedCtas, kMedThreads, 0, s>>>(pairs, tiles, P, pair_k);
    /* the BFS queue reuses pair_k's tail: [npairs] medians, then [ntiles] queue */
    int *queue = reinterpret_cast<int *>(pair_k + npairs);
    k_stitch_finalize<<<(nscenes + 63) / 64, 64, 0, s>>>(scenes, nscenes, tiles, P, ntile_labels,
                                                        pair_k, tile_k, comp_off, sout, queue);
    return cuda_fail(cudaGetLastError(), "stitch kernels");
}

int launch_merge(const ScenePlan *scenes, const ScenePlan *h_scenes, int nscenes,
                 const TileDesc *tiles, const SolverPlanes &P, const double *tile_k,
                 const unsigned *comp_off, const SceneOut *sout, cudaStream_t s)
{
    for (int i = 0; i < nscenes; ++i) {
        long long n = (long long)h_scenes[i].nrow * h_scenes[i].ncol;
        int blocks = (int)std::min<long long>((n + 255) / 256, 148LL * 16);
        k_merge<<<blocks, 256, 0, s>>>(scenes, i, tiles, P, tile_k, comp_off, sout);
    }
    return cuda_fail(cudaGetLastError(), "k_merge");
}

}  // namespace cuphu
