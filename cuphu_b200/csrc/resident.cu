/*
 * resident.cu -- the mixed-precision Laplace solve of tiles whose PCG state
 * fits on the chip.
 *
 * k_solve (laplace.cu) streams every plane of the state through each block
 * once per PCG iteration.  A tile of the usual size (about 1000 x 1000
 * pixels, 24 MB of state) fits into the shared and tensor memory of the
 * chip, so this kernel loads a tile once per IRLS pass and keeps it there:
 * between two iterations only the rims of the work items and one partial sum
 * per block cross the L2.
 *
 *  - A tile is run by a group of blocks, one block per SM.  Each block holds
 *    up to kResItems work items (16 rows x 64 columns): p with its halo ring
 *    and the two arc-weight planes in shared memory; dx, r, M^-1 and q in
 *    tensor memory (TMEM, used as a 256 KB register file: every thread keeps
 *    the 16 words of its four pixels of an item in 16 columns of its lane).
 *  - An iteration is k_solve's single-synchronisation mixed pass with the
 *    same operations per pixel and the same reduction tree, so every result
 *    is bit-identical to k_solve's.
 *  - The tree sums items j, j + 256, ... per slot j, then the 256 slots by a
 *    butterfly over the slot's lane bits (16, 8, 4, 2, 1) and its warp bits
 *    (4, 2, 1).  A group of 2^g blocks assigns the slots so that the first
 *    8 - g levels of that butterfly stay inside a block: a block publishes
 *    one partial per dot product, and every block finishes the tree for
 *    itself.
 *  - Partials and rims travel as 16-byte packets that carry the number of
 *    their exchange (one 128-bit store each, so data and number arrive
 *    together).  A reader polls the packets it needs; there is no barrier
 *    and no memory fence inside an iteration.  Packets alternate between two
 *    buffers; a block overwrites one only after it has seen the partials of
 *    the exchange in between, which every reader of the old packet publishes
 *    after reading it.
 *  - Every wait is bounded: when it runs out the error status is set, which
 *    ends all other waits, and the kernel returns.
 *
 * What bounds it, and why this split, stands at k_resident.
 */
#include "resident.cuh"

namespace cuphu {
namespace {
constexpr int kResItems = kResItemsMixed;
constexpr int kResCols = 16;   /* dx, r, M^-1 and q of four pixels */
}  // namespace
}  // namespace cuphu
#include "resident_dev.cuh"

namespace cuphu {
namespace {

constexpr int kRimF = 2 * kRim;                         /* r and M^-1 of the halo ring */
constexpr int kResItemF = kPnN + kWdN + kWrN + kRimF;   /* floats of an item */

constexpr size_t kResSmem = (size_t)kResItems * kResItemF * 4 + kResSharedB;
static_assert(kResSmem <= 232448, "shared memory of a block");

__device__ __forceinline__ float *pn_of(int i)
{
    return reinterpret_cast<float *>(res_items()) + i * kResItemF;
}
__device__ __forceinline__ float *wd_of(int i) { return pn_of(i) + kPnN; }
__device__ __forceinline__ float *wr_of(int i) { return pn_of(i) + kPnN + kWdN; }
__device__ __forceinline__ float2 *rim_state(int i)
{
    return reinterpret_cast<float2 *>(pn_of(i) + kPnN + kWdN + kWrN);
}
__device__ __forceinline__ uint32_t tm_of(const ResCtx &C, int i)
{
    return C.tm + (uint32_t)(i / kResEngines) * kResCols;
}

/* rim packets: q of a pixel and the exchange number, 8 bytes each (the two
 * of a vector store need not arrive together) */
__device__ __forceinline__ unsigned long long rim_packet(float q, unsigned seq)
{
    return (unsigned long long)__float_as_uint(q) | ((unsigned long long)seq << 32);
}
__device__ __forceinline__ void rim_store2(unsigned long long *p, float a, float b, unsigned seq)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(rim_packet(a, seq)),
                 "l"(rim_packet(b, seq))
                 : "memory");
}
__device__ __forceinline__ void rim_store(unsigned long long *p, float q, unsigned seq)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(rim_packet(q, seq)) : "memory");
}
__device__ __forceinline__ unsigned long long rim_load(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void rim_void(int k)
{
    rim_store(res_shared().K.A.rim + blockIdx.x * kResItems * 2 * kRim + k, 0.f, 0u);
}

/* columns of an item: dx 0..3, r 4..7, M^-1 8..11, q 12..15 */
constexpr int kTmDx = 0, kTmR = 4, kTmQ = 12;

/* Load an item after an assembly or a residual replacement: dx = 0, q = 0,
 * r from the residual plane; with `pass_start` also the weights, M^-1 and
 * p = 0.  Weights beyond the tile's last arcs and pixels beyond its columns
 * read as zero, so the iterations need no edge tests. */
__device__ __forceinline__ void load_item(const ResCtx &C, int i, bool pass_start)
{
    const TileDesc &T = res_shared().T;
    const int li = res_shared().li[i];
    const int r0b = (li / T.nbx) * kItemBy, c0b = (li % T.nbx) * kItemBx;
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    const int r = r0b + ty, c0 = c0b + tx * kItemVx;
    const bool own = r < T.nr && c0 < T.nc;
    float *Pn = pn_of(i), *WD = wd_of(i), *WR = wr_of(i);
    float rv[4] = {0.f, 0.f, 0.f, 0.f};
    if (own) {
        ld4((const float *)res_shared().K.P.z + T.pix + (size_t)r * T.pitch + c0, rv);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (c0 + j >= T.nc) rv[j] = 0.f;
    }
    __syncwarp();
    const float zr[8] = {0.f, 0.f, 0.f, 0.f, rv[0], rv[1], rv[2], rv[3]};
    tm_st8(tm_of(C, i), zr);
    float m[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   /* M^-1, q = 0 */
    if (pass_start) {
        for (int k = C.tid; k < kPnN; k += kItemThreads) Pn[k] = 0.f;
        /* the item's own arcs, the down arcs of the row above and the right
         * arcs of the column left of it */
        float wdn[4] = {0.f, 0.f, 0.f, 0.f}, wrt[4] = {0.f, 0.f, 0.f, 0.f};
        if (own) {
            const size_t o = T.pix + (size_t)r * T.pitch + c0;
            if (r < T.nr - 1) ld4(res_shared().K.P.wd + o, wdn);
            ld4(res_shared().K.P.wr + o, wrt);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (c0 + j >= T.nc) wdn[j] = 0.f;
                if (c0 + j >= T.nc - 1) wrt[j] = 0.f;
            }
        }
        st4(WD + (ty + 1) * kItemBx + tx * kItemVx, wdn);
        st4(WR + ty * kWrW2 + 4 + tx * kItemVx, wrt);
        float up[4] = {0.f, 0.f, 0.f, 0.f};
        if (own && r > 0) {
            ld4(res_shared().K.P.wd + T.pix + (size_t)(r - 1) * T.pitch + c0, up);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (c0 + j >= T.nc) up[j] = 0.f;
        }
        if (ty == 0) st4(WD + tx * kItemVx, up);
        float lf = 0.f;
        if (own && c0 > 0) lf = ldc(res_shared().K.P.wr + T.pix + (size_t)r * T.pitch + c0 - 1);
        if (tx == 0) WR[ty * kWrW2 + 3] = lf;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (own && c0 + j < T.nc)
                m[j] = rcp_pre(diag32(r, c0 + j, T.nr, T.nc, wdn[j], up[j], wrt[j],
                                      j == 0 ? lf : wrt[j - 1]));
        __syncwarp();
        tm_st8(tm_of(C, i) + 8, m);
    } else {
        tm_st4(tm_of(C, i) + kTmQ, m + 4);
    }
}

/* r and M^-1 of a rim pixel right after an assembly or replacement, from the
 * planes (zero outside the tile) */
__device__ __forceinline__ float2 fresh_rim(const ResCtx &C, int gr, int gc)
{
    const TileDesc &T = res_shared().T;
    if (gr < 0 || gr >= T.nr || gc < 0 || gc >= T.nc) return make_float2(0.f, 0.f);
    const size_t o = T.pix + (size_t)gr * T.pitch + gc;
    const float dn = gr < T.nr - 1 ? ldc(res_shared().K.P.wd + o) : 0.f;
    const float up = gr > 0 ? ldc(res_shared().K.P.wd + o - T.pitch) : 0.f;
    const float rt = gc < T.nc - 1 ? ldc(res_shared().K.P.wr + o) : 0.f;
    const float lf = gc > 0 ? ldc(res_shared().K.P.wr + o - 1) : 0.f;
    return make_float2(ldc((const float *)res_shared().K.P.z + o),
                       rcp_pre(diag32(gr, gc, T.nr, T.nc, dn, up, rt, lf)));
}

/* this thread's rim packets of the block's items, asked for ahead of use */
struct RimAsk {
    unsigned long long v[kResPerEngine];
};
__device__ __forceinline__ void rim_ask(const ResCtx &C, unsigned seq, RimAsk &A)
{
#pragma unroll
    for (int x = 0; x < kResPerEngine; ++x) {
        const int i = x * kResEngines + C.eng;
        if (C.rim_at >= 0 && i < res_shared().nloc) {
            const unsigned base = res_shared().nbr[i][C.rim_nb];
            if (base != ~0u) A.v[x] = rim_load(res_shared().K.A.rim + base + (seq & 1u) * kRim + C.rim_pk);
        }
    }
}

/* first half of an iteration: r -= alpha q, dx += alpha p, p = M^-1 r + beta p
 * of the block's items and their halo rings.  A: the rim
 * packets of exchange `seq`, asked for before its totals were waited for. */
__device__ __forceinline__ bool half1(const ResCtx &C, float alpha, float beta, unsigned seq, const RimAsk &A)
{
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    const int so = (ty + 1) * kPnW + 4 + tx * kItemVx;
    const float2 a2 = pf2(alpha, alpha), na2 = pf2(-alpha, -alpha), b2 = pf2(beta, beta);
    for (int i = C.eng; i < res_shared().nloc; i += kResEngines) {
        uint32_t t[16];
        tm_ld16(tm_of(C, i), t);
        float *Pn = pn_of(i);
        float pv[4], nd[8];
        { const float4 p = *reinterpret_cast<const float4 *>(Pn + so);
          pv[0] = p.x; pv[1] = p.y; pv[2] = p.z; pv[3] = p.w; }
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const float2 p2 = pf2(pv[j], pv[j + 1]);
            const float2 x2 = __ffma2_rn(a2, p2, pf2(__uint_as_float(t[j]), __uint_as_float(t[j + 1])));
            const float2 r2 = __ffma2_rn(na2, pf2(__uint_as_float(t[12 + j]), __uint_as_float(t[13 + j])),
                                         pf2(__uint_as_float(t[4 + j]), __uint_as_float(t[5 + j])));
            const float2 z2 = __fmul2_rn(r2, pf2(__uint_as_float(t[8 + j]), __uint_as_float(t[9 + j])));
            const float2 n2 = __ffma2_rn(b2, p2, z2);
            nd[j] = x2.x; nd[j + 1] = x2.y;
            nd[4 + j] = r2.x; nd[5 + j] = r2.y;
            pv[j] = n2.x; pv[j + 1] = n2.y;
        }
        *reinterpret_cast<float4 *>(Pn + so) = make_float4(pv[0], pv[1], pv[2], pv[3]);
        tm_st8(tm_of(C, i), nd);
    }
    tm_wait_st();
    bool ok = true;
    if (C.rim_at >= 0) {
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= res_shared().nloc) continue;
            const unsigned base = res_shared().nbr[i][C.rim_nb];
            if (base == ~0u) continue;   /* outside the tile: p stays zero */
            float *p = pn_of(i) + C.rim_at;
            unsigned long long v = A.v[x];
            if ((unsigned)(v >> 32) != seq) {
                Waiter w(res_shared().K.ctl, res_shared().K.sp.timeout_ns);
                do {
                    if (!w.turn()) {
                        ok = false;
                        break;
                    }
                    v = rim_load(res_shared().K.A.rim + base + (seq & 1u) * kRim + C.rim_pk);
                } while ((unsigned)(v >> 32) != seq);
            }
            float2 *st = rim_state(i) + (C.tid - (kItemThreads - kRim));
            const float2 rm = *st;
            const float r = __fmaf_rn(-alpha, __uint_as_float((unsigned)v), rm.x);
            st->x = r;
            *p = __fmaf_rn(beta, *p, __fmul_rn(r, rm.y));
        }
    }
    return __syncthreads_and(ok);
}

/* the first half right after an assembly or replacement: nothing to update,
 * p = M^-1 r + beta p */
__device__ __noinline__ void half1_fresh()
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    (void)K;
    const float beta = (float)sh.beta;
    const int so = (C.tid / kItemTx + 1) * kPnW + 4 + (C.tid % kItemTx) * kItemVx;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        uint32_t t[8];
        tm_ld8(tm_of(C, i) + kTmR, t);
        float *Pn = pn_of(i);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            Pn[so + j] = __fmaf_rn(beta, Pn[so + j],
                                   __fmul_rn(__uint_as_float(t[j]), __uint_as_float(t[4 + j])));
        if (C.rim_at >= 0 && sh.nbr[i][C.rim_nb] != ~0u) {
            const int li = sh.li[i];
            const float2 rm = fresh_rim(C, (li / sh.T.nbx) * kItemBy - 1 + C.rim_at / kPnW,
                                        (li % sh.T.nbx) * kItemBx - 4 + C.rim_at % kPnW);
            rim_state(i)[C.tid - (kItemThreads - kRim)] = rm;
            float *p = Pn + C.rim_at;
            *p = __fmaf_rn(beta, *p, __fmul_rn(rm.x, rm.y));
        }
        __syncwarp();
    }
    __syncthreads();
}

/* second half: q = A p, the item's four dot products, the rim packets and the
 * block's partials of exchange `seq` */
__device__ __forceinline__ void half2(const ResCtx &C, unsigned seq)
{
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    const int so = (ty + 1) * kPnW + 4 + tx * kItemVx;
    for (int i = C.eng; i < res_shared().nloc; i += kResEngines) {
        const float *Pn = pn_of(i), *WD = wd_of(i), *WR = wr_of(i);
        uint32_t t[8];
        tm_ld8(tm_of(C, i) + kTmR, t);
        float rv[4], m[4], zn[4], pn[4], up[4], dn[4], wdn[4], wup[4], wrt[4], qv[4], mq[4];
        auto s4 = [](const float *p, float v[4]) {
            const float4 f = *reinterpret_cast<const float4 *>(p);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        };
        s4(Pn + so, pn);
        s4(Pn + so - kPnW, up);
        s4(Pn + so + kPnW, dn);
        const float lf = Pn[so - 1], rt = Pn[so + 4];
        s4(WD + (ty + 1) * kItemBx + tx * kItemVx, wdn);
        s4(WD + ty * kItemBx + tx * kItemVx, wup);
        s4(WR + ty * kWrW2 + 4 + tx * kItemVx, wrt);
        const float wlf = WR[ty * kWrW2 + 3 + tx * kItemVx];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            rv[j] = __uint_as_float(t[j]);
            m[j] = __uint_as_float(t[4 + j]);
        }
        /* the operations of k_solve's interior pass, two pixels each */
#pragma unroll
        for (int j = 0; j < kItemVx; j += 2) {
            const float2 xa = pf2(pn[j], pn[j + 1]);
            const float2 xl = pf2(j == 0 ? lf : pn[j - 1], pn[j]);
            const float2 xr = pf2(pn[j + 1], j + 2 == kItemVx ? rt : pn[j + 2]);
            const float2 wl = pf2(j == 0 ? wlf : wrt[j - 1], wrt[j]);
            float2 y = __fmul2_rn(pf2(kLapEpsF, kLapEpsF), xa);
            y = __ffma2_rn(pf2(wdn[j], wdn[j + 1]), psub(xa, pf2(dn[j], dn[j + 1])), y);
            y = __ffma2_rn(pf2(wup[j], wup[j + 1]), psub(xa, pf2(up[j], up[j + 1])), y);
            y = __ffma2_rn(pf2(wrt[j], wrt[j + 1]), psub(xa, xr), y);
            y = __ffma2_rn(wl, psub(xa, xl), y);
            const float2 md = pf2(m[j], m[j + 1]);
            const float2 y2 = __fmul2_rn(y, md), z2 = __fmul2_rn(pf2(rv[j], rv[j + 1]), md);
            qv[j] = y.x; qv[j + 1] = y.y;
            mq[j] = y2.x; mq[j + 1] = y2.y;
            zn[j] = z2.x; zn[j + 1] = z2.y;
        }
        tm_st4(tm_of(C, i) + kTmQ, qv);
        /* rims for the neighbouring items: rows 0 and 15, columns 0 and 63 */
        unsigned long long *rim =
            res_shared().K.A.rim + ((blockIdx.x * kResItems + i) * 2 + (seq & 1u)) * kRim;
        if (ty == 0 || ty == kItemBy - 1) {
            unsigned long long *d = rim + (ty == 0 ? 0 : kItemBx) + tx * kItemVx;
            rim_store2(d, qv[0], qv[1], seq);
            rim_store2(d + 2, qv[2], qv[3], seq);
        }
        if (tx == 0) rim_store(rim + 2 * kItemBx + ty, qv[0], seq);
        if (tx == kItemTx - 1) rim_store(rim + 2 * kItemBx + kItemBy + ty, qv[3], seq);
        double acc[kNComp];
        dot4_df2(pn, qv, zn, qv, acc[1], acc[2]);
        dot4_df2(qv, mq, rv, zn, acc[3], acc[0]);
        const double v = warp_scatter4(acc);   /* lane 8c: the warp's component c */
        if ((C.lane & 7) == 0) res_shared().red[i][C.lane >> 3][C.warp & 7] = v;
        __syncwarp();
    }
    tm_wait_st();
    __syncthreads();
    block_partials(C, kNComp);
    send_partials(C, kNComp, seq);
}

/* x += dx (+ alpha p with `update`) of the block's items */
__device__ __noinline__ void fold_items(bool update)
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    (void)K;
    const float alpha = (float)sh.alpha;
    const TileDesc &T = res_shared().T;
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    for (int i = C.eng; i < res_shared().nloc; i += kResEngines) {
        float dx[4];
        tm_ld4(tm_of(C, i) + kTmDx, dx);
        const int li = res_shared().li[i];
        const int r = (li / T.nbx) * kItemBy + ty, c0 = (li % T.nbx) * kItemBx + tx * kItemVx;
        if (r < T.nr && c0 < T.nc) {
            double *x = res_shared().K.P.x + T.pix + (size_t)r * T.pitch + c0;
            const float *p = pn_of(i) + (ty + 1) * kPnW + 4 + tx * kItemVx;
            double xv[4];
            ld4(x, xv);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (c0 + j >= T.nc) continue;
                const float d = update ? __fmaf_rn(alpha, p[j], dx[j]) : dx[j];
                xv[j] = xv[j] + (double)d;
            }
            st4(x, xv);
        }
        __syncwarp();
    }
}

/* assembly (or, without `assemble`, the true residual) of the block's items,
 * and their sums of r.z */
template <bool WLS>
__device__ __noinline__ void init_items(bool zero_x,
                                        bool assemble)
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    (void)K;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        double v = phase_init<float, WLS>(sh.T, sh.li[i], K.P, zero_x, assemble, (float *)K.P.z,
                                          C.tid);
        __syncwarp();
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (C.lane == 0) sh.red[i][0][C.warp & 7] = v;
    }
    __syncthreads();
}

__device__ __noinline__ void load_items(bool pass_start)
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    (void)K;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) load_item(C, i, pass_start);
    tm_wait_st();
    __syncthreads();
}

__device__ __noinline__ void reweight_items(float delta)
{
    const ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    const int tid = (int)threadIdx.x % kItemThreads;
    for (int i = (int)threadIdx.x / kItemThreads; i < sh.nloc; i += kResEngines)
        phase_rw<float>(sh.T, sh.li[i], K.P, delta, tid);
}

__device__ __noinline__ void final_items()
{
    const ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    const int tid = (int)threadIdx.x % kItemThreads;
    for (int i = (int)threadIdx.x / kItemThreads; i < sh.nloc; i += kResEngines)
        phase_final<float>(sh.T, sh.li[i], K.P, tid);
}

/* PCG iterations of a pass from a fresh residual (the first half of pass
 * sh.k is done) to the next replacement or the tile's stop.  In a function
 * of its own without calls: everything it uses stays in registers. */
enum { kStop, kReplace, kGaveUp };
__device__ __noinline__ int iterate()
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    (void)K;
    const SolveParams &sp = K.sp;
    TileState &S = sh.S;
    unsigned seq = sh.seq + 1;
    int k = sh.k;
    half2(C, seq);
    bool fresh = true;
    while (true) {
        /* the scalars of the next pass from the totals of this one, as in
         * k_solve: the stop test on the true r.z of an update, then alpha and
         * the recurrence for beta */
        RimAsk A;
        rim_ask(C, seq, A);
        double t[kNComp];
        if (!totals<kNComp>(C, seq, t)) return kGaveUp;
        ++k;
        if (threadIdx.x == 0) {
            double rz = S.rz;
            int act = 1;
            if (!fresh) {
                const int it = S.iter + 1;
                S.iter = it;
                if (t[0] < S.thr || it >= sp.max_iter) act = 0;
                else S.rz = rz = t[0];
            }
            double alpha = 0.0, beta = 0.0;
            if (act) {
                if (t[1] <= 0.0) {
                    act = 0;
                } else {
                    alpha = rz / t[1];
                    const double rzn =
                        __fma_rn(alpha * alpha, t[3], __fma_rn(-2.0 * alpha, t[2], rz));
                    beta = rzn > 0.0 ? rzn / rz : 0.0;
                }
            }
            sh.alpha = (float)alpha;
            sh.beta = (float)beta;
            sh.active = act;
            sh.k = k;
            sh.seq = seq;
        }
        __syncthreads();
        if (!sh.active) return kStop;
        if (sp.replace_every > 0 && k % sp.replace_every == 0) return kReplace;
        if (!half1(C, (float)sh.alpha, (float)sh.beta, seq, A)) return kGaveUp;
        half2(C, ++seq);
        fresh = false;
        if ((k & 63) == 63 && threadIdx.x == 0 && sh.member == 0) atomicAdd(&K.ctl->progress, 1u);
    }
}

/* r.z of a new residual, summed over the group (in warp 0); the barrier
 * publishes the residual itself */
template <bool WLS>
__device__ __noinline__ bool new_residual(bool zero_x,
                                          bool assemble, double &rz)
{
    init_items<WLS>(zero_x, assemble);
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    (void)K;
    const unsigned seq = sh.seq + 1;
    block_partials(C, 1);
    send_partials(C, 1, seq);
    if (!totals<1>(C, seq, &rz)) return false;
    if (threadIdx.x == 0) sh.seq = seq;
    return group_sync();
}

/* Run all IRLS passes of one tile; false: a wait ran out. */
template <bool WLS>
__device__ __forceinline__ bool run_tile()
{
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    const SolveParams &sp = K.sp;
    TileState &S = sh.S;
    setup_items();
    if (!group_sync(true)) return false;
    for (int outer = 0; outer <= sp.n_irls; ++outer) {
        double rz;
        if (!new_residual<WLS>(outer == 0 && !(WLS && sp.warm), true, rz)) return false;
        if (threadIdx.x == 0) {
            S = start_state(rz, sp);
            sh.alpha = 0.0;
            sh.beta = 0.0;
            sh.active = S.active;
            sh.k = 0;
        }
        load_items(true);
        while (sh.active) {
            half1_fresh();
            const int why = iterate();
            if (why == kGaveUp) return false;
            if (why == kStop) break;
            /* x += dx + alpha p, then the true residual replaces the
             * recursive one */
            fold_items(true);
            if (!group_sync()) return false;
            if (!new_residual<WLS>(false, false, rz)) return false;
            if (threadIdx.x == 0) {
                const int it = S.iter + 1;
                S.iter = it;
                if (rz < S.thr || it >= sp.max_iter) {
                    sh.active = 0;
                } else {
                    sh.beta = (float)(rz / S.rz);
                    S.rz = rz;
                }
                sh.alpha = 0.0;
            }
            load_items(false);
        }
        count_pass(outer);
        fold_items(false);
        if (!group_sync()) return false;
        if (outer < sp.n_irls) {
            reweight_items(sp.deltas[outer]);
            if (!group_sync()) return false;
        }
    }
    if (!WLS) final_items();
    return true;
}

template <bool WLS>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const __grid_constant__ ResParams K)
{
    resident_blocks(K, [] { return run_tile<WLS>(); });
}

}  // namespace

int launch_resident_mixed(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                          SolverCtl *ctl, const SolveParams &sp, cudaStream_t s)
{
    ResParams K = {tiles, A, P, ctl, sp};
    K.P.dx = nullptr;   /* the increment lives in TMEM */
    return sp.wls ? resident_start(k_resident<true>, kResSmem, K, s)
                  : resident_start(k_resident<false>, kResSmem, K, s);
}

}  // namespace cuphu
