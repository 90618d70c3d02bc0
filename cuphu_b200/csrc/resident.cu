/*
 * resident.cu -- the mixed-precision Laplace solve of tiles whose PCG state
 * fits on the chip.
 *
 * k_solve (laplace.cu) streams every plane of the state through each block
 * once per PCG iteration.  A tile of the usual size (about 1000 x 1000
 * pixels, 24 MB of state) fits into the shared and tensor memory of the
 * chip, so this kernel loads a tile once per IRLS pass and keeps it there:
 * between two iterations only the rims of the blocks' regions and one
 * partial sum per block and dot product cross the L2.
 *
 *  - A tile is run by a group of blocks, one block per SM.  Each holds a
 *    region of up to 16 work items (16 rows x 64 columns each): p with a
 *    halo ring and the two arc-weight planes in shared memory; dx, r, M^-1
 *    and q in tensor memory (TMEM, used as a 256 KB register file: every
 *    thread keeps the 16 words of its four pixels of an item in 16 columns
 *    of its lane); r and M^-1 of the ring in registers.
 *  - An iteration is k_solve's single-synchronisation mixed pass with the
 *    same FP32 operations per pixel.  The dot products are summed in FP64
 *    (the products of two floats are exact there), over a thread's pixels,
 *    the block and the group; k_solve splits the products in FP32 instead
 *    (2^-44 of the sum of the magnitudes), so the scalars agree to about
 *    1e-14 and the iterates, almost always, to the last bit.
 *  - Partials and rims travel as packets that carry the number of their
 *    exchange, written by one store, so data and number arrive together.  A
 *    reader polls the packets it needs; there is no barrier and no memory
 *    fence inside an iteration.  Packets alternate between two buffers; a
 *    block overwrites one only after it has seen the partials of the exchange
 *    in between, which every reader of the old packet publishes after reading
 *    it.
 *  - Every wait is bounded: when it runs out the error status is set, which
 *    ends all other waits, and the kernel returns.
 *
 * What bounds it (967 x 967, 144 blocks of 7 x 1 items, 11.0 k cycles =
 * 5.5 us per iteration; k_solve took 25 us): the second half 5.0 k, bound by
 * no single pipe (290 warp instructions per item in both halves, 20 of them
 * FP32-to-FP64 conversions at a quarter of the issue rate, and 33 of the
 * load-store unit; FP32 dots would take 3.8 k, neighbours by shuffle 6.1 k,
 * and asking for the next item's tensor-memory words ahead changes nothing);
 * the exchange 2.5 k from the last store to the totals, of which 1.3 k are the
 * least that one store and one load of a line another SM has just written
 * take; the first half 1.3 k, sending 1.2 k, the scalars 0.6 k.
 * Regions instead of items dealt out by the slots of k_solve's reduction tree
 * cut the rims of this tile from 1280 to 352 pixels per block and use all
 * SMs, and one FP64 sum per thread replaces a warp tree per item over FP32
 * products split by FMA: 8.2 -> 6.6 us, the rest is the exchange's polling
 * (poll_together).  512 x 512 (2 items per block): 3.3 us, k_solve 15.8;
 * 96 x 128 (1 item): 2.7, k_solve 12.7.
 */
#include "resident.cuh"

namespace cuphu {
namespace {
constexpr int kResItems = kResItemsMixed;
struct ResOwn {
    double red[16][kNComp];             /* warp sums */
    double tot[16][kNComp];             /* warp sums of an exchange */
    int4 item[kResItems];               /* places of the items in the p, down and right arc
                                           arrays, and the region's sides they lie on */
    int2 org[kResItems];                /* the items' first row and column in the region */
    int na, nb;                         /* rows and columns of items of this block's region */
    int r0, c0;                         /* its first pixel in the tile */
    int pw, ww, rw;                     /* row lengths of the p, down and right arc arrays */
    int owd, owr;                       /* offsets of the arc arrays from the p array */
    int side[4];                        /* blocks above, below, left, right (-1: none) */
};
}  // namespace
}  // namespace cuphu
#include "resident_dev.cuh"

namespace cuphu {
namespace {

constexpr int kResCols = 16;   /* TMEM columns of an item: dx, r, M^-1 and q of four pixels */
constexpr int kResPerEngine = kResItems / kResEngines;
static_assert(2 * kResEngines * kResPerEngine * kResCols <= kTmemCols, "TMEM columns");
/* floats of a region of a x b items: p with a ring (four columns each side,
 * for alignment), the down arcs with the row above, the right arcs with four
 * columns to the left */
__host__ __device__ constexpr int region_floats(int a, int b)
{
    return (16 * a + 2) * (64 * b + 8) + (16 * a + 1) * 64 * b + 16 * a * (64 * b + 4);
}
constexpr int most_floats()
{
    int m = 0;
    for (int a = 1; a <= kResItems; ++a)
        for (int b = 1; b <= kResMaxB && a * b <= kResItems; ++b)
            m = region_floats(a, b) > m ? region_floats(a, b) : m;
    return m;
}
constexpr size_t kResSmem = (size_t)most_floats() * 4 + kResSharedB;
static_assert(kResSmem <= 232448, "shared memory of a block");

/* ── rims ─────────────────────────────────────────────────────────────────
 * Rim packets of a block: [parity][side][position], q of a pixel and the
 * exchange number, 8 bytes each (the two of a vector store need not arrive
 * together).  Sides of the writer: 0 its top row, 1 bottom row, 2 left
 * column, 3 right column. */
constexpr int kSide = 256;                  /* packets of a side */
constexpr int kRimN = 2 * 4 * kSide;        /* packets of a block */
constexpr int kMyRims = 2;                  /* ring pixels of a thread at most */
static_assert(2 * (64 * kResMaxB + 16 * kResItems / kResMaxB) <= kMyRims * kResThreads &&
                  2 * (64 + 16 * kResItems) <= kMyRims * kResThreads, "ring of the largest region");

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

/* columns of an item: dx 0..3, r 4..7, M^-1 8..11, q 12..15 */
constexpr int kTmDx = 0, kTmR = 4, kTmQ = 12;

/* A thread's view of its block. */
struct ResCtx {
    int eng, tid, warp, lane;
    int ty, tx;            /* row and first column / 4 of its pixels in an item */
    uint32_t tm;           /* its TMEM columns of its engine's first item */
};
__device__ __forceinline__ ResCtx make_ctx()
{
    const int warp = threadIdx.x >> 5, tid = (int)threadIdx.x % kItemThreads;
    return ResCtx{(int)threadIdx.x / kItemThreads, tid, warp, (int)threadIdx.x & 31,
                  tid / kItemTx, tid % kItemTx,
                  res_shared().tmem + ((uint32_t)(warp & 3) << 21) +
                      (uint32_t)(warp >> 2) * (kResPerEngine * kResCols)};
}
__device__ __forceinline__ float *p_array() { return reinterpret_cast<float *>(res_items()); }
__device__ __forceinline__ uint32_t tm_of(const ResCtx &C, int i)
{
    return C.tm + (uint32_t)(i / kResEngines) * kResCols;
}
/* this thread's offsets within an item in the p, down arc (row above) and
 * right arc arrays */
struct Place {
    int p, wd, wr;
};
__device__ __forceinline__ Place place_of(const ResCtx &C)
{
    const ResOwn &o = res_shared().own;
    return Place{C.ty * o.pw + C.tx * kItemVx, C.ty * o.ww + C.tx * kItemVx,
                 C.ty * o.rw + C.tx * kItemVx};
}
/* the sides of an item that this thread's pixels touch: bit 0 top, 1 bottom,
 * 2 left, 3 right */
__device__ __forceinline__ int sides_of(const ResCtx &C)
{
    return (C.ty == 0 ? 1 : 0) | (C.ty == kItemBy - 1 ? 2 : 0) | (C.tx == 0 ? 4 : 0) |
           (C.tx == kItemTx - 1 ? 8 : 0);
}
/* first row and column of the block's item i in the tile */
__device__ __forceinline__ void item_origin(int i, int &r, int &c)
{
    const ResOwn &o = res_shared().own;
    r = o.r0 + o.org[i].x;
    c = o.c0 + o.org[i].y;
}

/* A ring pixel of the region: its place in the p array, its packet and its
 * place in the tile. */
struct Rim {
    int at;                /* -1: none */
    unsigned pk;           /* packet, without the parity */
    int gr, gc;
};
__device__ __forceinline__ Rim rim_of(int q)
{
    const ResOwn &o = res_shared().own;
    const int w = o.nb * kItemBx, h = o.na * kItemBy;
    int side, pos, row, col;
    if (q < w) { side = 0; pos = q; row = -1; col = q; }
    else if (q < 2 * w) { side = 1; pos = q - w; row = h; col = pos; }
    else if (q < 2 * w + h) { side = 2; pos = q - 2 * w; row = pos; col = -1; }
    else if (q < 2 * w + 2 * h) { side = 3; pos = q - 2 * w - h; row = pos; col = w; }
    else return Rim{-1, 0u, 0, 0};
    const int blk = o.side[side];
    if (blk < 0) return Rim{-1, 0u, 0, 0};   /* outside the tile: p stays zero */
    /* the neighbour's facing side: its bottom row for the row above, ... */
    return Rim{(row + 1) * o.pw + 4 + col, (unsigned)(blk * kRimN + (side ^ 1) * kSide + pos),
               o.r0 + row, o.c0 + col};
}
__device__ __forceinline__ const unsigned long long *rim_src(const Rim &R, unsigned seq)
{
    return res_shared().K.A.rim + R.pk + (seq & 1u) * (4 * kSide);
}

/* ── sums over the group ──────────────────────────────────────────────────
 * A block's mailbox: [parity][member][component] packets. */
constexpr int kMailN = 2 * kNComp * kResMaxBlocks;
__device__ __forceinline__ ulonglong2 *mail_of(int block, unsigned seq, int m, int c)
{
    return res_shared().K.A.mail + (size_t)block * kMailN + (seq & 1u) * (kNComp * kResMaxBlocks) +
           m * kNComp + c;
}

/* Sum the threads' values over the block and send the sums to every block of
 * the group.  A block stores its packets into every mailbox, its own
 * included (8 KB per block and exchange for 128 blocks): one hop.  An
 * iteration at 512 x 512 (128 blocks) takes 3.3 us; with two hops over a grid
 * of 12 x 11 blocks (one warp, few messages) 4.1, and more with a block per
 * component that collects and publishes, or with every block polling the
 * members' own copies (128 readers of each line). */
template <int NCOMP>
__device__ __forceinline__ void send_sums(const ResCtx &C, const double acc[kNComp], unsigned seq)
{
    ResShared &sh = res_shared();
    if constexpr (NCOMP == kNComp) {
        const double v = warp_scatter4(acc);   /* lane 8c: the warp's component c */
        if ((C.lane & 7) == 0) sh.own.red[C.warp][C.lane >> 3] = v;
    } else {
        double v = acc[0];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (C.lane == 0) sh.own.red[C.warp][0] = v;
    }
    __syncthreads();
    /* every warp sums the sixteen warps' values; lane l ends with component
     * l % 4 and sends it to the members l / 4 + 8 w, ... */
    const int c = C.lane & 3, k = C.lane >> 2;
    double v = c < NCOMP ? sh.own.red[k][c] + sh.own.red[k + 8][c] : 0.0;
#pragma unroll
    for (int off = 16; off >= 4; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (c < NCOMP)
        for (int d = threadIdx.x >> 2; d < (int)sh.nact; d += kResThreads / 4)
            packet_store(mail_of(sh.phys[d], seq, sh.member, c),
                         (unsigned long long)__double_as_longlong(v), (unsigned long long)seq);
}

/* The sums of exchange `seq` over the group, in warp 0 (every block adds the
 * members' partials in the same order).  Thread t polls packets t and t + 512
 * of its block's mailbox. */
template <int NCOMP>
__device__ __forceinline__ bool totals(const ResCtx &C, unsigned seq, double out[NCOMP])
{
    ResShared &sh = res_shared();
    const int c = C.lane & 3, cc = c < NCOMP ? c : 0, n = (int)sh.nact;
    const int m = threadIdx.x >> 2, m2 = m + kResThreads / 4;
    bool ok = true;
    double v = 0.0;
    if (8 * C.warp < n) {
        const bool n0 = m < n, n1 = m2 < n, two = 8 * C.warp + kResThreads / 4 < n;
        const ulonglong2 *p0 = mail_of(blockIdx.x, seq, n0 ? m : 0, cc);
        const ulonglong2 *p1 = mail_of(blockIdx.x, seq, n1 ? m2 : 0, cc);
        unsigned long long a0, b0, a1 = 0, b1 = seq;
        ok = poll_together(sh, [&] {
            packet_load(p0, a0, b0);
            if (two) packet_load(p1, a1, b1);
            return (!n0 || b0 == (unsigned long long)seq) && (!n1 || b1 == (unsigned long long)seq);
        });
        if (n0 && c < NCOMP) v = __longlong_as_double((long long)a0);
        if (n1 && c < NCOMP) v += __longlong_as_double((long long)a1);
    }
#pragma unroll
    for (int off = 16; off >= 4; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (C.lane < NCOMP) sh.own.tot[C.warp][C.lane] = v;
    ok = __syncthreads_and(ok);
    if (C.warp == 0) {
        const int k = C.lane >> 2;
        v = c < NCOMP ? sh.own.tot[k][c] + sh.own.tot[k + 8][c] : 0.0;
#pragma unroll
        for (int off = 16; off >= 4; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
#pragma unroll
        for (int j = 0; j < NCOMP; ++j) out[j] = __shfl_sync(0xffffffffu, v, j);
    }
    return ok;
}

/* ── an IRLS pass's phases ────────────────────────────────────────────────── */

/* Load the block's items after an assembly or a residual replacement: dx = 0,
 * q = 0, r from the residual plane; with `pass_start` also the weights, M^-1
 * and p = 0.  Weights beyond the tile's last arcs and pixels beyond its columns
 * read as zero, so the iterations need no edge tests. */
__device__ __noinline__ void load_items(bool pass_start)
{
    const ResCtx C = make_ctx();
    const ResShared &sh = res_shared();
    const SolverPlanes &P = sh.K.P;
    const TileDesc &T = sh.T;
    float *p = p_array(), *WD = p + sh.own.owd, *WR = p + sh.own.owr;
    const Place at = place_of(C);
    const int sides = sides_of(C);
    if (pass_start)
        for (int k = threadIdx.x; k < sh.own.owd; k += kResThreads) p[k] = 0.f;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        int r, c0;
        item_origin(i, r, c0);
        r += C.ty;
        c0 += C.tx * kItemVx;
        const int4 it = sh.own.item[i];
        const bool own = r < T.nr && c0 < T.nc;
        const size_t o = T.pix + (size_t)r * T.pitch + c0;
        float zr[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   /* dx, r */
        if (own) {
            ld4((const float *)P.z + o, zr + 4);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (c0 + j >= T.nc) zr[4 + j] = 0.f;
        }
        __syncwarp();
        tm_st8(tm_of(C, i) + kTmDx, zr);
        float m[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};    /* M^-1, q */
        if (!pass_start) {
            tm_st4(tm_of(C, i) + kTmQ, m + 4);
            continue;
        }
        /* the item's own arcs; the region's first row and column also bring
         * the down arcs of the row above and the right arcs on the left */
        float wdn[4] = {0.f, 0.f, 0.f, 0.f}, wrt[4] = {0.f, 0.f, 0.f, 0.f};
        float up[4] = {0.f, 0.f, 0.f, 0.f}, lf = 0.f;
        if (own) {
            if (r < T.nr - 1) ld4(P.wd + o, wdn);
            if (r > 0) ld4(P.wd + o - T.pitch, up);
            ld4(P.wr + o, wrt);
            if (c0 > 0) lf = ldc(P.wr + o - 1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (c0 + j >= T.nc) wdn[j] = up[j] = 0.f;
                if (c0 + j >= T.nc - 1) wrt[j] = 0.f;
                if (c0 + j < T.nc)
                    m[j] = rcp_pre(diag32(r, c0 + j, T.nr, T.nc, wdn[j], up[j], wrt[j],
                                          j == 0 ? lf : wrt[j - 1]));
            }
        }
        st4(WD + it.y + at.wd + sh.own.ww, wdn);
        st4(WR + it.z + at.wr, wrt);
        if (sides & it.w & 1) st4(WD + it.y + at.wd, up);
        if (sides & it.w & 4) WR[it.z + at.wr - 1] = lf;
        __syncwarp();
        tm_st8(tm_of(C, i) + 8, m);
    }
    tm_wait_st();
    __syncthreads();
}

/* r and M^-1 of a ring pixel right after an assembly or replacement, from the
 * planes (zero outside the tile) */
__device__ __forceinline__ float2 fresh_rim(int gr, int gc)
{
    const ResShared &sh = res_shared();
    const TileDesc &T = sh.T;
    if (gr < 0 || gr >= T.nr || gc < 0 || gc >= T.nc) return make_float2(0.f, 0.f);
    const SolverPlanes &P = sh.K.P;
    const size_t o = T.pix + (size_t)gr * T.pitch + gc;
    const float dn = gr < T.nr - 1 ? ldc(P.wd + o) : 0.f;
    const float up = gr > 0 ? ldc(P.wd + o - T.pitch) : 0.f;
    const float rt = gc < T.nc - 1 ? ldc(P.wr + o) : 0.f;
    const float lf = gc > 0 ? ldc(P.wr + o - 1) : 0.f;
    return make_float2(ldc((const float *)P.z + o),
                       rcp_pre(diag32(gr, gc, T.nr, T.nc, dn, up, rt, lf)));
}

/* first half of an iteration: r -= alpha q, dx += alpha p, p = M^-1 r + beta p
 * of the block's items (alpha = 0 and q = 0 right after an assembly or
 * replacement) */
__device__ __forceinline__ void half1_items(const ResCtx &C, float alpha, float beta)
{
    const int nloc = res_shared().nloc;
    float *p0 = p_array();
    const float2 a2 = pf2(alpha, alpha), na2 = pf2(-alpha, -alpha), b2 = pf2(beta, beta);
    const int at = place_of(C).p;
    uint32_t tm = C.tm;
    for (int i = C.eng; i < nloc; i += kResEngines, tm += kResCols) {
        uint32_t t[16];
        tm_ld16(tm, t);
        float4 *pp = reinterpret_cast<float4 *>(p0 + res_shared().own.item[i].x + at);
        const float4 po = *pp;
        float pv[4] = {po.x, po.y, po.z, po.w}, nd[8];
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
        *pp = make_float4(pv[0], pv[1], pv[2], pv[3]);
        tm_st8(tm, nd);
    }
    tm_wait_st();
}

/* second half: q = A p, the dot products (summed over the thread's pixels in
 * FP64), the rim packets and the block's sums of exchange `seq` */
__device__ __forceinline__ void half2(const ResCtx &C, unsigned seq)
{
    const ResShared &sh = res_shared();
    const int nloc = sh.nloc, pw = sh.own.pw, ww = sh.own.ww;
    const float *p0 = p_array(), *wd0 = p0 + sh.own.owd, *wr0 = p0 + sh.own.owr;
    unsigned long long *rim = sh.K.A.rim + (blockIdx.x * kRimN + (seq & 1u) * (4 * kSide));
    const Place at = place_of(C);
    const int sides = sides_of(C);
    uint32_t tm = C.tm;
    double acc[kNComp] = {0.0, 0.0, 0.0, 0.0};
    auto s4 = [](const float *p, float v[4]) {
        const float4 f = *reinterpret_cast<const float4 *>(p);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    };
    for (int i = C.eng; i < nloc; i += kResEngines, tm += kResCols) {
        const int4 it = sh.own.item[i];
        uint32_t t[8];
        tm_ld8(tm + kTmR, t);
        float rv[4], m[4], zn[4], pn[4], up[4], dn[4], wdn[4], wup[4], wrt[4], qv[4], mq[4];
        const float *Pn = p0 + it.x + at.p, *WD = wd0 + it.y + at.wd, *WR = wr0 + it.z + at.wr;
        s4(Pn, pn);
        s4(Pn - pw, up);
        s4(Pn + pw, dn);
        const float lf = Pn[-1], rt = Pn[4], wlf = WR[-1];
        s4(WD + ww, wdn);
        s4(WD, wup);
        s4(WR, wrt);
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
        tm_st4(tm + kTmQ, qv);
        const int edge = sides & it.w;
        if (edge) {   /* rims for the neighbouring blocks */
            const int2 g = sh.own.org[i];
            if (edge & 3) {
                unsigned long long *d = rim + (edge & 1 ? 0 : kSide) + g.y + C.tx * kItemVx;
                rim_store2(d, qv[0], qv[1], seq);
                rim_store2(d + 2, qv[2], qv[3], seq);
                if ((edge & 3) == 3) {
                    rim_store2(d + kSide, qv[0], qv[1], seq);
                    rim_store2(d + kSide + 2, qv[2], qv[3], seq);
                }
            }
            if (edge & 4) rim_store(rim + 2 * kSide + g.x + C.ty, qv[0], seq);
            if (edge & 8) rim_store(rim + 3 * kSide + g.x + C.ty, qv[3], seq);
        }
#pragma unroll
        for (int j = 0; j < kItemVx; ++j) {
            const double q = (double)qv[j], z = (double)zn[j];
            acc[0] = __fma_rn((double)rv[j], z, acc[0]);
            acc[1] = __fma_rn((double)pn[j], q, acc[1]);
            acc[2] = __fma_rn(z, q, acc[2]);
            acc[3] = __fma_rn(q, (double)mq[j], acc[3]);
        }
        __syncwarp();
    }
    tm_wait_st();
    send_sums<kNComp>(C, acc, seq);
}

/* x += dx (+ alpha p with `update`) of the block's items */
__device__ __noinline__ void fold_items(bool update)
{
    const ResCtx C = make_ctx();
    const ResShared &sh = res_shared();
    const float alpha = (float)sh.alpha;
    const TileDesc &T = sh.T;
    const int at = place_of(C).p;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        float dx[4];
        tm_ld4(tm_of(C, i) + kTmDx, dx);
        int r, c0;
        item_origin(i, r, c0);
        r += C.ty;
        c0 += C.tx * kItemVx;
        if (r < T.nr && c0 < T.nc) {
            double *x = sh.K.P.x + T.pix + (size_t)r * T.pitch + c0;
            const float *p = p_array() + sh.own.item[i].x + at;
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

/* PCG iterations of a pass from a fresh residual to the next replacement or the
 * tile's stop.  In a function of its own without calls: everything it uses
 * stays in registers. */
enum { kStop, kReplace, kGaveUp };
__device__ __noinline__ int iterate()
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    const SolveParams &sp = sh.K.sp;
    TileState &S = sh.S;
    unsigned seq = sh.seq;
    int k = sh.k;
    float *p0 = p_array();
    Rim R[kMyRims];
    float2 rm[kMyRims];   /* r and M^-1 of the thread's ring pixels */
    half1_items(C, 0.f, (float)sh.beta);
#pragma unroll
    for (int n = 0; n < kMyRims; ++n) {
        R[n] = rim_of((int)threadIdx.x + n * kResThreads);
        rm[n] = make_float2(0.f, 0.f);
        if (R[n].at >= 0) {
            rm[n] = fresh_rim(R[n].gr, R[n].gc);
            p0[R[n].at] = __fmaf_rn((float)sh.beta, p0[R[n].at], __fmul_rn(rm[n].x, rm[n].y));
        }
    }
    __syncthreads();
    half2(C, ++seq);
    bool fresh = true;
    while (true) {
        /* the rim packets are asked for before the totals are waited for */
        unsigned long long pk[kMyRims];
#pragma unroll
        for (int n = 0; n < kMyRims; ++n)
            if (R[n].at >= 0) pk[n] = rim_load(rim_src(R[n], seq));
        double t[kNComp];
        if (!totals<kNComp>(C, seq, t)) return kGaveUp;
        ++k;
        /* the scalars of the next pass from the totals of this one, as in
         * k_solve: the stop test on the true r.z of an update, then alpha and
         * the recurrence for beta */
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
        if (threadIdx.x == kResThreads - 1 && (k & 7) == 0 && sh.member == 0)
            atomicAdd(&sh.K.ctl->progress, 1u);   /* while thread 0 forms the scalars */
        __syncthreads();
        if (!sh.active) return kStop;
        if (sp.replace_every > 0 && k % sp.replace_every == 0) return kReplace;
        const float alpha = (float)sh.alpha, beta = (float)sh.beta;
        half1_items(C, alpha, beta);
        bool ok = true;
#pragma unroll
        for (int n = 0; n < kMyRims; ++n) {
            if (R[n].at < 0) continue;
            if ((unsigned)(pk[n] >> 32) != seq) {
                Waiter w(sh.K.ctl, sp.timeout_ns);
                do {
                    if (!w.turn()) {
                        ok = false;
                        break;
                    }
                    pk[n] = rim_load(rim_src(R[n], seq));
                } while ((unsigned)(pk[n] >> 32) != seq);
            }
            rm[n].x = __fmaf_rn(-alpha, __uint_as_float((unsigned)pk[n]), rm[n].x);
            p0[R[n].at] = __fmaf_rn(beta, p0[R[n].at], __fmul_rn(rm[n].x, rm[n].y));
        }
        if (!__syncthreads_and(ok)) return kGaveUp;
        half2(C, ++seq);
        fresh = false;
    }
}

/* Assembly (or, without `assemble`, the true residual) of the block's items;
 * r.z over the group (in warp 0).  The barrier publishes the residual. */
template <bool WLS>
__device__ __noinline__ bool new_residual(bool zero_x, bool assemble, double &rz)
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    double acc[kNComp] = {0.0, 0.0, 0.0, 0.0};
    for (int i = C.eng; i < sh.nloc; i += kResEngines)
        acc[0] += phase_init<float, WLS>(sh.T, sh.li[i], sh.K.P, zero_x, assemble,
                                         (float *)sh.K.P.z, C.tid);
    __syncwarp();
    const unsigned seq = sh.seq + 1;
    send_sums<1>(C, acc, seq);
    if (!totals<1>(C, seq, &rz)) return false;
    if (threadIdx.x == 0) sh.seq = seq;
    return group_sync();
}

__device__ __noinline__ void reweight_items(float delta)
{
    const ResShared &sh = res_shared();
    const int tid = (int)threadIdx.x % kItemThreads;
    for (int i = (int)threadIdx.x / kItemThreads; i < sh.nloc; i += kResEngines)
        phase_rw<float>(sh.T, sh.li[i], sh.K.P, delta, tid);
}

__device__ __noinline__ void final_items()
{
    const ResShared &sh = res_shared();
    const int tid = (int)threadIdx.x % kItemThreads;
    for (int i = (int)threadIdx.x / kItemThreads; i < sh.nloc; i += kResEngines)
        phase_final<float>(sh.T, sh.li[i], sh.K.P, tid);
}

/* the block's region of a tile: member m of a grid of regions of a x b items */
__device__ __forceinline__ void begin_tile(const ResTile &G)
{
    ResShared &sh = res_shared();
    ResOwn &o = sh.own;
    const TileDesc &T = sh.T;
    const int nby = T.nitems / T.nbx, ra = sh.member / G.rcols, rb = sh.member % G.rcols;
    o.na = min(G.a, nby - ra * G.a);
    o.nb = min(G.b, T.nbx - rb * G.b);
    o.r0 = ra * G.a * kItemBy;
    o.c0 = rb * G.b * kItemBx;
    o.pw = 64 * G.b + 8;
    o.ww = 64 * G.b;
    o.rw = 64 * G.b + 4;
    o.owd = (16 * G.a + 2) * o.pw;
    o.owr = o.owd + (16 * G.a + 1) * o.ww;
    sh.nloc = o.na * o.nb;
    o.side[0] = ra > 0 ? sh.member - G.rcols : -1;
    o.side[1] = (ra + 1) * G.a < nby ? sh.member + G.rcols : -1;
    o.side[2] = rb > 0 ? sh.member - 1 : -1;
    o.side[3] = (rb + 1) * G.b < T.nbx ? sh.member + 1 : -1;
}

/* the block's item list, its neighbours' block numbers; the packets of an
 * earlier tile are voided */
__device__ __noinline__ void setup_items()
{
    ResShared &sh = res_shared();
    ResOwn &o = sh.own;
    if ((int)threadIdx.x < sh.nloc) {
        const int ia = (int)threadIdx.x / o.nb, ib = (int)threadIdx.x % o.nb;
        sh.li[threadIdx.x] = (o.r0 / kItemBy + ia) * sh.T.nbx + o.c0 / kItemBx + ib;
        o.org[threadIdx.x] = make_int2(ia * kItemBy, ib * kItemBx);
        o.item[threadIdx.x] =
            make_int4((ia * kItemBy + 1) * o.pw + 4 + ib * kItemBx,
                      ia * kItemBy * o.ww + ib * kItemBx, ia * kItemBy * o.rw + 4 + ib * kItemBx,
                      (ia == 0 ? 1 : 0) | (ia == o.na - 1 ? 2 : 0) | (ib == 0 ? 4 : 0) |
                          (ib == o.nb - 1 ? 8 : 0));
    }
    if (threadIdx.x < 4 && o.side[threadIdx.x] >= 0)
        o.side[threadIdx.x] = sh.phys[o.side[threadIdx.x]];
    for (int k = threadIdx.x; k < kRimN; k += kResThreads)
        rim_store(sh.K.A.rim + blockIdx.x * kRimN + k, 0.f, 0u);
    for (int k = threadIdx.x; k < kMailN; k += kResThreads)
        packet_store(sh.K.A.mail + (size_t)blockIdx.x * kMailN + k, 0ull, 0ull);
    if (threadIdx.x == 0) sh.seq = 0u;
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
    resident_blocks(K, [](const ResTile &R) { begin_tile(R); }, [] { return run_tile<WLS>(); });
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
