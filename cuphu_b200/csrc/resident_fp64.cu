/*
 * resident_fp64.cu -- the FP64 Laplace solve of tiles whose PCG state fits on
 * the chip; bit-identical to k_solve's FP64 form (laplace.cu), hence to the
 * CPU oracle.
 *
 * The same scheme as resident.cu with the FP64 form's two reductions per
 * iteration.  p with its halo ring and the arc weights (as doubles, so the
 * stencil converts nothing) are in shared memory; x, r, the diagonal and its
 * reciprocal in tensor memory; q = A p stays in registers between the two
 * halves.  The first half folds p = z + beta p and forms q and p.q; the
 * second applies alpha and forms z = r / diag and r.z.  A rim packet carries
 * z of a pixel and is sent with the exchange of r.z.
 *
 * z = r / diag is needed twice per iteration.  It comes from the stored
 * correctly rounded reciprocal by two correction steps, the second of which
 * rounds correctly (P. Markstein, "Computation of elementary functions on the
 * IBM RISC System/6000 processor", IBM J. Res. Develop. 34(1), 1990): five
 * FP64 operations in place of a division of some thirty.
 *
 * The split is by the slots of k_solve's reduction tree, so that the sums are
 * k_solve's to the bit: sums items j, j + 256, ... per slot j, then the 256
 * slots by a butterfly over the slot's lane bits (16, 8, 4, 2, 1) and its
 * warp bits (4, 2, 1).  A group of 2^g blocks deals the slots out so that
 * the first 8 - g levels of that butterfly stay inside a block: a block
 * publishes one partial, and every block finishes the tree for itself.
 *
 * What bounds it: two exchanges per iteration (see resident.cu), and with 8
 * items per block the shared-memory and tensor-memory latency of the two
 * halves.  Per iteration 5.5 us at 256 x 256, 6.2 us at 512 x 512, 11.1 us at
 * 967 x 967; the streaming form took 22, 28 and 50 us.
 */
#include "quotient.cuh"
#include "resident_geom.cuh"

namespace cuphu {
namespace {
constexpr int kResItems = kResItems64;
struct ResOwn {
    double red[kResItems][8];           /* warp sums per item */
    double tot[16];                     /* warp sums of an exchange */
    unsigned nbr[kResItems][4];         /* packet base of the rim sources: above,
                                           below, left, right (~0: outside) */
    int g;                              /* group of 2^g members */
    int slow;                           /* some quotient of the block needs IEEE divisions */
};
}  // namespace
}  // namespace cuphu
#include "resident_dev.cuh"

namespace cuphu {
namespace {

constexpr int kResCols = 32;   /* TMEM columns of an item: x, r, diag and 1/diag of four pixels */
constexpr int kResPerEngine = kResItems / kResEngines;
constexpr int kRim = 2 * kItemBx + 2 * kItemBy;         /* halo pixels of an item */
/* Rows of an item's arrays: the first two of every thread's four pixels, then
 * the other two (so a warp reads 16-byte pieces without bank conflicts; four
 * doubles in place cost two passes per read), then the halo columns: p has
 * one on each side, the right arcs one on the left. */
constexpr int kPnW = kItemBx + 2;
constexpr int kPnN = (kItemBy + 2) * kPnW;
constexpr int kWdN = (kItemBy + 1) * kItemBx;           /* down arcs, one row above */
constexpr int kWrW = kItemBx + 2;
constexpr int kWrN = kItemBy * kWrW;
constexpr int kHalf = kItemBx / 2, kLeft = kItemBx, kRight = kItemBx + 1;
__device__ __forceinline__ int col_at(int c)            /* place of column c in a row */
{
    return ((c >> 1) & 1) * kHalf + (c >> 2) * 2 + (c & 1);
}
static_assert(2 * kResEngines * kResPerEngine * kResCols <= kTmemCols, "TMEM columns");
constexpr int kResItemD = kPnN + kWdN + kWrN;   /* doubles of an item */
constexpr size_t kResSmem = (size_t)kResItems * kResItemD * 8 + kResSharedB;
static_assert(kResSmem <= 232448, "shared memory of a block");

/* A thread's view of its block. */
struct ResCtx {
    int eng, tid, warp, lane;
    int rim_at, rim_nb, rim_pk;   /* this thread's rim pixel of an item: place in the p array
                                     (-1: none), neighbour, packet */
    int rim_r, rim_c;             /* its row and column in the item (-1 .. 16, -1 .. 64) */
    uint32_t tm;           /* this thread's TMEM columns of its engine's first item */
};

__device__ __forceinline__ ResCtx make_ctx()
{
    const int warp = threadIdx.x >> 5;
    const int eng = (int)threadIdx.x / kItemThreads, tid = (int)threadIdx.x % kItemThreads;
    /* the halo ring of an item is the work of an engine's last 160 threads:
     * the rows above and below (the neighbour's last and first row), the
     * columns left and right (its last and first column) */
    int rim_at = -1, rim_nb = 0, rim_pk = 0, rim_r = 0, rim_c = 0;
    const int h = tid - (kItemThreads - kRim);
    if (h >= 2 * kItemBx + kItemBy) {
        rim_r = h - 2 * kItemBx - kItemBy; rim_c = kItemBx;
        rim_at = (rim_r + 1) * kPnW + kRight; rim_nb = 3; rim_pk = 2 * kItemBx + rim_r;
    } else if (h >= 2 * kItemBx) {
        rim_r = h - 2 * kItemBx; rim_c = -1;
        rim_at = (rim_r + 1) * kPnW + kLeft; rim_nb = 2; rim_pk = 2 * kItemBx + kItemBy + rim_r;
    } else if (h >= kItemBx) {
        rim_r = kItemBy; rim_c = h - kItemBx;
        rim_at = (kItemBy + 1) * kPnW + col_at(rim_c); rim_nb = 1; rim_pk = rim_c;
    } else if (h >= 0) {
        rim_r = -1; rim_c = h;
        rim_at = col_at(h); rim_nb = 0; rim_pk = kItemBx + h;
    }
    return ResCtx{eng, tid, warp, (int)threadIdx.x & 31, rim_at, rim_nb, rim_pk, rim_r, rim_c,
                  res_shared().tmem + ((uint32_t)(warp & 3) << 21) +
                      (uint32_t)(warp >> 2) * (kResPerEngine * kResCols)};
}

__device__ __forceinline__ double *pn_of(int i)
{
    return reinterpret_cast<double *>(res_items()) + i * kResItemD;
}
__device__ __forceinline__ double *wd_of(int i) { return pn_of(i) + kPnN; }
__device__ __forceinline__ double *wr_of(int i) { return pn_of(i) + kPnN + kWdN; }
__device__ __forceinline__ uint32_t tm_of(const ResCtx &C, int i)
{
    return C.tm + (uint32_t)(i / kResEngines) * kResCols;
}
/* columns of an item: x, r, diag and 1/diag (4 each) of the first two pixels,
 * then of the other two */
constexpr int kTmHalf = 16;

/* rim packets: z of a pixel and the exchange number */
__device__ __forceinline__ ulonglong2 *rim_at(unsigned base)
{
    return reinterpret_cast<ulonglong2 *>(res_shared().K.A.rim) + base;
}
__device__ __forceinline__ void rim_store(ulonglong2 *p, double z, unsigned seq)
{
    packet_store(p, (unsigned long long)__double_as_longlong(z), (unsigned long long)seq);
}
__device__ __forceinline__ void rim_void(int k)
{
    rim_store(rim_at(blockIdx.x * kResItems * 2 * kRim + k), 0.0, 0u);
}

__device__ __forceinline__ void unpack2(const uint32_t *t, double v[2])
{
    v[0] = __hiloint2double((int)t[1], (int)t[0]);
    v[1] = __hiloint2double((int)t[3], (int)t[2]);
}
__device__ __forceinline__ void pack2(const double v[2], float *f)
{
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        f[2 * j] = __int_as_float(__double2loint(v[j]));
        f[2 * j + 1] = __int_as_float(__double2hiint(v[j]));
    }
}
__device__ __forceinline__ void lds2(const double *p, double v[2])
{
    const double2 a = *reinterpret_cast<const double2 *>(p);
    v[0] = a.x; v[1] = a.y;
}
__device__ __forceinline__ void sts2(double *p, const double v[2])
{
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
}

/* A block's mailbox: [parity][member m] packets, four copies of each (64
 * bytes): four lanes store and read one packet, whole sectors at a time.
 * (With one lane in four: 7.9 us per iteration at 512 x 512 instead of 6.2.) */
constexpr int kCopies = 4;
constexpr int kMailN = 2 * kResMembers * kCopies;
__device__ __forceinline__ ulonglong2 *mail_of(int block, unsigned seq, int m)
{
    return res_shared().K.A.mail + (size_t)block * kMailN +
           ((seq & 1u) * kResMembers + m) * kCopies + (threadIdx.x & 3);
}

/* The block's partial, after a barrier that follows the items' warp sums: the
 * items' partials (lanes 2 i + h hold the half tree of warp parity h), the
 * slot sums (items of a slot in order) and the butterfly levels inside the
 * block.  Every warp forms it, so that all can send it at once. */
__device__ __forceinline__ double block_partial(const ResCtx &C)
{
    const ResOwn &own = res_shared().own;
    const int i = C.lane >> 1, h = C.lane & 1, nloc = res_shared().nloc;
    double v = 0.0;
    if (i < nloc) {
        const double *w = own.red[i];
        v = (w[h] + w[h + 4]) + (w[h + 2] + w[h + 6]);
    }
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    const int slog = 8 - own.g, S = 1 << slog, sub = C.lane & (S - 1);
    double a = 0.0;
    for (int k = 0; k < nloc; k += S) {
        const double x = __shfl_sync(0xffffffffu, v, (2 * (k + sub)) & 31);
        if (k + sub < nloc) a += x;
    }
    for (int off = S >> 1; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    return a;
}

/* Send the block's partial to every block of the group: threads 4 d .. 4 d + 3
 * to member d's mailbox. */
__device__ __forceinline__ void send_partial(double v, unsigned seq)
{
    const ResShared &sh = res_shared();
    const int d = threadIdx.x >> 2;
    if (d < (1 << sh.own.g) && sh.phys[d] != 0xffffu)
        packet_store(mail_of(sh.phys[d], seq, sh.member),
                     (unsigned long long)__double_as_longlong(v), (unsigned long long)seq);
}

/* Wait for exchange `seq` and finish the tree; the total is returned in warp
 * 0.  One hop: every member stores its packet into every mailbox, and threads
 * 32 w + 4 h .. + 3 poll the packet of member 16 h + w of their block's
 * mailbox.  The members' bits combine from the top: three levels across the
 * lanes, four across the warps. */
__device__ __forceinline__ bool total(const ResCtx &C, unsigned seq, double &out)
{
    ResShared &sh = res_shared();
    bool ok = true;
    const int m = ((C.lane >> 2) << 4) | C.warp;
    unsigned long long lo = 0, hi;
    const bool need = m < (1 << sh.own.g) && sh.phys[m] != 0xffffu;
    const unsigned who = __ballot_sync(0xffffffffu, need);
    if (who) {
        const int any = __shfl_sync(0xffffffffu, m, __ffs(who) - 1);
        const ulonglong2 *p = mail_of(blockIdx.x, seq, need ? m : any);
        ok = poll_together(sh, [&] {
            packet_load(p, lo, hi);
            return hi == (unsigned long long)seq;
        });
        if (!need) lo = 0;
    }
    double v = __longlong_as_double((long long)lo);
#pragma unroll
    for (int off = 16; off >= 4; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (C.lane == 0) sh.own.tot[C.warp] = v;
    ok = __syncthreads_and(ok);
    if (C.warp == 0) {
        v = C.lane < 16 ? sh.own.tot[C.lane] : 0.0;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        out = v;
    }
    return ok;
}

/* this block's items of the tile, their rim sources; the packets of an
 * earlier tile are voided */
__device__ __noinline__ void setup_items()
{
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    const TileDesc &T = sh.T;
    if (threadIdx.x < kResItems) {
        const int i = threadIdx.x, slog = 8 - sh.own.g;
        const int u = ((i & ((1 << slog) - 1)) << sh.own.g) | sh.member;
        const int li = 256 * (i >> slog) + res_slot(u);
        sh.li[i] = li;
        if (i < sh.nloc) {
            const int row = li / T.nbx, col = li % T.nbx;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int n = -1;
                if (k == 0 && row > 0) n = li - T.nbx;
                if (k == 1 && li + T.nbx < T.nitems) n = li + T.nbx;
                if (k == 2 && col > 0) n = li - 1;
                if (k == 3 && col + 1 < T.nbx) n = li + 1;
                unsigned base = ~0u;
                if (n >= 0) {
                    const int v = res_u(n & 255), m = v & ((1 << sh.own.g) - 1);
                    base = ((unsigned)sh.phys[m] * kResItems + ((n >> 8) << slog) + (v >> sh.own.g)) *
                           2 * kRim;
                }
                sh.own.nbr[i][k] = base;
            }
        }
    }
    for (int k = threadIdx.x; k < sh.nloc * 2 * kRim; k += kResThreads)
        rim_void(k);
    for (int k = threadIdx.x; k < kMailN; k += kResThreads)
        packet_store(K.A.mail + (size_t)blockIdx.x * kMailN + k, 0ull, 0ull);
    if (threadIdx.x == 0) sh.seq = 0u;
}

/* Load an item at the start of a pass: x, r and the diagonal from the planes,
 * the weights as doubles, p = 0.  Weights beyond the tile's last arcs read as
 * zero, so the iterations need no edge tests. */
__device__ __noinline__ void load_items()
{
    const ResCtx C = make_ctx();
    const ResShared &sh = res_shared();
    const SolverPlanes &P = sh.K.P;
    const TileDesc &T = sh.T;
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    bool odd = false;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        const int li = sh.li[i];
        const int r = (li / T.nbx) * kItemBy + ty, c0 = (li % T.nbx) * kItemBx + tx * kItemVx;
        const bool own = r < T.nr && c0 < T.nc;
        const size_t o = T.pix + (size_t)r * T.pitch + c0;
        double *Pn = pn_of(i), *WD = wd_of(i), *WR = wr_of(i);
        double xv[4] = {0.0, 0.0, 0.0, 0.0}, rv[4] = {0.0, 0.0, 0.0, 0.0};
        double dv[4] = {1.0, 1.0, 1.0, 1.0}, yv[4];
        float wdn[4] = {0.f, 0.f, 0.f, 0.f}, wrt[4] = {0.f, 0.f, 0.f, 0.f};
        float up[4] = {0.f, 0.f, 0.f, 0.f}, lf = 0.f;
        if (own) {
            ld4(P.x + o, xv);
            ld4((const double *)P.r + o, rv);
            ld4((const double *)P.diag + o, dv);
            if (r < T.nr - 1) ld4(P.wd + o, wdn);
            if (r > 0) ld4(P.wd + o - T.pitch, up);
            ld4(P.wr + o, wrt);
            if (c0 > 0) lf = ldc(P.wr + o - 1);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (c0 + j >= T.nc) {
                xv[j] = rv[j] = 0.0;
                dv[j] = 1.0;
                wdn[j] = up[j] = 0.f;
            }
            if (c0 + j >= T.nc - 1) wrt[j] = 0.f;
            yv[j] = dv[j] >= 0x1p-100 && dv[j] <= 0x1p100 ? __drcp_rn(dv[j]) : 0.0;
            odd = odd || yv[j] == 0.0 || res_odd(rv[j]);
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float f[16];
            pack2(xv + 2 * h, f);
            pack2(rv + 2 * h, f + 4);
            pack2(dv + 2 * h, f + 8);
            pack2(yv + 2 * h, f + 12);
            tm_st8(tm_of(C, i) + h * kTmHalf, f);
            tm_st8(tm_of(C, i) + h * kTmHalf + 8, f + 8);
        }
        for (int k = C.tid; k < kPnN; k += kItemThreads) Pn[k] = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = col_at(tx * kItemVx + j);
            WD[(ty + 1) * kItemBx + c] = (double)wdn[j];
            WR[ty * kWrW + c] = (double)wrt[j];
            if (ty == 0) WD[c] = (double)up[j];
        }
        if (tx == 0) WR[ty * kWrW + kLeft] = (double)lf;
        __syncwarp();
    }
    tm_wait_st();
    odd = __syncthreads_or(odd);
    if (threadIdx.x == 0) res_shared().own.slow = odd;
    __syncthreads();
}

/* x of the block's items back to its plane */
__device__ __noinline__ void store_items()
{
    const ResCtx C = make_ctx();
    const ResShared &sh = res_shared();
    const TileDesc &T = sh.T;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        double xv[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t t[8];
            tm_ld8(tm_of(C, i) + h * kTmHalf, t);
            unpack2(t, xv + 2 * h);
        }
        const int li = sh.li[i];
        const int r = (li / T.nbx) * kItemBy + C.tid / kItemTx;
        const int c0 = (li % T.nbx) * kItemBx + (C.tid % kItemTx) * kItemVx;
        if (r < T.nr && c0 < T.nc) st4(sh.K.P.x + T.pix + (size_t)r * T.pitch + c0, xv);
        __syncwarp();
    }
}

/* the warp's share of an item's sum */
__device__ __forceinline__ void item_sum(const ResCtx &C, int i, double v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (C.lane == 0) res_shared().own.red[i][C.warp & 7] = v;
}

/* this thread's rim packets of the block's items, asked for ahead of use */
struct RimAsk {
    unsigned long long lo[kResPerEngine], hi[kResPerEngine];
};
__device__ __forceinline__ void rim_ask(const ResCtx &C, unsigned seq, RimAsk &A)
{
    const ResShared &sh = res_shared();
#pragma unroll
    for (int x = 0; x < kResPerEngine; ++x) {
        const int i = x * kResEngines + C.eng;
        A.lo[x] = 0;
        A.hi[x] = seq;
        if (C.rim_at >= 0 && i < sh.nloc) {
            const unsigned base = sh.own.nbr[i][C.rim_nb];
            if (base != ~0u)
                packet_load(rim_at(base + (seq & 1u) * kRim + C.rim_pk), A.lo[x], A.hi[x]);
        }
    }
}

/* p = z + beta p of the block's items */
template <bool SLOW> __device__ __forceinline__ void fold_own(const ResCtx &C, double beta)
{
    const ResShared &sh = res_shared();
    const int so = (C.tid / kItemTx + 1) * kPnW + (C.tid % kItemTx) * 2;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        double *Pn = pn_of(i) + so;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t t[16];
            tm_ld16(tm_of(C, i) + h * kTmHalf, t);
            double rv[2], dv[2], yv[2], pv[2];
            unpack2(t + 4, rv);
            unpack2(t + 8, dv);
            unpack2(t + 12, yv);
            lds2(Pn + h * kHalf, pv);
#pragma unroll
            for (int j = 0; j < 2; ++j)
                pv[j] = __fma_rn(beta, pv[j],
                                 SLOW ? __ddiv_rn(rv[j], dv[j]) : quotient(rv[j], dv[j], yv[j]));
            sts2(Pn + h * kHalf, pv);
            __syncwarp();
        }
    }
}
__device__ __noinline__ void slow_fold()
{
    const ResCtx C = make_ctx();
    fold_own<true>(C, res_shared().beta);
}

/* the rim packets of an item: z of its first and last rows and columns */
__device__ __forceinline__ void send_rims(const ResCtx &C, int i, const double zv[4], unsigned seq)
{
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    ulonglong2 *rim = rim_at(((blockIdx.x * kResItems + i) * 2 + (seq & 1u)) * kRim);
    if (ty == 0 || ty == kItemBy - 1) {
        ulonglong2 *d = rim + (ty == 0 ? 0 : kItemBx) + tx * kItemVx;
#pragma unroll
        for (int j = 0; j < 4; ++j) rim_store(d + j, zv[j], seq);
    }
    if (tx == 0) rim_store(rim + 2 * kItemBx + ty, zv[0], seq);
    if (tx == kItemTx - 1) rim_store(rim + 2 * kItemBx + kItemBy + ty, zv[3], seq);
}

/* z = r / diag, the rims and r.z of the block's items by IEEE divisions */
__device__ __noinline__ void slow_update(unsigned seq)
{
    const ResCtx C = make_ctx();
    const ResShared &sh = res_shared();
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        double zv[4], acc = 0.0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t t[16];
            tm_ld16(tm_of(C, i) + h * kTmHalf, t);
            double rv[2], dv[2];
            unpack2(t + 4, rv);
            unpack2(t + 8, dv);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                zv[2 * h + j] = __ddiv_rn(rv[j], dv[j]);
                acc = __fma_rn(rv[j], zv[2 * h + j], acc);
            }
            __syncwarp();
        }
        send_rims(C, i, zv, seq);
        __syncwarp();
        item_sum(C, i, acc);
    }
    __syncthreads();
}

/* p = z + beta p of the items' halo rings (z from the plane right after an
 * assembly, else from the packets of exchange `seq`) */
__device__ __forceinline__ bool fold_rims(const ResCtx &C, double beta, bool first, unsigned seq,
                                          const RimAsk &A)
{
    const ResShared &sh = res_shared();
    bool ok = true;
    if (C.rim_at >= 0) {
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= sh.nloc) continue;
            const unsigned base = sh.own.nbr[i][C.rim_nb];
            if (base == ~0u) continue;   /* outside the tile: p stays zero */
            double z;
            if (first) {
                const int li = sh.li[i], gr = (li / sh.T.nbx) * kItemBy + C.rim_r;
                const int gc = (li % sh.T.nbx) * kItemBx + C.rim_c;
                z = gr < sh.T.nr && gc < sh.T.nc
                        ? ldc((const double *)sh.K.P.z + sh.T.pix + (size_t)gr * sh.T.pitch + gc)
                        : 0.0;
            } else {
                unsigned long long lo = A.lo[x], hi = A.hi[x];
                if (hi != (unsigned long long)seq) {
                    Waiter w(sh.K.ctl, sh.K.sp.timeout_ns);
                    do {
                        if (!w.turn()) {
                            ok = false;
                            break;
                        }
                        packet_load(rim_at(base + (seq & 1u) * kRim + C.rim_pk), lo, hi);
                    } while (hi != (unsigned long long)seq);
                }
                z = __longlong_as_double((long long)lo);
            }
            double *p = pn_of(i) + C.rim_at;
            *p = __fma_rn(beta, *p, z);
        }
    }
    return __syncthreads_and(ok);
}

/* PCG iterations of a pass, from its assembly to the tile's stop; false: a
 * wait ran out.  In a function of its own without calls: everything it uses
 * stays in registers. */
__device__ __noinline__ bool iterate()
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    TileState &S = sh.S;
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    const int row = (ty + 1) * kPnW, so = row + tx * 2;
    /* left neighbour of the first pixel, right neighbour of the last */
    const int so_l = tx > 0 ? so + kHalf - 1 : row + kLeft;
    const int so_r = tx < kItemTx - 1 ? so + 2 : row + kRight;
    const int wo = ty * kWrW + tx * 2, wo_l = tx > 0 ? wo + kHalf - 1 : ty * kWrW + kLeft;
    unsigned seq = sh.seq;
    RimAsk A;
    bool first = true;
    while (true) {
        if (sh.own.slow) {
            slow_fold();
            if (!first) rim_ask(C, seq, A);
        } else {
            fold_own<false>(C, sh.beta);
        }
        if (!fold_rims(C, sh.beta, first, seq, A)) return false;
        first = false;
        /* q = A p and p.q, in k_solve's order (an arc outside the tile has
         * weight zero and adds nothing) */
        /* set to zero: with values left open for items the block does not hold,
         * the compiler kept all of q in local memory */
        double q[kResPerEngine][4] = {};
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= sh.nloc) continue;
            const double *Pn = pn_of(i), *WD = wd_of(i), *WR = wr_of(i);
            double acc = 0.0, xl = Pn[so_l], wl = WR[wo_l];   /* left pixel and arc */
            double pn[2], nx[2];
            lds2(Pn + so, pn);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double up[2], dn[2], wdn[2], wup[2], wrt[2];
                if (h == 0) lds2(Pn + so + kHalf, nx);
                else nx[0] = Pn[so_r];
                lds2(Pn + so - kPnW + h * kHalf, up);
                lds2(Pn + so + kPnW + h * kHalf, dn);
                lds2(WD + (ty + 1) * kItemBx + tx * 2 + h * kHalf, wdn);
                lds2(WD + ty * kItemBx + tx * 2 + h * kHalf, wup);
                lds2(WR + wo + h * kHalf, wrt);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const double xa = pn[j], xr = j == 0 ? pn[1] : nx[0];
                    double y = (double)kLapEpsF * xa;
                    y = __fma_rn(wdn[j], xa - dn[j], y);
                    y = __fma_rn(wup[j], xa - up[j], y);
                    y = __fma_rn(wrt[j], xa - xr, y);
                    y = __fma_rn(wl, xa - xl, y);
                    q[x][2 * h + j] = y;
                    acc = __fma_rn(xa, y, acc);
                    xl = xa;
                    wl = wrt[j];
                }
                pn[0] = nx[0];
                pn[1] = nx[1];
            }
            item_sum(C, i, acc);
        }
        __syncthreads();
        send_partial(block_partial(C), ++seq);
        double tot;
        if (!total(C, seq, tot)) return false;
        if (threadIdx.x == 0) {
            if (tot <= 0.0) sh.active = 0;
            else sh.alpha = quotient_any(S.rz, tot);
        }
        __syncthreads();
        if (!sh.active) break;
        /* x += alpha p, r -= alpha q, z = r / diag, r.z; the rims' z */
        const double alpha = sh.alpha;
        bool odd = false;
        ++seq;
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= sh.nloc) continue;
            double zv[4], acc = 0.0;
            bool mine = false;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t t[16];
                tm_ld16(tm_of(C, i) + h * kTmHalf, t);
                double xv[2], rv[2], dv[2], yv[2], pv[2];
                unpack2(t, xv);
                unpack2(t + 4, rv);
                unpack2(t + 8, dv);
                unpack2(t + 12, yv);
                lds2(pn_of(i) + so + h * kHalf, pv);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    xv[j] = __fma_rn(alpha, pv[j], xv[j]);
                    rv[j] = __fma_rn(-alpha, q[x][2 * h + j], rv[j]);
                    mine = mine || __double2hiint(yv[j]) == 0 || res_odd(rv[j]);
                    const double z = quotient(rv[j], dv[j], yv[j]);
                    zv[2 * h + j] = z;
                    acc = __fma_rn(rv[j], z, acc);
                }
                float f[8];
                pack2(xv, f);
                pack2(rv, f + 4);
                __syncwarp();
                tm_st8(tm_of(C, i) + h * kTmHalf, f);
            }
            odd = odd || mine;
            if (!mine) send_rims(C, i, zv, seq);   /* else slow_update does */
            __syncwarp();
            item_sum(C, i, acc);
        }
        tm_wait_st();
        odd = __syncthreads_or(odd);
        if (odd) slow_update(seq);
        if (threadIdx.x == 0) sh.own.slow = odd;
        send_partial(block_partial(C), seq);
        rim_ask(C, seq, A);
        if (!total(C, seq, tot)) return false;
        if (threadIdx.x == 0) {
            const int it = S.iter + 1;
            S.iter = it;
            if (tot < S.thr || it >= sh.K.sp.max_iter) {
                sh.active = 0;
            } else {
                sh.beta = quotient_any(tot, S.rz);
                S.rz = tot;
            }
            if ((it & 7) == 0 && sh.member == 0) atomicAdd(&sh.K.ctl->progress, 1u);
        }
        __syncthreads();
        if (!sh.active) break;
    }
    if (threadIdx.x == 0) sh.seq = seq;
    return true;
}

/* b, diag, r, z and r.z of the block's items; the group's r.z (in warp 0).
 * The barrier publishes the planes. */
template <bool WLS> __device__ __noinline__ bool assemble(bool zero_x, double &rz)
{
    const ResCtx C = make_ctx();
    ResShared &sh = res_shared();
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        const double v = phase_init<double, WLS>(sh.T, sh.li[i], sh.K.P, zero_x, true,
                                                 (double *)sh.K.P.z, C.tid);
        __syncwarp();
        item_sum(C, i, v);
    }
    __syncthreads();
    const unsigned seq = sh.seq + 1;
    send_partial(block_partial(C), seq);
    if (!total(C, seq, rz)) return false;
    if (threadIdx.x == 0) sh.seq = seq;
    return group_sync();
}

__device__ __noinline__ void reweight_items(float delta)
{
    const ResShared &sh = res_shared();
    const int tid = (int)threadIdx.x % kItemThreads;
    for (int i = (int)threadIdx.x / kItemThreads; i < sh.nloc; i += kResEngines)
        phase_rw<double>(sh.T, sh.li[i], sh.K.P, delta, tid);
}

__device__ __noinline__ void final_items()
{
    const ResShared &sh = res_shared();
    const int tid = (int)threadIdx.x % kItemThreads;
    for (int i = (int)threadIdx.x / kItemThreads; i < sh.nloc; i += kResEngines)
        phase_final<double>(sh.T, sh.li[i], sh.K.P, tid);
}

/* Run all IRLS passes of one tile; false: a wait ran out. */
template <bool WLS> __device__ __forceinline__ bool run_tile()
{
    ResShared &sh = res_shared();
    const SolveParams &sp = sh.K.sp;
    setup_items();
    if (!group_sync(true)) return false;
    for (int outer = 0; outer <= sp.n_irls; ++outer) {
        double rz;
        if (!assemble<WLS>(outer == 0 && !(WLS && sp.warm), rz)) return false;
        if (threadIdx.x == 0) {
            sh.S = start_state(rz, sp);
            sh.beta = 0.0;
            sh.active = sh.S.active;
        }
        load_items();
        if (sh.active && !iterate()) return false;
        count_pass(outer);
        store_items();
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
__global__ void __launch_bounds__(kResThreads, 1) k_resident64(const __grid_constant__ ResParams K)
{
    resident_blocks(
        K,
        [](const ResTile &R) {
            ResShared &sh = res_shared();
            sh.own.g = R.g;
            sh.nloc = res_count(sh.T.nitems, sh.member, R.g);
        },
        [] { return run_tile<WLS>(); });
}

}  // namespace

int launch_resident_fp64(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                         SolverCtl *ctl, const SolveParams &sp, cudaStream_t s)
{
    const ResParams K = {tiles, A, P, ctl, sp};
    return sp.wls ? resident_start(k_resident64<true>, kResSmem, K, s)
                  : resident_start(k_resident64<false>, kResSmem, K, s);
}

}  // namespace cuphu
