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
#include "solver.cuh"
#include "resident.cuh"

#include <algorithm>
#include <cmath>
#include <cuda/atomic>
#include <vector>

namespace cuphu {

constexpr int kResEngines = 2;                          /* 256-thread engines per block */
constexpr int kResThreads = kResEngines * kItemThreads;
constexpr int kResPerEngine = kResItems / kResEngines;
constexpr int kRim = 2 * kItemBx + 2 * kItemBy;         /* halo pixels of an item */
constexpr int kPnW = kItemBx + 8;                       /* p row: 4 columns each side */
constexpr int kPnN = (kItemBy + 2) * kPnW;
constexpr int kWdN = (kItemBy + 1) * kItemBx;           /* down arcs, one row above */
constexpr int kWrW2 = kItemBx + 4;                      /* right arcs, 4 columns left */
constexpr int kWrN = kItemBy * kWrW2;
constexpr int kRimF = 2 * kRim;                         /* r and M^-1 of the halo ring */
constexpr int kResItemF = kPnN + kWdN + kWrN + kRimF;   /* floats of an item */
constexpr int kTmemCols = 512;
static_assert(2 * kResEngines * kResPerEngine * 16 <= kTmemCols, "TMEM columns");

/* The kernel's parameters. */
struct ResParams {
    const TileDesc *tiles;
    ResidentArgs A;
    SolverPlanes P;
    SolverCtl *ctl;
    SolveParams sp;
};

/* What the threads of a block share about the tile in progress.  Nothing of
 * it is kept in registers or on the stack: the block's shared memory leaves
 * next to no L1, so a spilled word costs a trip to the L2. */
struct ResShared {
    ResParams K;
    double red[kResItems][kNComp][8];   /* warp sums per item and component */
    double part[kNComp];                /* the block's partials */
    double tot[kResThreads / 32][kNComp];   /* warp sums of an exchange */
    TileDesc T;
    TileState S;                        /* the tile's PCG scalars (thread 0) */
    unsigned *bar;                      /* barrier of the group */
    unsigned bar_target, nact;
    int g, member, nloc;                /* group of 2^g, this block's member, its items */
    int skip;                           /* failure test: do not arrive at the next barrier */
    unsigned nbr[kResItems][4];         /* packet base of the rim sources: above,
                                           below, left, right (~0: outside) */
    int li[kResItems];
    unsigned short phys[kResMembers];
    float alpha, beta;
    int active, k;                      /* pass number of the IRLS pass's solve */
    unsigned seq;                       /* number of the last exchange */
    uint32_t tmem;
};
/* The block's dynamic shared memory: ResShared, then the items.  Every
 * function starts from here, so its accesses are shared-memory accesses with
 * 32-bit addresses (through a pointer argument they would be generic ones, at
 * twice the instructions). */
extern __shared__ __align__(128) char res_smem[];
constexpr int kResSharedB = (int)((sizeof(ResShared) + 127) & ~(size_t)127);
__device__ __forceinline__ ResShared &res_shared() { return *reinterpret_cast<ResShared *>(res_smem); }
__device__ __forceinline__ float *res_items()
{
    return reinterpret_cast<float *>(res_smem + kResSharedB);
}
constexpr size_t kResSmem = (size_t)kResItems * kResItemF * 4 + kResSharedB;
static_assert(kResSmem <= 232448, "shared memory of a block");

/* ── 128-bit packets ───────────────────────────────────────────────────── */
__device__ __forceinline__ void packet_store(void *p, unsigned long long lo, unsigned long long hi)
{
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}"
                 ::"l"(p), "l"(lo), "l"(hi)
                 : "memory");
}
__device__ __forceinline__ void packet_load(const void *p, unsigned long long &lo,
                                            unsigned long long &hi)
{
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
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

/* ── tensor memory as a register file ──────────────────────────────────────
 * A warp reaches the 32 lanes of its quarter (warp % 4); the warps that
 * share a quarter use different columns. */
__device__ __forceinline__ void tm_ld16(uint32_t a, uint32_t v[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15}, [%16];\n tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15])
        : "r"(a)
        : "memory");
}
__device__ __forceinline__ void tm_ld8(uint32_t a, uint32_t v[8])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n "
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7])
        : "r"(a)
        : "memory");
}
__device__ __forceinline__ void tm_ld4(uint32_t a, float v[4])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n "
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
        : "r"(a)
        : "memory");
}
__device__ __forceinline__ void tm_st8(uint32_t a, const float v[8])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
        : "memory");
}
__device__ __forceinline__ void tm_st4(uint32_t a, const float v[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a),
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
}
__device__ __forceinline__ void tm_wait_st()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
/* columns of an item: dx 0..3, r 4..7, M^-1 8..11, q 12..15 */
constexpr int kTmDx = 0, kTmR = 4, kTmQ = 12;

/* ── bounded waits ─────────────────────────────────────────────────────── */
struct Waiter {
    SolverCtl *ctl;
    long long limit_ns;
    unsigned long long t0;
    unsigned n;
    __device__ Waiter(SolverCtl *c, long long l) : ctl(c), limit_ns(l), t0(0), n(0) {}
    /* one more turn of a polling loop; false: give up (timeout, or another
     * block gave up) */
    __device__ __forceinline__ bool turn()
    {
        if ((++n & 63u) != 0) return true;
        if (*(volatile int *)&ctl->err) return false;
        const unsigned long long t = globaltimer();
        if (t0 == 0) {
            t0 = t;
        } else if ((long long)(t - t0) > limit_ns) {
            atomicExch(&ctl->err, 1);
            return false;
        }
        return true;
    }
};

/* Barrier over the blocks of a tile's group: the counter only grows, and
 * barrier number n is passed at n x (blocks of the group).  With
 * `any_progress` the wait may outlast the limit as long as some block of
 * the launch still finishes exchanges (a block that is free early waits here for
 * partners that are still in an earlier tile). */
__device__ __noinline__ bool group_sync(bool any_progress = false)
{
    ResShared &sh = res_shared();
    SolverCtl *ctl = sh.K.ctl;
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> cnt(*sh.bar);
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> beat(ctl->progress);
        const unsigned target = sh.bar_target + sh.nact;
        sh.bar_target = target;
        __threadfence();
        if (!sh.skip) cnt.fetch_add(1u, cuda::memory_order_acq_rel);
        sh.skip = 0;
        Waiter w(ctl, sh.K.sp.timeout_ns);
        unsigned seen = beat.load(cuda::memory_order_relaxed);
        while ((int)(cnt.load(cuda::memory_order_acquire) - target) < 0) {
            if (any_progress && (w.n & 63u) == 62u) {
                const unsigned b = beat.load(cuda::memory_order_relaxed);
                if (b != seen) {
                    seen = b;
                    w.t0 = 0;
                }
            }
            if (!w.turn()) {
                ok = false;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_and(ok);
}

/* ── geometry of a group ───────────────────────────────────────────────────
 * u = the slot's bits in the order the tree combines them (lane bits 4..0,
 * then warp bits 2..0); member = the low g bits of u, sub = the rest.  Local
 * items are numbered level by level (items 256 j + slot), and the last,
 * partial level is a prefix of the subs (res_last). */
__host__ __device__ __forceinline__ int res_slot(int u) { return ((u >> 3) & 31) | ((u & 7) << 5); }
__host__ __device__ __forceinline__ int res_u(int slot) { return ((slot & 31) << 3) | (slot >> 5); }
/* subs of member m that hold an item in a last level of `rem` items */
__host__ __device__ __forceinline__ int res_last(int rem, int m, int g)
{
    const int lanes = rem - 32 * (m & 7);          /* lanes of this warp in use */
    const int hi = m >> 3, step = g - 3;
    if (lanes <= hi) return 0;
    const int l = lanes < 32 ? lanes : 32;
    return (l - hi + (1 << step) - 1) >> step;
}
__host__ __device__ __forceinline__ int res_count(int nitems, int m, int g)
{
    return ((nitems >> 8) << (8 - g)) + res_last(nitems & 255, m, g);
}

/* A thread's view of its block. */
struct ResCtx {
    int eng, tid, warp, lane;
    int rim_at, rim_nb, rim_pk;   /* this thread's rim pixel of an item: place in the p array
                                     (-1: none), neighbour, packet */
    uint32_t tm;           /* this thread's TMEM columns of its engine's first item */

    __device__ __forceinline__ float *pn(int i) const { return res_items() + i * kResItemF; }
    __device__ __forceinline__ float *wd(int i) const { return pn(i) + kPnN; }
    __device__ __forceinline__ float *wr(int i) const { return pn(i) + kPnN + kWdN; }
    __device__ __forceinline__ float2 *rim(int i) const
    {
        return reinterpret_cast<float2 *>(pn(i) + kPnN + kWdN + kWrN);
    }
    __device__ __forceinline__ uint32_t tmem(int i) const
    {
        return tm + (uint32_t)(i / kResEngines) * 16u;
    }
};

__device__ __forceinline__ ResCtx make_ctx()
{
    const int warp = threadIdx.x >> 5;
    const int eng = (int)threadIdx.x / kItemThreads, tid = (int)threadIdx.x % kItemThreads;
    /* the halo ring of an item is the work of an engine's last 160 threads:
     * the rows above and below (the neighbour's last and first row), the
     * columns left and right (its last and first column) */
    int rim_at = -1, rim_nb = 0, rim_pk = 0;
    const int h = tid - (kItemThreads - kRim);
    if (h >= 2 * kItemBx + kItemBy) {
        const int r = h - 2 * kItemBx - kItemBy;
        rim_at = (r + 1) * kPnW + 4 + kItemBx; rim_nb = 3; rim_pk = 2 * kItemBx + r;
    } else if (h >= 2 * kItemBx) {
        const int r = h - 2 * kItemBx;
        rim_at = (r + 1) * kPnW + 3; rim_nb = 2; rim_pk = 2 * kItemBx + kItemBy + r;
    } else if (h >= kItemBx) {
        rim_at = (kItemBy + 1) * kPnW + 4 + h - kItemBx; rim_nb = 1; rim_pk = h - kItemBx;
    } else if (h >= 0) {
        rim_at = 4 + h; rim_nb = 0; rim_pk = kItemBx + h;
    }
    return ResCtx{eng, tid, warp, (int)threadIdx.x & 31, rim_at, rim_nb, rim_pk,
                  res_shared().tmem + ((uint32_t)(warp & 3) << 21) +
                      (uint32_t)(warp >> 2) * kResPerEngine * 16u};
}

/* A block's mailbox: [parity][member m][component] packets, in the order in
 * which the threads read them (thread 32 w + 4 h + c: member 16 h + w,
 * component c). */
constexpr int kMailN = 2 * kNComp * kResMembers;
__device__ __forceinline__ ulonglong2 *mail_of(const ResCtx &C, int block, unsigned seq, int m, int c)
{
    return res_shared().K.A.mail + (size_t)block * kMailN + (seq & 1u) * (kNComp * kResMembers) +
           ((m & 15) << 5) + ((m >> 4) << 2) + c;
}

/* The block's partials into sh.part: warp c forms the items' partials of
 * component c (lanes 2 i + h hold the half tree of warp parity h), then the
 * slot sums (items of a slot in order) and the butterfly levels inside the
 * block. */
__device__ __forceinline__ void block_partials(const ResCtx &C, int ncomp)
{
    if (C.warp >= ncomp) return;
    const int c = C.warp, i = C.lane >> 1, h = C.lane & 1;
    double v = 0.0;
    if (i < res_shared().nloc) {
        const double *w = res_shared().red[i][c];
        v = (w[h] + w[h + 4]) + (w[h + 2] + w[h + 6]);
    }
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    const int slog = 8 - res_shared().g, S = 1 << slog, sub = C.lane & (S - 1);
    double a = 0.0;
    for (int k = 0; k < res_shared().nloc; k += S) {
        const double x = __shfl_sync(0xffffffffu, v, (2 * (k + sub)) & 31);
        if (k + sub < res_shared().nloc) a += x;
    }
    for (int off = S >> 1; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if (C.lane == 0) res_shared().part[c] = a;
}

/* Send the block's partials to every block of the group and ask for nothing
 * yet: thread 4 d + c stores component c into member d's mailbox. */
__device__ __forceinline__ void send_partials(const ResCtx &C, int ncomp, unsigned seq)
{
    static_assert(kResThreads == kNComp * kResMembers, "one packet per thread");
    __syncthreads();
    const int d = threadIdx.x >> 2, c = threadIdx.x & 3;
    if (c < ncomp && d < (1 << res_shared().g)) {
        const unsigned ph = res_shared().phys[d];
        if (ph != 0xffffu)
            packet_store(mail_of(C, ph, seq, res_shared().member, c),
                         (unsigned long long)__double_as_longlong(res_shared().part[c]),
                         (unsigned long long)seq);
    }
}

/* Wait for exchange `seq` and finish the tree; the totals are returned in warp
 * 0.  One hop: every member stores its packets into every mailbox (8 KB per
 * block and exchange), and a thread polls one packet of its own block's
 * mailbox.  Measured for 128 blocks, from the stores to the totals: 1900 cycles,
 * against 4900 when one block per component collects and publishes (two
 * hops) and 7500 when every block polls the members' own copies (128 readers
 * of each line).  The members' bits combine
 * from the top: three levels across the lanes, four across the warps. */
template <int NCOMP>
__device__ __forceinline__ bool totals(const ResCtx &C, unsigned seq, double out[NCOMP])
{
    const int c = C.lane & 3, m = ((C.lane >> 2) << 4) | C.warp;
    unsigned long long lo = 0;
    bool ok = true;
    if (c < NCOMP && m < (1 << res_shared().g) && res_shared().phys[m] != 0xffffu) {
        const ulonglong2 *p = mail_of(C, blockIdx.x, seq, m, c);
        unsigned long long hi;
        packet_load(p, lo, hi);
        if (hi != (unsigned long long)seq) {
            Waiter w(res_shared().K.ctl, res_shared().K.sp.timeout_ns);
            do {
                if (!w.turn()) {
                    ok = false;
                    break;
                }
                packet_load(p, lo, hi);
            } while (hi != (unsigned long long)seq);
        }
    }
    __syncwarp();
    double v = __longlong_as_double((long long)lo);
#pragma unroll
    for (int off = 16; off >= 4; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (C.lane < NCOMP) res_shared().tot[C.warp][C.lane] = v;
    ok = __syncthreads_and(ok);
    if (C.warp == 0) {
        const int k = C.lane >> 2;
        v = c < NCOMP ? res_shared().tot[k][c] + res_shared().tot[k + 8][c] : 0.0;
#pragma unroll
        for (int off = 16; off >= 4; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
#pragma unroll
        for (int j = 0; j < NCOMP; ++j) out[j] = __shfl_sync(0xffffffffu, v, j);
    }
    return ok;
}

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
    float *Pn = C.pn(i), *WD = C.wd(i), *WR = C.wr(i);
    float rv[4] = {0.f, 0.f, 0.f, 0.f};
    if (own) {
        ld4((const float *)res_shared().K.P.z + T.pix + (size_t)r * T.pitch + c0, rv);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (c0 + j >= T.nc) rv[j] = 0.f;
    }
    __syncwarp();
    const float zr[8] = {0.f, 0.f, 0.f, 0.f, rv[0], rv[1], rv[2], rv[3]};
    tm_st8(C.tmem(i), zr);
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
        tm_st8(C.tmem(i) + 8, m);
    } else {
        tm_st4(C.tmem(i) + kTmQ, m + 4);
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
        tm_ld16(C.tmem(i), t);
        float *Pn = C.pn(i);
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
        tm_st8(C.tmem(i), nd);
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
            float *p = C.pn(i) + C.rim_at;
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
            float2 *st = C.rim(i) + (C.tid - (kItemThreads - kRim));
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
    const float beta = sh.beta;
    const int so = (C.tid / kItemTx + 1) * kPnW + 4 + (C.tid % kItemTx) * kItemVx;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        uint32_t t[8];
        tm_ld8(C.tmem(i) + kTmR, t);
        float *Pn = C.pn(i);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            Pn[so + j] = __fmaf_rn(beta, Pn[so + j],
                                   __fmul_rn(__uint_as_float(t[j]), __uint_as_float(t[4 + j])));
        if (C.rim_at >= 0 && sh.nbr[i][C.rim_nb] != ~0u) {
            const int li = sh.li[i];
            const float2 rm = fresh_rim(C, (li / sh.T.nbx) * kItemBy - 1 + C.rim_at / kPnW,
                                        (li % sh.T.nbx) * kItemBx - 4 + C.rim_at % kPnW);
            C.rim(i)[C.tid - (kItemThreads - kRim)] = rm;
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
        const float *Pn = C.pn(i), *WD = C.wd(i), *WR = C.wr(i);
        uint32_t t[8];
        tm_ld8(C.tmem(i) + kTmR, t);
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
        tm_st4(C.tmem(i) + kTmQ, qv);
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
    const float alpha = sh.alpha;
    const TileDesc &T = res_shared().T;
    const int ty = C.tid / kItemTx, tx = C.tid % kItemTx;
    for (int i = C.eng; i < res_shared().nloc; i += kResEngines) {
        float dx[4];
        tm_ld4(C.tmem(i) + kTmDx, dx);
        const int li = res_shared().li[i];
        const int r = (li / T.nbx) * kItemBy + ty, c0 = (li % T.nbx) * kItemBx + tx * kItemVx;
        if (r < T.nr && c0 < T.nc) {
            double *x = res_shared().K.P.x + T.pix + (size_t)r * T.pitch + c0;
            const float *p = C.pn(i) + (ty + 1) * kPnW + 4 + tx * kItemVx;
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
        if (!half1(C, sh.alpha, sh.beta, seq, A)) return kGaveUp;
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

/* this block's items of the tile, their rim sources; the packets of an
 * earlier tile are voided */
__device__ __noinline__ void setup_items()
{
    ResShared &sh = res_shared();
    const ResParams &K = sh.K;
    const TileDesc &T = sh.T;
    if (threadIdx.x < kResItems) {
        const int i = threadIdx.x, slog = 8 - sh.g;
        const int u = ((i & ((1 << slog) - 1)) << sh.g) | sh.member;
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
                    const int v = res_u(n & 255), m = v & ((1 << sh.g) - 1);
                    base = ((unsigned)sh.phys[m] * kResItems + ((n >> 8) << slog) + (v >> sh.g)) *
                           2 * kRim;
                }
                sh.nbr[i][k] = base;
            }
        }
    }
    for (int k = threadIdx.x; k < sh.nloc * 2 * kRim; k += kResThreads)
        rim_store(K.A.rim + blockIdx.x * kResItems * 2 * kRim + k, 0.f, 0u);
    for (int k = threadIdx.x; k < kMailN; k += kResThreads)
        packet_store(K.A.mail + (size_t)blockIdx.x * kMailN + k, 0ull, 0ull);
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
            sh.alpha = 0.f;
            sh.beta = 0.f;
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
                sh.alpha = 0.f;
            }
            load_items(false);
        }
        if (sh.member == 0 && threadIdx.x == 0) {
            atomicAdd(&K.ctl->progress, 1u);
            atomicAdd(&K.ctl->px_iters, (unsigned long long)S.iter *
                                            (unsigned long long)((long long)sh.T.nr * sh.T.nc));
            atomicMax(&sp.pass_iters[outer], S.iter);
        }
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
__global__ void __launch_bounds__(kResThreads, 1)
    k_resident(const __grid_constant__ ResParams K)
{
    ResShared &sh = res_shared();
    for (int k = threadIdx.x; k < (int)(sizeof(ResParams) / 4); k += kResThreads)
        reinterpret_cast<uint32_t *>(&sh.K)[k] = reinterpret_cast<const uint32_t *>(&K)[k];
    const int warp = threadIdx.x >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&sh.tmem)),
                     "n"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int w0 = K.A.blk_off[blockIdx.x], w1 = K.A.blk_off[blockIdx.x + 1];
    for (int w = w0; w < w1; ++w) {
        const ResWork W = K.A.work[w];
        const ResTile R = K.A.sched[W.sched];
        __syncthreads();   /* the last tile's reads of sh are done */
        for (int k = threadIdx.x; k < (1 << R.g); k += kResThreads)
            sh.phys[k] = K.A.phys[R.phys0 + k];
        if (threadIdx.x == 0) {
            sh.T = K.tiles[R.tile];
            sh.bar = K.A.bars + W.sched;
            sh.bar_target = 0u;
            sh.nact = (unsigned)R.nact;
            sh.g = R.g;
            sh.member = W.member;
            sh.nloc = res_count(sh.T.nitems, W.member, R.g);
            sh.skip = w == w0 && (int)blockIdx.x == K.sp.skip_block;
        }
        __syncthreads();
        if (!run_tile<WLS>()) break;
    }
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem),
                     "n"(kTmemCols));
}

/* ── host: which tiles, on which blocks ─────────────────────────────────── */

/* most items any block of a group of 2^g holds */
static int res_most(int nitems, int g)
{
    int most = 0;
    for (int m = 0; m < (1 << g); ++m) most = std::max(most, res_count(nitems, m, g));
    return most;
}

bool resident_fits(int nitems) { return res_most(nitems, kResMaxG) <= kResItems; }

/* Choose the group sizes and the schedule.  An iteration of a tile costs about
 * c0 + c1 x (most items of one block): c0 the exchange, c1 one item (both
 * measured, in us).  Small groups spread the exchange over more work per block
 * and let many tiles run side by side; large ones shorten a tile's
 * iteration.  The bound k on the items of a block that gives the smallest
 * estimated makespan over the job's tiles is taken. */
void plan_resident(const std::vector<TileDesc> &tiles, int nblk, ResidentPlan &R)
{
    constexpr double c0 = 3.8, c1 = 0.6;
    R = ResidentPlan();
    std::vector<int> fit;
    for (int t = 0; t < (int)tiles.size(); ++t)
        if (resident_fits(tiles[t].nitems) && nblk >= (1 << kResMaxG)) fit.push_back(t);
        else R.streamed.push_back(t);
    if (fit.empty()) return;
    auto shape = [&](int nitems, int k, int &g, int &most) {
        for (g = 3; g < kResMaxG; ++g)
            if ((most = res_most(nitems, g)) <= k) return;
        most = res_most(nitems, g);
    };
    auto active = [&](int nitems, int g) {
        int a = 0;
        for (int m = 0; m < (1 << g); ++m) a += res_count(nitems, m, g) > 0;
        return a;
    };
    int best_k = kResItems;
    double best = 0.0;
    for (int k = 1; k <= kResItems; ++k) {
        double area = 0.0, longest = 0.0;
        for (int t : fit) {
            int g, most;
            shape(tiles[t].nitems, k, g, most);
            const int a = active(tiles[t].nitems, g);
            const double d = std::sqrt((double)tiles[t].nitems) * (c0 + c1 * most);
            /* groups that do not pack waste the blocks left over */
            area += d / (nblk / a);
            longest = std::max(longest, d);
        }
        const double est = std::max(area, longest);
        if (k == 1 || est < best) {
            best = est;
            best_k = k;
        }
    }
    struct Job { int t, g, a; double d; };
    std::vector<Job> jobs;
    for (int t : fit) {
        int g, most;
        shape(tiles[t].nitems, best_k, g, most);
        jobs.push_back({t, g, active(tiles[t].nitems, g),
                        std::sqrt((double)tiles[t].nitems) * (c0 + c1 * most)});
    }
    std::stable_sort(jobs.begin(), jobs.end(), [](const Job &a, const Job &b) { return a.d > b.d; });
    /* longest first onto the blocks that are free first; blocks process
     * their tiles in this order, so the first unfinished tile of the order
     * always has all its blocks */
    std::vector<double> load(nblk, 0.0);
    std::vector<std::vector<ResWork>> per(nblk);
    std::vector<int> idx(nblk);
    for (const Job &j : jobs) {
        for (int b = 0; b < nblk; ++b) idx[b] = b;
        std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return load[a] < load[b]; });
        const double start = load[idx[j.a - 1]];
        const int sched = (int)R.sched.size();
        R.sched.push_back({j.t, j.g, j.a, (int)R.phys.size()});
        int used = 0;
        for (int m = 0; m < (1 << j.g); ++m) {
            if (res_count(tiles[j.t].nitems, m, j.g) == 0) {
                R.phys.push_back(0xffff);
                continue;
            }
            const int b = idx[used++];
            R.phys.push_back((unsigned short)b);
            per[b].push_back({sched, m});
            load[b] = start + j.d;
        }
    }
    R.blk_off.push_back(0);
    for (int b = 0; b < nblk; ++b) {
        R.work.insert(R.work.end(), per[b].begin(), per[b].end());
        R.blk_off.push_back((int)R.work.size());
    }
    /* blocks without work at the end of the grid are not launched */
    R.nblk = nblk;
    while (R.nblk > 1 && per[R.nblk - 1].empty()) --R.nblk;
}

size_t resident_rim_bytes(int nblk) { return (size_t)nblk * kResItems * 2 * kRim * 8; }
size_t resident_mail_bytes(int nblk) { return (size_t)nblk * kMailN * sizeof(ulonglong2); }

template <bool WLS> static int launch_resident_t(const ResParams &K, cudaStream_t s)
{
    auto kern = k_resident<WLS>;
    CUPHU_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kResSmem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(K.A.nblk);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = kResSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   /* all blocks resident: they wait on one another */
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUPHU_TRY_CUDA(cudaLaunchKernelEx(&cfg, kern, K));
    return 0;
}

int launch_resident(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                    SolverCtl *ctl, const SolveParams &sp, cudaStream_t s)
{
    ResParams K = {tiles, A, P, ctl, sp};
    K.P.dx = nullptr;   /* the increment lives in TMEM */
    return sp.wls ? launch_resident_t<true>(K, s) : launch_resident_t<false>(K, s);
}

}  // namespace cuphu
