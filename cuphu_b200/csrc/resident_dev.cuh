/*
 * resident_dev.cuh -- what the two on-chip solver kernels (resident.cu: mixed
 * precision, resident_fp64.cu) share: the block's shared state, packets,
 * tensor memory, bounded waits, the group's barrier and geometry, and the
 * exchange of partial sums.  A kernel's file defines kResItems (items of a
 * block) and kResCols (TMEM columns of an item) before it includes this; all
 * of it has internal linkage.
 */
#include "resident_geom.cuh"
#include "solver.cuh"

#include <cuda/atomic>

namespace cuphu {
namespace {

constexpr int kResEngines = 2;                          /* 256-thread engines per block */
constexpr int kResThreads = kResEngines * kItemThreads;
constexpr int kResPerEngine = kResItems / kResEngines;
constexpr int kRim = 2 * kItemBx + 2 * kItemBy;         /* halo pixels of an item */
constexpr int kPnW = kItemBx + 8;                       /* p row: 4 columns each side */
constexpr int kPnN = (kItemBy + 2) * kPnW;
constexpr int kWdN = (kItemBy + 1) * kItemBx;           /* down arcs, one row above */
constexpr int kWrW2 = kItemBx + 4;                      /* right arcs, 4 columns left */
constexpr int kWrN = kItemBy * kWrW2;
constexpr int kTmemCols = 512;
static_assert(2 * kResEngines * kResPerEngine * kResCols <= kTmemCols, "TMEM columns");

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
    double alpha, beta;                 /* the mixed solve's are floats */
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
__device__ __forceinline__ char *res_items() { return res_smem + kResSharedB; }
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

/* A thread's view of its block. */
struct ResCtx {
    int eng, tid, warp, lane;
    int rim_at, rim_nb, rim_pk;   /* this thread's rim pixel of an item: place in the p array
                                     (-1: none), neighbour, packet */
    uint32_t tm;           /* this thread's TMEM columns of its engine's first item */
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
                      (uint32_t)(warp >> 2) * (kResPerEngine * kResCols)};
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

/* void the k-th rim packet of this block (each kernel has its own kind) */
__device__ __forceinline__ void rim_void(int k);

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
        rim_void(k);
    for (int k = threadIdx.x; k < kMailN; k += kResThreads)
        packet_store(K.A.mail + (size_t)blockIdx.x * kMailN + k, 0ull, 0ull);
    if (threadIdx.x == 0) sh.seq = 0u;
}

/* The body of both kernels: take tensor memory, run this block's part of its
 * tiles in order, give the tensor memory back. */
template <typename Run> __device__ __forceinline__ void resident_blocks(const ResParams &K, Run run)
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
        if (!run()) break;
    }
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem),
                     "n"(kTmemCols));
}

/* a tile's pass is over: count it (one thread per tile) */
__device__ __forceinline__ void count_pass(int outer)
{
    ResShared &sh = res_shared();
    if (sh.member != 0 || threadIdx.x != 0) return;
    atomicAdd(&sh.K.ctl->progress, 1u);
    atomicAdd(&sh.K.ctl->px_iters, (unsigned long long)sh.S.iter *
                                       (unsigned long long)((long long)sh.T.nr * sh.T.nc));
    atomicMax(&sh.K.sp.pass_iters[outer], sh.S.iter);
}

template <typename Kern>
int resident_start(Kern kern, size_t smem, const ResParams &K, cudaStream_t s)
{
    CUPHU_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(K.A.nblk);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   /* all blocks resident: they wait on one another */
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUPHU_TRY_CUDA(cudaLaunchKernelEx(&cfg, kern, K));
    return 0;
}

}  // namespace
}  // namespace cuphu
