/*
 * resident_dev.cuh -- what the two on-chip solver kernels (resident.cu: mixed
 * precision, resident_fp64.cu) share: the block's shared state, packets,
 * tensor memory, bounded waits, the group's barrier, and the launch.  A kernel's file defines ResOwn (its own part of the shared state)
 * before it includes this; all of it has internal linkage.
 */
#include "solver.cuh"

#include <cuda/atomic>

namespace cuphu {
namespace {

constexpr int kResEngines = 2;                          /* 256-thread engines per block */
constexpr int kResThreads = kResEngines * kItemThreads;
constexpr int kTmemCols = 512;
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
    ResOwn own;                         /* the kernel's own part */
    TileDesc T;
    TileState S;                        /* the tile's PCG scalars (thread 0) */
    unsigned *bar;                      /* barrier of the group */
    unsigned bar_target, nact;          /* blocks of the group */
    int member, nloc;                   /* this block's member number and items */
    int skip;                           /* failure test: do not arrive at the next barrier */
    int li[kResItemsMixed];             /* the items, by number in the tile */
    unsigned short phys[kResMaxBlocks]; /* the members' blocks */
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

/* Poll until `there()` holds in every lane of the warp; all lanes read in every
 * turn.  (Where each lane leaves the loop by itself, the lanes still waiting
 * issue their reads one after the other, over 1000 cycles each: at 512 x 512
 * an iteration took 4.4 us instead of 3.3.)  false: gave up. */
template <typename There>
__device__ __forceinline__ bool poll_together(ResShared &sh, There there)
{
    Waiter w(sh.K.ctl, sh.K.sp.timeout_ns);
    while (true) {
        const bool t = there();
        if (__all_sync(0xffffffffu, t)) return true;
        if (!__all_sync(0xffffffffu, w.turn())) return false;
    }
}

/* Barrier over the blocks of a tile's group: the counter only grows, and
 * barrier number n is passed at n x (blocks of the group).  With
 * `any_progress` the wait may outlast the limit as long as some block of
 * the launch still finishes exchanges (a block that is free early waits here for
 * partners that are still in an earlier tile).  Every running tile counts its
 * progress up after each eighth iteration, whatever follows it, so the limit
 * only has to cover eight iterations with their residual replacements (0.3 ms
 * for tiles of 1000 x 1000 pixels, two side by side). */
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

/* The body of both kernels: take tensor memory, run this block's part of its
 * tiles in order, give the tensor memory back.  begin(R) sets the kernel's
 * own part for a tile (one thread); run() returns false when a wait ran
 * out. */
template <typename Begin, typename Run>
__device__ __forceinline__ void resident_blocks(const ResParams &K, Begin begin, Run run)
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
        for (int k = threadIdx.x; k < R.nmem; k += kResThreads)
            sh.phys[k] = K.A.phys[R.phys0 + k];
        if (threadIdx.x == 0) {
            sh.T = K.tiles[R.tile];
            sh.bar = K.A.bars + W.sched;
            sh.bar_target = 0u;
            sh.nact = (unsigned)R.nact;
            sh.member = W.member;
            begin(R);
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
