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
 */
#include "resident.cuh"

namespace cuphu {
namespace {
constexpr int kResItems = kResItems64;
constexpr int kResCols = 32;   /* x, r, diag and 1/diag of four pixels */
}  // namespace
}  // namespace cuphu
#include "resident_dev.cuh"

namespace cuphu {
namespace {

constexpr int kResItemD = kPnN + kWdN + kWrN;   /* doubles of an item */
constexpr size_t kResSmem = (size_t)kResItems * kResItemD * 8 + kResSharedB;
static_assert(kResSmem <= 232448, "shared memory of a block");

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
/* columns of an item */
constexpr int kTmX = 0, kTmR = 8, kTmD = 16, kTmY = 24;

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

__device__ __forceinline__ void unpack4(const uint32_t *t, double v[4])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __hiloint2double((int)t[2 * j + 1], (int)t[2 * j]);
}
__device__ __forceinline__ void tm_st4d(uint32_t a, const double v[4])
{
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        f[2 * j] = __int_as_float(__double2loint(v[j]));
        f[2 * j + 1] = __int_as_float(__double2hiint(v[j]));
    }
    tm_st8(a, f);
}
__device__ __forceinline__ void lds4(const double *p, double v[4])
{
    const double2 a = reinterpret_cast<const double2 *>(p)[0];
    const double2 b = reinterpret_cast<const double2 *>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

/* r / d from y = RN(1/d).  The correction steps are exact where nothing
 * underflows or overflows; a residual outside [2^-900, 2^900] and a diagonal
 * outside [2^-100, 2^100] (y = 0 marks it) take the IEEE division. */
__device__ __forceinline__ double quotient(double r, double d, double y)
{
    const double q0 = __dmul_rn(r, y);
    const double q1 = __fma_rn(__fma_rn(-q0, d, r), y, q0);
    double q = __fma_rn(__fma_rn(-q1, d, r), y, q1);
    const unsigned e = ((unsigned)__double2hiint(r) & 0x7fffffffu) - (123u << 20);
    if ((e > (1800u << 20) || __double2hiint(y) == 0) && r != 0.0) q = __ddiv_rn(r, d);
    return q;
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
        }
        __syncwarp();
        tm_st4d(tm_of(C, i) + kTmX, xv);
        tm_st4d(tm_of(C, i) + kTmR, rv);
        tm_st4d(tm_of(C, i) + kTmD, dv);
        tm_st4d(tm_of(C, i) + kTmY, yv);
        for (int k = C.tid; k < kPnN; k += kItemThreads) Pn[k] = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            WD[(ty + 1) * kItemBx + tx * kItemVx + j] = (double)wdn[j];
            WR[ty * kWrW2 + 4 + tx * kItemVx + j] = (double)wrt[j];
            if (ty == 0) WD[tx * kItemVx + j] = (double)up[j];
        }
        if (tx == 0) WR[ty * kWrW2 + 3] = (double)lf;
        __syncwarp();
    }
    tm_wait_st();
    __syncthreads();
}

/* x of the block's items back to its plane */
__device__ __noinline__ void store_items()
{
    const ResCtx C = make_ctx();
    const ResShared &sh = res_shared();
    const TileDesc &T = sh.T;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        uint32_t t[8];
        tm_ld8(tm_of(C, i) + kTmX, t);
        double xv[4];
        unpack4(t, xv);
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
    if (C.lane == 0) res_shared().red[i][0][C.warp & 7] = v;
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
            const unsigned base = sh.nbr[i][C.rim_nb];
            if (base != ~0u)
                packet_load(rim_at(base + (seq & 1u) * kRim + C.rim_pk), A.lo[x], A.hi[x]);
        }
    }
}

/* p = z + beta p of the block's items and their halo rings (z of the rims
 * from the plane right after an assembly, else from the packets of exchange
 * `seq`) */
__device__ __forceinline__ bool fold_p(const ResCtx &C, double beta, bool first, unsigned seq,
                                       const RimAsk &A)
{
    const ResShared &sh = res_shared();
    const int so = (C.tid / kItemTx + 1) * kPnW + 4 + (C.tid % kItemTx) * kItemVx;
    for (int i = C.eng; i < sh.nloc; i += kResEngines) {
        uint32_t t[16], u[8];
        tm_ld16(tm_of(C, i) + kTmR, t);
        tm_ld8(tm_of(C, i) + kTmY, u);
        double rv[4], dv[4], yv[4], pv[4];
        unpack4(t, rv);
        unpack4(t + 8, dv);
        unpack4(u, yv);
        double *Pn = pn_of(i) + so;
        lds4(Pn, pv);
#pragma unroll
        for (int j = 0; j < 4; ++j) pv[j] = __fma_rn(beta, pv[j], quotient(rv[j], dv[j], yv[j]));
        reinterpret_cast<double2 *>(Pn)[0] = make_double2(pv[0], pv[1]);
        reinterpret_cast<double2 *>(Pn)[1] = make_double2(pv[2], pv[3]);
        __syncwarp();
    }
    bool ok = true;
    if (C.rim_at >= 0) {
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= sh.nloc) continue;
            const unsigned base = sh.nbr[i][C.rim_nb];
            if (base == ~0u) continue;   /* outside the tile: p stays zero */
            double z;
            if (first) {
                const int li = sh.li[i], gr = (li / sh.T.nbx) * kItemBy - 1 + C.rim_at / kPnW;
                const int gc = (li % sh.T.nbx) * kItemBx - 4 + C.rim_at % kPnW;
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
    const int so = (ty + 1) * kPnW + 4 + tx * kItemVx;
    unsigned seq = sh.seq;
    RimAsk A;
    bool first = true;
    while (true) {
        if (!fold_p(C, sh.beta, first, seq, A)) return false;
        first = false;
        /* q = A p and p.q, in k_solve's order (an arc outside the tile has
         * weight zero and adds nothing) */
        double q[kResPerEngine][4];
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= sh.nloc) continue;
            const double *Pn = pn_of(i), *WD = wd_of(i), *WR = wr_of(i);
            double pn[4], up[4], dn[4], wdn[4], wup[4], wrt[4];
            lds4(Pn + so, pn);
            lds4(Pn + so - kPnW, up);
            lds4(Pn + so + kPnW, dn);
            lds4(WD + (ty + 1) * kItemBx + tx * kItemVx, wdn);
            lds4(WD + ty * kItemBx + tx * kItemVx, wup);
            lds4(WR + ty * kWrW2 + 4 + tx * kItemVx, wrt);
            const double lf = Pn[so - 1], rt = Pn[so + 4], wlf = WR[ty * kWrW2 + 3 + tx * kItemVx];
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double xa = pn[j];
                const double xl = j == 0 ? lf : pn[j - 1], xr = j == 3 ? rt : pn[j + 1];
                double y = (double)kLapEpsF * xa;
                y = __fma_rn(wdn[j], xa - dn[j], y);
                y = __fma_rn(wup[j], xa - up[j], y);
                y = __fma_rn(wrt[j], xa - xr, y);
                y = __fma_rn(j == 0 ? wlf : wrt[j - 1], xa - xl, y);
                q[x][j] = y;
                acc = __fma_rn(xa, y, acc);
            }
            item_sum(C, i, acc);
        }
        __syncthreads();
        block_partials(C, 1);
        send_partials(C, 1, ++seq);
        double tot[1];
        if (!totals<1>(C, seq, tot)) return false;
        if (threadIdx.x == 0) {
            if (tot[0] <= 0.0) sh.active = 0;
            else sh.alpha = S.rz / tot[0];
        }
        __syncthreads();
        if (!sh.active) break;
        /* x += alpha p, r -= alpha q, z = r / diag, r.z; the rims' z */
        const double alpha = sh.alpha;
        ++seq;
#pragma unroll
        for (int x = 0; x < kResPerEngine; ++x) {
            const int i = x * kResEngines + C.eng;
            if (i >= sh.nloc) continue;
            uint32_t t[16], u[16];
            tm_ld16(tm_of(C, i) + kTmX, t);
            tm_ld16(tm_of(C, i) + kTmD, u);
            double xv[4], rv[4], dv[4], yv[4], pv[4], zv[4], acc = 0.0;
            unpack4(t, xv);
            unpack4(t + 8, rv);
            unpack4(u, dv);
            unpack4(u + 8, yv);
            lds4(pn_of(i) + so, pv);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                xv[j] = __fma_rn(alpha, pv[j], xv[j]);
                rv[j] = __fma_rn(-alpha, q[x][j], rv[j]);
                zv[j] = quotient(rv[j], dv[j], yv[j]);
                acc = __fma_rn(rv[j], zv[j], acc);
            }
            __syncwarp();
            tm_st4d(tm_of(C, i) + kTmX, xv);
            tm_st4d(tm_of(C, i) + kTmR, rv);
            ulonglong2 *rim = rim_at(((blockIdx.x * kResItems + i) * 2 + (seq & 1u)) * kRim);
            if (ty == 0 || ty == kItemBy - 1) {
                ulonglong2 *d = rim + (ty == 0 ? 0 : kItemBx) + tx * kItemVx;
#pragma unroll
                for (int j = 0; j < 4; ++j) rim_store(d + j, zv[j], seq);
            }
            if (tx == 0) rim_store(rim + 2 * kItemBx + ty, zv[0], seq);
            if (tx == kItemTx - 1) rim_store(rim + 2 * kItemBx + kItemBy + ty, zv[3], seq);
            __syncwarp();
            item_sum(C, i, acc);
        }
        tm_wait_st();
        __syncthreads();
        block_partials(C, 1);
        send_partials(C, 1, seq);
        rim_ask(C, seq, A);
        if (!totals<1>(C, seq, tot)) return false;
        if (threadIdx.x == 0) {
            const int it = S.iter + 1;
            S.iter = it;
            if (tot[0] < S.thr || it >= sh.K.sp.max_iter) {
                sh.active = 0;
            } else {
                sh.beta = tot[0] / S.rz;
                S.rz = tot[0];
            }
            if ((it & 63) == 63 && sh.member == 0) atomicAdd(&sh.K.ctl->progress, 1u);
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
    block_partials(C, 1);
    send_partials(C, 1, seq);
    if (!totals<1>(C, seq, &rz)) return false;
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
    resident_blocks(K, [] { return run_tile<WLS>(); });
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
