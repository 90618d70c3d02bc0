/*
 * solver.cuh -- device functions the Laplace solver's kernels share: vector
 * access, the mixed solve's preconditioner and dots, and the per-pass phases
 * (assembly / true residual, IRLS reweight, anchor + congruence) of one work
 * item.  laplace.cu streams the items of a job through its blocks;
 * resident.cu keeps a tile's items on the chip.  Both call these functions,
 * so their results agree bit for bit.
 */
#pragma once

#include "kernels.cuh"

namespace cuphu {

/* ── vector access helpers (L2-coherent loads of in-kernel-written data) ── */
__device__ __forceinline__ void ld4(const float *p, float v[4])
{
    float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void ld4(const double *p, double v[4])
{
    double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
    double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void st4(float *p, const float v[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st4(double *p, const double v[4])
{
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
}
template <typename T> __device__ __forceinline__ T ldc(const T *p) { return __ldcg(p); }

/* warp sums of four values by a reduce-scatter tree: after the xor-16 and
 * xor-8 steps each lane holds one component (lanes 8c..8c+7 component c),
 * then three plain levels; every lane of group c returns the warp's sum of
 * component c (the same value in all eight lanes) */
__device__ __forceinline__ double warp_scatter4(const double a[kNComp])
{
    static_assert(kNComp == 4, "four components");
    const int lane = threadIdx.x & 31;
    const bool hi16 = lane & 16, hi8 = lane & 8;
    const double r0 = __shfl_xor_sync(0xffffffffu, hi16 ? a[0] : a[2], 16);
    const double r1 = __shfl_xor_sync(0xffffffffu, hi16 ? a[1] : a[3], 16);
    const double k0 = (hi16 ? a[2] : a[0]) + r0;
    const double k1 = (hi16 ? a[3] : a[1]) + r1;
    const double r2 = __shfl_xor_sync(0xffffffffu, hi8 ? k0 : k1, 8);
    double v = (hi8 ? k1 : k0) + r2;
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct ItemXY {
    int r, c0, ty, tx;
};

__device__ __forceinline__ ItemXY item_xy(const TileDesc &T, int li, int tid)
{
    ItemXY q;
    int iby = li / T.nbx, ibx = li % T.nbx;
    q.ty = tid / kItemTx;
    q.tx = tid % kItemTx;
    q.r = iby * kItemBy + q.ty;
    q.c0 = ibx * kItemBx + q.tx * kItemVx;
    return q;
}

/* ── mixed-precision preconditioner and dots ─────────────────────────────
 * diag32: the Jacobi diagonal as an FP32 sum of the positive in-tile arc
 * weights (down, up, right, left) plus eps; rcp_pre: its reciprocal by the
 * hardware approximation (rcp.approx, within 1 ulp).  M^-1 = rcp_pre(diag32)
 * is the preconditioner of the mixed solve: every place that forms
 * z = M^-1 r (the INIT/true-residual phase, an item's own pixels, its halo
 * ring) evaluates these two functions on the same weights, so all blocks
 * agree on M bit for bit and no division is needed. */
__device__ __forceinline__ float diag32(int r, int c, int nr, int nc, float wdn, float wup,
                                        float wrt, float wlf)
{
    float ws = 0.0f;
    if (r < nr - 1 && wdn > 0.0f) ws = __fadd_rn(ws, wdn);
    if (r > 0 && wup > 0.0f) ws = __fadd_rn(ws, wup);
    if (c < nc - 1 && wrt > 0.0f) ws = __fadd_rn(ws, wrt);
    if (c > 0 && wlf > 0.0f) ws = __fadd_rn(ws, wlf);
    return __fadd_rn(ws, kLapEpsF);
}

__device__ __forceinline__ float rcp_pre(float d)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return y;
}

/* sum_j a[j] b[j] over a thread's four pixels with FP64 accuracy and no
 * per-element conversion: each FP32 product is split exactly into
 * p + e (e = fma(a, b, -p)), the p are summed with Knuth's TwoSum (the
 * rounding error of each addition recovered exactly), and the small terms
 * in FP32; hi + lo is then converted once.  For products in FP32's normal
 * range the error is ~2^-44 of the sum of the magnitudes, far below what
 * the FP64 tree reduction over a tile rounds away. */
__device__ __forceinline__ double dot4_df(const float a[4], const float b[4])
{
    float hi = __fmul_rn(a[0], b[0]);
    float lo = __fmaf_rn(a[0], b[0], -hi);
#pragma unroll
    for (int j = 1; j < 4; ++j) {
        const float p = __fmul_rn(a[j], b[j]);
        const float e = __fmaf_rn(a[j], b[j], -p);
        const float s = __fadd_rn(hi, p);
        const float bp = __fsub_rn(s, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(p, bp));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(e, err));
    }
    return (double)hi + (double)lo;
}

/* paired FP32 arithmetic (two lanes per instruction, IEEE round-to-nearest
 * per lane, the same results as the scalar operations) */
__device__ __forceinline__ float2 pf2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b)   /* a - b, one rounding */
{
    return __ffma2_rn(b, pf2(-1.0f, -1.0f), a);
}

/* two dot4_df sums at once, lane 0 for (a0, b0) and lane 1 for (a1, b1):
 * the same operations, so each result equals dot4_df's */
__device__ __forceinline__ void dot4_df2(const float a0[4], const float b0[4], const float a1[4],
                                         const float b1[4], double &r0, double &r1)
{
    float2 a = pf2(a0[0], a1[0]), b = pf2(b0[0], b1[0]);
    float2 hi = __fmul2_rn(a, b);
    float2 lo = __ffma2_rn(a, b, pf2(-hi.x, -hi.y));
#pragma unroll
    for (int j = 1; j < 4; ++j) {
        a = pf2(a0[j], a1[j]);
        b = pf2(b0[j], b1[j]);
        const float2 p = __fmul2_rn(a, b);
        const float2 e = __ffma2_rn(a, b, pf2(-p.x, -p.y));
        const float2 sm = __fadd2_rn(hi, p);
        const float2 bp = psub(sm, hi);
        const float2 err = __fadd2_rn(psub(hi, psub(sm, bp)), psub(p, bp));
        hi = sm;
        lo = __fadd2_rn(lo, __fadd2_rn(e, err));
    }
    r0 = (double)hi.x + (double)lo.x;
    r1 = (double)hi.y + (double)lo.y;
}

/* ── INIT / true residual: b, diag (A10) and r = b - A x, rz partial ────────
 * zero_x: first pass (x = 0, r = b).  write_diag: assemble pass (else the
 * stored diag is reused: residual replacement).  FP64 mode: z = r / diag
 * goes to zout.  Mixed mode: the FP32 residual r goes to zout (its
 * double-buffered residual plane), the preconditioner is M^-1 =
 * rcp_pre(diag32) recomputed from the weights, and the partial r.z comes
 * from dot4_df.  With P.bvec (mixed mode) the assemble pass stores the
 * right-hand side b and the replacements of the same IRLS pass read it back
 * instead of rebuilding it from the wrapped phase (the same doubles either
 * way).  The thread's row and the rows above and below of x and of the arc
 * weights arrive as 16-byte vectors; only the phase (scene layout) is read
 * element by element.  The arithmetic and its order are the oracle's. */
template <typename V, bool WLS>
__device__ double phase_init(const TileDesc &T, int li, const SolverPlanes &P, bool zero_x,
                             bool write_diag, V *zout, int tid)
{
    ItemXY q = item_xy(T, li, tid);
    if (q.r >= T.nr || q.c0 >= T.nc) return 0.0;
    double *x = P.x + T.pix;
    V *rr = (V *)P.r + T.pix;
    V *dg = (V *)P.diag + T.pix;
    const float *wd = P.wd + T.pix, *wr = P.wr + T.pix;
    const float *ph = T.ph;
    /* WLS mode: per-arc targets or an explicit right-hand side */
    const float *gdp = (WLS && P.gd) ? P.gd + T.pix : nullptr;
    const float *grp = (WLS && P.gr) ? P.gr + T.pix : nullptr;
    const float *rhsp = (WLS && P.rhs) ? P.rhs + T.pix : nullptr;
    const double eps = (double)kLapEpsF;
    const int r = q.r, nr = T.nr, nc = T.nc, pitch = T.pitch, pp = T.ph_pitch;
    const size_t prow = (size_t)r * pitch;
    const bool has_dn = r < nr - 1, has_up = r > 0;
    const bool has_l = q.c0 > 0, has_r = q.c0 + kItemVx < nc;
    /* the down arcs of this row and of the row above (the up arcs), the
     * right arcs of this row and the one left of the thread's columns; the
     * last row of wd and the last column of wr are zero, so the vectors
     * stay inside the tile's rows */
    float wdn[4], wup[4] = {0.f, 0.f, 0.f, 0.f}, wrt[4];
    ld4(wd + prow + q.c0, wdn);
    if (has_up) ld4(wd + prow - pitch + q.c0, wup);
    ld4(wr + prow + q.c0, wrt);
    const float wlf = has_l ? ldc(wr + prow + q.c0 - 1) : 0.0f;
    double xv[4], xdn[4] = {0.0, 0.0, 0.0, 0.0}, xup[4] = {0.0, 0.0, 0.0, 0.0};
    double xl = 0.0, xr = 0.0;
    if (!zero_x) {
        ld4(x + prow + q.c0, xv);
        if (has_dn) ld4(x + prow + pitch + q.c0, xdn);
        if (has_up) ld4(x + prow - pitch + q.c0, xup);
        if (has_l) xl = ldc(x + prow + q.c0 - 1);
        if (has_r) xr = ldc(x + prow + q.c0 + kItemVx);
    }
    V rv[4], dv[4], zv[4];
    float zf[4];   /* mixed: z = M^-1 r of the thread's pixels */
    if (!write_diag && sizeof(V) == 8) ld4(dg + prow + q.c0, dv);
    double *bvp = P.bvec ? P.bvec + T.pix + prow + q.c0 : nullptr;
    const bool b_stored = bvp && !write_diag;
    double bst[4];
    if (b_stored) ld4((const double *)bvp, bst);
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < kItemVx; ++j) {
        int c = q.c0 + j;
        if (c >= nc) {
            rv[j] = (V)0;
            zv[j] = (V)0;
            zf[j] = 0.0f;
            if (write_diag) dv[j] = (V)0;
            if (zero_x) xv[j] = 0.0;
            bst[j] = 0.0;
            continue;
        }
        const float w_dn = wdn[j], w_up = wup[j], w_rt = wrt[j];
        const float w_lf = j == 0 ? wlf : wrt[j - 1];
        double bv = 0.0, ws = 0.0;
        float ws32 = 0.0f;   /* mixed: diag32's sum, in its order */
        if (b_stored) {
            bv = bst[j];
            if (has_dn && w_dn > 0.0f) ws32 = __fadd_rn(ws32, w_dn);
            if (has_up && w_up > 0.0f) ws32 = __fadd_rn(ws32, w_up);
            if (c < nc - 1 && w_rt > 0.0f) ws32 = __fadd_rn(ws32, w_rt);
            if (c > 0 && w_lf > 0.0f) ws32 = __fadd_rn(ws32, w_lf);
        } else {
            const size_t gi = (size_t)r * pp + c, pi = prow + c;
            float pa = gdp ? 0.0f : __ldg(ph + gi);
            if (has_dn && w_dn > 0.0f) {
                float g = gdp ? ldc(gdp + pi) : lap_wrap_pi(__ldg(ph + gi + pp) - pa);
                bv = __fma_rn(-(double)w_dn, (double)g, bv);
                ws += w_dn;
                ws32 = __fadd_rn(ws32, w_dn);
            }
            if (has_up && w_up > 0.0f) {
                float g = gdp ? ldc(gdp + pi - pitch) : lap_wrap_pi(pa - __ldg(ph + gi - pp));
                bv = __fma_rn((double)w_up, (double)g, bv);
                ws += w_up;
                ws32 = __fadd_rn(ws32, w_up);
            }
            if (c < nc - 1 && w_rt > 0.0f) {
                float g = grp ? ldc(grp + pi) : lap_wrap_pi(__ldg(ph + gi + 1) - pa);
                bv = __fma_rn(-(double)w_rt, (double)g, bv);
                ws += w_rt;
                ws32 = __fadd_rn(ws32, w_rt);
            }
            if (c > 0 && w_lf > 0.0f) {
                float g = grp ? ldc(grp + pi - 1) : lap_wrap_pi(pa - __ldg(ph + gi - 1));
                bv = __fma_rn((double)w_lf, (double)g, bv);
                ws += w_lf;
                ws32 = __fadd_rn(ws32, w_lf);
            }
            if (rhsp) bv = (double)ldc(rhsp + pi);
            bst[j] = bv;
        }
        double d = write_diag ? ws + eps : (double)dv[j];
        double y;
        if (zero_x) {
            y = 0.0;
            xv[j] = 0.0;
        } else {
            const double xa = xv[j];
            const double x_l = j == 0 ? xl : xv[j - 1];
            const double x_r = j == kItemVx - 1 ? xr : xv[j + 1];
            y = eps * xa;
            if (has_dn)     y = __fma_rn((double)w_dn, xa - xdn[j], y);
            if (has_up)     y = __fma_rn((double)w_up, xa - xup[j], y);
            if (c < nc - 1) y = __fma_rn((double)w_rt, xa - x_r, y);
            if (c > 0)      y = __fma_rn((double)w_lf, xa - x_l, y);
        }
        V rs = (V)(bv - y);
        if constexpr (sizeof(V) == 8) {
            V ds = (V)d;
            double z = (double)rs / (double)ds;
            acc = __fma_rn((double)rs, z, acc);
            rv[j] = rs;
            zv[j] = (V)z;
            if (write_diag) dv[j] = ds;
        } else {
            const float d32 = __fadd_rn(ws32, kLapEpsF);
            rv[j] = rs;
            zf[j] = __fmul_rn((float)rs, rcp_pre(d32));
            zv[j] = rs;
            if (write_diag) dv[j] = (V)d32;
        }
    }
    if constexpr (sizeof(V) == 4) acc = dot4_df((const float *)rv, zf);
    if (sizeof(V) == 8) st4(rr + prow + q.c0, rv);
    st4(zout + T.pix + prow + q.c0, zv);
    if (write_diag && sizeof(V) == 8) st4(dg + prow + q.c0, dv);
    if (bvp && write_diag) st4(bvp, bst);
    if (zero_x) {
        st4(x + prow + q.c0, xv);
        if (P.dx) {
            const float zero[4] = {0.f, 0.f, 0.f, 0.f};
            st4(P.dx + T.pix + prow + q.c0, zero);
        }
    }
    return acc;
}

/* ── IRLS reweight (A13): w = w0 / sqrt(e^2 + delta^2) ───────────────────── */
template <typename V>
__device__ void phase_rw(const TileDesc &T, int li, const SolverPlanes &P, float delta, int tid)
{
    ItemXY q = item_xy(T, li, tid);
    if (q.r >= T.nr || q.c0 >= T.nc) return;
    const double *x = P.x + T.pix;
    const double dd = (double)delta * (double)delta;
    const int r = q.r, nr = T.nr, nc = T.nc, pitch = T.pitch, pp = T.ph_pitch;
    size_t prow = (size_t)r * pitch;
    float wdo[4], wro[4];
#pragma unroll
    for (int j = 0; j < kItemVx; ++j) {
        int c = q.c0 + j;
        wdo[j] = 0.0f; wro[j] = 0.0f;
        if (c >= nc) continue;
        size_t pi = prow + c, gi = (size_t)r * pp + c;
        double xa = ldc(x + pi);
        float pa = __ldg(T.ph + gi);
        if (r < nr - 1) {
            float w0 = __ldg(P.w0d + T.pix + pi);
            if (w0 > 0.0f) {
                float g = lap_wrap_pi(__ldg(T.ph + gi + pp) - pa);
                double e = (ldc(x + pi + pitch) - xa) - (double)g;
                wdo[j] = (float)((double)w0 / __dsqrt_rn(__fma_rn(e, e, dd)));
            }
        }
        if (c < nc - 1) {
            float w0 = __ldg(P.w0r + T.pix + pi);
            if (w0 > 0.0f) {
                float g = lap_wrap_pi(__ldg(T.ph + gi + 1) - pa);
                double e = (ldc(x + pi + 1) - xa) - (double)g;
                wro[j] = (float)((double)w0 / __dsqrt_rn(__fma_rn(e, e, dd)));
            }
        }
    }
    st4(P.wd + T.pix + prow + q.c0, wdo);
    st4(P.wr + T.pix + prow + q.c0, wro);
}

/* ── anchor + congruence (A14) ────────────────────────────────────────── */
template <typename V>
__device__ void phase_final(const TileDesc &T, int li, const SolverPlanes &P, int tid)
{
    ItemXY q = item_xy(T, li, tid);
    if (q.r >= T.nr || q.c0 >= T.nc) return;
    const double *x = P.x + T.pix;
    double off = (double)__ldg(T.ph) - ldc(x);
    size_t prow = (size_t)q.r * T.pitch;
    float uo[4] = {0.f, 0.f, 0.f, 0.f}, co[4] = {0.f, 0.f, 0.f, 0.f};
    int ko[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < kItemVx; ++j) {
        int c = q.c0 + j;
        if (c >= T.nc) continue;
        float ph = __ldg(T.ph + (size_t)q.r * T.ph_pitch + c);
        double u = ldc(x + prow + c) + off;
        double d = u - (double)ph;
        double k = rint(d / kTwoPiD);
        co[j] = (float)u;
        uo[j] = __fmaf_rn(kTwoPiF, (float)k, ph);
        ko[j] = (int)k;
    }
    *reinterpret_cast<float4 *>(P.unw + T.pix + prow + q.c0) = make_float4(uo[0], uo[1], uo[2], uo[3]);
    if (P.cyc)
        *reinterpret_cast<int4 *>(P.cyc + T.pix + prow + q.c0) = make_int4(ko[0], ko[1], ko[2], ko[3]);
    if (P.cont)
        *reinterpret_cast<float4 *>(P.cont + T.pix + prow + q.c0) = make_float4(co[0], co[1], co[2], co[3]);
}

/* first scalars of a solve from the tile's initial r.z */
__device__ __forceinline__ TileState start_state(double rz, const SolveParams &sp)
{
    TileState S;
    S.rz = rz;
    S.rz0 = rz;
    S.thr = (double)sp.tol * (double)sp.tol * rz;
    S.alpha = 0.0;
    S.beta = 0.0;
    S.iter = 0;
    S.active = (rz > 0.0 && sp.max_iter > 0) ? 1 : 0;
    return S;
}

}  // namespace cuphu
