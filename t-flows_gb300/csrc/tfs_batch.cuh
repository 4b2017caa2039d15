// tfs_batch.cuh -- many independent systems in one persistent launch.
//
// Each system of a batch is solved, start to finish, by one thread-block
// cluster (C CTAs on C SMs, 2 <= C <= 16).  Clusters take systems from a
// queue sorted by decreasing size (longest first), so a batch of uneven
// systems packs onto the GPU and small systems fill the gaps left by large
// ones.  Inside a cluster every synchronisation is the hardware cluster
// barrier, and every reduction sums one partial per CTA through distributed
// shared memory in CTA-rank order: there are no spin-waits, and a system's
// result depends only on (C, threads per CTA), never on which cluster ran it
// or on what else was in the batch -- a system gives bitwise the same result
// alone and in any mix.
//
// Methods: CG and BiCG (A, not A^T, on the shadow system) with no or diagonal
// preconditioning, and CG (hence the reference's BiCG, whose iterates are
// CG's) with DIC preconditioning: the factor (Prec_Form.f90:32-40) and both
// triangular sweeps (Prec_Solve.f90:46-67) run level by level over the
// system's DIC level schedule, the cluster's threads sharing each level's
// rows and the cluster barrier between levels; every row keeps the
// reference's arithmetic.  Binary64 (the reference's per-row arithmetic) or
// mixed precision (binary32 iteration, binary64 reliable updates, as
// tfs_mixed.cuh; the factor formed in binary64 and rounded once).
#pragma once
#include <cooperative_groups.h>

#include "tfs_kernels.cuh"

namespace tfs {

namespace cg = cooperative_groups;

// One system of a batch (device memory, written by the host per solve).
struct BatchSys {
    SellDev A;
    const double *val;        // SELL binary64 values (gathered by the kernel)
    float *val32;             // SELL binary32 values (mixed)
    const int *vmap;          // SELL -> CSR position
    int nnz_pad;
    const int *perm;          // internal -> natural row
    Vec64 V;
    Vec32 F;
    const double *val_csr;    // caller's CSR values (natural order)
    const double *b;          // caller's right-hand side (natural order)
    double *x;                // caller's x (natural order, in/out)
    double *r_out;            // r1 on return (natural order)
    double tol;
    int niter_max;
    int prec;
    const int *lvl_begin;     // DIC level schedule (prec 2): first row of every level, n_levels + 1
    int n_levels;
    // outputs
    int niter_out, status, early, true_res;
    double ini_res, fin_res;
};

static_assert(sizeof(BatchSys) % 8 == 0, "copied to shared memory by words of eight bytes");

struct BatchCtl {
    unsigned int head;        // next queue position
    unsigned int pad;
};

#define TFS_BATCH_MAX_TPB 512
// CTAs of 512 threads an SM is to hold: one (128 registers, no spilling), two
// (64, some spilling) or three (42).  More hold more systems at once, each
// slower for it.  `asked`: the CTAs of the whole batch, in 512 threads, for each
// SM; `work`: the same with every system counted by its rows over the largest's,
// which is what there is to do beside the largest.  Measured, one / two / three,
// ms, 60 iterations (systems log-uniform in a range of cells):
//   DIC, whose level barriers leave most to wait for: two as soon as one does not
//   hold the batch, three where two do not, unless the rows of a thread are many
//   and the largest system dominates:
//     mixed    24 of 2k to 30k, 8 x 512 (asked 1.3)   10.6   7.1   7.6
//              64 of 2k to 30k, 8 x 512 (3.4)         26.7  12.7  12.0
//             110 of 2k to 30k, 8 x 512 (5.8)         43.0  22.7  19.5
//              64 of 20k to 200k, 8 x 512 (3.4; work 1.3)  61.1  37.9  42.8
//             100 of 20k to 200k, 8 x 512 (5.3; work 2.1)  91.6  56.3  52.8
//     binary64 64 of 2k to 30k, 8 x 512                35.8  19.3  17.7
//             110 of 2k to 30k, 8 x 512                58.3  32.2  28.9
//   binary64 without DIC: two where the work asked is more than one holds:
//             110 of 2k to 30k, 8 x 512 (work 2.0)     12.0   8.8   8.7
//              64 of 20k to 200k, 8 x 512 (1.3)        29.7  26.2  32.9
//              64 of 5k to 500k, 8 x 512 (0.7)         366   490   655
//              64 of 5k to 500k, 16 x 512 (1.5)        337   341   478
//             256 of 5k to 500k, 8 x 512 (2.9)        1267  1043  1127
//   mixed without DIC: two past TFS_BATCH_ROOMY CTAs an SM:
//              24 of 5k to 91k, 8 x 512               9.6  14.0
//              96 of up to 500k, 16 x 512             235   197
#define TFS_BATCH_ROOMY 3
#define TFS_BATCH_WIDE_ROWS 16      // rows of a thread from which the largest system's own time counts
#define TFS_BATCH_WIDE_WORK 1.6

// Sum of NV values over the cluster: block sum, one partial per CTA in
// shared memory, cluster barrier, the C partials added in rank order.  The
// totals are valid in thread 0 of every CTA (all get the same bits), which
// alone goes on with them: a binary64 instruction occupies a quarter of an
// SM's narrow binary64 pipe for 64 cycles a warp, and when every thread
// added the partials and took the divisions and square roots of an iteration
// itself, those hundred instructions in 16 warps were most of a small
// system's iteration.  Two partial slots alternate, so a slot is rewritten
// only after the next barrier, by which time every reader of its previous
// contents is done.
//
// AT is the type of the per-thread partials: binary64, or binary32 in the
// mixed solves, whose warp sums are compensated pairs (warp_sum_f2), turned
// into binary64 a lane per warp by the first warp.
template <int NV, typename AT = double>
__device__ __forceinline__ void cluster_sum(const AT (&in)[NV], double (&v)[NV], double (*s_part)[4],
                                            int &parity, cg::cluster_group &cl)
{
    __shared__ double sm[NV][TFS_BATCH_MAX_TPB / 32];
    __shared__ float smf[NV][2][TFS_BATCH_MAX_TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        if constexpr (sizeof(AT) == 4) {
            float hi, lo;
            warp_sum_f2(in[k], hi, lo);
            if (lane == 0) { smf[k][0][warp] = hi; smf[k][1][warp] = lo; }
        } else {
            double w = in[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) w = w + __shfl_down_sync(FULL, w, o);
            if (lane == 0) sm[k][warp] = w;
        }
    }
    __syncthreads();
    if (warp == 0) {
        if constexpr (sizeof(AT) == 4) {
#pragma unroll
            for (int k = 0; k < NV; k++)
                if (lane < nw) sm[k][lane] = (double)smf[k][0][lane] + (double)smf[k][1][lane];
            __syncwarp();
        }
        if (lane < NV) {   // one value a lane
            double s = sm[lane][0];
            for (int w = 1; w < nw; w++) s = s + sm[lane][w];
            s_part[parity][lane] = s;
        }
    }
    cl.sync();
    if (warp == 0) {
        const unsigned C = cl.num_blocks();
        double s = 0.0;
        if (lane < NV) {
#pragma unroll 8
            for (unsigned r = 0; r < C; r++) {
                double(*rp)[4] = cl.map_shared_rank(s_part, r);
                s = s + rp[parity][lane];
            }
        }
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = __shfl_sync(FULL, s, k);
    }
    parity ^= 1;
}

// The vectors of arithmetic VT, by name.  S lies in shared memory and each
// phase of a solve takes the few pointers that it uses: thirty-odd pointers
// kept in registers through the whole solve were spilled, and with them the
// solve's own values.
template <typename VT>
__device__ __forceinline__ auto &batch_vecs(BatchSys &S)
{
    if constexpr (sizeof(VT) == 4) return S.F;
    else return S.V;
}
template <typename VT>
__device__ __forceinline__ const VT *batch_val(const BatchSys &S)
{
    if constexpr (sizeof(VT) == 4) return S.val32;
    else return S.val;
}

// The whole solve of one system by the calling cluster.  VT = double:
// binary64 with the reference's per-row arithmetic; VT = float: mixed.
// Per-thread dot-product partial: binary64 fma in the binary64 solves (the
// values are binary64 already), binary32 fmaf in the mixed ones.
template <typename AccT, typename VT>
__device__ __forceinline__ AccT acc_fma(VT a, VT b, AccT c)
{
    if constexpr (sizeof(AccT) == 4) return fmaf((float)a, (float)b, c);
    else return fma((double)a, (double)b, c);
}

// DIC factor of one system (binary64, Prec_Form.f90:32-40): levels
// ascending, the cluster's threads sharing each level's rows, the cluster
// barrier between levels (its release/acquire makes every CTA's stores
// visible; gathers read past L1).
__device__ void batch_dic_form(const SellDev &A, const double *val, double *d, const int *lvl_begin, int nl,
                               int gtid, int stride, cg::cluster_group &cl)
{
    for (int l = 0; l < nl; l++) {
        const int r1 = __ldg(lvl_begin + l + 1);
        for (int i = __ldg(lvl_begin + l) + gtid; i < r1; i += stride) {
            const RowGeom g = row_geom(A, i);
            if (g.len == 0) { d[i] = 1.0; continue; }
            double s = __ldg(val + g.off + (g.dpos << 5));
            for (int j = 0; j < g.dpos; j++) {
                const int ee = g.off + (j << 5);
                const double a = __ldg(val + ee);
                s = s - __ldcg(d + __ldg(A.col + ee)) * a * a;
            }
            d[i] = 1.0 / s;
        }
        cl.sync();
    }
}

// z = M^-1 r with the DIC factor d (Prec_Solve.f90:46-67): forward sweep
// into y, levels ascending, then y / (D + TINY) and the backward sweep into
// z, levels descending; returns the thread's partial of (r, z).  r must be
// complete (a cluster barrier after its stores).
template <typename VT, typename AccT>
__device__ AccT batch_dic_apply(const SellDev &A, const VT *val, const VT *d, const VT *r, VT *y, VT *z,
                                const int *lvl_begin, int nl, int gtid, int stride, cg::cluster_group &cl)
{
    for (int l = 0; l < nl; l++) {
        const int r1 = __ldg(lvl_begin + l + 1);
        for (int i = __ldg(lvl_begin + l) + gtid; i < r1; i += stride) {
            const RowGeom g = row_geom(A, i);
            if (g.len == 0) { y[i] = (VT)0; continue; }
            VT s = __ldcg(r + i);
            for (int j = 0; j < g.dpos; j++) {
                const int ee = g.off + (j << 5);
                s = s - __ldg(val + ee) * __ldcg(y + __ldg(A.col + ee));
            }
            y[i] = s * __ldcg(d + i);
        }
        cl.sync();
    }
    AccT rz = (AccT)0;
    for (int l = nl - 1; l >= 0; l--) {
        const int r1 = __ldg(lvl_begin + l + 1);
        for (int i = __ldg(lvl_begin + l) + gtid; i < r1; i += stride) {
            const RowGeom g = row_geom(A, i);
            if (g.len == 0) { z[i] = (VT)0; continue; }
            const VT di = __ldcg(d + i);
            VT s = __ldcg(y + i) / (di + (VT)TINY);
            for (int j = g.dpos + 1; j < g.len; j++) {
                const int ee = g.off + (j << 5);
                s = s - __ldg(val + ee) * __ldcg(z + __ldg(A.col + ee));
            }
            const VT zi = s * di;
            z[i] = zi;
            if constexpr (sizeof(AccT) == 4) rz = fmaf((float)__ldcg(r + i), (float)zi, rz);
            else rz = fma((double)__ldcg(r + i), (double)zi, rz);
        }
        cl.sync();
    }
    return rz;
}

// q = A p over the thread's rows (gtid, gtid + stride, ...) and its partial
// of (p, q).  Uniform slice widths up to 8 (hex meshes) run software-pipelined
// as k_spmv_pq_pipe does: the next row's columns are loaded while the gathers
// and values of the current one are in flight.  Gathers past L1: other CTAs
// of the cluster wrote p.
template <typename VT, typename AccT>
__device__ __forceinline__ void batch_spmv(const SellDev &A, const VT *__restrict__ val, const VT *p, VT *q, AccT &pq,
                                           int n_int, int gtid, int stride)
{
    if (A.width > 0 && A.width <= 8) {
        constexpr int W = 8;
        int nk[W];
        uint32_t ninfo = 0u;
        auto cols = [&](int i) {
            const int off = (i & ~31) * A.width + (i & 31);
            ninfo = __ldg(A.rowinfo + i);
#pragma unroll
            for (int j = 0; j < W; j++)
                if (j < A.width) nk[j] = __ldg(A.col + off + 32 * j);
        };
        if (gtid < n_int) cols(gtid);
        for (int i = gtid; i < n_int; i += stride) {
            const int off = (i & ~31) * A.width + (i & 31), len = (int)(ninfo & 0xffffu);
            VT x[W], a[W];
#pragma unroll
            for (int j = 0; j < W; j++)
                if (j < len) {
                    x[j] = __ldcg(p + nk[j]);
                    a[j] = __ldg(val + off + 32 * j);
                }
            const VT pi = p[i];
            if (i + stride < n_int) cols(i + stride);
            VT s = (VT)0;
#pragma unroll
            for (int j = 0; j < W; j++)
                if (j < len) s = s + a[j] * x[j];
            q[i] = s;
            pq = acc_fma(pi, s, pq);
        }
        return;
    }
    for (int i = gtid; i < n_int; i += stride) {
        const RowGeom g = row_geom(A, i);
        const VT s = row_accum<false, VT, VT, VT, false, 4>((VT)0, A.col, val, p, g.off, 0, g.len);
        q[i] = s;
        pq = acc_fma(p[i], s, pq);
    }
}

// What thread 0 of a CTA keeps and hands to the others, in shared memory.
struct BatchLead {
    double alfa, beta;                            // for every thread
    int need, done;                               // (two words: each is read while thread 0 may already write the other)
    double err, ini, rho, rho_old, r_true;        // thread 0's own
    int status, niter_out, early, true_res;
};

// r = b - A x in binary64 (b in V.u1), the iteration's residual and, unless
// DIC sweeps do it, z = M^-1 r; the thread's partials of ||r||^2 and rho.
template <int METHOD, typename VT>
__device__ __forceinline__ void batch_true_residual(BatchSys &S, int gtid, int stride, double &e2, double &rz)
{
    constexpr bool MIXED = sizeof(VT) == 4;
    const SellDev A = S.A;
    const double *const val = S.val, *const b = S.V.u1, *const x = S.V.x;
    double *const r64 = S.V.r;
    auto &W = batch_vecs<VT>(S);
    VT *const rT = W.r, *const z = W.z, *const r2 = W.r2, *const z2 = W.z2;
    const VT *const d = W.d;
    e2 = 0.0;
    rz = 0.0;
    for (int i = gtid; i < A.n_int; i += stride) {
        const RowGeom g = row_geom(A, i);
        const double r = row_accum<true, double, double, double, false, 4>(b[i], A.col, val, x, g.off, 0, g.len);
        r64[i] = r;
        e2 = fma(r, r, e2);
        const VT rt = (VT)r;
        if (MIXED) rT[i] = rt;
        if (METHOD == 2) continue;   // z and (r, z) from the sweeps
        const VT zt = rt / d[i];
        z[i] = zt;
        if (METHOD == 1) {
            // The shadow residual equals r1 (see k_mx_true): reset both.
            r2[i] = rt;
            z2[i] = zt;
            rz = fma((double)zt, (double)rt, rz);
        } else {
            rz = fma((double)rt, (double)zt, rz);
        }
    }
}

// z = M^-1 r by the DIC sweeps; the thread's partial of (r, z).
template <typename VT, typename AccT>
__device__ __forceinline__ AccT batch_sweeps(BatchSys &S, int gtid, int stride, cg::cluster_group &cl)
{
    cl.sync();
    const SellDev A = S.A;
    auto &W = batch_vecs<VT>(S);
    return batch_dic_apply<VT, AccT>(A, batch_val<VT>(S), (const VT *)W.d, W.r, W.y, W.z, S.lvl_begin, S.n_levels,
                                     gtid, stride, cl);
}

template <int METHOD, typename VT>
__device__ void batch_solve_one(BatchSys &S, BatchSys &out, BatchLead &L, cg::cluster_group &cl, double (*s_part)[4],
                                int &parity)
{
    constexpr bool MIXED = sizeof(VT) == 4;
    using AccT = VT;
    const int stride = (int)cl.num_blocks() * (int)blockDim.x;
    const int gtid = (int)cl.block_rank() * (int)blockDim.x + (int)threadIdx.x;
    const int n_int = S.A.n_int;
    // METHOD 2: the CG sequence with DIC preconditioning (its own instance,
    // so that the DIC sweeps add no registers to the other kernels)
    constexpr bool dic = METHOD == 2;
    const bool lead = threadIdx.x == 0;
    auto &W = batch_vecs<VT>(S);

    // b, x0 in internal order, d, ||b|| (Cg.f90:48-58).  The values were
    // gathered into SELL order by k_batch_gather before this launch.
    {
        double acc = 0.0;
        {
            const int *const perm = S.perm;
            const double *const b = S.b, *const x0 = S.x;
            double *const r = S.V.r, *const u = S.V.u1, *const x = S.V.x;
            for (int i = gtid; i < n_int; i += stride) {
                const int o = __ldg(perm + i);
                double bi = 0.0, xi = 0.0;
                if (o >= 0) { bi = b[o]; xi = x0[o]; }
                r[i] = bi;
                u[i] = bi;
                x[i] = xi;
                acc = fma(bi, bi, acc);
            }
        }
        {
            const SellDev A = S.A;
            const double *const val = S.val;
            const bool diag = S.prec == 1;
            double *const d = S.V.d;
            float *const d32 = S.F.d, *const e = S.F.e;
            for (int i = gtid; i < n_int; i += stride) {
                const RowGeom g = row_geom(A, i);
                const double di = (diag && g.len > 0) ? val[g.off + (g.dpos << 5)] : 1.0;
                d[i] = di;
                if (MIXED) { d32[i] = (float)di; e[i] = 0.f; }
            }
        }
        if (dic) {
            cl.sync();
            const SellDev A = S.A;
            batch_dic_form(A, S.val, S.V.d, S.lvl_begin, S.n_levels, gtid, stride, cl);
            if (MIXED) {
                const double *const d = S.V.d;
                float *const d32 = S.F.d;
                for (int i = gtid; i < n_int; i += stride) d32[i] = (float)__ldcg(d + i);
            }
        }
        const double a1[1] = {acc};
        double v1[1];
        cluster_sum<1>(a1, v1, s_part, parity, cl);
        if (lead) {
            const double bnrm2 = sqrt(v1[0]);
            L.done = bnrm2 < S.tol;
            if (L.done && cl.block_rank() == 0) {
                // Early exit 1: x, r1 untouched, ini_res untouched (Cg.f90:55-58).
                out.niter_out = 0; out.early = 1; out.fin_res = bnrm2; out.status = TFS_OK; out.true_res = 0;
            }
        }
        __syncthreads();
        if (L.done) return;
    }
    {
        double e2, rz;
        batch_true_residual<METHOD, VT>(S, gtid, stride, e2, rz);
        if (dic) rz = (double)batch_sweeps<VT, double>(S, gtid, stride, cl);
        const double a2[2] = {e2, rz};
        double v2[2];
        cluster_sum<2>(a2, v2, s_part, parity, cl);
        if (lead) {
            const double err = sqrt(v2[0]);
            L.err = L.ini = L.r_true = err;
            L.rho = v2[1];
            L.true_res = 1;
            L.status = TFS_OK;
            L.niter_out = L.early = 0;
            bool stop = false;
            if (!(err <= DBL_MAX)) { L.status = TFS_ERR_NONFINITE; L.niter_out = (S.niter_max > 0 ? S.niter_max : 0) + 1; stop = true; }
            else if (err < S.tol) { L.early = 2; stop = true; }
            else if (S.niter_max <= 0) { L.niter_out = 1; stop = true; }
            L.done = stop;
            L.beta = 0.0;
        }
        __syncthreads();
    }

    for (int iter = 1; !L.done; iter++) {
        // p = z + beta p (Cg.f90:114-123; both directions for BiCG).
        {
            const VT betaT = (VT)L.beta;
            const VT *const z = W.z, *const z2 = W.z2;
            VT *const p = W.p, *const p2 = W.p2;
            for (int i0 = gtid; i0 < n_int; i0 += 2 * stride) {
                const int i1 = i0 + stride;
                const bool ok1 = i1 < n_int;
                // z past L1: with DIC other threads of the cluster wrote it
                const VT z0 = __ldcg(z + i0), p0 = p[i0], z1 = ok1 ? __ldcg(z + i1) : (VT)0, p1 = ok1 ? p[i1] : (VT)0;
                VT a0 = (VT)0, b0 = (VT)0, a1 = (VT)0, b1 = (VT)0;
                if (METHOD == 1) {
                    a0 = z2[i0]; b0 = p2[i0];
                    if (ok1) { a1 = z2[i1]; b1 = p2[i1]; }
                }
                p[i0] = iter == 1 ? z0 : z0 + betaT * p0;
                if (METHOD == 1) p2[i0] = iter == 1 ? a0 : a0 + betaT * b0;
                if (ok1) {
                    p[i1] = iter == 1 ? z1 : z1 + betaT * p1;
                    if (METHOD == 1) p2[i1] = iter == 1 ? a1 : a1 + betaT * b1;
                }
            }
        }
        cl.sync();
        // q = A p and alpha (Cg.f90:128-153 / Bicg.f90:136-165).
        {
            AccT pq = (AccT)0;
            const SellDev A = S.A;
            const VT *const val = batch_val<VT>(S), *const p = W.p;
            VT *const q = W.q;
            if (METHOD == 1) {
                const VT *const p2 = W.p2;
                VT *const q2 = W.q2;
                for (int i = gtid; i < n_int; i += stride) {
                    const RowGeom g = row_geom(A, i);
                    VT s1 = (VT)0, s2 = (VT)0;
                    row_accum2<false, VT, VT, VT>(s1, s2, A.col, val, p, p2, g.off, 0, g.len);
                    q[i] = s1;
                    q2[i] = s2;
                    pq = acc_fma(p2[i], s1, pq);
                }
            } else {
                batch_spmv<VT, AccT>(A, val, p, q, pq, n_int, gtid, stride);
            }
            const AccT a1[1] = {pq};
            double v1[1];
            cluster_sum<1, AccT>(a1, v1, s_part, parity, cl);
            if (lead) L.alfa = L.rho / v1[0];
            __syncthreads();
        }
        // x (or e) += alpha p, r -= alpha q, z = M^-1 r, ||r||, next rho.
        {
            const double alfa = L.alfa;
            const VT alfaT = (VT)alfa;
            AccT e2a = (AccT)0, rza = (AccT)0;
            VT *const r = W.r, *const z = W.z, *const r2 = W.r2, *const z2 = W.z2;
            const VT *const p = W.p, *const q = W.q, *const q2 = W.q2, *const d = W.d;
            double *const x = S.V.x;
            float *const e = S.F.e;
            if (METHOD == 1) {
                for (int i = gtid; i < n_int; i += stride) {
                    if (MIXED) e[i] = fmaf((float)alfaT, (float)p[i], e[i]);
                    else x[i] = x[i] + alfa * (double)p[i];
                    const VT r1 = r[i] - alfaT * q[i];
                    r[i] = r1;
                    const VT dT = d[i];
                    const VT z1 = r1 / dT;
                    z[i] = z1;
                    e2a = acc_fma(r1, r1, e2a);
                    const VT rs = r2[i] - alfaT * q2[i];
                    r2[i] = rs;
                    z2[i] = rs / dT;
                    rza = acc_fma(z1, rs, rza);
                }
            } else {
                for (int i0 = gtid; i0 < n_int; i0 += 4 * stride) {
                    VT pv[4], rv[4], qv[4], dv[4];
                    double xv[4];
                    float ev[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int i = i0 + k * stride < n_int ? i0 + k * stride : i0;
                        pv[k] = p[i]; rv[k] = r[i]; qv[k] = q[i];
                        if (!dic) dv[k] = d[i];
                        if (MIXED) ev[k] = e[i]; else xv[k] = x[i];
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int i = i0 + k * stride;
                        if (i >= n_int) continue;
                        if (MIXED) e[i] = fmaf((float)alfaT, (float)pv[k], ev[k]);
                        else x[i] = xv[k] + alfa * (double)pv[k];
                        const VT r1 = rv[k] - alfaT * qv[k];
                        r[i] = r1;
                        e2a = acc_fma(r1, r1, e2a);
                        if (dic) continue;
                        const VT z1 = r1 / dv[k];
                        z[i] = z1;
                        rza = acc_fma(r1, z1, rza);
                    }
                }
            }
            if (dic) rza = batch_sweeps<VT, AccT>(S, gtid, stride, cl);
            const AccT a3[2] = {e2a, rza};
            double v3[2];
            cluster_sum<2, AccT>(a3, v3, s_part, parity, cl);
            if (lead) {
                const double est = sqrt(v3[0]);
                L.err = est;
                L.rho_old = L.rho;
                L.rho = v3[1];
                L.need = MIXED && (!(est <= DBL_MAX) || est < S.tol || est < 0.1 * L.r_true || iter >= S.niter_max);
            }
        }
        if (MIXED) __syncthreads();
        if (MIXED && L.need) {
            {
                double *const x = S.V.x;
                float *const e = S.F.e;
                for (int i = gtid; i < n_int; i += stride) {
                    x[i] = x[i] + (double)e[i];
                    e[i] = 0.f;
                }
            }
            cl.sync();
            double e2, rz;
            batch_true_residual<METHOD, VT>(S, gtid, stride, e2, rz);
            if (dic) rz = (double)batch_sweeps<VT, double>(S, gtid, stride, cl);
            const double a4[2] = {e2, rz};
            double v4[2];
            cluster_sum<2>(a4, v4, s_part, parity, cl);
            if (lead) {
                L.r_true = L.err = sqrt(v4[0]);
                L.rho = v4[1];
                L.true_res++;
            }
        }
        if (lead) {
            bool stop = true;
            if (!(L.err <= DBL_MAX)) { L.status = TFS_ERR_NONFINITE; L.niter_out = (S.niter_max > 0 ? S.niter_max : 0) + 1; }
            else if (L.err < S.tol) L.niter_out = iter;
            else if (iter >= S.niter_max) L.niter_out = iter + 1;
            else {
                stop = false;
                L.beta = L.rho / L.rho_old;
            }
            L.done = stop;
        }
        __syncthreads();
    }
    cl.sync();
    // x and r1 back to natural order.
    {
        const int *const perm = S.perm;
        double *const xo = S.x, *const ro = S.r_out;
        const double *const x = S.V.x, *const r = S.V.r;
        for (int i = gtid; i < n_int; i += stride) {
            const int o = __ldg(perm + i);
            if (o >= 0) { xo[o] = x[i]; ro[o] = r[i]; }
        }
    }
    if (cl.block_rank() == 0 && lead) {
        out.niter_out = L.niter_out; out.status = L.status; out.early = L.early; out.true_res = L.true_res;
        out.ini_res = L.ini; out.fin_res = L.err;
    }
}

// SELL values of every system from the callers' CSR values (blockIdx.y =
// system), and the queue head reset for the launch that follows.
__global__ void k_batch_gather(BatchSys *sys, BatchCtl *ctl, int mixed)
{
    const BatchSys &S = sys[blockIdx.y];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ctl->head = 0u;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < S.nnz_pad; e += gridDim.x * blockDim.x) {
        int m = __ldg(S.vmap + e);
        double v = m >= 0 ? S.val_csr[m] : 0.0;
        ((double *)S.val)[e] = v;
        if (mixed) S.val32[e] = (float)v;
    }
}

template <int METHOD, typename VT, int PER_SM>
__global__ void __launch_bounds__(TFS_BATCH_MAX_TPB, PER_SM)
k_batch(BatchSys *sys, const int *order, int n_sys, BatchCtl *ctl)
{
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double s_part[2][4];
    __shared__ int s_sys;
    __shared__ BatchSys s_S;
    __shared__ BatchLead s_L;
    int parity = 0;
    for (;;) {
        if (cl.block_rank() == 0 && threadIdx.x == 0) s_sys = (int)atomicAdd(&ctl->head, 1u);
        cl.sync();
        const int q = *cl.map_shared_rank(&s_sys, 0);
        cl.sync();   // every CTA has read rank 0's s_sys before it changes
        if (q >= n_sys) break;
        BatchSys &S = sys[order[q]];
        for (int k = threadIdx.x; k < (int)(sizeof(BatchSys) / 8); k += blockDim.x)
            ((unsigned long long *)&s_S)[k] = ((const unsigned long long *)&S)[k];
        __syncthreads();
        batch_solve_one<METHOD, VT>(s_S, S, s_L, cl, s_part, parity);
        cl.sync();
    }
}

}  // namespace tfs
