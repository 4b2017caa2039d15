// tfs_cg_resident.cuh -- the binary64 CG loop with the diagonal (or no)
// preconditioner (Cg.f90:96-176) of a small system as one kernel: every
// thread owns one row and keeps its matrix entries, x, r, z, p and d in
// registers for the whole solve, and the blocks, all resident (a cooperative
// launch), meet twice an iteration to exchange their partial sums.
//
// The three kernels of an iteration (k_cg_p, k_spmv_pq, k_cg_update) spend a
// small system's time on the kernel boundaries, the round of the conditional
// node and the reload of what the previous kernel had in registers.  Here an
// iteration is bound by two exchanges through L2 and by the binary64
// instructions between them (a row's 28 of the product alone take 2.7 us at
// 256 rows a multiprocessor).  An iteration, us: 1,320 rows 19.1 -> 9.0,
// 32^3 17.4 -> 10.3, 38,912 rows (a block per multiprocessor) 18.0 -> 10.6,
// 77,658 rows (two, the most that are resident) 23.7 -> 19.5.
//
// The blocks start with a roll call.  That they are all resident is what a
// cooperative launch promises; how long it takes beside other work -- a batch,
// another handle, kernels of the caller's -- is not said anywhere.  A call not
// answered in full in some 10 ms is given up by all of them; nothing has been
// touched, nothing is stored, and the host launches the per-iteration kernels
// instead, which give the same bits.  After the call every block runs, and a
// wait that runs out is an error.  (The loop in the same graph, for the device
// to fall back on, would cost every solve the 10 us of a conditional node.)
//
// Bitwise the same as those kernels: the same row sums, the block sums and
// the sum over the blocks' partials in the same order.  A block forms p of a
// gathered row itself, z + beta p_old (the two operations of k_cg_p), which
// takes the place of a third exchange an iteration.
#pragma once
#include "tfs_kernels.cuh"

namespace tfs {

// A block's partial sum and the number of the exchange it belongs to, read
// and written as one 128-bit access.
struct alignas(16) CgSlot {
    double v;
    unsigned long long seq;
};

// Looks, of about a microsecond, that a wait for the other blocks takes at
// most: in the roll call, and in an exchange, whose blocks all run and are at
// most a row's work apart.  (Looks, not time: a context that is switched off
// the GPU does not look.)
#define CG_ROLL_LOOKS (1u << 14)
#define CG_RESIDENT_LOOKS (1u << 21)

// DevState::roll: blocks that have answered the call, and
#define CG_ROLL_COUNT 0x0000ffffu
#define CG_ROLL_LOST 0x40000000u       // a wait of an exchange ran out
#define CG_ROLL_ENDED 0x20000000u      // block 0 has written the outcome

// Whether all `blocks` blocks run; by one thread of each, to the same answer.
__device__ __forceinline__ bool cg_roll_call(unsigned *roll, unsigned blocks, unsigned looks)
{
    unsigned v = atomicAdd(roll, 1u) + 1u;
    for (unsigned k = 0;;) {
        if (v & CG_ROLL_GIVEN_UP) return false;
        if ((v & CG_ROLL_COUNT) == blocks) return true;
        if (k++ < looks) {
            __nanosleep(100);
            v = *(volatile unsigned *)roll;
        } else {
            const unsigned was = atomicCAS(roll, v, v | CG_ROLL_GIVEN_UP);   // at most `blocks` times
            v = was == v ? v | CG_ROLL_GIVEN_UP : was;
        }
    }
}

// (An exchange, not a store: a store reached the other blocks 2 us later, a
// 32^3 iteration 11.8 us with a store, 11.2 with a fence after it, 10.2.)
__device__ __forceinline__ void cg_slot_put(CgSlot *s, double v, unsigned long long seq)
{
    asm volatile("{ .reg .b128 t, u; mov.b128 t, {%1, %2}; atom.relaxed.gpu.global.exch.b128 u, [%0], t; }"
                 : : "l"(s), "l"(__double_as_longlong(v)), "l"(seq) : "memory");
}
__device__ __forceinline__ void cg_slot_get(const CgSlot *s, double &v, unsigned long long &seq)
{
    long long b;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(b), "=l"(seq) : "l"(s) : "memory");
    v = __longlong_as_double(b);
}
// The values of the slots s[0 .. NV - 1] once exchange seq has reached them,
// `mine` lanes only; the warp stays together.  False: the wait ran out.
// (Up to 100 ns between two looks: without, the looks themselves cost a
// system of two blocks a multiprocessor 0.5 to 1 us an iteration.)
template <int NV>
__device__ __forceinline__ bool cg_slot_wait(const CgSlot *s, bool mine, unsigned long long seq, double (&v)[NV],
                                             unsigned looks)
{
    for (unsigned k = 0;; k++) {
        unsigned long long got[NV];
        bool ok = true;
        if (mine) {
#pragma unroll
            for (int j = 0; j < NV; j++) cg_slot_get(s + j, v[j], got[j]);
#pragma unroll
            for (int j = 0; j < NV; j++) ok = ok && got[j] == seq;
        }
        if (__all_sync(FULL, ok)) return true;
        if (k >= looks) return false;
        __nanosleep(100);
    }
}

// Sums of NV (1 or 2) values over the warp, each as block_sum takes it
// (lane l + lane l + 16, then 8, 4, 2, 1); two share the binary64 adds:
// value 0 ends in lane 0, value 1 in lane 16.
template <int NV>
__device__ __forceinline__ double cg_warp_sum(const double (&v)[NV])
{
    const int lane = threadIdx.x & 31;
    double w;
    if constexpr (NV == 2) {
        const double got = __shfl_xor_sync(FULL, lane < 16 ? v[1] : v[0], 16);
        w = (lane < 16 ? v[0] : v[1]) + got;
    } else {
        w = v[0] + __shfl_down_sync(FULL, v[0], 16);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) w = w + __shfl_down_sync(FULL, w, o);
    return w;
}

// Block sum of NV values: lane k of warp 0 returns value k's.
template <int NV>
__device__ __forceinline__ double cg_block_sum(const double (&v)[NV], double (*sm)[TFS_TPB / 32])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double w = cg_warp_sum<NV>(v);
    if ((lane & 15) == 0 && lane < 16 * NV) sm[lane >> 4][warp] = w;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < NV) {
        s = sm[threadIdx.x][0];
#pragma unroll
        for (int k = 1; k < TFS_TPB / 32; k++) s = s + sm[threadIdx.x][k];
    }
    return s;
}

// Second half of an exchange, after the partials of exchange seq are waited
// for: warp sums of the partials (thread t takes blocks t, t + 256, ...) as
// grid_publish takes them, into sm.  Warps without a block have nothing to
// add.
template <int NV>
__device__ __forceinline__ void cg_partial_sums(const double (&a)[NV], double (*sm)[TFS_TPB / 32], int warps)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < warps) {
        const double w = cg_warp_sum<NV>(a);
        if ((lane & 15) == 0 && lane < 16 * NV) sm[lane >> 4][warp] = w;
    }
}
__device__ __forceinline__ double cg_total(const double *sm, int warps)
{
    double s = sm[0];
    for (int k = 1; k < warps; k++) s = s + sm[k];
    return warps < TFS_TPB / 32 ? s + 0.0 : s;   // (the other warps' sums are zeros)
}

// slots: 3 gridDim.x, the partials of (p, q), then pairs (r, r), (r, z);
// epoch: the last exchange number of the solves before.  p of odd
// iterations lies in V.p, of even ones in V.q.  W >= every row's entries.
template <int W>
__global__ void __launch_bounds__(TFS_TPB)
k_cg_resident(SellDev A, const double *__restrict__ val, Vec64 V, DevState *st, CgSlot *slots,
              unsigned long long *epoch)
{
    __shared__ double sm[2][TFS_TPB / 32], s_scalar;
    __shared__ int s_run, s_lost;
    const int tid = threadIdx.x, G = gridDim.x, warps = G < TFS_TPB ? (G + 31) / 32 : TFS_TPB / 32;
    const int i = blockIdx.x * TFS_TPB + tid;
    // tfs_diag_resident: the last block misses the call (1) or withholds its
    // partial of the first exchange (2)
    const int diag = blockIdx.x == G - 1 ? st->resident_diag : 0;
    const unsigned looks = st->resident_looks ? st->resident_looks : CG_RESIDENT_LOOKS;
    if (tid == 0) {
        s_run = st->done == 0 && diag != 1 &&
                cg_roll_call(&st->roll, (unsigned)G, min(looks, CG_ROLL_LOOKS));
        s_lost = 0;
    }
    __syncthreads();
    if (!s_run) return;
    const RowGeom g = row_geom(A, i);
    double a[W];
    int k[W];
#pragma unroll
    for (int j = 0; j < W; j++) {
        a[j] = 0.0;
        k[j] = 0;
        if (j < g.len) {
            a[j] = val[g.off + 32 * j];
            k[j] = __ldg(A.col + g.off + 32 * j);
        }
    }
    const double d = V.d[i], tol = st->tol;
    double x = V.x[i], r = V.r[i], z = V.z[i], p = 0.0, beta = 0.0, alfa = 0.0, rho = st->rho, err = 0.0;
    const int niter = st->niter_max, loop_limit = st->loop_limit;
    const unsigned long long e0 = *(volatile unsigned long long *)epoch;
    unsigned long long seq = e0, t_spmv = 0ull, spmv_ns = 0ull;
    __threadfence();   // the reads above, before block 0 (which ends last) writes the same words
    int it = 1, loops = 0, done = 0, status = TFS_OK, niter_out = 0;
    CgSlot *const sq = slots, *const sz = slots + G;
    // z, r of the prologue are visible (an earlier kernel's)
    for (;;) {
        double *const pn = it & 1 ? V.p : V.q;
        const double *const po = it & 1 ? V.q : V.p;
        double zg[W], pg[W];
#pragma unroll
        for (int j = 0; j < W; j++) {
            zg[j] = 0.0;
            pg[j] = 0.0;
            if (j < g.len) {
                zg[j] = __ldcg(V.z + k[j]);
                if (it > 1) pg[j] = __ldcg(po + k[j]);
            }
        }
        if (it > 1) {
            // beta = rho / rho_old, the norm and the outcome (finish_iteration)
            if (tid == 0) {
                const double rho_new = cg_total(sm[1], warps);
                s_scalar = rho_new / rho;
                rho = rho_new;
            }
            if (tid == 32) {
                err = sqrt(cg_total(sm[0], warps));
                const int was = it - 1;
                if (!(err <= DBL_MAX)) {
                    status = TFS_ERR_NONFINITE;
                    done = 1;
                    niter_out = (niter > 0 ? niter : 0) + 1;
                } else if (err < tol) {
                    done = 1;
                    niter_out = was;
                } else if (was >= niter) {
                    done = 1;
                    niter_out = was + 1;
                } else if (loops >= loop_limit) {
                    done = 1;
                    status = TFS_ERR_TIMEOUT;
                    niter_out = was + 1;
                }
                if (done) s_run = 0;
            }
            __syncthreads();
            if (!s_run) break;
            beta = s_scalar;
        }
        if (blockIdx.x == 0 && tid == 0) t_spmv = gtimer();
        p = it == 1 ? z : z + beta * p;
        pn[i] = p;
        double q = 0.0;
        if (it == 1) {
#pragma unroll
            for (int j = 0; j < W; j++)
                if (j < g.len) q = q + a[j] * zg[j];
        } else {
#pragma unroll
            for (int j = 0; j < W; j++)
                if (j < g.len) q = q + a[j] * (zg[j] + beta * pg[j]);
        }
        // (p, q) and alpha
        seq++;
        {
            const double v[1] = {fma(p, q, 0.0)};
            const double s = cg_block_sum<1>(v, sm);
            if (tid == 0 && !(diag && it == 1)) cg_slot_put(sq + blockIdx.x, s, seq);
            double t[1] = {0.0};
            for (int b0 = tid & ~31; b0 < G; b0 += TFS_TPB) {
                const int b = b0 + (tid & 31);
                double u[1] = {0.0};
                if (!cg_slot_wait<1>(sq + b, b < G, seq, u, looks)) s_lost = 1;
                t[0] = t[0] + u[0];
            }
            __syncthreads();
            cg_partial_sums<1>(t, sm, warps);
            __syncthreads();
            if (tid == 0) s_scalar = rho / cg_total(sm[0], warps);
            __syncthreads();
            alfa = s_scalar;
        }
        if (s_lost) break;
        if (blockIdx.x == 0 && tid == 0) spmv_ns += gtimer() - t_spmv;
        r = r - alfa * q;
        z = r / d;
        V.z[i] = z;
        seq++;
        {
            const double v[2] = {fma(r, r, 0.0), fma(r, z, 0.0)};
            const double s = cg_block_sum<2>(v, sm);
            if (tid < 2) {
                __threadfence();   // z and p of this block, before its partials
                cg_slot_put(sz + 2 * blockIdx.x + tid, s, seq);
            }
            x = x + alfa * p;
            double t[2] = {0.0, 0.0};
            for (int b0 = tid & ~31; b0 < G; b0 += TFS_TPB) {
                const int b = b0 + (tid & 31);
                double u[2] = {0.0, 0.0};
                if (!cg_slot_wait<2>(sz + 2 * b, b < G, seq, u, looks)) s_lost = 1;
                t[0] = t[0] + u[0];
                t[1] = t[1] + u[1];
            }
            __threadfence();       // the partials, before the others' z and p
            __syncthreads();
            cg_partial_sums<2>(t, sm, warps);
            loops++;
            it++;
            __syncthreads();
        }
        if (s_lost) break;
    }
    V.x[i] = x;
    V.r[i] = r;
    // The outcome: block 0's, unless a wait of any block ran out.  Others may
    // not have found the same (in the last exchange a block can miss the others'
    // partials after it has put its own): whichever of the two comes last at
    // the roll word sees the other there and leaves the error standing.
    bool lost = s_lost != 0;
    if (blockIdx.x == 0 && !lost) {
        if (tid == 32) {
            st->error = err;
            st->fin_res = err;
            st->status = status;
            st->niter_out = niter_out;
            st->iter = it - 1;
        }
        if (tid == 0) {
            st->loops = loops;
            st->alpha = alfa;
            st->spmv_ns = spmv_ns;
            st->spmv_n = loops;
        }
        __syncthreads();
    }
    if (tid == 0) {
        if (blockIdx.x == 0 && !lost) {
            __threadfence();
            lost = (atomicOr(&st->roll, CG_ROLL_ENDED) & CG_ROLL_LOST) != 0;
        } else if (lost) {
            atomicOr(&st->roll, CG_ROLL_LOST);
        }
        if (lost) {
            __threadfence();
            st->status = TFS_ERR_TIMEOUT;
            st->niter_out = it + 1;
            st->loops = loops;
        }
        if (lost || blockIdx.x == 0) {
            st->done = 1;
            atomicMax(epoch, e0 + 2ull * (unsigned)loop_limit + 8ull);
        }
    }
}

}  // namespace tfs
