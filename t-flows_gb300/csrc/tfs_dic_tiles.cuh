// tfs_dic_tiles.cuh -- the DIC sweeps (Prec_Solve.f90:46-67) tile by tile:
// one thread block sweeps a compact tile of rows together with the closure of
// the rows it depends on (tfs_dic_tiles_plan.h), so a sweep is one launch
// whose blocks never wait for one another, instead of one dependent launch
// per level.
//
// What bounds the level kernels is the chain of 31 launches of an
// application on the 128^3 system (about 3 us each, two thirds of a 155 us
// iteration); the tiles stream their entries instead, 1.32 times as many:
//   - the swept vector of the tile and its closure lives in shared memory,
//     indexed by 16-bit local slots, rows in level order; a level step costs
//     shared-memory gathers and one named barrier;
//   - the entries (values, D and local indices, packed in sweep order, most
//     entries first inside a level so that slices of 32 rows carry little
//     padding) come through a ring in rounds of up to TILE_ROWS rows, one
//     bulk copy (cp.async.bulk) a round into a place fixed by the plan,
//     issued by a copy lane as the rounds it overwrites are released;
//   - the vectors move between the solver's row order and the slots by
//     threads of their own, level by level and in the order of the rows:
//     loaders bring every row's right-hand side by a 4- or 8-byte cp.async
//     into its slot, storers (binary32) take the own rows out;
//   - every row of the closure is swept, only the tile's own rows are stored.
//     In binary64 the forward sweep stores the backward start values
//     y / (D + TINY) by tile_quotient; in binary32 it stores y and the
//     backward sweep divides.
// An application alone, us, level kernels -> tiles: 128^3 binary32 98 -> 51,
// binary64 219 -> 141; 64^3 52 -> 19 and 92 -> 39.  In binary64 the pipe
// bounds it (77 us of the 141 at 128^3 are its instructions alone); in
// binary32 and on small meshes the chain of a level's gathers, products and
// barrier does, about 0.5 us a level (128^3: 35% of the DRAM's rate, 45% of
// the issue slots).  Slower: rounds of 1024 rows, two or three tiles a
// multiprocessor (57 and 78 us), row words in a register queue moved along
// every round (each move waits for its load), operands loaded before the
// barrier (64), a seven-way switch over the widths unrolled four times (it
// leaves the instruction cache).
// Every row does exactly sweep_row's operations in sweep_row's order, so the
// sweeps are bitwise those of the level kernels.
//
// Every wait is on the block's own copies or its own warps, and bounded as in
// the one-block DIC: a wait that runs out raises the block's abort flag,
// after which no copy is issued and no slot is read, and the solve ends with
// TFS_ERR_TIMEOUT.  The copy lane stays until what it issued has landed,
// whether the sweep was finished, called off or never begun (tile_copy_walk).
#pragma once
#include "tfs_dic_block.cuh"
#include "tfs_dic_tiles_plan.h"
#include "tfs_spmv.cuh"

namespace tfs {

constexpr int TILE_TPB = TILE_ROWS + 2 * TILE_MOVERS + 32;   // row threads, loaders, storers and a copy warp
constexpr int TILE_QUIT = 2;                              // abort flag of a sweep that has nothing to do
constexpr int TILE_BATCH = 8;                             // list rounds whose rows a mover holds at once

// One direction of a plan on the device.
struct TileDev {
    const TileRound *rounds;
    const int *tile_round;
    const uint32_t *rows;
    const int *vbeg;
    unsigned char *packed;
    const int *tile_list;
    const uint8_t *lists;
    const uint32_t *list_row;
    const uint16_t *list_slot;
    int max_slots, max_rounds, max_lists, ring_bytes;
};

// s <- *p asynchronously (4 or 8 bytes).
template <typename T>
__device__ __forceinline__ void tile_cp_async(uint32_t s, const T *p)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" : : "r"(s), "l"(p), "n"(sizeof(T)) : "memory");
}
// Arrive on bar once every cp.async of this thread so far has landed.
__device__ __forceinline__ void tile_cp_arrive(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" : : "r"(dicb_smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tile_cp_wait_all() { asm volatile("cp.async.wait_all;" : : : "memory"); }
// Prefetch of `bytes` (a multiple of 16, from a 16-byte boundary) into L2.
__device__ __forceinline__ void tile_prefetch(const void *p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" : : "l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tile_row_sync()
{
    asm volatile("bar.sync 1, %0;" : : "n"(TILE_ROWS) : "memory");
}

// Whether x / d may be taken as tile_quotient does: x's exponent in a range
// where nothing under- or overflows for the d that tile_recip admits.
__device__ __forceinline__ bool tile_in_range(double x)
{
    return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 223u < 1600u;
}
// 1 / d rounded for tile_quotient, 0 where it must not be used: d + TINY is
// not d, or d is outside 2^-40 .. 2^40.
template <typename T>
__device__ __forceinline__ T tile_recip(T d)
{
    const T lim = (T)1099511627776.0, a = d < (T)0 ? -d : d;
    return d + (T)TINY == d && a < lim && a * lim > (T)1 ? (T)1 / d : (T)0;
}
// y / (d + TINY) for y = s d rounded (Prec_Solve.f90:55-57), rc =
// tile_recip(d): the division's correctly rounded result from two FMAs.
// y - s d is exact (the rounding error of a product), at most half an ulp of
// y; s + (y - s d) rc therefore differs from y / d by at most 2^-(2p+1) for
// y, d scaled to [1, 2) (p bits, rc off by at most 2^-(p+1)), while no
// quotient of two p-bit numbers lies that close to the midpoint of two p-bit
// numbers: the FMA rounds it as the division does (the argument of
// Markstein, IBM J. Res. Dev. 34, 1990).  A binary64 division takes about
// ten instructions of GB300's narrow binary64 pipe.
template <typename T>
__device__ __forceinline__ T tile_quotient(T s, T y, T d, T rc)
{
    if (rc != (T)0 && tile_in_range(y)) return fma_t(fma_t(-d, s, y), rc, s);
    return y / (d + (T)TINY);
}

// acc minus the row's products in order; si, sv: its first index and value,
// W: the slice's width rounded up to even, odd: it was odd, cnt <= W: the
// row's entries.  Every index, value and gather is issued before the chain.
// In binary64 the chain ends at the row's last entry: an update predicated
// off still takes its turn in GB300's narrow binary64 pipe.
template <typename T, int W>
__device__ __forceinline__ T tile_row(T acc, const T *s, const uint16_t *si, const T *sv, int cnt, bool odd)
{
    T a[W], x[W];
#pragma unroll
    for (int j = 0; j < W; j++) {
        x[j] = (T)0;
        a[j] = (T)0;
        if (j < W - 1 || !odd) {
            x[j] = s[si[32 * j]];
            a[j] = sv[32 * j];
        }
    }
#pragma unroll
    for (int j = 0; j < W; j++) {
        if (sizeof(T) == 8 && j >= cnt) break;
        if (j < cnt) acc = acc - a[j] * x[j];
    }
    return acc;
}

// dicb_mbar_wait with its loop out of line: the sweep's code is to stay in
// the instruction cache.
__device__ __noinline__ bool tile_wait_slow(uint64_t *bar, unsigned parity, volatile int *abort, unsigned long long wait_ns)
{
    return dicb_mbar_wait(bar, parity, abort, wait_ns);
}
// The copy lane's wait for a release: it looks at the abort flag between two
// tests that do not suspend it (try_wait may for a good part of a
// millisecond, which a sweep with nothing to do would spend leaving).
__device__ __forceinline__ bool tile_wait_empty(uint64_t *bar, unsigned parity, volatile int *abort, unsigned long long wait_ns)
{
    const unsigned long long t0 = gtimer();
    for (;;) {
        unsigned ok;
        asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok) : "r"(dicb_smem_addr(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (*abort) return false;
        if (gtimer() - t0 > wait_ns) {
            *abort = 1;
            return false;
        }
    }
}
__device__ __forceinline__ bool tile_wait(uint64_t *bar, unsigned parity, volatile int *abort, unsigned long long wait_ns)
{
    return dicb_mbar_test(bar, parity) || tile_wait_slow(bar, parity, abort, wait_ns);
}

// What the copy lane does for a round (tile_copy_walk).
struct TileCopy {
    const uint4 *tab;
    unsigned char *ring;
    const unsigned char *packed;
    uint64_t *full, *empty;
    volatile int *abort;
    unsigned long long wait_ns;
    uint4 c;                            // the round that back() looked at last
    __device__ int back(int k)
    {
        c = tab[k];
        return (int)(c.y >> 16 & 0xffu);
    }
    __device__ bool released(int k)
    {
        return tile_wait_empty(empty + k % TILE_BARS, (unsigned)(k / TILE_BARS) & 1u, abort, wait_ns);
    }
    __device__ bool off() { return *abort != 0; }
    __device__ void issue(int k)
    {
        uint64_t *bar = full + k % TILE_BARS;
        const unsigned bytes = (c.y & 0xffffu) * 16u;
        dicb_mbar_expect(bar, bytes);
        dicb_bulk(ring + (c.w & 0xffffu) * 128u, packed + 16 * (size_t)c.x, bytes, bar);
    }
    // (bounded as every wait, but the flag is not asked)
    __device__ void landed(int k)
    {
        const unsigned long long t0 = gtimer();
        while (!dicb_mbar_test(full + k % TILE_BARS, (unsigned)(k / TILE_BARS) & 1u) && gtimer() - t0 < wait_ns) {
        }
    }
};

// The vectors between global memory and the tile's slots, by two sets of
// TILE_MOVERS threads (m: this one's number in its set), level by level: the
// loaders every row's right-hand side, asynchronously; the storers the own
// rows of every level as soon as it is swept.  A mover's rows of the next
// TILE_BATCH list rounds are in flight: each is read again for the round
// TILE_BATCH on as soon as it is used.
template <typename T, bool STORE>
__device__ __forceinline__ void tile_move(const TileDev &P, int m, const T *src, T *dst, T *s, const uint8_t *lists,
                                          uint64_t *loaded, uint64_t *done, const DevState *st, volatile int *abort)
{
    const int l0 = __ldg(P.tile_list + blockIdx.x), n = __ldg(P.tile_list + blockIdx.x + 1) - l0;
    const uint32_t *rows = P.list_row + (size_t)l0 * TILE_MOVERS + m;
    const uint16_t *slots = P.list_slot + (size_t)l0 * TILE_MOVERS + m;
    uint32_t w[TILE_BATCH], k[TILE_BATCH];
    auto row = [&](int q, uint32_t &wq, uint32_t &kq) {
        wq = TILE_NO_ROW;
        kq = 0;
        if (q < n) {
            wq = __ldg(rows + (size_t)q * TILE_MOVERS);
            kq = __ldg(slots + (size_t)q * TILE_MOVERS);
        }
    };
#pragma unroll
    for (int u = 0; u < TILE_BATCH; u++) row(u, w[u], k[u]);
    const uint32_t s_at = dicb_smem_addr(s);
    cudaGridDependencySynchronize();
    const unsigned long long diag = st->dicb_wait_ns;
    const unsigned long long wait_ns = diag ? diag : TFS_DICB_WAIT_NS;
    if (st->done) return;
    for (int q0 = 0; q0 < n; q0 += TILE_BATCH) {
#pragma unroll
        for (int u = 0; u < TILE_BATCH; u++) {
            if (q0 + u >= n) break;
            const uint8_t l = lists[q0 + u];
            if (STORE) {
                tile_wait(done + (l & 127u), 0u, abort, wait_ns);
                if (w[u] & TILE_OWN) dst[w[u] & TILE_ROW_MASK] = s[k[u]];
            } else {
                if ((w[u] & TILE_ROW_MASK) != TILE_NO_ROW)
                    tile_cp_async(s_at + k[u] * (uint32_t)sizeof(T), src + (w[u] & TILE_ROW_MASK));
                if (l & 128u) tile_cp_arrive(loaded + (l & 127u));
            }
            row(q0 + u + TILE_BATCH, w[u], k[u]);
        }
    }
    if (!STORE) tile_cp_wait_all();
}

// The packed bytes of a direction are filled by k_tile_fill; src: the
// right-hand side (DIR 0: b; DIR 1: what DIR 0 wrote); dst: DIR 0: y in
// binary32, the backward start values y / (D + TINY) in binary64; DIR 1: z.
// All vectors in internal row order.  In binary32 the movers store (the
// backward sweep divides); in binary64, where the pipe and not the stores
// bounds the sweep, the row threads do, since only they hold the operands
// of tile_quotient.
template <typename T, int DIR>
__global__ void __launch_bounds__(TILE_TPB, 1)
k_dic_tile(TileDev P, const T *__restrict__ src, T *__restrict__ dst, DevState *st)
{
    constexpr bool MOVED = sizeof(T) == 4;
    constexpr int DIAGS = tile_diags(DIR, sizeof(T));
    extern __shared__ __align__(128) unsigned char tile_smem[];
    T *s = reinterpret_cast<T *>(tile_smem);
    unsigned char *ring = tile_smem + ((P.max_slots * (int)sizeof(T) + 127) & ~127);
    uint4 *tab = reinterpret_cast<uint4 *>(ring + P.ring_bytes);
    uint8_t *lists = reinterpret_cast<uint8_t *>(tab + P.max_rounds);
    uint64_t *full = reinterpret_cast<uint64_t *>(lists + ((P.max_lists + 15) & ~15)), *empty = full + TILE_BARS;
    uint64_t *loaded = empty + TILE_BARS, *done = loaded + TILE_MAX_LEVELS;
    volatile int *abort = reinterpret_cast<volatile int *>(done + TILE_MAX_LEVELS);
    const int tid = threadIdx.x;
    const int c0 = __ldg(P.tile_round + blockIdx.x), rounds = __ldg(P.tile_round + blockIdx.x + 1) - c0;
    for (int k = tid; k < rounds; k += TILE_TPB) tab[k] = __ldg(reinterpret_cast<const uint4 *>(P.rounds + c0 + k));
    {
        const int l0 = __ldg(P.tile_list + blockIdx.x), n = __ldg(P.tile_list + blockIdx.x + 1) - l0;
        for (int k = tid; k < n; k += TILE_TPB) lists[k] = __ldg(P.lists + l0 + k);
    }
    if (tid < TILE_BARS) {
        dicb_mbar_init(full + tid, 1);              // the copy lane's arrival (+ the copy's bytes)
        dicb_mbar_init(empty + tid, TILE_SLICES);   // every row warp's
    }
    if (tid < TILE_MAX_LEVELS) {
        dicb_mbar_init(loaded + tid, TILE_MOVERS);  // every mover's, once its loads have landed
        dicb_mbar_init(done + tid, 1);              // one row thread's
    }
    if (tid == 0) *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
    __syncthreads();
    cudaTriggerProgrammaticLaunchCompletion();
    if (tid >= TILE_ROWS + 32 + TILE_MOVERS) {
        if (MOVED) tile_move<T, true>(P, tid - TILE_ROWS - 32 - TILE_MOVERS, src, dst, s, lists, loaded, done, st, abort);
        return;
    }
    if (tid >= TILE_ROWS + 32) {
        tile_move<T, false>(P, tid - TILE_ROWS - 32, src, dst, s, lists, loaded, done, st, abort);
        return;
    }
    if (tid >= TILE_ROWS) {
        // The copy lane.  The packed rounds are not written inside the
        // solve's loop: it starts before the dependency wait.
        if (tid != TILE_ROWS) return;
        const unsigned long long diag = st->dicb_wait_ns;
        const unsigned long long wait_ns = diag ? diag : TFS_DICB_WAIT_NS;
        if (diag) return;                   // tfs_diag_dic_timeout: stage nothing
        {   // the movers' lists on their way into L2
            const int l0 = __ldg(P.tile_list + blockIdx.x), n = __ldg(P.tile_list + blockIdx.x + 1) - l0;
            tile_prefetch(P.list_row + (size_t)l0 * TILE_MOVERS, (unsigned)n * TILE_MOVERS * 4u);
            tile_prefetch(P.list_slot + (size_t)l0 * TILE_MOVERS, (unsigned)n * TILE_MOVERS * 2u);
        }
        TileCopy copy{tab, ring, P.packed, full, empty, abort, wait_ns, make_uint4(0u, 0u, 0u, 0u)};
        tile_copy_walk(rounds, copy);
        return;
    }
    const int warp = tid >> 5, lane = tid & 31;
    const uint32_t *words = P.rows + (size_t)c0 * TILE_ROWS + tid;
    cudaGridDependencySynchronize();
    const unsigned long long diag = st->dicb_wait_ns;
    const unsigned long long wait_ns = diag ? diag : TFS_DICB_WAIT_NS;
    if (st->done) {   // nothing to sweep: the copy lane issues no more
        if (tid == 0) *abort = TILE_QUIT;
        return;
    }
    if (DIR == 0 && blockIdx.x == 0 && tid == 0) st->t_sweep0 = gtimer();
    int level = 0;
    bool ok = tile_wait(loaded, 0u, abort, wait_ns);
#pragma unroll 1
    for (int q = 0; q < rounds; q++) {
        const uint4 c = tab[q];
        const int bar = q % TILE_BARS;
        const uint32_t w = MOVED ? 0u : __ldg(words + (size_t)q * TILE_ROWS);   // used after the barrier below
        ok = tile_wait(full + bar, (unsigned)(q / TILE_BARS) & 1u, abort, wait_ns) && ok;
        T acc = (T)0, y = (T)0, d = (T)1, rc = (T)0;
        const int slices = (int)(c.z >> 16);
        if (ok && warp < slices) {
            const unsigned char *at = ring + (c.w & 0xffffu) * 128u;
            const uint32_t head = reinterpret_cast<const uint32_t *>(at)[warp];
            const int cnt = at[TILE_HEAD + tid], width = (int)(head >> 16), e0 = (int)(head & 0xffffu) * 32 + lane;
            const T *sd = reinterpret_cast<const T *>(at + TILE_HEAD + 32 * slices) + tid;
            const T *sv = sd - tid + 32 * slices * DIAGS + e0;
            const uint16_t *si = reinterpret_cast<const uint16_t *>(at + (c.w >> 16) * 16u) + e0;
            T *own = s + (c.z & 0xffffu) + tid;
            d = sd[0];
            if (DIAGS == 2) rc = sd[32 * slices];
            acc = *own;
            if (DIR == 1 && MOVED) acc = acc / (d + (T)TINY);
            const bool odd = width & 1;
            if (width > 6) {
                for (int j = 0; j < cnt; j++) acc = acc - sv[32 * j] * s[si[32 * j]];
            } else if (width > 4) {
                acc = tile_row<T, 6>(acc, s, si, sv, cnt, odd);
            } else if (width > 2) {
                acc = tile_row<T, 4>(acc, s, si, sv, cnt, odd);
            } else if (width > 0) {
                acc = tile_row<T, 2>(acc, s, si, sv, cnt, odd);
            }
            y = acc * d;
            *own = y;
        }
        __syncwarp();
        if (lane == 0) dicb_mbar_arrive(empty + bar);   // done with the round's bytes
        if (c.y >> 24) {
            if (q + 1 < rounds) ok = tile_wait(loaded + level + 1, 0u, abort, wait_ns) && ok;
            tile_row_sync();                            // this level's rows visible to the next
            if (MOVED && tid == 0) dicb_mbar_arrive(done + level);
            level++;
        }
        if (!MOVED && (w & TILE_OWN)) dst[w & TILE_ROW_MASK] = DIR == 0 ? tile_quotient(acc, y, d, rc) : y;
    }
    tile_row_sync();
    if (tid == 0 && *abort) {
        st->status = TFS_ERR_TIMEOUT;
        st->done = 1;
        st->niter_out = st->iter + 1;
    }
}

// D (with its reciprocal, tile_diags) and the values of one direction into round
// `round` of the packed rounds, from the factor d (internal row order) and the
// caller's values; a thread a slot.
template <typename T, int DIR>
__device__ __forceinline__ void tile_fill_round(const TileDev &P, int round, const DevParams *prm,
                                                const double *__restrict__ d)
{
    const uint4 c = __ldg(reinterpret_cast<const uint4 *>(P.rounds + round));
    const int t = threadIdx.x, slices = (int)(c.z >> 16);
    const size_t slot = (size_t)round * TILE_ROWS + t;
    const uint32_t w = __ldg(P.rows + slot);
    if ((w & TILE_ROW_MASK) == TILE_NO_ROW) return;
    unsigned char *at = P.packed + 16 * (size_t)c.x;
    const uint32_t head = reinterpret_cast<const uint32_t *>(at)[t >> 5];
    T *td = reinterpret_cast<T *>(at + TILE_HEAD + 32 * slices);
    const T di = (T)d[w & TILE_ROW_MASK];
    td[t] = di;
    if (tile_diags(DIR, sizeof(T)) == 2) td[32 * slices + t] = tile_recip(di);
    const double *val = prm->val_csr + __ldg(P.vbeg + slot);
    const int cnt = (int)((w >> TILE_CNT_SHIFT) & 15u);
    T *tv = td + 32 * slices * tile_diags(DIR, sizeof(T)) + (head & 0xffffu) * 32 + (t & 31);
    for (int j = 0; j < cnt; j++) tv[32 * j] = (T)val[j];
}

// Both directions' rounds, n0 of them forward; a block a round.  (One launch:
// a second one was 5 of the 15 us that packing adds to a small solve.)
template <typename T>
__global__ void __launch_bounds__(TILE_ROWS)
k_tile_fill(TileDev P0, TileDev P1, int n0, const DevParams *prm, const double *__restrict__ d)
{
    const int b = blockIdx.x;
    if (b < n0) tile_fill_round<T, 0>(P0, b, prm, d);
    else tile_fill_round<T, 1>(P1, b - n0, prm, d);
}

// rho = (r, z) after tiled sweeps, with the terms and the order of
// k_sweep0_rho (which sweeps level 0 as well): a thread adds r_i z_i of one
// row of level 0, then of the rows above it over a grid-stride loop.
template <typename T>
__global__ void __launch_bounds__(TFS_TPB)
k_rho_l0(const T *__restrict__ r, const T *__restrict__ z, int l0_rows, int n_int, DevState *st, double *part)
{
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const bool stop = (st->done) != 0;
    const int i = blockIdx.x * TFS_TPB + threadIdx.x;
    T acc = (T)0;
    if (i < l0_rows) {
        if constexpr (sizeof(T) == 4) acc = fmaf(r[i], z[i], acc);
        else acc = fma(r[i], z[i], acc);
    }
    const int stride = gridDim.x * TFS_TPB;
    int k = l0_rows + i;
    for (; k + 3 * stride < n_int; k += 4 * stride) {   // four rows' loads in flight
        T a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; q++) { a[q] = r[k + q * stride]; b[q] = z[k + q * stride]; }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if constexpr (sizeof(T) == 4) acc = fmaf(a[q], b[q], acc);
            else acc = fma(a[q], b[q], acc);
        }
    }
    for (; k < n_int; k += stride) {
        if constexpr (sizeof(T) == 4) acc = fmaf(r[k], z[k], acc);
        else acc = fma(r[k], z[k], acc);
    }
    if (stop) return;
    double v[1];
    bool last;
    if constexpr (sizeof(T) == 4) {
        const float av[1] = {acc};
        last = grid_reduce_f<1>(av, v, part, &st->counter);
    } else {
        v[0] = acc;
        last = grid_reduce<1, false>(v, part, &st->counter);
    }
    if (last) {
        st->rho = v[0];
        if (st->iter > 1) publish_beta(st);
        st->sweep_ns += gtimer() - st->t_sweep0;
        st->sweep_n += 1;
    }
}

}  // namespace tfs
