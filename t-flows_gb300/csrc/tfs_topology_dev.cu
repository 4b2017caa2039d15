// tfs_topology_dev.cu -- Matrix_Mod_Topology on the device.
//
// The reference builds the compressed-row topology of its matrix once per
// mesh on the host (Matrix_Mod/Topology.f90:2-127): stencil widths from the
// faces (:33-41), row starts with the diagonal first (:54-59), off-diagonal
// columns in face order (:62-71), every row sorted ascending and its
// diagonal located (:75-82), the mirror position of every entry (:85-103)
// and the two entry positions of every interior face (:106-121).  The same
// arrays come out of this file, bit for bit, built on the device:
//
//   k_topo_count        stencil widths; the integer atomic that counts an
//                       entry also numbers it within its row
//   k_scan_*            row starts: exclusive prefix sum of the widths (a
//                       three-pass scan: per block, block totals, add back)
//   k_topo_fill         every entry's face side into its numbered slot
//   k_topo_sort         each row sorted ascending by its columns (a row holds
//                       distinct cell numbers, so the sorted row is unique
//                       whatever order the slots were filled in): col, dia
//                       and pos, which is where an entry's face side says
//   k_topo_mir          mir(p): the position of the entry of the same face's
//                       other side
//
// What bounds it is the scattered access to 12.8 M face sides (128^3 mesh,
// random cell numbers): one atomic, two reads and two writes each.  The
// entries carry their face sides through the sort so that neither mir nor
// pos is searched for (three row searches an entry and face before), the
// sort runs in registers with its output staged in shared memory, and the
// widths, numbers and face sides live in the output arrays until those are
// due, so that a call allocates nothing (17 MB before).  What is
// read or written once goes past the caches' replacement (ld/st .cs), which
// keeps the randomly accessed arrays in L2.  128^3 mesh: 570 us a call, 1,021
// with the searches (600 without the cache hints).
//
// The faces must join distinct pairs of distinct cells (each stored entry
// then belongs to exactly one face side; where several faces join a pair all
// the same, every one of its entries gets the pair's first place as mir and
// every face its last as pos, as row searches give them), as meshes from the
// reference's
// generators do; every array is 1-based, as in the reference.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "tfs_internal.h"

namespace {

constexpr int kTB = 256;

constexpr int kRowMax = 8;     // entries of a row sorted in registers

// The error flag and the entry count of the call in progress (one at a time:
// g_topo_mutex).  A device variable of the library, so that a call allocates
// nothing: cudaMalloc and cudaFree took up to 0.2 ms of it.
struct TopoState {
    int bad, total;
    int twice;        // a pair of cells is joined by more than one face
};
__device__ TopoState g_topo;
std::mutex g_topo_mutex;

__global__ void k_topo_reset() { g_topo = TopoState{0, 0, 0}; }

__global__ void k_topo_zero(int n, int *width)
{
    if (g_topo.bad) return;
    for (int c = blockIdx.x * kTB + threadIdx.x; c < n; c += gridDim.x * kTB) width[c] = 0;
}

// Widths without the diagonal, and every interior face side's number in its
// row (rank, 2 n_faces; 0 for a boundary face).
__global__ void k_topo_count(int n_faces, const int *__restrict__ fc, int *width, int *rank)
{
    if (g_topo.bad) return;
    for (int s = blockIdx.x * kTB + threadIdx.x; s < n_faces; s += gridDim.x * kTB) {
        const int c1 = __ldcs(fc + 2 * s), c2 = __ldcs(fc + 2 * s + 1);
        int r1 = 0, r2 = 0;
        if (c2 > 0) {
            r1 = atomicAdd(width + c1 - 1, 1);
            r2 = atomicAdd(width + c2 - 1, 1);
        }
        __stcs(rank + 2 * s, r1);
        __stcs(rank + 2 * s + 1, r2);
    }
}

// Exclusive scan, pass 1: each block scans kTB * 4 elements, one more each
// for the row's diagonal, and writes its total.
__global__ void k_scan_block(int n, const int *__restrict__ in, int *out, int *block_sum)
{
    if (g_topo.bad) return;
    __shared__ int sm[kTB];
    const int base = blockIdx.x * kTB * 4;
    int v[4], t = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int i = base + threadIdx.x * 4 + q;
        v[q] = i < n ? 1 + in[i] : 0;
        t += v[q];
    }
    sm[threadIdx.x] = t;
    __syncthreads();
    for (int o = 1; o < kTB; o <<= 1) {   // inclusive scan of the thread totals
        const int a = threadIdx.x >= o ? sm[threadIdx.x - o] : 0;
        __syncthreads();
        sm[threadIdx.x] += a;
        __syncthreads();
    }
    int run = sm[threadIdx.x] - t;        // exclusive prefix of this thread
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int i = base + threadIdx.x * 4 + q;
        if (i < n) out[i] = run;
        run += v[q];
    }
    if (threadIdx.x == kTB - 1) block_sum[blockIdx.x] = sm[kTB - 1];
}

// Pass 2 (one block): exclusive scan of the block totals in place, a run of
// them a thread; the grand total goes to g_topo.
__global__ void __launch_bounds__(1024) k_scan_totals(int nb, int *block_sum)
{
    if (g_topo.bad) return;
    __shared__ int sm[32];
    const int per = (nb + 1023) / 1024, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b0 = min(nb, (int)threadIdx.x * per), b1 = min(nb, b0 + per);
    int t = 0;
    for (int b = b0; b < b1; b++) t += block_sum[b];
    int incl = t;
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += a;
    }
    if (lane == 31) sm[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int w = sm[lane];
        int wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += a;
        }
        sm[lane] = wi - w;
        if (lane == 31) g_topo.total = wi;
    }
    __syncthreads();
    int run = sm[warp] + incl - t;
    for (int b = b0; b < b1; b++) {
        const int v = block_sum[b];
        block_sum[b] = run;
        run += v;
    }
}

// Pass 3: row(c) = 1 + exclusive prefix (in row1 already within its block);
// row(n+1) = 1 + total.
__global__ void k_scan_add(int n, const int *__restrict__ block_sum, int *row1)
{
    if (g_topo.bad) return;
    for (int i = blockIdx.x * kTB + threadIdx.x; i <= n; i += gridDim.x * kTB)
        row1[i] = i < n ? 1 + row1[i] + block_sum[i / (kTB * 4)] : 1 + g_topo.total;
}

// Every entry's face side (face << 1 | side of the row's own cell) at its
// row's start + its number; the slot of the diagonal, the row's last, is
// left alone.
__global__ void k_topo_fill(int n_faces, const int *__restrict__ fc, const int *__restrict__ rank,
                            const int *__restrict__ row1, int *side)
{
    if (g_topo.bad) return;
    for (int s = blockIdx.x * kTB + threadIdx.x; s < n_faces; s += gridDim.x * kTB) {
        const int c1 = __ldcs(fc + 2 * s), c2 = __ldcs(fc + 2 * s + 1);
        if (c2 > 0) {
            const int r1 = __ldcs(rank + 2 * s), r2 = __ldcs(rank + 2 * s + 1);
            side[__ldg(row1 + c1 - 1) - 1 + r1] = 2 * s;
            side[__ldg(row1 + c2 - 1) - 1 + r2] = 2 * s + 1;
        }
    }
}

// Rows sorted: col1, dia1, pos1, and side (in place: the sorted entries'
// face sides, -1 for the diagonal).  One thread a row; the block's rows are
// one contiguous range of entries, brought in and out through shared memory
// when every row has at most kRowMax entries, else sorted where they are.
__global__ void __launch_bounds__(kTB)
k_topo_sort(int n_cells, const int *__restrict__ fc, const int *__restrict__ row1, int *col1, int *side, int *dia1,
            int *pos1)
{
    if (g_topo.bad) return;
    __shared__ int sc[kTB * kRowMax], ss[kTB * kRowMax];
    for (int c0 = blockIdx.x * kTB; c0 < n_cells; c0 += gridDim.x * kTB) {
        const int c = c0 + threadIdx.x;
        const int first = row1[c0] - 1, end = row1[min(n_cells, c0 + kTB)] - 1;
        const int b = c < n_cells ? row1[c] - 1 : end, e = c < n_cells ? row1[c + 1] - 1 : end, len = e - b;
        if (__syncthreads_or(len > kRowMax)) {
            if (c < n_cells) {
                side[e - 1] = -1;
                for (int a = b; a < e; a++) col1[a] = side[a] < 0 ? c + 1 : __ldg(fc + (side[a] ^ 1));
                for (int a = b + 1; a < e; a++) {
                    const int v = col1[a], w = side[a];
                    int k = a - 1;
                    while (k >= b && col1[k] > v) {
                        col1[k + 1] = col1[k];
                        side[k + 1] = side[k];
                        k--;
                    }
                    col1[k + 1] = v;
                    side[k + 1] = w;
                }
                for (int p = e - 1, last = e; p >= b; p--) {   // last: of the entries of this column
                    if (p + 1 < e && col1[p] == col1[p + 1]) g_topo.twice = 1;
                    else last = p + 1;
                    if (side[p] < 0) dia1[c] = p + 1;
                    else pos1[side[p]] = last;
                }
            }
            __syncthreads();
            continue;
        }
        for (int p = first + threadIdx.x; p < end; p += kTB) ss[p - first] = __ldcs(side + p);
        __syncthreads();
        if (c < n_cells) {
            int v[kRowMax], w[kRowMax];
#pragma unroll
            for (int q = 0; q < kRowMax; q++) {
                w[q] = q < len - 1 ? ss[b - first + q] : -1;
                v[q] = q < len - 1 ? __ldg(fc + (w[q] ^ 1)) : q == len - 1 ? c + 1 : INT32_MAX;
            }
            // odd-even transposition: kRowMax rounds sort kRowMax entries
#pragma unroll
            for (int r = 0; r < kRowMax; r++)
#pragma unroll
                for (int q = r & 1; q + 1 < kRowMax; q += 2)
                    if (v[q] > v[q + 1]) {
                        const int tv = v[q], tw = w[q];
                        v[q] = v[q + 1];
                        w[q] = w[q + 1];
                        v[q + 1] = tv;
                        w[q + 1] = tw;
                    }
            bool twice = false;
#pragma unroll
            for (int q = 0; q < kRowMax; q++)
                if (q < len) {
                    sc[b - first + q] = v[q];
                    ss[b - first + q] = w[q];
                    if (w[q] < 0) dia1[c] = b + q + 1;
                    else pos1[w[q]] = b + q + 1;
                    if (q > 0) twice = twice || v[q] == v[q - 1];
                }
            if (twice) {
                g_topo.twice = 1;
                for (int q = len - 2, last = len; q >= 0; q--) {
                    if (sc[b - first + q] != sc[b - first + q + 1]) last = q + 1;
                    if (ss[b - first + q] >= 0) pos1[ss[b - first + q]] = b + last;
                }
            }
        }
        __syncthreads();
        for (int p = first + threadIdx.x; p < end; p += kTB) {
            __stcs(col1 + p, sc[p - first]);
            __stcs(side + p, ss[p - first]);
        }
        __syncthreads();
    }
}

// mir(p) in place of the entry's face side: the position of the same face's
// other entry (the first of its pair), or the diagonal's own.
__global__ void k_topo_mir(const int *__restrict__ pos1, const int *__restrict__ row1, const int *__restrict__ col1,
                           int *mir1)
{
    if (g_topo.bad) return;
    const int n = g_topo.total;
    const bool twice = g_topo.twice != 0;
    for (int p = blockIdx.x * kTB + threadIdx.x; p < n; p += gridDim.x * kTB) {
        const int s = __ldcs(mir1 + p);
        int m = s < 0 ? p + 1 : __ldg(pos1 + (s ^ 1));
        if (twice && s >= 0)
            for (const int row = __ldg(row1 + __ldg(col1 + p) - 1); m > row && col1[m - 2] == col1[m - 1];) m--;
        __stcs(mir1 + p, m);
    }
}

// Faces are checked before anything is built: 1 <= c1 <= n_cells,
// c2 <= n_cells, c1 != c2.  Any violation sets g_topo.bad, and every kernel after
// this one returns at once, so that the host need not wait in between.
__global__ void k_topo_check(int n_cells, int n_faces, const int *__restrict__ fc)
{
    for (int s = blockIdx.x * kTB + threadIdx.x; s < n_faces; s += gridDim.x * kTB) {
        const int c1 = fc[2 * s], c2 = fc[2 * s + 1];
        if (c1 < 1 || c1 > n_cells || c2 > n_cells || c2 == c1) atomicOr(&g_topo.bad, 1);
    }
}

}  // namespace

extern "C" int tfs_topology_build_device(int32_t n_cells, int32_t n_faces, const int32_t *d_faces_c,
                                         int32_t *d_row1, int32_t *d_col1, int32_t *d_dia1,
                                         int32_t *d_mir1, int32_t *d_pos1, int32_t *nnz_out)
{
    if (n_cells <= 0 || n_faces < 0 || !d_row1 || !d_col1 || !d_dia1 || !d_mir1 || !nnz_out ||
        (n_faces > 0 && (!d_faces_c || !d_pos1)))
        return TFS_ERR_ARG;
    if ((int64_t)n_cells + 2 * (int64_t)n_faces > INT32_MAX) return TFS_ERR_ARG;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return tfs_engine_error(e, "cudaGetDevice");
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return tfs_engine_error(e, "cudaDeviceGetAttribute");
    auto grid = [&](int64_t items) {
        int64_t b = (items + kTB - 1) / kTB;
        if (b > (int64_t)sms * 16) b = (int64_t)sms * 16;
        return (int)(b < 1 ? 1 : b);
    };
    const int nb = (n_cells + kTB * 4 - 1) / (kTB * 4);
    // The widths wait in dia1, the block totals and then the entries' face
    // sides in mir1, the face sides' numbers in pos1.
    int *bsum = d_mir1;
    std::lock_guard<std::mutex> lock(g_topo_mutex);
    k_topo_reset<<<1, 1>>>();
    if (n_faces > 0) k_topo_check<<<grid(n_faces), kTB>>>(n_cells, n_faces, d_faces_c);
    k_topo_zero<<<grid(n_cells), kTB>>>(n_cells, d_dia1);
    if (n_faces > 0) k_topo_count<<<grid(n_faces), kTB>>>(n_faces, d_faces_c, d_dia1, d_pos1);
    k_scan_block<<<nb, kTB>>>(n_cells, d_dia1, d_row1, bsum);
    k_scan_totals<<<1, 1024>>>(nb, bsum);
    k_scan_add<<<grid((int64_t)n_cells + 1), kTB>>>(n_cells, bsum, d_row1);
    if (n_faces > 0) k_topo_fill<<<grid(n_faces), kTB>>>(n_faces, d_faces_c, d_pos1, d_row1, d_mir1);
    k_topo_sort<<<grid(n_cells), kTB>>>(n_cells, d_faces_c, d_row1, d_col1, d_mir1, d_dia1, d_pos1);
    k_topo_mir<<<grid((int64_t)n_cells + 2 * (int64_t)n_faces), kTB>>>(d_pos1, d_row1, d_col1, d_mir1);
    e = cudaGetLastError();
    TopoState out{0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&out, g_topo, sizeof out);
    if (e != cudaSuccess) return tfs_engine_error(e, "tfs_topology_build_device");
    if (out.bad) {
        tfs_set_error_text("tfs_topology_build_device: a face has a cell number out of range or c1 == c2");
        return TFS_ERR_TOPOLOGY;
    }
    *nnz_out = out.total;
    return TFS_OK;
}
