// tfs_assemble.cu -- matrix values assembled on the device from per-face
// coefficients through the face -> entry map (Matrix_Type%pos).
//
// The reference fills A%val face by face (NewUVW.f90:366-384,
// Compute_Pressure_Simple.f90:100-113): an interior face s between cells c1
// and c2 updates the entries (c1,c2) and (c2,c1) found through pos(1,s) and
// pos(2,s) and the two diagonals found through dia; a boundary face of a
// contributing type adds to the diagonal of c1; a cell loop then adds the
// inertial term to every diagonal (NewUVW.f90:500-505).  Every stored entry
// except the diagonal is touched by one face; a diagonal receives one
// addition per face of its cell, in face order.
//
// Here one thread owns one cell (one matrix row): it walks the faces of its
// cell in ascending face order -- a list built once per mesh on the host --
// updates the off-diagonal entries of its own row and sums its diagonal in
// exactly the reference's order, so the values are bitwise those of the
// sequential loops, and no two threads write the same entry.
//
// The path is bound by memory: four coefficients a face, the values twice.
// Cells numbered at random scatter both, so the cells are taken in the order
// of their first faces instead of their numbers: the 32 cells of a warp then
// share the sectors of their coefficients, and the face codes and entry
// offsets, stored in that order column by column, are read coalesced.  Only
// the rows of the values stay scattered; a warp brings its 32 rows into
// shared memory eight lanes a row, updates them there and writes them back
// the same way, a few 128-byte lines an access instead of 32.  On the 128^3
// mesh (random cell numbers, 6.5 M faces) an assembly takes 307 us, the 45 us
// reset of the values included (818 us when the cells were taken by number
// and each thread walked its row in global memory); its floor is about 110 us
// with the scattered rows' unused sectors counted, and what it waits for is
// latency: 64 registers, a few of them spilled, for four blocks per
// multiprocessor and four faces' coefficients in flight (eight faces 371 us
// at three blocks, 420 at four; five blocks 364).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "tfs_internal.h"

namespace {

constexpr int kTB = 256;
constexpr int kRow = 8;              // entries of a row held in shared memory
constexpr uint16_t kBoundary = 0xffffu;   // entry offset of a boundary face

// The mesh's faces by cell, in the order of the cells' first faces; slices of
// 32 cells, incidence j of lane t at slice_off + 32 j + t.
struct FaceMapDev {
    int n_cells;
    const int *cell, *begin;         // cell number, its row's first entry
    const uint32_t *info;            // entries of the row | offset of the diagonal << 16
    const int *count;                // faces of the cell
    const int *slice_off;
    const uint32_t *code;            // face << 1 | side (0: the cell is the face's c1)
    const uint16_t *off;             // offset in the row of the entry the face updates
};

// The cell's faces on its row `v` (its own memory or shared), diagonal dv;
// kBatch faces' coefficients are in flight at once.
template <int kBatch = 4, typename Row>
__device__ __forceinline__ double assemble_row(const FaceMapDev &F, Row v, double dv, int e0, int n,
                                               const double *__restrict__ off12, const double *__restrict__ off21,
                                               const double *__restrict__ dia12, const double *__restrict__ dia21)
{
    for (int j0 = 0; j0 < n; j0 += kBatch) {
        uint32_t code[kBatch];
        uint16_t at[kBatch];
        double o[kBatch], d[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; q++)
            if (j0 + q < n) {
                code[q] = __ldcs(F.code + e0 + 32 * (j0 + q));
                at[q] = __ldcs(F.off + e0 + 32 * (j0 + q));
            }
#pragma unroll
        for (int q = 0; q < kBatch; q++)
            if (j0 + q < n) {
                const uint32_t s = code[q] >> 1;
                d[q] = __ldg((code[q] & 1u ? dia21 : dia12) + s);
                o[q] = 0.0;
                if (at[q] != kBoundary) o[q] = __ldg((code[q] & 1u ? off21 : off12) + s);
            }
#pragma unroll
        for (int q = 0; q < kBatch; q++)
            if (j0 + q < n) {
                if (at[q] != kBoundary) {
                    v[at[q]] = v[at[q]] - o[q];
                    dv = dv + d[q];
                } else if (d[q] != 0.0) {
                    dv = dv + d[q];
                }
            }
    }
    return dv;
}

// A row of more entries than the shared rows hold, in place.
__device__ __noinline__ double assemble_long_row(const FaceMapDev &F, double *v, double dv, int e0, int n,
                                                 const double *off12, const double *off21, const double *dia12,
                                                 const double *dia21)
{
    return assemble_row(F, v, dv, e0, n, off12, off21, dia12, dia21);
}

// Cells that come in the order of their rows (a structured numbering): a row a
// thread, in place and face by face.  The rows of a warp are one run of memory
// and its coefficients nearly so, so the caches serve a walk along them, and
// what counts is how many warps walk: 128^3 lexicographic 132 us, with two
// faces in flight 142 to 153, four 157 to 190; with the rows through shared
// memory (k_assemble_faces) 197, by cell number with the incidence lists 165.
__global__ void __launch_bounds__(kTB, 4)
k_assemble_ordered(FaceMapDev F, const double *__restrict__ off12, const double *__restrict__ off21,
                   const double *__restrict__ dia12, const double *__restrict__ dia21,
                   const double *__restrict__ cell, double *val)
{
    for (int k = blockIdx.x * kTB + threadIdx.x; k < F.n_cells; k += gridDim.x * kTB) {
        double *const v = val + __ldg(F.begin + k);
        const int dia = (int)(__ldg(F.info + k) >> 16), n = __ldg(F.count + k);
        double dv = assemble_row<1>(F, v, v[dia], __ldg(F.slice_off + (k >> 5)) + (k & 31), n, off12,
                                    off21, dia12, dia21);
        if (cell) dv = dv + __ldg(cell + __ldg(F.cell + k));
        v[dia] = dv;
    }
}

__global__ void __launch_bounds__(kTB, 4)
k_assemble_faces(FaceMapDev F, const double *__restrict__ off12, const double *__restrict__ off21,
                 const double *__restrict__ dia12, const double *__restrict__ dia21,
                 const double *__restrict__ cell, double *val)
{
    __shared__ double sm[kTB / 32][32][kRow + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_slices = (F.n_cells + 31) >> 5;
    for (int s = blockIdx.x * (kTB / 32) + warp; s < n_slices; s += gridDim.x * (kTB / 32)) {
        const int k = 32 * s + lane;
        const bool mine = k < F.n_cells;
        const int begin = mine ? __ldg(F.begin + k) : 0;
        const uint32_t info = mine ? __ldg(F.info + k) : 0u;
        const int n = mine ? __ldg(F.count + k) : 0, e0 = __ldg(F.slice_off + s) + lane;
        const int len = (int)(info & 0xffffu), dia = (int)(info >> 16);
        const double add = cell && mine ? __ldg(cell + __ldg(F.cell + k)) : 0.0;
        if (__reduce_max_sync(0xffffffffu, (unsigned)len) > (unsigned)kRow) {   // long rows: in place
            if (mine) {
                double dv = assemble_long_row(F, val + begin, val[begin + dia], e0, n, off12, off21, dia12, dia21);
                if (cell) dv = dv + add;
                val[begin + dia] = dv;
            }
            continue;
        }
        const int e = lane & 7;
#pragma unroll 4
        for (int g = 0; g < 8; g++) {
            const int r = 4 * g + (lane >> 3);
            const int rb = __shfl_sync(0xffffffffu, begin, r), rl = __shfl_sync(0xffffffffu, len, r);
            if (e < rl) sm[warp][r][e] = val[rb + e];
        }
        __syncwarp();
        if (mine) {
            double *v = sm[warp][lane];
            double dv = assemble_row(F, v, v[dia], e0, n, off12, off21, dia12, dia21);
            if (cell) dv = dv + add;
            v[dia] = dv;
        }
        __syncwarp();
#pragma unroll 4
        for (int g = 0; g < 8; g++) {
            const int r = 4 * g + (lane >> 3);
            const int rb = __shfl_sync(0xffffffffu, begin, r), rl = __shfl_sync(0xffffffffu, len, r);
            if (e < rl) val[rb + e] = sm[warp][r][e];
        }
        __syncwarp();
    }
}

}  // namespace

struct FaceMap {
    int n_faces = 0;
    bool ordered = false;   // most cells come one after the other by number
    int *cell = nullptr, *begin = nullptr, *count = nullptr, *slice_off = nullptr;   // FaceMapDev
    uint32_t *info = nullptr, *code = nullptr;
    uint16_t *off = nullptr;
    int64_t bytes = 0;
};

void tfs_faces_free(tfs_handle *h)
{
    if (!h || !h->faces) return;
    FaceMap *F = h->faces;
    for (void *p : {(void *)F->cell, (void *)F->begin, (void *)F->count, (void *)F->slice_off, (void *)F->info,
                    (void *)F->code, (void *)F->off})
        if (p) cudaFree(p);
    h->device_bytes -= F->bytes;
    delete F;
    h->faces = nullptr;
}

extern "C" int tfs_faces_register(tfs_handle *h, int32_t n_faces, const int32_t *faces_c,
                                  const int32_t *pos1)
{
    if (!h || n_faces < 0 || (n_faces > 0 && (!faces_c || !pos1))) return TFS_ERR_ARG;
    const int n = h->n;
    // Validate against the registered topology: cell numbers in range, the
    // positions of an interior face inside the rows of c1 and c2 and off the
    // diagonal, boundary faces with c2 <= 0.  On the way the cells are put in
    // the order of their first faces, those without one at the end.  (What a
    // cell needs in one place: its faces are all over the mesh, and each visit
    // is a miss.)
    struct Cell {
        int place = -1, faces = 0;
    };
    std::vector<Cell> cells(n);
    std::vector<int> order;
    order.reserve(n);
    auto visit = [&](int c) {
        Cell &q = cells[c];
        if (q.place < 0) {
            q.place = (int)order.size();
            order.push_back(c);
        }
        return &q;
    };
    for (int s = 0; s < n_faces; s++) {
        const int c1 = faces_c[2 * s], c2 = faces_c[2 * s + 1];
        if (c1 < 1 || c1 > n || c2 > n) {
            tfs_set_error_text("tfs_faces_register: cell number out of range");
            return TFS_ERR_ARG;
        }
        if (c2 > 0) {
            const int p1 = pos1[2 * s] - 1, p2 = pos1[2 * s + 1] - 1;
            if (p1 < h->row0[c1 - 1] || p1 >= h->row0[c1] || p1 == h->dia0[c1 - 1] ||
                p2 < h->row0[c2 - 1] || p2 >= h->row0[c2] || p2 == h->dia0[c2 - 1]) {
                tfs_set_error_text("tfs_faces_register: pos does not match the registered topology");
                return TFS_ERR_ARG;
            }
        }
        visit(c1 - 1)->faces++;
        if (c2 > 0) visit(c2 - 1)->faces++;
    }
    for (int c = 0; c < n; c++) visit(c);
    const int n_slices = (n + 31) / 32;
    std::vector<int> slice_off(n_slices + 1, 0), begin(n), count(n);
    std::vector<uint32_t> info(n);
    int64_t total = 0;
    for (int s = 0; s < n_slices; s++) {
        int width = 0;
        for (int k = 32 * s; k < std::min(n, 32 * s + 32); k++) {
            const int c = order[k];
            width = std::max(width, cells[c].faces);
            begin[k] = h->row0[c];
            count[k] = cells[c].faces;
            info[k] = (uint32_t)(h->row0[c + 1] - h->row0[c]) | (uint32_t)(h->dia0[c] - h->row0[c]) << 16;
        }
        slice_off[s] = (int)total;
        total += 32 * (int64_t)width;
        if (total > INT32_MAX) {
            tfs_set_error_text("tfs_faces_register: too many faces");
            return TFS_ERR_ARG;
        }
    }
    slice_off[n_slices] = (int)total;
    // (from here on: the place of the cell's next incidence, its row's start)
    struct Next {
        uint32_t at;
        int row;
    };
    std::vector<Next> next(n);
    for (int k = 0; k < n; k++) next[order[k]] = Next{(uint32_t)(slice_off[k >> 5] + (k & 31)), begin[k]};
    std::vector<uint32_t> code((size_t)total + 1, 0u);
    std::vector<uint16_t> off((size_t)total + 1, 0);
    auto add = [&](int c, uint32_t f, int at) {
        Next &q = next[c];
        code[q.at] = f;
        off[q.at] = at < 0 ? kBoundary : (uint16_t)(at - q.row);
        q.at += 32;
    };
    for (int s = 0; s < n_faces; s++) {   // ascending s: each cell's list ends up sorted
        const int c1 = faces_c[2 * s], c2 = faces_c[2 * s + 1];
        add(c1 - 1, (uint32_t)s << 1, c2 > 0 ? pos1[2 * s] - 1 : -1);
        if (c2 > 0) add(c2 - 1, (uint32_t)s << 1 | 1u, pos1[2 * s + 1] - 1);
    }
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return tfs_engine_error(e, "cudaSetDevice");
    tfs_faces_free(h);
    FaceMap *F = new FaceMap();
    F->n_faces = n_faces;
    int follow = 0;
    for (int k = 1; k < n; k++) follow += order[k] == order[k - 1] + 1;
    F->ordered = 2 * (int64_t)follow > n;
    h->faces = F;
    auto up = [&](auto **dst, const auto &src) -> cudaError_t {
        const size_t bytes = sizeof(src[0]) * std::max<size_t>(src.size(), 1);
        cudaError_t err = cudaMalloc((void **)dst, bytes);
        if (err != cudaSuccess) return err;
        F->bytes += (int64_t)bytes;
        h->device_bytes += (int64_t)bytes;
        return cudaMemcpyAsync(*dst, src.data(), sizeof(src[0]) * src.size(), cudaMemcpyHostToDevice, h->stream);
    };
    if ((e = up(&F->cell, order)) != cudaSuccess || (e = up(&F->begin, begin)) != cudaSuccess ||
        (e = up(&F->info, info)) != cudaSuccess || (e = up(&F->count, count)) != cudaSuccess ||
        (e = up(&F->slice_off, slice_off)) != cudaSuccess || (e = up(&F->code, code)) != cudaSuccess ||
        (e = up(&F->off, off)) != cudaSuccess) {
        cudaStreamSynchronize(h->stream);
        tfs_faces_free(h);
        return tfs_engine_error(e, "tfs_faces_register upload");
    }
    // The host vectors go out of scope: wait for the copies.
    e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return tfs_engine_error(e, "tfs_faces_register");
    return TFS_OK;
}

extern "C" int tfs_assemble_faces_device(tfs_handle *h, const double *d_off12, const double *d_off21,
                                         const double *d_dia12, const double *d_dia21,
                                         const double *d_cell, double *d_val)
{
    if (!h || !h->faces || !d_val) return TFS_ERR_ARG;
    FaceMap *F = h->faces;
    if (F->n_faces > 0 && (!d_off12 || !d_off21 || !d_dia12 || !d_dia21)) return TFS_ERR_ARG;
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return tfs_engine_error(e, "cudaSetDevice");
    const int n = h->n;
    int blocks = (n + kTB - 1) / kTB;
    if (blocks > h->sm_count * 16) blocks = h->sm_count * 16;
    if (blocks < 1) blocks = 1;
    const FaceMapDev D{n, F->cell, F->begin, F->info, F->count, F->slice_off, F->code, F->off};
    auto kernel = F->ordered ? k_assemble_ordered : k_assemble_faces;
    kernel<<<blocks, kTB, 0, h->stream>>>(D, d_off12, d_off21, d_dia12, d_dia21, d_cell, d_val);
    e = cudaGetLastError();
    if (e != cudaSuccess) return tfs_engine_error(e, "k_assemble_faces launch");
    return TFS_OK;
}
