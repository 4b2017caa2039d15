// tfs_dic_tiles_plan.h -- host-side plan of the tiled DIC sweeps
// (tfs_dic_tiles.cuh): a partition of the rows into compact tiles and, per
// sweep direction, everything one thread block needs to sweep its tile with
// no other block's help.  No CUDA calls: the engine includes it, and the
// host compiler builds it on its own for the tests.
//
// A row's value in a triangular sweep depends only on the rows reached from
// it through entries on the swept side (its closure).  Under the numbering an
// unstructured mesh generator leaves, where neighbours' numbers are in no
// particular order, closures are short: a compact tile of 24^3 cells of a
// hexahedral mesh and the closure of its rows are 1.32 times the tile.  A
// block that sweeps its tile's closure level by level in shared memory
// therefore waits for nobody, at the price of computing a third of the rows
// twice -- with the same operations in the same order, so to the same bits.
// Under a structured mesh's own numbering closures reach through the whole
// mesh; then there is no plan (tiles = 0).
//
// The partition: graph distances to a few far-apart rows (landmarks) as
// coordinates, and recursive bisection of the rows at the median along the
// coordinates' direction of largest variance.  On a 128^3 hexahedral mesh and
// 152 tiles the tiles with their closures hold 1.32 n rows (six landmarks;
// 1.45 n with four, 1.31 n with eight; cubes of the same size 1.32 n; halves
// of a breadth-first order instead 1.35 n).
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <utility>
#include <vector>

namespace tfs {

constexpr int TILE_ROWS = 512;           // rows of a round (a row per thread); a multiple of 32, at most 992
constexpr int TILE_SLICES = TILE_ROWS / 32;
constexpr uint32_t TILE_ROW_MASK = 0x03ffffffu;  // row word: internal row,
constexpr int TILE_CNT_SHIFT = 26;               // entries on the swept side (0..15) << 26,
constexpr uint32_t TILE_OWN = 0x80000000u;       // own row of the tile (its value is stored)
constexpr uint32_t TILE_NO_ROW = TILE_ROW_MASK;  // no row
constexpr int TILE_MAX_CNT = 15;
constexpr int TILE_MAX_ROUNDS = 512;     // rounds of one tile and direction
constexpr int TILE_MAX_SLOTS = 65504;    // slots of one tile: 16-bit entry indices
constexpr int TILE_MAX_LEVELS = 64;      // deeper schedules have long closures
constexpr int TILE_BARS = 16;            // rounds staged ahead at most
constexpr int TILE_MOVERS = 224;         // threads that move vectors one way: rows of a list round
constexpr int TILE_MAX_LISTS = 1024;     // list rounds of one tile and direction
constexpr int TILE_HEAD = 128;           // bytes of a round's head: a word per slice

// One round: up to TILE_ROWS slots (slices of 32 rows) of one level of one
// tile.  Its packed bytes, one bulk copy: a word per slice (its first entry /
// 32 in the round | its width << 16), every slot's number of entries (a
// byte), D of every slot, in binary64 and
// forward also the rounded reciprocal of D of every slot, the values, then
// the 16-bit local slots of the entries (column-major inside a slice).
//   x  first packed byte / 16 (over the whole direction)
//   y  packed bytes / 16 | rounds back to the one whose release makes room
//      in the ring << 16 (0: none) | last round of its level << 24
//   z  first slot in the tile | slices << 16
//   w  place in the ring / 128 | place of the indices in the round / 16 << 16
struct TileRound {
    uint32_t x, y, z, w;
};

// The rows of a level are moved between the vectors and the slots in another
// order than they are swept in: by internal row, so that a warp's accesses
// fall into few 128-byte lines (sorted by entry count, as they are swept, a
// warp touches about 28; by row about 9).  A list round is up to TILE_MOVERS
// rows of one level.

// One sweep direction.
struct TileDir {
    std::vector<int> tile_round;         // first round of every tile (n_tiles + 1)
    std::vector<TileRound> rounds;
    std::vector<uint32_t> rows;          // row word per round and thread
    std::vector<int> vbeg;               // CSR position of that row's first entry
    std::vector<uint8_t> packed;         // every round's packed bytes, D and values left zero
    std::vector<int> tile_list;          // first list round of every tile (n_tiles + 1)
    std::vector<uint8_t> lists;          // per list round: level of the tile | last of the level << 7
    std::vector<uint32_t> list_row;      // per list round and thread: internal row, own row flag
    std::vector<uint16_t> list_slot;     // and the row's slot
};

// A plan in values of `ts` bytes.
struct TilePlan {
    int tiles = 0;                       // 0: no plan
    int ts = 0;
    int max_slots = 0;                   // slots of the largest tile
    int max_rounds = 0;                  // rounds of the tile with most
    int max_lists = 0;                   // list rounds of the tile with most
    int ring_bytes = 0;                  // the ring of packed rounds
    int smem_bytes = 0;                  // dynamic shared memory of a sweep
    double redundancy = 0.0;             // rows swept per row, the larger direction
    TileDir dir[2];                      // forward, backward

    // Device bytes of its arrays.
    int64_t bytes() const
    {
        int64_t b = 0;
        for (const TileDir &D : dir)
            b += (int64_t)(4 * (D.tile_round.size() + D.tile_list.size() + D.rows.size() + D.vbeg.size() +
                                D.list_row.size()) +
                           2 * D.list_slot.size() + D.packed.size() + D.lists.size() +
                           sizeof(TileRound) * D.rounds.size());
        return b;
    }
};

// Dynamic shared memory of a sweep: the tile's vector, the ring, the round
// table, the list table, the mbarriers (full and empty of the ring, loaded
// and done of every level) and the abort flag.
inline int tile_vec_bytes(int max_slots, int ts) { return (max_slots * ts + 127) & ~127; }
inline int tile_fixed_bytes(int max_slots, int max_rounds, int max_lists, int ts)
{
    return tile_vec_bytes(max_slots, ts) + max_rounds * (int)sizeof(TileRound) + ((max_lists + 15) & ~15) +
           (2 * TILE_BARS + 2 * TILE_MAX_LEVELS) * 8 + 16;
}

// Arrays of one value per slot before a round's values: D and, in binary64
// and forward, its reciprocal.
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int tile_diags(int dir, int ts) { return dir == 0 && ts == 8 ? 2 : 1; }

// Places a tile's rounds one after the other in a ring of `ring` bytes (a
// round never wraps) and notes for each how many rounds back the last one is
// that it overwrites; false when a round does not fit.  Two rounds at least
// fit beside each other when every round takes at most half the ring.
inline bool tile_place(TileRound *r, int n, int ring)
{
    std::vector<std::pair<int, int>> at(n);
    int head = 0;
    for (int k = 0; k < n; k++) {
        const int bytes = (int)((r[k].y & 0xffffu) * 16u + 127u) & ~127;
        if (bytes > ring) return false;
        if (head + bytes > ring) head = 0;
        at[k] = {head, head + bytes};
        int back = 0;
        for (int q = 1; q <= TILE_BARS && q <= k; q++) {
            const auto &o = at[k - q];
            if (q == TILE_BARS || (o.first < at[k].second && at[k].first < o.second)) { back = q; break; }
        }
        r[k].y = (r[k].y & 0xff00ffffu) | (uint32_t)back << 16;
        r[k].w = (r[k].w & 0xffff0000u) | (uint32_t)(head / 128);
        head += bytes;
    }
    return true;
}

// The copy lane's walk over a tile's rounds: the kernel's, and on the host its
// test's.  C: back(k) how many rounds back the last one is that round k
// overwrites (0: none); released(k) waits until the row warps have released
// round k, false when that wait ends otherwise; off() whether the sweep has
// been called off; issue(k) starts round k's copy; landed(k) waits for it.
//   - The flag is asked after the wait: in a sweep that is called off, rounds
//     are released that have not landed.
//   - The last rounds issued are waited for however the walk ends.  Those
//     before them have landed, since one of these overwrites them.  Asking the
//     flag whether to wait is not enough: a sweep that has nothing to do is
//     called off after its dependency wait, when the lane of a tile whose
//     rounds all fit the ring is long through, and the block would leave with
//     copies on their way into shared memory that is another's by then.
template <class C>
#ifdef __CUDACC__
__device__
#endif
inline void tile_copy_walk(int rounds, C &c)
{
    int k = 0;
    for (; k < rounds; k++) {
        const int back = c.back(k);
        if ((back && !c.released(k - back)) || c.off()) break;
        c.issue(k);
    }
    for (int q = k > TILE_BARS ? k - TILE_BARS : 0; q < k; q++) c.landed(q);
}

// Runs fn(k, thread) for k in [0, n) on up to `threads` host threads, fewer
// where the system refuses to start one.  An exception of fn ends the run and
// is thrown again here, once every thread is through.
template <class F>
inline void tile_parallel(int n, int threads, F fn)
{
    threads = std::max(1, std::min(threads, n));
    std::atomic<int> next{0};
    std::exception_ptr error;
    std::mutex mu;
    auto work = [&](int t) {
        try {
            for (int k; (k = next.fetch_add(1)) < n;) fn(k, t);
        } catch (...) {
            next = n;
            std::lock_guard<std::mutex> lock(mu);
            if (!error) error = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve((size_t)threads);
    try {
        for (int t = 1; t < threads; t++) pool.emplace_back(work, t);
    } catch (const std::exception &) {   // the threads there are do the work
    }
    work(0);
    for (auto &t : pool) t.join();
    if (error) std::rethrow_exception(error);
}

// Rows (in the order `pos`, which keeps mesh neighbours close) into `tiles`
// compact tiles of equal size; tile_of[k] for the row at position k.
inline void tile_partition(int n, const std::vector<int> &adj_ptr, const std::vector<int> &adj, int tiles,
                           int threads, std::vector<int> &tile_of)
{
    constexpr int L = 6;
    tile_of.assign(n, 0);
    if (tiles <= 1) return;
    // Landmarks: each the row farthest from the ones before (ties: largest
    // sum of distances); rows a landmark does not reach count as farthest.
    std::vector<float> X((size_t)n * L);
    {
        std::vector<int> d(n), q(n), mn(n, INT32_MAX);
        std::vector<long long> sum(n, 0);
        int s = 0;
        for (int l = 0; l < L; l++) {
            std::fill(d.begin(), d.end(), -1);
            int head = 0, tail = 0;
            q[tail++] = s;
            d[s] = 0;
            while (head < tail) {
                const int u = q[head++];
                for (int j = adj_ptr[u]; j < adj_ptr[u + 1]; j++)
                    if (d[adj[j]] < 0) {
                        d[adj[j]] = d[u] + 1;
                        q[tail++] = adj[j];
                    }
            }
            const int beyond = d[q[tail - 1]] + 1;
            int best = 0;
            for (int i = 0; i < n; i++) {
                if (d[i] < 0) d[i] = beyond;
                X[(size_t)i * L + l] = (float)d[i];
                mn[i] = std::min(mn[i], d[i]);
                sum[i] += d[i];
                if (mn[i] > mn[best] || (mn[i] == mn[best] && sum[i] > sum[best])) best = i;
            }
            s = best;
        }
    }
    struct Part {
        int a, b, t0, nt;
    };
    std::vector<int> id(n);
    for (int i = 0; i < n; i++) id[i] = i;
    std::vector<std::pair<float, int>> key(n);
    std::vector<Part> level(1, Part{0, n, 0, tiles}), next;
    while (!level.empty()) {
        next.assign(2 * level.size(), Part{0, 0, 0, 0});
        tile_parallel((int)level.size(), threads, [&](int k, int) {
            const Part p = level[k];
            if (p.nt == 1) {
                for (int i = p.a; i < p.b; i++) tile_of[id[i]] = p.t0;
                return;
            }
            // Direction of largest variance of a sample's coordinates.
            double m[L] = {}, S[L][L] = {}, w[L];
            const int step = std::max(1, (p.b - p.a) / 4096);
            int cnt = 0;
            for (int i = p.a; i < p.b; i += step, cnt++)
                for (int l = 0; l < L; l++) m[l] += X[(size_t)id[i] * L + l];
            for (int l = 0; l < L; l++) m[l] /= std::max(1, cnt);
            for (int i = p.a; i < p.b; i += step) {
                double v[L];
                for (int l = 0; l < L; l++) v[l] = X[(size_t)id[i] * L + l] - m[l];
                for (int r = 0; r < L; r++)
                    for (int c = 0; c < L; c++) S[r][c] += v[r] * v[c];
            }
            for (int l = 0; l < L; l++) w[l] = 1.0 + 0.1 * l;
            for (int it = 0; it < 64; it++) {
                double y[L], nn = 0.0;
                for (int r = 0; r < L; r++) {
                    y[r] = 0.0;
                    for (int c = 0; c < L; c++) y[r] += S[r][c] * w[c];
                    nn += y[r] * y[r];
                }
                if (!(nn > 0.0)) break;
                for (int r = 0; r < L; r++) w[r] = y[r] / std::sqrt(nn);
            }
            for (int i = p.a; i < p.b; i++) {
                float s = 0.f;
                for (int l = 0; l < L; l++) s += (float)w[l] * X[(size_t)id[i] * L + l];
                key[i] = {s, id[i]};
            }
            const int h = p.nt / 2, mid = p.a + (int)((int64_t)(p.b - p.a) * h / p.nt);
            std::nth_element(key.begin() + p.a, key.begin() + mid, key.begin() + p.b);
            for (int i = p.a; i < p.b; i++) id[i] = key[i].second;
            next[2 * k] = Part{p.a, mid, p.t0, h};
            next[2 * k + 1] = Part{mid, p.b, p.t0 + h, p.nt - h};
        });
        level.clear();
        for (const Part &p : next)
            if (p.nt > 0) level.push_back(p);
    }
}

// A partition, kept for a plan in the other arithmetic: finding it is two thirds
// of the work (128^3: 1.1 of 1.6 s on eight cores).
struct TilePartition {
    int tiles = 0;
    std::vector<int> tile_of;            // by position
};

// The plan for n rows given as 0-based CSR (row0, col0 ascending in a row,
// dia0), their DIC levels, an order that keeps mesh neighbours close (pos)
// and the internal row of every row.  tiles: how many; max_ratio: the most
// rows swept per row, beyond which there is no plan; ts: bytes of a value;
// optin: shared memory a block can have, ring_most: of it for the ring.
// kept: a partition of the same rows to use where it is into as many tiles, or
// to leave the new one in.  Throws std::bad_alloc where the host has no memory.
inline TilePlan tile_plan(int n, const std::vector<int> &row0, const std::vector<int> &col0,
                          const std::vector<int> &dia0, const std::vector<int32_t> &level,
                          const std::vector<int> &pos, const std::vector<int> &internal, int tiles,
                          double max_ratio, int ts, int optin, int ring_most, int threads,
                          TilePartition *kept = nullptr)
{
    TilePlan P;
    P.ts = ts;
    int n_levels = 0;
    for (int i = 0; i < n; i++) {
        n_levels = std::max(n_levels, level[i] + 1);
        if (dia0[i] - row0[i] > TILE_MAX_CNT || row0[i + 1] - dia0[i] - 1 > TILE_MAX_CNT ||
            (uint32_t)internal[i] >= TILE_NO_ROW)
            return P;
    }
    if (n < 1 || n_levels > TILE_MAX_LEVELS || tiles < 1) return P;
    tiles = std::min(tiles, n);
    // The closure of a ball of rows first: a structured numbering is told
    // from it before anything is partitioned.
    auto closure = [&](std::vector<int> &set, std::vector<int> &mark, int stamp, int dir, size_t most) {
        for (size_t h = 0; h < set.size() && set.size() <= most; h++) {
            const int i = set[h];
            const int a = dir == 0 ? row0[i] : dia0[i] + 1, b = dir == 0 ? dia0[i] : row0[i + 1];
            for (int j = a; j < b; j++)
                if (mark[col0[j]] != stamp) {
                    mark[col0[j]] = stamp;
                    set.push_back(col0[j]);
                }
        }
        return set.size() <= most;
    };
    std::vector<int> byp(n);
    for (int i = 0; i < n; i++) byp[pos[i]] = i;
    const size_t per = ((size_t)n + tiles - 1) / tiles;
    const size_t most = std::min<size_t>((size_t)((double)per * 2.0 * max_ratio) + 64, TILE_MAX_SLOTS);
    if (tiles > 1) {
        std::vector<int> mark(n, -1), ball;
        for (int dir = 0; dir < 2; dir++) {
            ball.assign(1, byp[n / 2]);
            mark[ball[0]] = dir;
            for (size_t h = 0; h < ball.size() && ball.size() < per; h++)
                for (int j = row0[ball[h]]; j < row0[ball[h] + 1] && ball.size() < per; j++)
                    if (mark[col0[j]] != dir) {
                        mark[col0[j]] = dir;
                        ball.push_back(col0[j]);
                    }
            if (!closure(ball, mark, dir, dir, most)) return P;
        }
    }
    TilePartition mine, &part = kept ? *kept : mine;
    std::vector<int> &tile_of = part.tile_of;
    if (part.tiles != tiles) {
        part.tiles = 0;
        std::vector<int> ptr(n + 1), adj(col0.size());
        ptr[0] = 0;
        for (int k = 0; k < n; k++) ptr[k + 1] = ptr[k] + (row0[byp[k] + 1] - row0[byp[k]]);
        const int blocks = std::min(64, n);
        tile_parallel(blocks, threads, [&](int b, int) {
            for (int k = (int)((int64_t)n * b / blocks); k < (int)((int64_t)n * (b + 1) / blocks); k++)
                for (int j = row0[byp[k]], q = ptr[k]; j < row0[byp[k] + 1]; j++, q++) adj[q] = pos[col0[j]];
        });
        tile_partition(n, ptr, adj, tiles, threads, tile_of);
        part.tiles = tiles;
    }
    std::vector<std::vector<int>> own(tiles);
    for (auto &o : own) o.reserve(per);
    for (int k = 0; k < n; k++) own[tile_of[k]].push_back(byp[k]);

    // Every tile and direction on its own, then joined.
    struct One {
        std::vector<TileRound> rounds;
        std::vector<uint32_t> rows;
        std::vector<int> vbeg;
        std::vector<uint8_t> packed, lists;
        std::vector<uint32_t> list_row;
        std::vector<uint16_t> list_slot;
        size_t swept = 0;
        int slots = 0;
    };
    std::vector<One> one(2 * (size_t)tiles);
    std::atomic<bool> fail{false};
    const int nt = std::max(1, std::min(threads, 2 * tiles));
    std::vector<std::vector<int>> marks(nt), locals(nt);
    tile_parallel(2 * tiles, nt, [&](int k, int t) {
        if (fail) return;
        const int tile = k >> 1, dir = k & 1;
        if (marks[t].empty()) {
            marks[t].assign(n, -1);
            locals[t].assign(n, 0);
        }
        std::vector<int> set = own[tile];
        for (int i : set) marks[t][i] = k;
        const size_t n_own = set.size();
        if (!closure(set, marks[t], k, dir, most)) {
            fail = true;
            return;
        }
        One &o = one[k];
        o.swept = set.size();
        // Level order (descending for the backward sweep); inside a level
        // by the number of entries, most first, so that slices carry little
        // padding, then by internal row.
        auto first = [&](int i) { return dir == 0 ? row0[i] : dia0[i] + 1; };
        auto count = [&](int i) { return dir == 0 ? dia0[i] - row0[i] : row0[i + 1] - dia0[i] - 1; };
        std::vector<std::pair<uint64_t, int>> key(set.size());
        for (size_t q = 0; q < set.size(); q++) {
            const int i = set[q];
            const uint64_t lv = dir == 0 ? level[i] : n_levels - 1 - level[i];
            key[q] = {lv << 40 | (uint64_t)(TILE_MAX_CNT - count(i)) << 32 | (uint64_t)(uint32_t)internal[i],
                      q < n_own ? i : -1 - i};
        }
        std::sort(key.begin(), key.end());
        std::vector<uint16_t> idx;
        std::vector<std::pair<uint32_t, uint16_t>> moved;
        int lv = 0;
        for (size_t a = 0; a < key.size(); lv++) {
            size_t b = a;
            while (b < key.size() && key[b].first >> 40 == key[a].first >> 40) b++;
            for (size_t r0 = a; r0 < b; r0 += TILE_ROWS) {
                const size_t r1 = std::min(b, r0 + TILE_ROWS), slot0 = (size_t)o.slots;
                const size_t slices = (r1 - r0 + 31) / 32, base = o.rows.size();
                uint32_t head[TILE_HEAD / 4] = {};
                uint8_t counts[TILE_ROWS] = {};
                o.rows.resize(base + TILE_ROWS, TILE_NO_ROW);
                o.vbeg.resize(base + TILE_ROWS, 0);
                idx.clear();
                for (size_t s = 0; s < slices; s++) {
                    const size_t q0 = r0 + 32 * s, q1 = std::min(r1, q0 + 32);
                    uint32_t width = 0;
                    for (size_t q = q0; q < q1; q++) {
                        const int i = key[q].second >= 0 ? key[q].second : -1 - key[q].second;
                        width = std::max(width, (uint32_t)count(i));
                        locals[t][i] = (int)(slot0 + (q - r0));
                        o.rows[base + (q - r0)] = (uint32_t)internal[i] | (uint32_t)count(i) << TILE_CNT_SHIFT |
                                                  (key[q].second >= 0 ? TILE_OWN : 0u);
                        o.vbeg[base + (q - r0)] = first(i);
                        counts[q - r0] = (uint8_t)count(i);
                    }
                    const size_t e0 = idx.size();
                    head[s] = (uint32_t)(e0 / 32) | width << 16;
                    idx.resize(e0 + 32 * (size_t)width, 0);
                    for (size_t q = q0; q < q1; q++) {
                        const int i = key[q].second >= 0 ? key[q].second : -1 - key[q].second;
                        for (int j = 0; j < count(i); j++)
                            idx[e0 + 32 * (size_t)j + (q - q0)] = (uint16_t)locals[t][col0[first(i) + j]];
                    }
                }
                const size_t values = 32 * slices * (size_t)tile_diags(dir, ts) + idx.size();
                const size_t at_idx = TILE_HEAD + 32 * slices + values * (size_t)ts;
                const size_t bytes = (at_idx + 2 * idx.size() + 15) & ~(size_t)15, at = o.packed.size();
                if (bytes / 16 > 0xffffu || at_idx / 16 > 0xffffu) {
                    fail = true;
                    return;
                }
                o.packed.resize(at + bytes, 0);
                std::memcpy(o.packed.data() + at, head, TILE_HEAD);
                std::memcpy(o.packed.data() + at + TILE_HEAD, counts, 32 * slices);
                if (!idx.empty()) std::memcpy(o.packed.data() + at + at_idx, idx.data(), 2 * idx.size());
                o.rounds.push_back(TileRound{(uint32_t)(at / 16), (uint32_t)(bytes / 16) | (r1 == b ? 1u << 24 : 0u),
                                             (uint32_t)slot0 | (uint32_t)slices << 16, (uint32_t)(at_idx / 16) << 16});
                o.slots += 32 * (int)slices;
                if (o.slots > TILE_MAX_SLOTS) {
                    fail = true;
                    return;
                }
            }
            moved.clear();
            for (size_t q = a; q < b; q++) {
                const int i = key[q].second >= 0 ? key[q].second : -1 - key[q].second;
                moved.push_back({(uint32_t)internal[i] << 1 | (key[q].second >= 0 ? 1u : 0u), (uint16_t)locals[t][i]});
            }
            std::sort(moved.begin(), moved.end());
            for (size_t q = 0; q < moved.size(); q += TILE_MOVERS) {
                const size_t base = o.list_row.size(), m = std::min<size_t>(TILE_MOVERS, moved.size() - q);
                o.lists.push_back((uint8_t)(lv | (q + TILE_MOVERS >= moved.size() ? 128 : 0)));
                o.list_row.resize(base + TILE_MOVERS, TILE_NO_ROW);
                o.list_slot.resize(base + TILE_MOVERS, 0);
                for (size_t e = 0; e < m; e++) {
                    o.list_row[base + e] = moved[q + e].first >> 1 | (moved[q + e].first & 1u ? TILE_OWN : 0u);
                    o.list_slot[base + e] = moved[q + e].second;
                }
            }
            a = b;
        }
        if (o.rounds.size() > (size_t)TILE_MAX_ROUNDS || o.lists.size() > (size_t)TILE_MAX_LISTS) fail = true;
    });
    if (fail) return P;
    int max_round = 0;
    for (int dir = 0; dir < 2; dir++) {
        size_t swept = 0;
        for (int t = 0; t < tiles; t++) {
            const One &o = one[2 * t + dir];
            swept += o.swept;
            P.max_slots = std::max(P.max_slots, o.slots);
            P.max_rounds = std::max(P.max_rounds, (int)o.rounds.size());
            P.max_lists = std::max(P.max_lists, (int)o.lists.size());
            for (const TileRound &r : o.rounds) max_round = std::max(max_round, (int)(r.y & 0xffffu) * 16);
        }
        P.redundancy = std::max(P.redundancy, (double)swept / n);
    }
    if (P.redundancy > max_ratio) return P;
    // The ring: what the rest leaves, at most ring_most, no more than all
    // rounds of a tile and at least 1.5 of the largest (most are half as
    // large).
    const int fixed = tile_fixed_bytes(P.max_slots, P.max_rounds, P.max_lists, ts);
    max_round = (max_round + 127) & ~127;
    P.ring_bytes = std::min(optin - fixed, std::max(ring_most, 2 * max_round)) & ~127;
    P.ring_bytes = (int)std::min<int64_t>(P.ring_bytes, (int64_t)max_round * std::max(2, P.max_rounds));
    if (2 * P.ring_bytes < 3 * max_round) return P;
    P.smem_bytes = fixed + P.ring_bytes;
    for (int dir = 0; dir < 2; dir++) {
        TileDir &D = P.dir[dir];
        D.tile_round.assign(1, 0);
        D.tile_list.assign(1, 0);
        std::vector<size_t> at(tiles + 1, 0);
        for (int t = 0; t < tiles; t++) {
            const One &o = one[2 * t + dir];
            at[t + 1] = at[t] + o.packed.size();
            D.tile_round.push_back(D.tile_round.back() + (int)o.rounds.size());
            D.tile_list.push_back(D.tile_list.back() + (int)o.lists.size());
        }
        D.lists.resize(D.tile_list.back());
        D.list_row.resize((size_t)D.tile_list.back() * TILE_MOVERS);
        D.list_slot.resize((size_t)D.tile_list.back() * TILE_MOVERS);
        if (at[tiles] / 16 > 0xffffffffull) return P;
        D.rows.resize((size_t)D.tile_round.back() * TILE_ROWS);
        D.vbeg.resize((size_t)D.tile_round.back() * TILE_ROWS);
        D.packed.resize(at[tiles]);
        D.rounds.resize(D.tile_round.back());
        tile_parallel(tiles, threads, [&](int t, int) {
            One &o = one[2 * t + dir];
            const size_t r0 = (size_t)D.tile_round[t];
            std::copy(o.rows.begin(), o.rows.end(), D.rows.begin() + (long)(r0 * TILE_ROWS));
            std::copy(o.vbeg.begin(), o.vbeg.end(), D.vbeg.begin() + (long)(r0 * TILE_ROWS));
            std::copy(o.packed.begin(), o.packed.end(), D.packed.begin() + (long)at[t]);
            const size_t l0 = (size_t)D.tile_list[t];
            std::copy(o.lists.begin(), o.lists.end(), D.lists.begin() + (long)l0);
            std::copy(o.list_row.begin(), o.list_row.end(), D.list_row.begin() + (long)(l0 * TILE_MOVERS));
            std::copy(o.list_slot.begin(), o.list_slot.end(), D.list_slot.begin() + (long)(l0 * TILE_MOVERS));
            tile_place(o.rounds.data(), (int)o.rounds.size(), P.ring_bytes);
            for (size_t c = 0; c < o.rounds.size(); c++) {
                D.rounds[r0 + c] = o.rounds[c];
                D.rounds[r0 + c].x += (uint32_t)(at[t] / 16);
            }
        });
    }
    P.tiles = tiles;
    return P;
}

// Tiles for n rows on `sms` multiprocessors: one tile per multiprocessor
// while a tile's rows (about 1.35 times its own) fit beside the ring in
// binary64, fewer where tiles would drop below about 1500 own rows (their
// closures would outweigh them).
inline int tile_count(int n, int sms)
{
    const int cap = 14400, least = 1536;
    if (n < 2 * least) return 1;
    if ((int64_t)n < (int64_t)least * sms) return n / least;
    return sms * (int)(((int64_t)n + (int64_t)sms * cap - 1) / ((int64_t)sms * cap));
}

}  // namespace tfs
