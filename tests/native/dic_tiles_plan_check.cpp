// Host check of the tiled DIC's plan (tfs_dic_tiles_plan.h): on random
// matrices -- symmetric and non-symmetric patterns, meshes and graphs, one
// tile and many -- every row is owned once, every chunk and slice is laid out
// as the kernel reads it, and sweeping the tiles one by one in plan order
// gives the sequential sweeps of Prec_Solve bit for bit.  A structured
// numbering, a row with too many entries and a deep schedule get no plan.
// Prints "ok" when everything holds.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <random>
#include <set>
#include <vector>

#include "tfs_dic_tiles_plan.h"

using namespace tfs;

static int fails = 0;
#define EXPECT(c)                                                        \
    do {                                                                 \
        if (!(c)) {                                                      \
            std::printf("line %d: %s\n", __LINE__, #c);                  \
            fails++;                                                     \
        }                                                                \
    } while (0)

struct Matrix {
    int n = 0;
    std::vector<int> row, col, dia, level, pos, internal;
    std::vector<double> val;
};

// Rows from neighbour sets; levels as the library computes them (a row waits
// for its lower entries and for the lower rows that hold it above their
// diagonal); the positions breadth first, the internal rows by level.
static Matrix make(const std::vector<std::set<int>> &nb, unsigned seed)
{
    std::mt19937 g(seed);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    Matrix m;
    m.n = (int)nb.size();
    m.row.assign(1, 0);
    for (int i = 0; i < m.n; i++) {
        std::set<int> s = nb[i];
        s.insert(i);
        for (int k : s) {
            if (k == i) m.dia.push_back((int)m.col.size());
            m.col.push_back(k);
            m.val.push_back(k == i ? 4.0 + u(g) : u(g));
        }
        m.row.push_back((int)m.col.size());
    }
    m.level.assign(m.n, 0);
    std::vector<std::vector<int>> dep(m.n);
    for (int i = 0; i < m.n; i++)
        for (int j = m.row[i]; j < m.row[i + 1]; j++)
            if (m.col[j] < i) dep[i].push_back(m.col[j]);
            else if (m.col[j] > i) dep[m.col[j]].push_back(i);
    for (int i = 0; i < m.n; i++)
        for (int k : dep[i]) m.level[i] = std::max(m.level[i], m.level[k] + 1);
    std::vector<int> order;
    m.pos.assign(m.n, -1);
    for (int s = 0; s < m.n; s++) {
        if (m.pos[s] >= 0) continue;
        size_t h = order.size();
        order.push_back(s);
        m.pos[s] = (int)h;
        for (; h < order.size(); h++)
            for (int j = m.row[order[h]]; j < m.row[order[h] + 1]; j++)
                if (m.pos[m.col[j]] < 0) {
                    m.pos[m.col[j]] = (int)order.size();
                    order.push_back(m.col[j]);
                }
    }
    std::vector<int> by(m.n);
    std::iota(by.begin(), by.end(), 0);
    std::sort(by.begin(), by.end(), [&](int a, int b) {
        return std::make_pair(m.level[a], m.pos[a]) < std::make_pair(m.level[b], m.pos[b]);
    });
    m.internal.assign(m.n, 0);
    for (int k = 0; k < m.n; k++) m.internal[by[k]] = 2 * k;   // gaps, as padding rows leave them
    return m;
}

static Matrix mesh(int a, int b, int c, bool permute, unsigned seed)
{
    const int n = a * b * c;
    std::mt19937 g(seed);
    std::vector<int> num(n);
    std::iota(num.begin(), num.end(), 0);
    if (permute) std::shuffle(num.begin(), num.end(), g);
    std::vector<std::set<int>> nb(n);
    auto at = [&](int i, int j, int k) { return num[i + a * (j + b * k)]; };
    auto join = [&](int p, int q) { nb[p].insert(q); nb[q].insert(p); };
    for (int k = 0; k < c; k++)
        for (int j = 0; j < b; j++)
            for (int i = 0; i < a; i++) {
                if (i + 1 < a) join(at(i, j, k), at(i + 1, j, k));
                if (j + 1 < b) join(at(i, j, k), at(i, j + 1, k));
                if (k + 1 < c) join(at(i, j, k), at(i, j, k + 1));
            }
    return make(nb, seed + 1);
}

static Matrix graph(int n, int degree, bool symmetric, unsigned seed)
{
    std::mt19937 g(seed);
    std::vector<std::set<int>> nb(n);
    for (int i = 0; i < n; i++)
        for (int d = 0; d < degree; d++) {
            // neighbours close by, so that closures stay local
            const int k = (i + 1 + (int)(g() % 40)) % n;
            if (k == i) continue;
            nb[i].insert(k);
            if (symmetric) nb[k].insert(i);
        }
    std::vector<int> num(n);
    std::iota(num.begin(), num.end(), 0);
    std::shuffle(num.begin(), num.end(), g);
    std::vector<std::set<int>> out(n);
    for (int i = 0; i < n; i++)
        for (int k : nb[i]) out[num[i]].insert(num[k]);
    return make(out, seed + 1);
}

static void check(const Matrix &m, int tiles, double ratio, bool want, int ts = 8, int optin = 232448)
{
    const TilePlan P = tile_plan(m.n, m.row, m.col, m.dia, m.level, m.pos, m.internal, tiles, ratio, ts, optin, 16384, 3);
    EXPECT((P.tiles > 0) == want);
    if (!P.tiles) return;
    EXPECT(P.max_slots <= TILE_MAX_SLOTS && P.max_rounds <= TILE_MAX_ROUNDS && P.redundancy <= ratio);
    EXPECT(P.smem_bytes == tile_fixed_bytes(P.max_slots, P.max_rounds, P.max_lists, ts) + P.ring_bytes && P.smem_bytes <= optin);
    EXPECT(P.ring_bytes % 128 == 0);
    std::mt19937 g(5);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    std::vector<double> d(m.n), b(m.n), y(m.n), z(m.n);
    for (int i = 0; i < m.n; i++) { d[i] = 0.2 + 0.1 * u(g); b[i] = u(g); }
    for (int i = 0; i < m.n; i++) {
        double s = b[i];
        for (int j = m.row[i]; j < m.dia[i]; j++) s = s - m.val[j] * y[m.col[j]];
        y[i] = s * d[i];
    }
    for (int i = m.n - 1; i >= 0; i--) {
        double s = y[i] / (d[i] + 1e-30);
        for (int j = m.dia[i] + 1; j < m.row[i + 1]; j++) s = s - m.val[j] * z[m.col[j]];
        z[i] = s * d[i];
    }
    const int n_int = 2 * m.n;
    std::vector<int> natural(n_int, -1);
    for (int i = 0; i < m.n; i++) natural[m.internal[i]] = i;
    std::vector<double> start(n_int, 0.0), out(n_int, 0.0);
    for (int dir = 0; dir < 2; dir++) {
        const TileDir &D = P.dir[dir];
        std::vector<int> owners(m.n, 0);
        EXPECT((int)D.tile_round.size() == P.tiles + 1 && D.tile_round.back() == (int)D.rounds.size());
        EXPECT(D.rows.size() == D.rounds.size() * TILE_ROWS && D.vbeg.size() == D.rows.size());
        uint32_t next_byte = 0;
        for (int t = 0; t < P.tiles; t++) {
            const int c0 = D.tile_round[t], nr = D.tile_round[t + 1] - c0;
            EXPECT(nr > 0 && nr <= P.max_rounds);
            std::vector<double> s(P.max_slots, 0.0);
            std::vector<char> done(P.max_slots, 0);
            std::vector<int> level_slots;
            std::vector<int> holder(P.ring_bytes / 128, -1);   // which round's bytes a part of the ring holds
            uint32_t local = 0;
            // the lists: every row of a level once, at its slot, own rows marked
            std::vector<std::vector<std::pair<uint32_t, int>>> listed(1);
            const int l0 = D.tile_list[t], nl = D.tile_list[t + 1] - l0;
            EXPECT(nl > 0 && nl <= P.max_lists);
            for (int q = 0; q < nl; q++) {
                EXPECT((D.lists[l0 + q] & 127) == (int)listed.size() - 1);
                for (int k = 0; k < TILE_MOVERS; k++) {
                    const size_t e = (size_t)(l0 + q) * TILE_MOVERS + k;
                    if ((D.list_row[e] & TILE_ROW_MASK) != TILE_NO_ROW)
                        listed.back().push_back({D.list_row[e], D.list_slot[e]});
                }
                if (D.lists[l0 + q] & 128) listed.emplace_back();
            }
            EXPECT(listed.back().empty());
            size_t tile_level = 0;
            std::vector<std::pair<uint32_t, int>> swept;
            for (int q = 0; q < nr; q++) {
                const TileRound c = D.rounds[c0 + q];
                const uint32_t bytes = (c.y & 0xffffu) * 16u, slices = c.z >> 16, values = slices * 32 * tile_diags(dir, ts);
                EXPECT(c.x * 16u == next_byte && (c.z & 0xffffu) == local && slices >= 1 && slices <= TILE_SLICES);
                next_byte += bytes;
                // its place in the ring: in bounds, and everything it
                // overwrites at least `back` rounds old
                const uint32_t at = (c.w & 0xffffu) * 128u, back = c.y >> 16 & 0xffu;
                EXPECT(at + bytes <= (uint32_t)P.ring_bytes && back <= TILE_BARS && (int)back <= q);
                EXPECT(q < TILE_BARS || back > 0);
                for (uint32_t k = at / 128; k < (at + bytes + 127) / 128; k++) {
                    EXPECT(holder[k] < 0 || (back > 0 && holder[k] <= q - (int)back));
                    holder[k] = q;
                }
                const uint8_t *pk = D.packed.data() + 16 * (size_t)c.x;
                const uint32_t *head = reinterpret_cast<const uint32_t *>(pk);
                const uint16_t *idx = reinterpret_cast<const uint16_t *>(pk + (c.w >> 16) * 16u);
                uint32_t off = 0;
                for (uint32_t w = 0; w < slices; w++) {
                    const int width = (int)(head[w] >> 16);
                    EXPECT((head[w] & 0xffffu) == off);
                    for (int lane = 0; lane < 32; lane++) {
                        const size_t slot = (size_t)(c0 + q) * TILE_ROWS + 32 * w + lane;
                        const uint32_t word = D.rows[slot], internal = word & TILE_ROW_MASK;
                        if (internal == TILE_NO_ROW) continue;
                        const int i = natural[internal];
                        EXPECT(i >= 0);
                        const int cnt = (int)((word >> TILE_CNT_SHIFT) & 15u);
                        EXPECT(cnt <= width && pk[TILE_HEAD + 32 * w + lane] == cnt);
                        EXPECT(cnt == (dir == 0 ? m.dia[i] - m.row[i] : m.row[i + 1] - m.dia[i] - 1));
                        double acc = dir == 0 ? b[i] : start[internal];
                        for (int j = 0; j < cnt; j++) {
                            const uint16_t k = idx[32 * (size_t)off + 32 * (size_t)j + lane];
                            EXPECT(done[k]);
                            acc = acc - m.val[D.vbeg[slot] + j] * s[k];
                        }
                        acc = acc * d[i];
                        const int me = (int)local + 32 * (int)w + lane;
                        s[me] = acc;
                        level_slots.push_back(me);
                        swept.push_back({word & (TILE_ROW_MASK | TILE_OWN), me});
                        if (word & TILE_OWN) {
                            owners[i]++;
                            out[internal] = dir == 0 ? acc / (d[i] + 1e-30) : acc;
                        }
                    }
                    for (int lane = 0; lane < 32 * width; lane++) EXPECT(idx[32 * (size_t)off + lane] < P.max_slots);
                    off += (uint32_t)width;
                }
                EXPECT((c.w >> 16) * 16u == TILE_HEAD + 32 * slices + (values + 32 * off) * (uint32_t)ts);
                EXPECT(bytes >= (c.w >> 16) * 16u + 64 * off);
                for (int k = 32 * (int)slices; k < TILE_ROWS; k++)
                    EXPECT((D.rows[(size_t)(c0 + q) * TILE_ROWS + k] & TILE_ROW_MASK) == TILE_NO_ROW);
                local += 32 * slices;
                EXPECT((int)local <= P.max_slots);
                if (c.y >> 24) {
                    for (int k : level_slots) done[k] = 1;   // visible after the level's barrier only
                    level_slots.clear();
                    EXPECT(tile_level < listed.size());
                    std::sort(swept.begin(), swept.end());
                    std::sort(listed[tile_level].begin(), listed[tile_level].end());
                    EXPECT(swept == listed[tile_level]);
                    tile_level++;
                    swept.clear();
                }
            }
            EXPECT(level_slots.empty() && tile_level + 1 == listed.size() && tile_level <= TILE_MAX_LEVELS);
        }
        EXPECT(next_byte == D.packed.size());
        for (int i = 0; i < m.n; i++) EXPECT(owners[i] == 1);
        if (dir == 0)
            for (int i = 0; i < m.n; i++) {
                EXPECT(out[m.internal[i]] == y[i] / (d[i] + 1e-30));
                start[m.internal[i]] = out[m.internal[i]];
            }
        else
            for (int i = 0; i < m.n; i++) EXPECT(out[m.internal[i]] == z[i]);
    }
}

int main()
{
    check(mesh(12, 11, 10, true, 1), 1, 2.2, true);
    check(mesh(12, 11, 10, true, 2), 3, 3.0, true);
    check(mesh(31, 17, 23, true, 3), 7, 2.2, true);
    check(mesh(40, 40, 40, true, 4), 41, 2.2, true);
    check(mesh(40, 40, 40, true, 4), 12, 2.2, true, 4);
    check(mesh(40, 40, 40, true, 4), 12, 2.2, false, 8, 64 << 10);   // the tiles' vector does not fit
    check(mesh(1, 1, 1, true, 5), 4, 2.2, true);
    check(mesh(300, 1, 1, true, 6), 5, 2.2, true);
    check(mesh(7, 1, 900, true, 7), 9, 2.2, true);
    check(graph(500, 3, true, 8), 1, 2.2, true);
    check(graph(4000, 2, true, 9), 6, 3.0, true);
    check(graph(4000, 2, false, 10), 6, 3.0, true);    // non-symmetric pattern
    check(graph(3000, 1, false, 11), 9, 3.0, true);    // rows without entries on a side, several components
    check(mesh(24, 24, 24, false, 12), 9, 2.2, false); // lexicographic: closures reach through the mesh
    check(mesh(20, 20, 20, false, 16), 5, 2.2, false); // the same with a schedule that is not too deep
    check(mesh(200, 2, 1, false, 13), 1, 2.2, false);  // a schedule deeper than TILE_MAX_LEVELS
    check(graph(400, 20, true, 14), 1, 2.2, false);    // rows of more than 15 entries on a side
    check(mesh(24, 24, 24, true, 15), 300, 1.5, false); // tiles too small for the ratio
    if (!fails) std::printf("ok\n");
    return fails ? 1 : 0;
}
