// Host check of a kept partition (tfs_dic_tiles_plan.h): a plan made with the
// partition of another arithmetic's, of another tile count's, or of a plan that
// did not come to be, is the plan made without one.  Prints "ok" when
// everything holds.
#include <cstdio>
#include <numeric>
#include <random>

#include "tfs_dic_tiles_plan.h"

using namespace tfs;

struct Mesh {   // k^3 cells numbered at random
    int n;
    std::vector<int> row, col, dia, level, pos, internal;
    explicit Mesh(int k) : n(k * k * k)
    {
        std::vector<int> num(n);
        std::iota(num.begin(), num.end(), 0);
        std::shuffle(num.begin(), num.end(), std::mt19937(11));
        std::vector<int> at(n);
        for (int c = 0; c < n; c++) at[num[c]] = c;
        row.assign(1, 0);
        level.assign(n, 0);
        const int step[3] = {1, k, k * k};
        for (int i = 0; i < n; i++) {
            std::vector<int> nb(1, i);
            const int c = at[i], x[3] = {c % k, c / k % k, c / (k * k)};
            for (int d = 0; d < 3; d++) {
                if (x[d] > 0) nb.push_back(num[c - step[d]]);
                if (x[d] + 1 < k) nb.push_back(num[c + step[d]]);
            }
            std::sort(nb.begin(), nb.end());
            for (int j : nb) {
                if (j == i) dia.push_back((int)col.size());
                if (j < i) level[i] = std::max(level[i], level[j] + 1);
                col.push_back(j);
            }
            row.push_back((int)col.size());
        }
        pos = at;
        internal.resize(n);
        std::iota(internal.begin(), internal.end(), 0);
    }
    TilePlan plan(int tiles, int ts, TilePartition *kept, double ratio = 3.0) const
    {
        return tile_plan(n, row, col, dia, level, pos, internal, tiles, ratio, ts, 227 << 10, 96 << 10, 4, kept);
    }
};

static bool same(const TilePlan &a, const TilePlan &b)
{
    bool ok = a.tiles == b.tiles && a.tiles > 0 && a.smem_bytes == b.smem_bytes && a.bytes() == b.bytes();
    for (int d = 0; d < 2 && ok; d++)
        ok = a.dir[d].rows == b.dir[d].rows && a.dir[d].packed == b.dir[d].packed && a.dir[d].vbeg == b.dir[d].vbeg &&
             a.dir[d].list_row == b.dir[d].list_row && a.dir[d].list_slot == b.dir[d].list_slot;
    return ok;
}

int main()
{
    int fails = 0;
    for (int k : {9, 16, 23}) {
        const Mesh m(k);
        const int tiles = std::max(1, m.n / 700);
        TilePartition kept;
        for (int t : {tiles, tiles + 3, tiles})
            for (int ts : {8, 4, 8})
                if (!same(m.plan(t, ts, &kept), m.plan(t, ts, nullptr)) || kept.tiles != t)
                    fails++, std::printf("%d^3, %d tiles of %d-byte values\n", k, t, ts);
        TilePartition refused;   // a ratio that no plan meets
        if (tiles > 1 && m.plan(tiles, 8, &refused, 1.0).tiles) fails++, std::printf("%d^3: a plan at ratio 1\n", k);
        if (!same(m.plan(tiles, 8, &refused), m.plan(tiles, 8, nullptr))) fails++, std::printf("%d^3 after a refusal\n", k);
    }
    if (!fails) std::printf("ok\n");
    return fails != 0;
}
