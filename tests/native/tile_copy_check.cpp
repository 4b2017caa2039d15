// Host check of the copy lane's walk (tile_copy_walk of
// tfs_dic_tiles_plan.h) against a model of the block around it: rounds placed
// by tile_place in rings that hold all of a tile's rounds or few, copies that
// land at any time, row warps that release a round at any time after it has
// landed -- or, once the sweep is called off, before --, and a call-off at
// any time, also after the lane has issued its last round.  No round may be
// issued into bytes or onto a barrier still in use, none after the call-off
// was seen, and nothing may be in flight when the walk returns.  Prints "ok"
// when everything holds.
#include <cstdio>
#include <random>
#include <set>
#include <vector>

#include "tfs_dic_tiles_plan.h"

using namespace tfs;

static int fails = 0;
#define EXPECT(c)                                                        \
    do {                                                                 \
        if (!(c) && fails++ < 20) std::printf("line %d: %s\n", __LINE__, #c); \
    } while (0)

struct Block {
    const std::vector<TileRound> &r;
    std::mt19937 &g;
    int steps_to_off;                    // the call-off comes after so many looks (negative: never)
    int issued = 0, landed_to = 0, released_to = 0;   // landed_to: every round before it has landed
    bool is_off = false;
    std::set<int> flying;

    bool chance(int of) { return g() % of == 0; }
    void elapse()
    {
        if (steps_to_off >= 0 && steps_to_off-- == 0) is_off = true;
        for (auto it = flying.begin(); it != flying.end();) it = chance(3) ? flying.erase(it) : std::next(it);
        while (landed_to < issued && !flying.count(landed_to)) landed_to++;
        if (!is_off && released_to < landed_to && chance(2)) released_to++;
    }
    int back(int k) { return (int)(r[k].y >> 16 & 0xffu); }
    bool released(int k)
    {
        for (int t = 0; t < 100000; t++) {
            elapse();
            if (is_off && chance(2)) released_to = issued;   // the row warps' last arrivals
            if (released_to > k) return true;
            if (is_off) return false;
        }
        EXPECT(!"a release that never comes");
        return false;
    }
    bool off()
    {
        elapse();
        return is_off;
    }
    void issue(int k)
    {
        EXPECT(!is_off && k == issued);
        const int a = (int)(r[k].w & 0xffffu) * 128, b = a + (int)(r[k].y & 0xffffu) * 16;
        for (int q = 0; q < k; q++) {
            const int c = (int)(r[q].w & 0xffffu) * 128, d = c + (int)(r[q].y & 0xffffu) * 16;
            if ((a < d && c < b) || q % TILE_BARS == k % TILE_BARS) EXPECT(q < released_to && !flying.count(q));
        }
        flying.insert(k);
        issued++;
    }
    void landed(int k)
    {
        EXPECT(k < issued);
        flying.erase(k);
        elapse();
    }
};

int main()
{
    std::mt19937 g(20260701u);
    for (int trial = 0; trial < 4000; trial++) {
        const int n = 1 + (int)(g() % 70), most = 1 + (int)(g() % 900);
        std::vector<TileRound> r(n, TileRound{0, 0, 0, 0});
        int total = 0;
        for (TileRound &x : r) {
            x.y = 1 + g() % most;
            total += ((int)x.y * 16 + 127) & ~127;
        }
        const int whole = std::min(total, 65535 * 128), half = ((most * 16 + 127) & ~127) * 2;
        EXPECT(tile_place(r.data(), n, g() % 2 ? whole : std::min(whole, half + 128 * (int)(g() % 200))) || total < half);
        // called off at some look, at once after the last issue, or never
        for (int when : {-1, 0, 1, (int)(g() % (2u * n)), (int)(g() % (8u * n)), n - 1, n, n + 1}) {
            Block b{r, g, when};
            tile_copy_walk(n, b);
            EXPECT(b.flying.empty());
            EXPECT(when >= 0 || b.issued == n);
        }
    }
    if (!fails) std::printf("ok\n");
    return fails != 0;
}
