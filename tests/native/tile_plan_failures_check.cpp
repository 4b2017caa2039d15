// Host check of the tiled DIC's plan (tfs_dic_tiles_plan.h) where the host
// runs short: with every start of a thread refused, or some, the plan is the
// one that one thread makes; with every allocation from some point on refused,
// whichever thread makes it, tile_plan throws std::bad_alloc in the calling
// thread and ends no process.  (pthread_create and operator new of this
// program.)  Prints "ok" when everything holds.
#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <numeric>
#include <random>

#include "tfs_dic_tiles_plan.h"

static std::atomic<int> threads_left{1 << 30}, news_left{1 << 30};

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg)
{
    using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    return threads_left-- > 0 ? real(t, a, f, arg) : EAGAIN;
}
void *operator new(size_t n)
{
    void *p = news_left-- > 0 ? std::malloc(n ? n : 1) : nullptr;
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

using namespace tfs;

// A k^3 mesh numbered at random.
struct Mesh {
    int n;
    std::vector<int> row, col, dia, level, pos, internal;
    explicit Mesh(int k) : n(k * k * k)
    {
        std::vector<int> num(n), at(n);
        std::iota(num.begin(), num.end(), 0);
        std::shuffle(num.begin(), num.end(), std::mt19937(7));
        for (int c = 0; c < n; c++) at[num[c]] = c;
        row.assign(1, 0);
        level.assign(n, 0);
        for (int i = 0; i < n; i++) {
            const int c = at[i], x = c % k, y = c / k % k, z = c / (k * k);
            std::vector<int> nb(1, i);
            if (x) nb.push_back(num[c - 1]);
            if (x + 1 < k) nb.push_back(num[c + 1]);
            if (y) nb.push_back(num[c - k]);
            if (y + 1 < k) nb.push_back(num[c + k]);
            if (z) nb.push_back(num[c - k * k]);
            if (z + 1 < k) nb.push_back(num[c + k * k]);
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
    TilePlan plan(int threads) const
    {
        return tile_plan(n, row, col, dia, level, pos, internal, 12, 3.0, 4, 227 << 10, 96 << 10, threads);
    }
};

static bool same(const TilePlan &a, const TilePlan &b)
{
    if (a.tiles != b.tiles || a.bytes() != b.bytes()) return false;
    for (int d = 0; d < 2; d++)
        if (a.dir[d].rows != b.dir[d].rows || a.dir[d].packed != b.dir[d].packed ||
            a.dir[d].list_slot != b.dir[d].list_slot || a.dir[d].tile_round != b.dir[d].tile_round)
            return false;
    return true;
}

int main()
{
    const Mesh m(22);
    const TilePlan one = m.plan(1);
    int fails = one.tiles != 12;
    for (int t : {0, 1, 5, 1 << 30}) {
        threads_left = t;
        if (!same(m.plan(8), one)) fails++, std::printf("%d threads: another plan\n", t);
    }
    int thrown = 0, through = 0;
    for (int k = 0; k < 6000; k = k < 40 ? k + 1 : k + k / 5) {
        news_left = k;
        try {
            const TilePlan p = m.plan(8);
            news_left = 1 << 30;
            through++;
            if (!same(p, one)) fails++, std::printf("%d allocations: another plan\n", k);
        } catch (const std::bad_alloc &) {
            news_left = 1 << 30;
            thrown++;
        }
    }
    if (thrown < 10) fails++, std::printf("%d of %d plans without memory\n", thrown, thrown + through);
    if (!fails) std::printf("ok\n");
    return fails != 0;
}
