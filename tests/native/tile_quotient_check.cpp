// Host check of tile_quotient (tfs_dic_tiles.cuh): for y = s d rounded and
// rc = 1 / d rounded, fma(fma(-d, s, y), rc, s) is y / d as the division
// rounds it, on random operands and on significands at the ends of their
// range, in binary32 and binary64.  Prints "ok" when every quotient agrees.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

template <class T>
static long differing(long n, int bits, unsigned seed)
{
    std::mt19937_64 g(seed);
    auto operand = [&]() {
        const uint64_t r = g();
        uint64_t m = r & ((1ull << bits) - 1);
        switch (r >> 58 & 7) {
        case 0: m = (1ull << bits) - 1 - (m & 15); break;   // significand near 2
        case 1: m = m & 15; break;                          // near 1
        case 2: m = 1ull << (m % (uint64_t)bits); break;    // one bit
        default: break;
        }
        const T v = std::ldexp((T)1 + (T)m * std::ldexp((T)1, -bits), (int)(r >> 54 & 15) - 8);
        return r >> 63 ? -v : v;
    };
    long bad = 0;
    for (long k = 0; k < n; k++) {
        const T s = operand(), d = operand();
        const volatile T y = s * d, rc = (T)1 / d, want = y / d;
        const T got = std::fma(std::fma(-d, s, (T)y), (T)rc, s);
        bad += got != want;
    }
    return bad;
}

int main()
{
    const long a = differing<float>(4000000, 23, 1), b = differing<double>(4000000, 52, 2);
    if (!a && !b) std::printf("ok\n");
    else std::printf("%ld %ld\n", a, b);
    return a || b;
}
