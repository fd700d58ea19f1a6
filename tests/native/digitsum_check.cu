// Host check of the conversions of digit sums to FP64 in hsr_digits.cuh
// (dg_value, one word and two), compiled for the host: sums next to powers of
// two, where the rounding carries through all bits, and seeded ones, against
// the same value in extended precision rounded to FP64 (ties away from zero).
// Prints "<sums> <wrong, one word> <wrong, two words>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../hsrq3in_gb300/csrc/hsr_digits.cuh"

using namespace hsr;

// |x| rounded to 53 bits, ties away from zero, from at most 128 bits.
static double rounded(unsigned __int128 a, bool negative, int e) {
    int drop = 0;
    while ((a >> drop) >> 53) ++drop;
    unsigned __int128 m = drop ? (a + ((unsigned __int128)1 << (drop - 1))) >> drop : a;
    const double v = std::ldexp((double)(unsigned long long)m, drop + e);
    return negative ? -v : v;
}

int main(int argc, char **argv) {
    const long long N = argc > 1 ? std::atoll(argv[1]) : 1000000LL;
    std::mt19937_64 rng(7);
    long long sums = 0, bad1 = 0, bad2 = 0;
    auto one = [&](long long T, int e) {
        const double want = rounded((unsigned __int128)(T < 0 ? -T : T), T < 0, e - 55), got = dg_value(T, e);
        if (got != want && bad1++ < 5) std::printf("one word %lld: got %a want %a\n", T, got, want);
    };
    auto two = [&](long long hi, long long lo, int e) {
        const __int128 t = (__int128)hi * ((__int128)1 << 36) + lo;
        unsigned __int128 a = (unsigned __int128)(t < 0 ? -t : t);
        // Bits below the leading 64 do not enter.
        for (int z = 0; (a >> 64) != 0 && z < 128; ++z)
            if ((a >> z) >> 64 == 0) {
                a = (a >> z) << z;
                break;
            }
        const double want = rounded(a, t < 0, e), got = dg_value(hi, lo, e);
        if (got != want && bad2++ < 5) std::printf("two words %lld %lld: got %a want %a\n", hi, lo, got, want);
    };
    for (int k = 0; k <= 62; ++k)
        for (long long d = -4; d <= 4; ++d) {
            const long long T = (1LL << k) + d;
            if (T < 0 || T > (1LL << 62)) continue;
            for (int e : {0, -900, 900}) {
                one(T, e);
                one(-T, e);
                two(T >> 10, T & 1023, e);
                two(-T, d, e);
                two(T, -d, e);
                two(0, T, e);
                two(0, -T, e);
            }
            sums += 42;
        }
    for (long long i = 0; i < N; ++i) {
        const long long T = (long long)(rng() >> 2) >> (rng() % 62), L = (long long)rng() >> (rng() % 40 + 8);
        one(rng() & 1 ? T : -T, (int)(rng() % 100) - 50);
        two(rng() & 1 ? T : -T, L, (int)(rng() % 100) - 50);
        sums += 2;
    }
    std::printf("%lld %lld %lld\n", sums, bad1, bad2);
    return bad1 != 0 || bad2 != 0;
}
