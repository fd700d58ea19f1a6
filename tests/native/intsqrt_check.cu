// Host check of the integer-pipe square root in hsr_device.cuh: ip_sqrt,
// compiled for the host, against the host's IEEE square root on seeded
// operands (random significands, significands near 1, near 2 and next to
// those of exact squares, the whole normal exponent range), and the quotient
// ip_quot takes from the root's own reciprocal (ip_recip_root) against the
// host's IEEE division.  Prints "<roots> <wrong roots> <quotients> <wrong quotients>".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../../hsrq3in_gb300/csrc/hsr_device.cuh"

using namespace hsr;

static unsigned long long bits_of(double x) {
    unsigned long long u;
    std::memcpy(&u, &x, 8);
    return u;
}
static double double_of(unsigned long long u) {
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}

int main(int argc, char **argv) {
    const long long N = argc > 1 ? std::atoll(argv[1]) : 20000000LL;
    std::mt19937_64 rng(20261205ULL);
    long long roots = 0, bad = 0, quots = 0, badq = 0;
    for (long long i = 0; i < N; ++i) {
        const unsigned long long ra = rng(), rb = rng(), rc = rng();
        const int mode = (int)(i % 6);
        unsigned long long f = ra & kSigMask;
        if (mode == 1) f |= 0xffffffffff000ULL;
        if (mode == 2) f &= 0xffULL;
        const int ex = mode == 3 ? 1 + (int)(rc % 2046) : 1023 + (int)(rc % 200) - 100;
        double x = double_of(((unsigned long long)ex << 52) | f);
        if (mode == 4) {                                          // next to the square of a 27-bit number
            const double r = (double)((ra >> 37) | (1ULL << 26));
            x = double_of(bits_of(r * r) + (rc >> 20) % 5 - 2);
        }
        if (mode == 5) {                                          // next to the square of a 53-bit number
            const double r = double_of((1023ULL << 52) | (ra & kSigMask));
            x = double_of(bits_of(r * r) + (rc >> 20) % 5 - 2);
        }
        unsigned long long y;
        const unsigned long long d = ip_sqrt(bits_of(x), y);
        ++roots;
        if (d != bits_of(std::sqrt(x))) {
            if (bad < 5) std::printf("root of %a: got %a want %a\n", x, double_of(d), std::sqrt(x));
            ++bad;
            continue;
        }
        const int ed = (int)(d >> 52), ea = ed - (int)((rc >> 40) % 60);
        if (ea < 1 || !ip_div_ok(ea, ed, d & kSigMask)) continue;
        const unsigned long long fa = rb & kSigMask, md = (d & kSigMask) | kHidden;
        const double q = double_of(ip_quot(fa | kHidden, md, ip_recip_root(d, y), ea - ed + 1023, 0ULL));
        const double a = double_of(((unsigned long long)ea << 52) | fa);
        ++quots;
        if (bits_of(q) != bits_of(a / double_of(d))) {
            if (badq < 5) std::printf("quotient %a / %a: got %a\n", a, double_of(d), q);
            ++badq;
        }
    }
    std::printf("%lld %lld %lld %lld\n", roots, bad, quots, badq);
    return bad != 0 || badq != 0;
}
