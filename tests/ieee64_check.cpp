// Checks csrc/ieee64.h on the host against the IEEE `/` and sqrt: exit code 0
// when every quotient and root is equal.  The device's seeds are imitated by
// the exact value with a relative error up to 2^-19.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "ieee64.h"

static uint64_t s = 88172645463325252ull;
static uint64_t rnd() {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}
static double bits(uint64_t u) {
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}
static double unit() { return (double)(rnd() >> 11) * 0x1p-53; }
// significands that stress rounding: random, few bits set, near a power of two
static uint64_t significand() {
    switch (rnd() % 4) {
        case 0: return (1ull << (rnd() % 52)) - 1;
        case 1: return ((1ull << 52) - 1) & ~((rnd() % 64));
        case 2: return rnd() % 64;
        default: return rnd() >> 12;
    }
}
static double value(int emin, int emax) {
    const uint64_t e = 1023 + emin + (int64_t)(rnd() % (uint64_t)(emax - emin + 1));
    return bits((e << 52) | (significand() & ((1ull << 52) - 1)));
}
static double seed_error() { return 1.0 + (2.0 * unit() - 1.0) * 0x1p-19; }

static long bad = 0;
static void check(const char *what, double x, double d, double got, double want) {
    if (got == want) return;
    if (bad++ < 10) std::printf("%s(%a, %a): %a, want %a\n", what, x, d, got, want);
}
static void check_root(double x) {
    const double want = std::sqrt(x);
    check("sqrt", x, 0.0, tsu::sqrt_from(x, 1.0 / want * seed_error()), want);
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 2000000;
    for (long i = 0; i < n; i++) {
        const bool wide = i & 1;
        const double d = value(wide ? -799 : -30, wide ? 799 : 30);
        double a = value(wide ? -799 : -60, wide ? 799 : 60);
        const int q = std::ilogb(a) - std::ilogb(d);
        if (q < -1000 || q > 1000) a = std::ldexp(a, -q);  // a representable quotient
        if (rnd() & 1) a = -a;
        if (tsu::mid(d) && tsu::recip_ok(d) && tsu::mid_or_zero(a)) {
            const double y = tsu::recip_from(d, 1.0 / d * seed_error());
            check("rcp", 1.0, d, y, 1.0 / d);
            check("quot", a, d, tsu::quot(a, d, y), a / d);
            // a first quotient that is off by up to a few thousand ulp
            const double q0 = a / d * (1.0 + (2.0 * unit() - 1.0) * 0x1p-40);
            check("quot_from", a, d, tsu::quot_from(a, d, y, q0), a / d);
        }
        check_root(value(wide ? -799 : -60, wide ? 799 : 60));
    }
    // Roots closest to a rounding boundary: with the root scaled to [2^52,
    // 2^53) and k its integer part, x = k (k + 1) + j is a multiple of 2^52 or
    // 2^53 for small even j.  k (k + 1) + j = 0 (mod 2^m) is solved bit by bit.
    for (int m = 52; m <= 53; m++)
        for (int j = -64; j <= 64; j += 2) {
            std::vector<uint64_t> ks = {0, 1};
            for (int b = 1; b < m; b++) {  // solutions mod 2^b -> mod 2^(b+1)
                std::vector<uint64_t> next;
                const uint64_t mask = (b + 1 == 64) ? ~0ull : ((1ull << (b + 1)) - 1);
                for (uint64_t k : ks)
                    for (int t = 0; t < 2; t++) {
                        const uint64_t c = k + ((uint64_t)t << b);
                        if (((c * (c + 1) + (uint64_t)(int64_t)j) & mask) == 0) next.push_back(c);
                    }
                ks.swap(next);
            }
            for (uint64_t k0 : ks)
                for (uint64_t k = k0; k < (1ull << 53); k += (1ull << m)) {
                    if (k < (1ull << 52)) continue;
                    const unsigned __int128 x = (unsigned __int128)k * (k + 1) + (__int128)j;
                    const uint64_t top = (uint64_t)(x >> m);  // x is a multiple of 2^m
                    const double v = (double)top;
                    if ((uint64_t)v != top) continue;  // not a double
                    for (int rep = 0; rep < 200; rep++)
                        for (int e = -2; e <= 2; e++) check_root(std::ldexp(v, m + 2 * 40 * e));
                }
        }
    for (int e = -300; e <= 300; e++)  // next to powers of two and four
        for (long u = -8; u <= 8; u++)
            for (int rep = 0; rep < 20; rep++) {
                uint64_t b;
                const double p = std::ldexp(1.0, e);
                std::memcpy(&b, &p, 8);
                check_root(bits(b + u));
            }
    std::printf("%ld wrong\n", bad);
    return bad ? 1 : 0;
}
