// Host-side check of int_math.cuh against the IEEE operations.
//   int_math_check N SEED -> "cases refused mismatches" for mulOnInts,
//   mulQuotOnInts and upwindSettled, one line each.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "int_math.cuh"

using namespace simplic;

static uint64_t gS;
static uint64_t rnd() {
    gS ^= gS << 13;
    gS ^= gS >> 7;
    gS ^= gS << 17;
    return gS;
}
static double dbl(uint64_t b) {
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}
static uint64_t bits(double x) {
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
}
// significands of several kinds: random, few bits, all ones, near powers of
// two; exponents around 1, over the whole range, at its ends
static uint64_t sample() {
    const uint64_t r = rnd();
    uint64_t f = rnd() & 0xfffffffffffffull;
    switch (r & 7) {
        case 0: f = 0; break;
        case 1: f = 0xfffffffffffffull; break;
        case 2: f = (rnd() & 0xff) << (rnd() % 45); break;
        case 3: f = 0xfffffffffffffull ^ ((rnd() & 0xff) << (rnd() % 45)); break;
        case 4: f &= ~((1ull << (rnd() % 52)) - 1); break;
        default: break;
    }
    uint64_t e;
    switch ((r >> 3) & 7) {
        case 0: e = rnd() & 0x7ff; break;
        case 1: e = rnd() % 70; break;
        case 2: e = 2047 - rnd() % 70; break;
        default: e = 1023 - 60 + rnd() % 120; break;
    }
    return ((r >> 63) << 63) | (e << 52) | (f & 0xfffffffffffffull);
}

int main(int argc, char** argv) {
    const long long n = argc > 1 ? std::atoll(argv[1]) : 1000000;
    gS = (argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1) * 0x9E3779B97F4A7C15ull + 1;
    long long refused[3] = {0, 0, 0}, bad[3] = {0, 0, 0};
    for (long long i = 0; i < n; ++i) {
        const uint64_t a = sample(), b = sample();
        uint64_t r, dv, q;
        if (!mulOnInts(a, b, r)) ++refused[0];
        else if (r != bits(dbl(a) * dbl(b))) ++bad[0];
        if (!mulQuotOnInts(a, b, dv, q)) {
            ++refused[1];
        } else {
            const volatile double p = dbl(a) * dbl(b);
            const volatile double w = p / dbl(b);
            if (dv != bits(p) || q != bits(w)) ++bad[1];
        }
        // upwind: also values close to each other and exact ties
        uint64_t c = b;
        if ((i & 3) == 1) c = (a & ~0xffffffffffffull) | (rnd() & 0xffffffffffffull);
        if ((i & 3) == 2) {  // lowest set bit of aN at the tie's place
            const int k = 1 + int(rnd() % 53);
            const int e = expFieldOf(a) - k;
            uint64_t f = k - 1 < 52 ? (rnd() & 0xfffffffffffffull & ~((1ull << (k - 1)) - 1)) | (1ull << (k - 1)) : 0;
            if (e > 0) c = (a & 0x8000000000000000ull) | (uint64_t(e) << 52) | f;
        }
        const int s = upwindSettled(a, c);
        const volatile double z = dbl(a) - dbl(c);
        const volatile double y = z + dbl(c);
        if (s == 0) ++refused[2];
        else if (bits(y) != (s > 0 ? a : 0ull)) ++bad[2];
    }
    for (int k = 0; k < 3; ++k) std::printf("%lld %lld %lld\n", n, refused[k], bad[k]);
    return 0;
}
