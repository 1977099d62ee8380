// Host-side check of divByRecip's integer quotient against the division.
//   int_div_check N SEED -> mismatches over N random pairs (significands of
//   several kinds, exponents to the ends of the range) and over all pairs of
//   the largest and smallest significands, where the estimate is furthest off.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "simplic_device.cuh"

using namespace simplic;

static uint64_t gS;
static uint64_t rnd() {
    gS ^= gS << 13;
    gS ^= gS >> 7;
    gS ^= gS << 17;
    return gS;
}
static double make(uint64_t f, int e, uint64_t s) {
    const uint64_t b = (s << 63) | (uint64_t(e) << 52) | (f & 0xfffffffffffffull);
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}
static uint64_t significand() {
    const uint64_t f = rnd() & 0xfffffffffffffull;
    switch (rnd() & 7) {
        case 0: return rnd() % 8;
        case 1: return 0xfffffffffffffull - rnd() % 8;
        case 2: return (rnd() & 0xff) << (rnd() % 45);
        case 3: return 0xfffffffffffffull ^ ((rnd() & 0xff) << (rnd() % 45));
        default: return f;
    }
}
static bool differs(double a, double b) {
    const double q = divByRecip(a, b, 1.0 / b), r = a / b;
    return std::memcmp(&q, &r, 8) != 0;
}

int main(int argc, char** argv) {
    const long long n = argc > 1 ? std::atoll(argv[1]) : 1000000;
    gS = (argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1) * 0x9E3779B97F4A7C15ull + 1;
    long long bad = 0;
    for (long long i = 0; i < n; ++i) {
        const int ea = (rnd() & 1) ? 1023 - 30 + int(rnd() % 60) : 1 + int(rnd() % 2046);
        const int eb = (rnd() & 1) ? 1023 - 30 + int(rnd() % 60) : 1 + int(rnd() % 2046);
        bad += differs(make(significand(), ea, rnd() & 1), make(significand(), eb, rnd() & 1));
    }
    for (uint64_t j = 0; j < 1500; ++j)
        for (uint64_t k = 0; k < 1500; ++k) {
            bad += differs(make(0xfffffffffffffull - j, 1023, 0), make(0xfffffffffffffull - k, 1023, 0));
            bad += differs(make(0xfffffffffffffull - j, 1023, 0), make(k, 1023, 0));
            bad += differs(make(j, 1023, 0), make(k, 1023, 1));
        }
    std::printf("%lld\n", bad);
}
