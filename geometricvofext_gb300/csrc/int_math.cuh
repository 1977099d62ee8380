// Double-precision products and quotients of the update on the integer pipe.
//
// An FP64 instruction takes an SM of this part 16 cycles per warp, a 32-bit
// integer one half a cycle or less, so a multiplication of two 53-bit
// significands as four 32-bit products with explicit round-to-nearest-even
// (about 35 integer instructions) costs less than the FP64 instruction it
// replaces, and runs beside the ones that are left.  Every function here
// returns the IEEE double of the operation it names, or false where an
// operand or the result is not a normal number; the caller then uses the
// operation itself.
#pragma once

#include <cstdint>

#include "simplic_device.cuh"

namespace simplic {

__host__ __device__ __forceinline__ int expFieldOf(uint64_t b) { return int((b >> 52) & 0x7ff); }

// The product of two 53-bit significands, left-aligned: its leading 64 bits in
// t (bit 63 set), whether anything is left below them, whether the product had
// 106 bits, and its low 53 bits.
struct SigProduct {
    uint64_t t;
    bool sticky, wide;
    uint64_t low53;
};
__host__ __device__ __forceinline__ SigProduct mulSignificands(uint64_t ma, uint64_t mb) {
    const uint32_t al = uint32_t(ma), ah = uint32_t(ma >> 32), bl = uint32_t(mb), bh = uint32_t(mb >> 32);
    const uint64_t p0 = uint64_t(al) * bl;
    const uint64_t p1 = uint64_t(ah) * bl + (p0 >> 32);
    const uint64_t p2 = uint64_t(al) * bh + uint32_t(p1);
    const uint64_t p3 = uint64_t(ah) * bh + (p1 >> 32) + (p2 >> 32);  // bits 64 .. 105
    const uint32_t w1 = uint32_t(p2), w0 = uint32_t(p0);              // bits 32 .. 63 and 0 .. 31
    SigProduct r;
    r.wide = (p3 >> 41) & 1u;
    const uint64_t t = (p3 << 22) | (w1 >> 10);  // bits 42 .. 105
    r.t = r.wide ? t : t << 1;                   // (the bit shifted in counts as sticky)
    r.sticky = ((w1 & 0x3ffu) | w0) != 0;
    r.low53 = (uint64_t(w1 & 0x1fffffu) << 32) | w0;
    return r;
}
// its leading 53 bits rounded to nearest even (2^53 when all are ones and it
// rounds up); up: away from zero
__host__ __device__ __forceinline__ uint64_t roundSignificand(const SigProduct& p, bool& up) {
    uint64_t m = p.t >> 11;
    const uint32_t rest = (uint32_t(p.t) & 0x7ffu) | (p.sticky ? 1u : 0u);
    const uint32_t inc = (rest + 0x3ffu + (uint32_t(m) & 1u)) >> 11;
    up = inc != 0;
    return m + inc;
}

// a b
__host__ __device__ __forceinline__ bool mulOnInts(uint64_t a, uint64_t b, uint64_t& r) {
    const int ea = expFieldOf(a), eb = expFieldOf(b);
    const uint64_t kFrac = 0xfffffffffffffull, kOne = 1ull << 52;
    const SigProduct p = mulSignificands((a & kFrac) | kOne, (b & kFrac) | kOne);
    bool up;
    const uint64_t m = roundSignificand(p, up);
    const int e = ea + eb - 1023 + (p.wide ? 1 : 0);
    r = ((uint64_t(uint32_t(e - 1)) << 52) + m) | ((a ^ b) & 0x8000000000000000ull);
    return ea > 0 && ea < 0x7ff && eb > 0 && eb < 0x7ff && e > 1 && e < 2045;
}

// dv = RN(x dt) and q = RN(dv / dt).  With x = mx 2^i, dt = mt 2^j and the
// product P = mx mt, dv = m 2^s (s = 52 or 53 places dropped) and dv / dt is
// x + (m 2^s - P) / mt units of x's last place, where |m 2^s - P| <= 2^(s-1):
//   s = 52: at most half a unit, and half only for mt = 2^52, where P is a
//     multiple of 2^52 and the remainder zero: q = x;
//   s = 53: q is x, or its neighbour on the side dv was rounded to when twice
//     the remainder exceeds mt (ties to even).  mx > 2^52 then (P >= 2^105 and
//     mt < 2^53), so both neighbours are one unit away.
__host__ __device__ __forceinline__ bool mulQuotOnInts(uint64_t x, uint64_t dt, uint64_t& dv, uint64_t& q) {
    const int ex = expFieldOf(x), et = expFieldOf(dt);
    const uint64_t kFrac = 0xfffffffffffffull, kOne = 1ull << 52;
    const uint64_t mt = (dt & kFrac) | kOne;
    const SigProduct p = mulSignificands((x & kFrac) | kOne, mt);
    bool up;
    const uint64_t m = roundSignificand(p, up);
    const int e = ex + et - 1023 + (p.wide ? 1 : 0);
    dv = ((uint64_t(uint32_t(e - 1)) << 52) + m) | ((x ^ dt) & 0x8000000000000000ull);
    const uint64_t rem2 = 2 * (up ? (1ull << 53) - p.low53 : p.low53);
    const bool off = p.wide && (rem2 > mt || (rem2 == mt && (x & 1u)));
    q = off ? (up ? x + 1 : x - 1) : x;
    return ex > 0 && ex < 0x7ff && et > 0 && et < 0x7ff && e > 1 && e < 2045;
}

// Whether RN(RN(aP - aN) + aN) is settled on the bits: +1 it is aP, -1 it is
// +0, 0 the operations decide.
//   * Of one sign with |aN| <= |aP|: the first result is aP - aN + d with |d| at
//     most half a unit of aP's last place, and the second rounds aP + d back to
//     aP unless d is exactly that half, which needs aP - aN midway between two
//     such units: with k = the difference of the exponents, aN's lowest set
//     bit at place k - 1.  (In aP's lower binade d is a quarter at most, a tie
//     that goes to the even aP at worst.)
//   * aN below a quarter unit of aP (55 binades): both results are aP; aP below
//     a quarter unit of aN: the first is -aN, the second +0.
// Both finite and normal, else 0.
__host__ __device__ __forceinline__ int upwindSettled(uint64_t bP, uint64_t bN) {
    const uint64_t kMag = 0x7fffffffffffffffull;
    const int eP = expFieldOf(bP), eN = expFieldOf(bN);
    if (eP == 0 || eN == 0 || eP == 0x7ff || eN == 0x7ff) return 0;
    const int k = eP - eN;
    if (k >= 55) return 1;
    if (k <= -55) return -1;
    if ((bP ^ bN) >> 63) return 0;
    if ((bN & kMag) > (bP & kMag)) return 0;
    const uint32_t lo = uint32_t(bN), hi = uint32_t(bN >> 32) | 0x100000u;  // with the implicit bit
#ifdef __CUDA_ARCH__
    const int low = lo ? __ffs(lo) - 1 : 31 + __ffs(hi);
#else
    const int low = lo ? __builtin_ctz(lo) : 32 + __builtin_ctz(hi);
#endif
    return low == k - 1 ? 0 : 1;
}

}  // namespace simplic
