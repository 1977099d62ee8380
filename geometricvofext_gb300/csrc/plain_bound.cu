// Conservative bounding of the plain FP64 form: advection::limitFlux and
// advection::boundFlux (src/SimPLIC/advection/advectionTemplates.C:118-349)
// with extendMarkedCells / netFlux / setDownwindFaces (advection.C:54-82,
// 224-288).  Built with -fmad=false.
//
// The reference walks the bounding set (mixed cells and their face
// neighbours) in ascending cell order, and a cell reads the flux corrections
// that earlier cells wrote during the same pass.  A cell only reads
// corrections on its own faces and only its face-adjacent cells write those,
// so the result is the same whenever every overshooting cell runs after its
// earlier face-adjacent overshooting neighbours and before its later ones.
// The kernel runs on every SM (cooperative launch, all blocks resident):
//   * candidates: the overshooting cells the update kernel listed, filtered to
//     the bounding set; their dependencies are found through per-cell stamps,
//     no sorting;
//   * dataflow: everything of a cell's loop that reads no correction is
//     computed for all overshooting cells at once; a cell then starts as soon
//     as the earlier neighbours it waits for have started -- the last of them
//     runs it next in the same warp (chains run through in one warp) and a
//     queue feeds the idle warps -- and polls for the corrections on the
//     faces it shares with them; the corrected-face lists are built
//     afterwards, off the dependency chains;
//   * corrections are applied per target cell in the reference's list order
//     (key = cell * 32 + position among the cell's first-iteration faces);
//   * the pass test max(alpha) - 1 > aTol || min(alpha) < -aTol is exactly
//     "some cell of the mesh overshoots": an exact counter of overshooting
//     cells replaces the global min / max.
// What bounds it is latency: dependent L2 accesses (0.4 us each), the FP64
// chain of a cell's loop (0.3 us) along chains of up to 70 cells a pass, and
// four barriers a pass (2-3 us each).  One GB300, kernel time before the
// records came ahead through shared memory, cells were handed over inside a
// block and the other phases took 8 lanes per cell -> after: 256^3 with 6,900
// overshooting cells in the first of three passes 0.81 -> 0.47 ms (dependency
// phases 0.64 -> 0.35), 128^3 (7,500) 0.32 -> 0.20 ms (0.14 -> 0.09), 96^3
// warped hexahedra (5,300) 0.71 -> 0.40 ms, 45^3 x 6 tetrahedra (3,400) 0.19
// -> 0.15 ms, 33^3 (31) 0.086 -> 0.078 ms.
// Blocks meet at a grid barrier whose wait is bounded (a timeout sets an
// error bit and ends the blocks that see it); every loop and every wait of
// the dependency phase is bounded too, and no block returns after the first
// barrier unless a bounded wait ran out, so all blocks take the same
// decisions from values that are final when read.
#include <cfloat>
#include <climits>

#include "plain_geom.cuh"
#include "simplic_kernels.h"

namespace simplic {

namespace {

constexpr double kATol = 100.0 * kSMALL;  // advectionTemplates.C:125,228

// a < -aTol || a > 1 + aTol on the bits (a NaN neither)
__device__ __forceinline__ bool overshoots(double a) {
    const long long b = bitsOf(a), mag = b & 0x7fffffffffffffffLL;
    return mag <= 0x7ff0000000000000LL && (b < 0 ? mag > bitsOf(kATol) : b > bitsOf(1.0 + kATol));
}
__device__ __forceinline__ unsigned long long globalNs() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// List append with one atomic per group of converged lanes: thousands of
// cells appending to one counter otherwise queue up on a single address.
__device__ __forceinline__ int aggAppend(int* ctr) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(ctr, __popc(m));
    base = __shfl_sync(m, base, leader);
    return base + __popc(m & ((1u << lane) - 1u));
}
__device__ __forceinline__ void aggAdd(int* ctr, int v) {
    const unsigned m = __activemask();
    const int total = __reduce_add_sync(m, v);
    if ((threadIdx.x & 31) == __ffs(m) - 1 && total) atomicAdd(ctr, total);
}

// A bounding list ran out of room: the error bit for the host, and which list
// in info[3] (the largest code seen).
// (code 2 is not produced: the dependency phase has no depth cap)
enum : int { kOvfOvershootList = 1, kOvfModList = 3, kOvfTouchedList = 4, kOvfCandidates = 5 };
__device__ __forceinline__ void boundOverflow(const StepArgs& a, const BoundBuffers& s, int code) {
    atomicOr(a.err, (uint32_t)kErrBoundOverflow);
    atomicMax(s.info + 3, code);
}

// A face whose correction a later cell of the pass waits for holds this
// NaN pattern (never produced by arithmetic here, which gives the canonical
// NaN) until the earlier cell stores the value.  The value is the flag: a
// 64-bit store is single-copy atomic, so no fence is needed on either side.
constexpr long long kCorrPending = (long long)0xfff4c0de0000f00dULL;
__device__ __forceinline__ long long ldRelaxed64(const double* p) {
    long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void stRelaxed64(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

__device__ __forceinline__ double curDVf(const DevMesh& m, int f, const double* phi, const double* aCur,
                                         const int8_t* status, const double* dvfI, const double* alphaB, double dt,
                                         const BoundBuffers& s, int stamp) {
    if (s.modStamp[f] == stamp) return s.dvfMod[f];
    return baseDVf(m, f, phi[f], aCur, status, dvfI, alphaB, dt);
}

// Grid-wide barrier for a cooperative launch.  Thread 0 of each block
// arrives on a counter that only grows (zeroed before every launch): the
// k-th barrier (k counted by every thread of the block, from 0) is complete
// when the counter reaches (k + 1) x blocks, and the block that brings it
// there advances the generation the others wait on.  The wait is bounded
// (s.spinLimit polls): a block that gives up sets the timeout bit and the
// barrier returns false to all its threads, and the kernel then ends that
// block at once -- nothing after a failed barrier may read what other blocks
// were to write before it.  The other blocks then give up at their next
// barrier, so the launch always ends.  s.barrierExtra (a test setting,
// normally 0) makes the barrier wait for arrivals that never come.
__device__ bool gridBarrier(const BoundBuffers& s, uint32_t* err, unsigned& k) {
    __shared__ int ok;
    __syncthreads();
    const unsigned target = (k + 1u) * (gridDim.x + unsigned(s.barrierExtra));
    ++k;
    if (threadIdx.x == 0) {
        ok = 1;
        volatile unsigned* gen = s.barGen;
        const unsigned g = *gen;
        __threadfence();
        const unsigned arrived = atomicAdd(s.barCount, 1u) + 1u;
        if (arrived == target) {
            atomicAdd((unsigned*)s.barGen, 1u);
        } else {
            long long spins = 0;
            while (*gen == g) {
                if (++spins > s.spinLimit) {
                    atomicOr(err, (uint32_t)kErrBarrierTimeout);
                    ok = 0;
                    break;
                }
                __nanosleep(32);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// Exact tests on IEEE bit patterns, on the integer pipe (a double compare
// costs as much as a double add on this part).  NaN is neither >= 0 nor < 0.
__device__ __forceinline__ bool geZero(double x) {  // x >= 0 (true for -0)
    const long long b = bitsOf(x);
    return b >= 0 ? b <= 0x7ff0000000000000LL : (b << 1) == 0;
}
__device__ __forceinline__ bool ltZero(double x) {  // x < 0
    const long long b = bitsOf(x);
    return b < 0 && (b << 1) != 0 && (b & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool isZero(double x) { return (bitsOf(x) << 1) == 0; }
__device__ __forceinline__ bool absLess(double x, double t) {  // |x| < t, t > 0 finite
    return (bitsOf(x) & 0x7fffffffffffffffLL) < bitsOf(t);
}
// fmin of two non-negative, non-NaN values
__device__ __forceinline__ double minNonNeg(double x, double y) { return bitsOf(x) <= bitsOf(y) ? x : y; }
__device__ __forceinline__ int expField(double x) { return int((bitsOf(x) >> 52) & 0x7ff); }

constexpr double kHalfATol = 0.5 * kATol;
constexpr double kUnitHi = 1.0 + kHalfATol;

// The body of the reference's cell loop (advectionTemplates.C:245-347) for
// one overshooting cell, run by a whole warp, lane k on the cell's k-th face
// (cells() order).  The corrections on this cell's faces are final (its
// earlier neighbours are done, its later ones have not started).  Every
// value is computed by the reference's operations in the reference's order,
// sums in face order through shuffles, so the corrections are bit for bit
// the serial loop's.  The latency of a dependency chain is the sum of its
// cells' loops, and a double operation takes tens of cycles here, so:
//   * everything that does not read a correction is computed for every
//     overshooting cell before the dependency phase (BoundLane /
//     BoundCellConst, kept per face slot and per cell), including the first
//     iteration's passing faces and flux shares as they are when no
//     correction has arrived -- reused when the corrections leave them
//     unchanged;
//   * the test "maxExtra / V > aTol" is decided on the bits of maxExtra
//     against aTol V (1 +- 2^-40), with the division only inside that band;
//   * the loop test on the next alpha1New is first decided on a product
//     estimate with a proved error bound (< 2^-46 + 2^-48 when it is
//     used), with the two divisions only when the estimate cannot decide;
//   * zero terms are left out of the face sums (a sum started at +0 never
//     becomes -0, so adding a zero never changes it).
struct BoundLane {
    int F;                   // face id
    bool on, own, down;      // a face of the cell; owner side; flux leaves the cell
    bool phPos;              // phi >= 0
    double dv, phdt, aPhdt;  // dVf at the start of the pass, phi dt, |phi dt|
    bool pass0;              // passing in the first iteration when no correction arrives
    double maxExtra0, through0;
};
struct alignas(16) BoundCellConst {
    double Vi, rVi;        // cell volume, 1 / V
    double ov0, fluid0;    // alphaOvershoot and fluid of the first iteration
    double num1;           // alpha.oldTime * rDeltaT (+ Su) - netFlux(dVf) / V * rDeltaT
    double den, rden;      // rDeltaT (- Sp), 1 / den
    double g;              // (1 / V) rDeltaT
    double tolLo, tolHi;   // aTol V (1 -+ 2^-40)
    int eNum1, eRden;      // exponent fields of num1, rden
    unsigned pm0, ownMask; // first-iteration passing faces without corrections; owner-side faces
    int nfc, pad;          // faces of the cell
    double pad2;           // to 16-byte multiples
};
static_assert(sizeof(BoundCellConst) == kBoundCellConstBytes, "per-candidate constant record size");
// A face of an overshooting candidate as the dependency phase reads it.
struct alignas(16) BoundSlot {
    double dv, phdt, max0, thr0;  // BoundLane's dv, phdt, maxExtra0, through0
    int F, succ;                  // face; later overshooting candidate across it when it is downwind, or -1
    int flags, pad;               // kSlot* bits
};
static_assert(sizeof(BoundSlot) == kBoundSlotBytes, "face slot size");
__device__ __forceinline__ uint8_t* recordOf(const BoundBuffers& s, int i) { return s.rec + size_t(i) * s.recBytes; }
__device__ __forceinline__ BoundSlot* slotsOf(const BoundBuffers& s, int i) {
    return reinterpret_cast<BoundSlot*>(recordOf(s, i) + kBoundCellConstBytes);
}
// Shared memory a warp has for records: four of a hexahedron, one of any cell.
constexpr int kWarpRecordBytes = 2048;
static_assert(boundRecordBytes(6) * 4 <= kWarpRecordBytes && boundRecordBytes(kMaxCellFaces) <= kWarpRecordBytes,
              "record buffers");
// A record into the warp's shared buffer, asynchronously; fetchWait makes it
// visible to the warp.
__device__ __forceinline__ void fetchRecord(uint8_t* buf, const BoundBuffers& s, int i, int lane) {
    const uint8_t* r = recordOf(s, i);
    for (int o = 16 * lane; o < s.recBytes; o += 512)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(buf + o))),
                     "l"(r + o)
                     : "memory");
}
__device__ __forceinline__ void fetchWait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// face-slot flags of an overshooting candidate
enum : uint8_t { kSlotOn = 1, kSlotOwn = 2, kSlotDown = 4, kSlotPhPos = 8, kSlotPass0 = 16, kSlotDep = 32 };

// maxExtra / V > aTol, maxExtra >= 0
__device__ __forceinline__ bool exceedsATol(double maxExtra, const BoundCellConst& kc) {
    const long long b = bitsOf(maxExtra);
    if (b > bitsOf(kc.tolHi) && b <= 0x7ff0000000000000LL) return true;
    if (b < bitsOf(kc.tolLo)) return false;
    return divByRecip(maxExtra, kc.Vi, kc.rVi) > kATol;
}

// The parts of the cell loop that read no correction, computed for every
// overshooting candidate before the dependency phase.  The cell's faces are
// on a group of lanes: lanes base .. base + 15 (two cells per warp) or the
// whole warp (base 0) when a cell of the mesh has more than 16 faces; gl is
// the lane's face, gbits the group's lane bits, nmax the most faces of a
// cell in the warp (every lane takes part in every shuffle).  The masks
// kept in kc are by face (bit k: face k).
__device__ __forceinline__ void boundCellPrep(int c, int nfc, int nmax, int base, unsigned gbits, int Fs, double ph,
                                              double dv, const DevMesh& m, const StepArgs& a, int gl, BoundLane& L,
                                              BoundCellConst& kc) {
    constexpr unsigned kAll = 0xffffffffu;
    L.on = gl < nfc;
    L.F = Fs & 0x7fffffff;
    L.own = L.on && Fs >= 0;
    L.phPos = geZero(ph);
    L.down = L.on && (L.own ? L.phPos : ltZero(ph));
    L.dv = dv;
    L.phdt = ph * a.dt;
    L.aPhdt = fabs(L.phdt);
    kc.ownMask = (__ballot_sync(kAll, L.own) >> base) & gbits;
    kc.nfc = nfc;
    kc.pad = 0;
    // netFlux(c, dVf) in face order: the same every iteration
    double nf1 = 0.0;
    for (int k = 0; k < nmax; ++k) {
        const double x = __shfl_sync(kAll, dv, base + k);
        if (k < nfc) {
            if ((kc.ownMask >> k) & 1u)
                nf1 += x;
            else
                nf1 -= x;
        }
    }
    const double al = a.aNew[c];  // updated only after the dependency phase
    kc.Vi = m.V[c];
    kc.rVi = m.rV[c];
    kc.ov0 = pos0(al - 1.0) * (al - 1.0) + neg0(al) * al;
    kc.fluid0 = kc.ov0 * kc.Vi;
    double num = a.aOld[c] * a.rDeltaT;
    if (a.Su) num = num + a.Su[c];
    kc.num1 = num - divByRecip(nf1, kc.Vi, kc.rVi) * a.rDeltaT;
    kc.den = a.Sp ? (a.rDeltaT - a.Sp[c]) : a.rDeltaT;
    kc.rden = 1.0 / kc.den;
    kc.g = kc.rVi * a.rDeltaT;  // (1 / V) rDeltaT
    // the band is relative: with a subnormal aTol V every test divides
    const double t = kATol * kc.Vi;
    const bool normal = expField(t) != 0;
    kc.tolLo = normal ? t * (1.0 - 0x1p-40) : 0.0;
    kc.tolHi = normal ? t * (1.0 + 0x1p-40) : __longlong_as_double(0x7ff0000000000000LL);
    kc.eNum1 = expField(kc.num1);
    kc.eRden = expField(kc.rden);
    // the first iteration with every correction zero
    L.pass0 = false;
    L.maxExtra0 = 0.0;
    if (L.down) {
        const double dVff = dv + 0.0;
        const double me = geZero(kc.fluid0) ? fabs(L.phdt - dVff) : fabs(dVff);
        if (exceedsATol(me, kc)) {
            L.pass0 = true;
            L.maxExtra0 = me;
        }
    }
    kc.pm0 = (__ballot_sync(kAll, L.pass0) >> base) & gbits;
    double dVftot = 0.0;
    for (int k = 0; k < nmax; ++k) {
        const double x = __shfl_sync(kAll, L.aPhdt, base + k);
        if ((kc.pm0 >> k) & 1u) dVftot += x;
    }
    L.through0 = L.pass0 ? fabs(kc.fluid0) * L.aPhdt / dVftot : 0.0;
}

// The loop itself, once the corrections it reads are final.  cr0 is the
// correction on this lane's face as the earlier overshooting cell across it
// left it -- read only when the face is downwind for that cell (hasDep),
// the only case in which it can write one; zero otherwise (a later
// neighbour writes only after this cell in the reference's order, an
// inactive one writes nothing).  Returns this lane's final correction;
// pmFirst gets the faces that pass in the first iteration; ahead() is called
// once, in the first iteration, for work that the loop's latency can hide.
template <class Ahead>
__device__ __forceinline__ double boundCellLoop(bool hasDep, double cr0, const BoundLane& L,
                                                const BoundCellConst& kc, const StepArgs& a, unsigned& pmFirst,
                                                Ahead&& ahead) {
    constexpr unsigned kAll = 0xffffffffu;
    double cr = cr0;
    double ov = kc.ov0, fluid = kc.fluid0;
    pmFirst = 0;
    unsigned sumOf = 0;            // the faces dVftot was last summed over
    double dVftot = 0.0, rTot = 0.0;
    // one iteration; false ends the loop
    const auto step = [&](bool first, bool last) -> bool {
        bool pass = false;
        double pmax = 0.0;
        if (first && !hasDep) {
            pass = L.pass0;
            pmax = L.maxExtra0;
        } else if (L.down) {
            const double dVff = L.dv + cr;
            // fabs(pos0(fluid) phi dt - dVff): pos0 is 1 or 0, and 0 phi dt - dVff
            // is -dVff up to the sign of a zero
            const double me = geZero(fluid) ? fabs(L.phdt - dVff) : fabs(dVff);
            if (exceedsATol(me, kc)) {
                pass = true;
                pmax = me;
            }
        }
        const unsigned pm = __ballot_sync(kAll, pass);
        double through = 0.0;
        if (first && pm == kc.pm0) {
            through = L.through0;  // the same faces, so the same dVftot
        } else {
            if (pm != sumOf) {
                dVftot = 0.0;
                for (unsigned mm = pm; mm; mm &= mm - 1u) dVftot += __shfl_sync(kAll, L.aPhdt, __ffs(mm) - 1);
                sumOf = pm;
                rTot = 1.0 / dVftot;
            }
            if (pass) through = divByRecip(fabs(fluid) * L.aPhdt, dVftot, rTot);
        }
        int passInc = 0;
        if (pass) {
            // pos0(maxExtra - through) of two values >= 0, on the bits (a NaN never)
            passInc = bitsOf(pmax) >= bitsOf(through) && bitsOf(pmax) <= 0x7ff0000000000000LL &&
                      (bitsOf(pmax) < 0x7ff0000000000000LL || bitsOf(through) < 0x7ff0000000000000LL);
            through = minNonNeg(through, pmax);
            // sign(phi) sign(fluid) through is +-through exactly
            cr = cr + ((L.phPos == geZero(fluid)) ? through : -through);
        }
        const int nPass = __popc(__ballot_sync(kAll, passInc));
        if (first) {
            pmFirst = pm;
            ahead();
        }
        // the next test ends the loop without reading alpha1New
        if (nPass == 0 || last) return false;
        double nf2 = 0.0;  // netFlux(c, dVfcorrectionValues), face order
        const unsigned nz = __ballot_sync(kAll, L.on && !isZero(cr));
        for (unsigned mm = nz; mm; mm &= mm - 1u) {
            const int k = __ffs(mm) - 1;
            const double x = __shfl_sync(kAll, cr, k);
            if ((kc.ownMask >> k) & 1u)
                nf2 += x;
            else
                nf2 -= x;
        }
        // estimate: |a1 - alpha1New| < 2^-48 (|num1| + |t2|) |rden| + 2^-50 (|a1| + 1),
        // and |a1| < 2 inside the window; with the exponent test that is
        // below 2^-46 + 2^-48, so |alphaOvershoot| < aTol / 2 + that < aTol
        const double t2 = nf2 * kc.g;
        const double a1 = (kc.num1 - t2) * kc.rden;
        const long long b1 = bitsOf(a1);
        const bool inWindow = b1 >= 0 ? b1 < bitsOf(kUnitHi) : (b1 & 0x7fffffffffffffffLL) < bitsOf(kHalfATol);
        if (inWindow && max(kc.eNum1, expField(t2)) + kc.eRden <= 2045) return false;
        double num = kc.num1;
        num = num - divByRecip(nf2, kc.Vi, kc.rVi) * a.rDeltaT;
        const double a1New = divByRecip(num, kc.den, kc.rden);
        // pos0(a1New - 1) (a1New - 1) + neg0(a1New) a1New up to the sign of a zero (NaN stays)
        const long long bn = bitsOf(a1New);
        if (bn >= bitsOf(1.0))
            ov = a1New - 1.0;
        else
            ov = ltZero(a1New) || (bn & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL ? a1New : 0.0;
        fluid = ov * kc.Vi;
        return !absLess(ov, kATol);
    };
    if (absLess(ov, kATol)) {
        ahead();
        return cr;
    }
    // (the first iteration apart: nine in ten cells have no other, and what
    // ahead() waits for is not waited for before it)
    if (step(true, false))
        for (int iter = 1; iter < 10 && step(false, iter == 9); ++iter) {
        }
    return cr;
}

// After the dependency phase, for the overshooting cells of a warp (a group
// of lanes each, lane gl on the cell's gl-th face; i < 0: no cell): the faces
// that passed in a cell's first iteration join the list of corrected faces
// (key cell * 32 + position, the reference's list order) with their new dVf,
// and the cells on both sides become targets of the pass.  No later cell
// changes the correction of such a face, as a face is downwind for one side
// only.
__device__ void boundCellLists(int i, int gl, const DevMesh& m, const StepArgs& a, const BoundBuffers& s, int lane,
                               int pass, int passStamp, int stamp) {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned below = (1u << lane) - 1u;
    const int c = i >= 0 ? s.cand[i] : 0;
    const unsigned pmFirst = i >= 0 ? s.candPm[i] : 0u;
    const bool first = (pmFirst >> gl) & 1u;
    int f = 0, t0 = -1, t1 = -1, c0 = passStamp, c1 = passStamp;
    bool fresh = false;
    if (first) {
        f = slotsOf(s, i)[gl].F;
        const double cr = s.corr[f];
        t0 = m.own[f];
        t1 = f < m.nfi ? m.nei[f] : -1;
        c0 = atomicExch(s.cellClaim + t0, passStamp);
        if (t1 >= 0) c1 = atomicExch(s.cellClaim + t1, passStamp);
        s.faceKey[f] = unsigned(c) * 32u + unsigned(__popc(pmFirst & ((1u << gl) - 1u)));
        s.faceStamp[f] = passStamp;
        const double nv = slotsOf(s, i)[gl].dv + cr;  // dv: the dVf the pass started from
        fresh = s.modStamp[f] != stamp;
        s.dvfMod[f] = nv;
        s.modStamp[f] = stamp;
    }
    const bool w0 = first && c0 != passStamp, w1 = first && c1 != passStamp;
    const unsigned bm = __ballot_sync(kAll, fresh), b0 = __ballot_sync(kAll, w0), b1 = __ballot_sync(kAll, w1);
    int mBase = 0, tBase = 0;
    if (lane == 0) {
        if (bm) mBase = atomicAdd(s.ctl + kCtlMod, __popc(bm));
        if (b0 | b1) tBase = atomicAdd(s.ctl + kCtlTouched0 + pass, __popc(b0) + __popc(b1));
    }
    mBase = __shfl_sync(kAll, mBase, 0);
    tBase = __shfl_sync(kAll, tBase, 0);
    if (fresh) {
        const int p = mBase + __popc(bm & below);
        if (p < s.modCap) s.modList[p] = f;
        else boundOverflow(a, s, kOvfModList);
    }
    const int p0 = tBase + __popc(b0 & below) + __popc(b1 & below);
    if (w0) {
        if (p0 < s.touchedCap) s.touched[p0] = t0;
        else boundOverflow(a, s, kOvfTouchedList);
    }
    if (w1) {
        const int p1 = p0 + (w0 ? 1 : 0);
        if (p1 < s.touchedCap) s.touched[p1] = t1;
        else boundOverflow(a, s, kOvfTouchedList);
    }
}

// queue entries carry the pass stamp, so stale ones never match
__device__ __forceinline__ void stQueue(unsigned long long* p, int passStamp, int i) {
    const unsigned long long v = (static_cast<unsigned long long>(unsigned(passStamp)) << 32) | unsigned(i);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ldQueue(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ldVol(const int* p) { return *(volatile const int*)p; }

__global__ void __launch_bounds__(256, 2) kBound(StepArgs a, BoundBuffers s) {
    constexpr unsigned kAll = 0xffffffffu;
    const DevMesh& m = a.m;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nth = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    const int gw = tid >> 5, nw = nth >> 5;
    const int stamp = s.stamp;  // step stamp
    unsigned barK = 0;          // grid barriers passed
    // Outside the dependency phase a cell takes a group of lanes, lane gl of it
    // on the cell's gl-th face: 8, 16 or 32 lanes as the mesh's cells have
    // faces.  These phases are latency and FP64 warp instructions, both per
    // warp, so more cells to a warp are as many times fewer of them.
    const int gsz = m.maxCellFaces <= 8 ? 8 : (m.maxCellFaces <= 16 ? 16 : 32);
    const int per = 32 / gsz, gl = lane & (gsz - 1), base = lane - gl;
    const unsigned gbits = gsz == 32 ? 0xffffffffu : (1u << gsz) - 1u;
    const bool clock0 = tid == 0;  // block 0 keeps the time profile
    __shared__ __align__(16) uint8_t recBuf[8][kWarpRecordBytes];  // per warp: records of the cells it may run next
    // a warp that waits for a cell from its own block: kMailIdle, or the cell
    // another warp gave it; kMailBusy otherwise
    __shared__ int mail[8];
    __shared__ int allRun;
    constexpr int kMailIdle = -1, kMailBusy = -2;
    const unsigned long long tStart = clock0 ? globalNs() : 0ull;
    unsigned long long tDep = 0ull;
    // Decisions before the first barrier read values no block modifies.
    const int ovCount = s.ovCount[0];  // overshooting cells of the whole mesh
    const int nList = s.ovCount[1];    // those of them in the bounding set
    // No overshooting cell, or none in the bounding set: no pass can change
    // anything (corrections only come from listed cells), so nothing to do.
    if (ovCount == 0 || nList == 0) return;
    if (nList > s.ovCap || 2 * nList > s.candCap) {
        if (tid == 0) boundOverflow(a, s, kOvfOvershootList);
        return;
    }
    // 1. candidates: the overshooting cells of the bounding set, as listed
    //    by the update
    for (int i = tid; i < nList; i += nth) {
        const int c = s.ovList[i];
        s.cand[i] = c;
        s.candIdx[c] = i;
        s.candMark[c] = stamp;
    }
    if (tid == 0) s.ctl[kCtlCand] = nList;
    if (!gridBarrier(s, a.err, barK)) return;

    int over = ovCount;  // overshooting cells in the whole mesh
    for (int pass = 0; pass < a.nAlphaBounds && pass < kMaxBoundPasses; ++pass) {
        if (over == 0) break;
        const int passStamp = stamp * kMaxBoundPasses + pass + 1;
        const int nCand = ldVol(s.ctl + kCtlCand);
        if (tid == 0) s.info[0] = pass + 1;
        // 2. the overshooting candidates (a group of lanes each, on the cell's
        //    faces in cells() order): per face the dVf the pass
        //    starts from (final here: earlier passes are complete), the
        //    earlier overshooting cell it waits for (when the face is
        //    downwind for that cell, the only case in which it writes a
        //    correction there) and the later one that waits for it; then the loop's
        //    parts that read no correction.  Cells that wait for nobody go to
        //    the front of the queue.
        {
            for (int r0 = gw * per; r0 < nCand; r0 += nw * per) {
                const int i = r0 + lane / gsz;
                const bool valid = i < nCand;
                const int c = s.cand[valid ? i : r0];
                const bool act = valid && overshoots(a.aNew[c]);
                if (!__any_sync(kAll, act)) continue;  // the same on every lane
                const int k0 = m.uniformFaces ? c * m.uniformFaces : m.cOff[c];
                const int nfc = !act ? 0 : (m.uniformFaces ? m.uniformFaces : m.cOff[c + 1] - k0);
                const int nmax = __reduce_max_sync(kAll, nfc);
                int Fs = 0, succ = -1;
                bool dep = false;
                double ph = 0.0, dv = 0.0;
                if (gl < nfc) {
                    const int f = m.cFaces[k0 + gl];
                    const int o = m.own[f];
                    const bool own = o == c;
                    const int nb = own ? (f < m.nfi ? m.nei[f] : -1) : o;
                    Fs = own ? f : int(unsigned(f) | 0x80000000u);
                    ph = a.phi[f];
                    dv = curDVf(m, f, a.phi, a.aCur, a.status, a.dvfI, a.alphaB, a.dt, s, stamp);
                    if (nb >= 0 && s.candMark[nb] == stamp && overshoots(a.aNew[nb])) {
                        if (nb < c && (own ? ltZero(ph) : geZero(ph))) {
                            dep = true;
                            s.corr[f] = __longlong_as_double(kCorrPending);  // until the earlier cell stores it
                        } else if (nb > c && (own ? geZero(ph) : ltZero(ph))) {
                            succ = s.candIdx[nb];
                        }
                    }
                }
                BoundLane L;
                BoundCellConst k;
                boundCellPrep(c, nfc, nmax, base, gbits, Fs, ph, dv, m, a, gl, L, k);
                const unsigned depMask = (__ballot_sync(kAll, dep) >> base) & gbits;
                if (L.on) {
                    BoundSlot v;
                    v.dv = L.dv;
                    v.phdt = L.phdt;
                    v.max0 = L.maxExtra0;
                    v.thr0 = L.through0;
                    v.F = L.F;
                    v.succ = succ;
                    v.flags = kSlotOn | (L.own ? kSlotOwn : 0) | (L.down ? kSlotDown : 0) |
                              (L.phPos ? kSlotPhPos : 0) | (L.pass0 ? kSlotPass0 : 0) | (dep ? kSlotDep : 0);
                    v.pad = 0;
                    slotsOf(s, i)[gl] = v;
                }
                if (gl == 0 && act) {
                    k.pad2 = 0.0;
                    *reinterpret_cast<BoundCellConst*>(recordOf(s, i)) = k;
                    s.candPending[i] = __popc(depMask);
                    s.actList[atomicAdd(s.ctl + kCtlActive0 + pass, 1)] = i;
                    if (depMask == 0) stQueue(s.readyQ + atomicAdd(s.ctl + kCtlFree0 + pass, 1), passStamp, i);
                }
            }
        }
        if (!gridBarrier(s, a.err, barK)) return;
        const int nAct = ldVol(s.ctl + kCtlActive0 + pass);
        // no listed cell overshoots: this and every later pass change nothing
        if (nAct == 0) break;
        // 3. dependencies as dataflow.  A cell may start once every earlier
        //    overshooting neighbour it waits for has started: the neighbour
        //    that starts last (by an atomic count) runs it next in the same
        //    warp, so a chain runs through in one warp; the others it releases
        //    go to the queue.  The correction values are their own flags (a
        //    face holds the pending NaN until the earlier cell stores it; a
        //    64-bit store is single-copy atomic), so a cell polls for what a
        //    neighbour in another warp is still computing -- that warp waits
        //    for nothing but cells that have started before it -- and takes
        //    the value of the cell its own warp has just run from registers.
        //    What a link of a chain costs is memory latency (about 0.4 us per
        //    dependent access; a cell's loop itself takes 0.3 us), so: the
        //    count goes ahead of the loop; the records of the cells that wait
        //    for this one come into shared memory meanwhile; and a released
        //    cell goes to a waiting warp of the same block through shared
        //    memory, to the queue (two atomics and two polls later in another
        //    block) only when there is none.
        //    Every wait is bounded: one that runs out sets the timeout bit and
        //    the warp stops; the others then stop at their own limits.
        const unsigned long long td0 = clock0 ? globalNs() : 0ull;
        {
            const int nFree = ldVol(s.ctl + kCtlFree0 + pass);
            const int wl = threadIdx.x >> 5;
            const bool taker = wl < 2;  // these two wait for the queue, the other six for cells of the block
            uint8_t* const bufs = recBuf[wl];
            const int nBuf = kWarpRecordBytes / s.recBytes;
            if (lane == 0) mail[wl] = kMailBusy;
            if (threadIdx.x == 0) allRun = 0;
            __syncthreads();
            volatile int* const vMail = mail;
            int longest = 0, starts = 0, h = gw;  // the first free cell without an atomic
            bool failed = false;
            for (;;) {
                int i = -1;
                if (h < nFree) {
                    i = int(unsigned(s.readyQ[h]));
                } else if (taker) {
                    if (lane == 0) {
                        const int e = atomicAdd(s.ctl + kCtlQHead0 + pass, 1);
                        for (long long spin = 0;; ++spin) {
                            const unsigned long long v = e < nAct ? ldQueue(s.readyQ + (s.candCap - 1 - e)) : 0ull;
                            if (unsigned(v >> 32) == unsigned(passStamp)) {
                                i = int(unsigned(v));
                                break;
                            }
                            if (ldVol(s.ctl + kCtlDone0 + pass) >= nAct) break;  // all done: entry e never comes
                            if (spin >= s.spinLimit) {
                                atomicOr(a.err, (uint32_t)kErrBarrierTimeout);
                                i = -3;
                                break;
                            }
                            __nanosleep(64);
                        }
                        if (i < 0) *(volatile int*)&allRun = 1;
                    }
                } else if (lane == 0) {
                    vMail[wl] = kMailIdle;
                    for (long long spin = 0;; ++spin) {
                        const int v = vMail[wl];
                        if (v >= 0) {
                            i = v;
                            break;
                        }
                        // (every cell has run, or a taker gave up: no mail comes any more)
                        if (*(volatile int*)&allRun) break;
                        if (spin >= 4 * s.spinLimit) {
                            atomicOr(a.err, (uint32_t)kErrBarrierTimeout);
                            break;
                        }
                        __nanosleep(32);
                    }
                    vMail[wl] = kMailBusy;
                }
                if (h >= nFree) i = __shfl_sync(kAll, i, 0);
                if (i < 0) break;
                ++starts;
                int gotF = -1;  // the face whose correction this warp has just formed, and that
                double gotCr = 0.0;
                int ran = 0, at = 0;  // cells run; the buffer with the cell's record
                fetchRecord(bufs, s, i, lane);
                while (i >= 0) {
                    fetchWait();
                    const uint8_t* const rec = bufs + at * s.recBytes;
                    const BoundCellConst k = *reinterpret_cast<const BoundCellConst*>(rec);
                    BoundSlot v;
                    v.flags = 0;
                    v.F = 0;
                    v.succ = -1;
                    v.dv = v.phdt = v.max0 = v.thr0 = 0.0;
                    if (lane < k.nfc) v = reinterpret_cast<const BoundSlot*>(rec + kBoundCellConstBytes)[lane];
                    const int succ = v.succ;
                    // count this cell as started for its successors, and fetch their records
                    // (under a predicate in one instruction: a select after the atomic
                    // would wait for it here)
                    int left = 0;
                    asm volatile(
                        "{\n .reg .pred p;\n setp.ge.s32 p, %2, 0;\n @p atom.relaxed.gpu.global.add.s32 %0, [%1], -1;\n}"
                        : "+r"(left)
                        : "l"(s.candPending + (succ >= 0 ? succ : 0)), "r"(succ)
                        : "memory");
                    const unsigned sm = __ballot_sync(kAll, succ >= 0);
                    __syncwarp();  // every lane has read the record: its buffer may be filled again
                    {
                        int b = 0;
                        for (unsigned mm = sm; mm && b < nBuf; mm &= mm - 1u, ++b)
                            fetchRecord(bufs + b * s.recBytes, s, __shfl_sync(kAll, succ, __ffs(mm) - 1), lane);
                    }
                    BoundLane L;
                    L.F = v.F;
                    L.dv = v.dv;
                    L.phdt = v.phdt;
                    L.maxExtra0 = v.max0;
                    L.through0 = v.thr0;
                    L.on = v.flags & kSlotOn;
                    L.own = v.flags & kSlotOwn;
                    L.down = v.flags & kSlotDown;
                    L.phPos = v.flags & kSlotPhPos;
                    L.pass0 = v.flags & kSlotPass0;
                    L.aPhdt = fabs(L.phdt);
                    const bool hasDep = v.flags & kSlotDep;
                    long long cv = 0;  // bits of +0
                    bool stuck = false;
                    if (hasDep) {
                        if (L.F == gotF) {
                            cv = bitsOf(gotCr);
                        } else {
                            for (long long spin = 0;; ++spin) {
                                cv = ldRelaxed64(s.corr + L.F);
                                if (cv != kCorrPending) break;
                                if (spin >= s.spinLimit) {
                                    atomicOr(a.err, (uint32_t)kErrBarrierTimeout);
                                    stuck = true;
                                    break;
                                }
                            }
                        }
                    }
                    if (__any_sync(kAll, stuck)) {
                        failed = true;
                        break;
                    }
                    unsigned pmFirst = 0, rm = 0;
                    double cr = boundCellLoop(hasDep, __longlong_as_double(cv), L, k, a, pmFirst, [&] {
                        // the cells this one was the last to wait for
                        rm = __ballot_sync(kAll, left == 1);
                        // one is this warp's next; the others go to waiting warps of the block or the queue
                        unsigned rest = rm & (rm - 1u);
                        while (rest) {
                            const int c = __shfl_sync(kAll, succ, __ffs(rest) - 1);
                            rest &= rest - 1u;
                            unsigned idle = __ballot_sync(kAll, lane < 8 && vMail[lane & 7] == kMailIdle);
                            bool given = false;
                            while (idle && !given) {
                                int old = 0;
                                if (lane == 0) old = atomicCAS(&mail[__ffs(idle) - 1], kMailIdle, c);
                                given = __shfl_sync(kAll, old, 0) == kMailIdle;
                                idle &= idle - 1u;
                            }
                            if (!given && lane == 0)
                                stQueue(s.readyQ + (s.candCap - 1 - atomicAdd(s.ctl + kCtlQTail0 + pass, 1)), passStamp,
                                        c);
                        }
                    });
                    if (bitsOf(cr) == kCorrPending) cr = __longlong_as_double(0x7fffffffffffffffLL);
                    // only downwind faces can carry this cell's corrections, and
                    // each face is downwind for one side only: the face's one writer
                    if (L.down) stRelaxed64(s.corr + L.F, cr);
                    if (lane == 0) s.candPm[i] = pmFirst;
                    ++ran;
                    i = -1;
                    if (rm) {
                        const int src = __ffs(rm) - 1;
                        i = __shfl_sync(kAll, succ, src);
                        gotF = __shfl_sync(kAll, L.F, src);
                        gotCr = __shfl_sync(kAll, cr, src);
                        at = __popc(sm & ((1u << src) - 1u));
                        if (at >= nBuf) {  // no buffer was left for it
                            fetchWait();
                            at = 0;
                            fetchRecord(bufs, s, i, lane);
                        }
                    }
                }
                fetchWait();  // nothing is in flight when the buffers are filled again
                longest = max(longest, ran);
                if (lane == 0) atomicAdd(s.ctl + kCtlDone0 + pass, ran);
                if (failed) break;
                if (h < nFree) {
                    if (lane == 0) h = nw + atomicAdd(s.ctl + kCtlFreeHead0 + pass, 1);
                    h = __shfl_sync(kAll, h, 0);
                }
            }
            if (lane == 0 && failed) *(volatile int*)&allRun = 1;
            if (lane == 0 && longest > 0) {
                atomicMax(s.info + 4, longest);
                atomicAdd(s.ctl + kCtlStarts0 + pass, starts);
            }
        }
        if (!gridBarrier(s, a.err, barK)) return;
        // a bounded wait ran out (the timeout bit was set before any block
        // reached this barrier, so every block leaves here)
        if (*(volatile uint32_t*)a.err & kErrBarrierTimeout) return;
        if (clock0) tDep += globalNs() - td0;
        // 3b. the corrected-face list and the targets of every overshooting cell
        for (int q0 = gw * per; q0 < nAct; q0 += nw * per) {
            const int q = q0 + lane / gsz;
            boundCellLists(q < nAct ? s.actList[q] : -1, gl, m, a, s, lane, pass, passStamp, stamp);
        }
        if (!gridBarrier(s, a.err, barK)) return;
        // 4. alpha of every target cell, its updates in list order
        //    (advectionTemplates.C:164-192: own -= corr/V, nei += corr/V).
        //    A group of lanes per target, lane gl on its gl-th face; a
        //    corrected face's rank is the number of corrected faces of the
        //    cell with a smaller key, and the group adds the terms up in
        //    rank order.  Targets of the bounding set join the candidates
        //    (extendMarkedCells).  Loops and shuffles run on the whole warp.
        const int nT = min(ldVol(s.ctl + kCtlTouched0 + pass), s.touchedCap);
        {
            const unsigned hmask = gbits << base;
            for (int r0 = gw * per; r0 < nT; r0 += nw * per) {
                const int r = r0 + lane / gsz;
                const bool valid = r < nT;
                const int t = valid ? s.touched[r] : 0;
                bool hit = false, ownSide = false, nbMixed = false;
                unsigned key = 0xffffffffu;
                double term = 0.0, at = 0.0;
                if (valid) {
                    const int k0 = m.uniformFaces ? t * m.uniformFaces : m.cOff[t];
                    const int nfc = m.uniformFaces ? m.uniformFaces : m.cOff[t + 1] - k0;
                    at = a.aNew[t];
                    const double Vt = m.V[t], rVt = m.rV[t];
                    if (gl < nfc) {
                        const int2 sl = m.cSlot[k0 + gl];
                        const int g = sl.y & 0x7fffffff;
                        nbMixed = sl.x >= 0 && a.status[sl.x] != kStNotMixed;
                        if (s.faceStamp[g] == passStamp) {
                            hit = true;
                            key = s.faceKey[g];
                            ownSide = sl.y >= 0;
                            term = divByRecip(s.corr[g], Vt, rVt);
                        }
                    }
                }
                const unsigned hits = __ballot_sync(0xffffffffu, hit) & hmask;
                const bool need = (__ballot_sync(0xffffffffu, nbMixed) & hmask) != 0;
                int rank = 0;
                for (int j = 0; j < gsz; ++j) {
                    const unsigned kj = __shfl_sync(0xffffffffu, key, base + j);
                    if (((hits >> (base + j)) & 1u) && kj < key) ++rank;
                }
                const bool before = overshoots(at);
                const int nHits = __reduce_max_sync(kAll, __popc(hits));
                for (int e = 0; e < nHits; ++e) {
                    const unsigned who = __ballot_sync(0xffffffffu, hit && rank == e) & hmask;
                    const int src = who ? __ffs(who) - 1 : lane;
                    const double x = __shfl_sync(0xffffffffu, term, src);
                    const bool o = __shfl_sync(0xffffffffu, ownSide, src);
                    if (who) {
                        if (o) at -= x;
                        else at += x;
                    }
                }
                if (valid && gl == 0) {
                    a.aNew[t] = at;
                    aggAdd(s.ctl + kCtlOverDelta0 + pass, int(overshoots(at)) - int(before));
                    const bool inSet = need || a.status[t] != kStNotMixed;
                    if (inSet && s.candMark[t] != stamp && atomicExch(s.candMark + t, stamp) != stamp) {
                        const int p = aggAppend(s.ctl + kCtlCand);
                        if (2 * (p + 1) <= s.candCap) {
                            s.cand[p] = t;
                            s.candIdx[t] = p;
                        } else {
                            boundOverflow(a, s, kOvfCandidates);
                        }
                    }
                }
            }
        }
        if (!gridBarrier(s, a.err, barK)) return;
        over += ldVol(s.ctl + kCtlOverDelta0 + pass);
        if (tid == 0) {
            if (nAct > s.info[1]) s.info[1] = nAct;
            const int starts = ldVol(s.ctl + kCtlStarts0 + pass);
            if (starts > s.info[2]) s.info[2] = starts;
            s.info[5] += nAct;
        }
    }
    // alphaPhi = dVf / dt of every face the bounding changed this step
    const int nMod = min(ldVol(s.ctl + kCtlMod), s.modCap);
    for (int i = tid; i < nMod; i += nth) {
        const int f = s.modList[i];
        a.alphaPhi[f] = s.dvfMod[f] / a.dt;
    }
    if (clock0) {
        s.info[6] = int(tDep / 1000ull);
        s.info[7] = int((globalNs() - tStart) / 1000ull);
    }
}

}  // namespace

cudaError_t launchBound(const StepArgs& a, const BoundBuffers& b, cudaStream_t st) {
    // all blocks must be resident at once for the grid barrier: one or two
    // blocks per SM, as the occupancy calculator allows
    int dev = 0, sms = 0, perSm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kBound, 256, 0);
    if (e != cudaSuccess) return e;
    if (perSm < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int grid = sms * (perSm >= 2 ? 2 : 1);
    StepArgs aa = a;
    BoundBuffers bb = b;
    void* args[] = {&aa, &bb};
    return cudaLaunchCooperativeKernel((const void*)kBound, dim3(grid), dim3(256), args, 0, st);
}

}  // namespace simplic
