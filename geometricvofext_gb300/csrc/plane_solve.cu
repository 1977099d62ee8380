// Plane constant of every mixed cell (cutCell::findSignedDistance,
// cutCell.C:611-799), a group of lanes per cell (plane_group.cuh).  Built
// with -fmad=false.
//
// One GB300, kernel time with one thread per cell -> a group per cell -> with
// the work left out that plane_group.cuh lists (deformation field; interface
// cells in brackets) -> a warp per cell on short lists:
//   24^3 hex (331) 0.861 -> 0.167 -> 0.101 -> 0.049 ms
//   33^3 hex (617) 0.880 -> 0.224 -> 0.138 -> 0.066 ms
//   128^3 hex (30,189) 1.451 -> 1.345 -> 0.660 ms
//   256^3 hex (35,452) 1.636 -> 1.628 -> 0.764 ms
//   96^3 warped hex (7,146) 0.985 -> 0.406 -> 0.348 ms
//   24^3 with 2:1 refinement (755), three solves: 20.8 -> 2.16 -> 1.56 -> 1.24 ms
// At the large sizes the FP64 pipe is about 80% busy.
#include "plane_group.cuh"
#include "simplic_kernels.h"

#include <mutex>

namespace simplic {

namespace {

// Warps are independent, so a block is only the unit shared memory is handed
// out in: two warps keep the largest workspace within the static limit.
constexpr int kPlaneThreads = 64;

// Lists of up to this many cells per SM leave FP64 pipes idle when the warps
// are filled (four pipes an SM, busy half the time with one warp each): there a
// warp takes one cell, a group a cut (teamSignedDistance).  Filled warps
// against one cell each, ms: hexahedra 365 cells 0.105 / 0.055, 936 0.140 /
// 0.069, 1,778 0.140 / 0.097, 2,296 0.113 / 0.131; warped hexahedra 387 0.158 /
// 0.099, 1,054 0.215 / 0.181, 1,578 0.192 / 0.200; tetrahedra 560 0.120 /
// 0.083, 1,131 0.122 / 0.123, 2,016 0.123 / 0.236.  152 SMs: the line is 1,216.
constexpr int kTeamPerSm = 8;

// One instantiation per cell class (workspace caps K, G lanes per cell); a
// launch handles the mixed cells of its class.  With SPLIT the workspace is
// the splitWarpedFace one.
// Six blocks per SM (168 registers, a few spilled) against four (200
// registers): 0.80 against 0.82 ms at 128^3, 0.35 against 0.44 on the warped
// 96^3 mesh; eight blocks spill more and gain nothing.
template <class K, int G, bool SPLIT>
__global__ void __launch_bounds__(kPlaneThreads, 6) kPlaneSolve(DevMesh m, PlaneArgs p, int cls) {
    __shared__ GroupShared<K, G> shared[kPlaneThreads / 32];
    constexpr int kCells = 32 / G;
    const int nm = *p.nMixed;
    const int mask = SPLIT ? m.splitClassMask : m.classMask;
    const uint8_t* cellCls = SPLIT ? m.splitClass : m.cellClass;
    GroupCell<K, G> w;
    w.sh = shared + (threadIdx.x >> 5);
    w.lane = threadIdx.x & 31;
    w.g = min(w.lane / G, kCells - 1);
    w.base = w.g * G;
    w.l = w.lane - w.base;  // >= G on the lanes left over
    uint32_t err = 0;
    // warps are dealt out one per block before any block gets a second
    const int warps = gridDim.x * (kPlaneThreads / 32);
    const int first = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const bool team = kCells > 1 && nm <= p.teamMax;
    const int cells = team ? 1 : kCells;  // of a warp
    for (int q = first; q * cells < nm; q += warps) {
        const int k = team ? q : q * kCells + w.g;
        bool act = k < nm;
        const int i = act && p.rest ? p.rest[k] : k;
        const int c = act ? p.mixed[i] : 0;
        if (act && mask != (1 << cls) && cellCls[c] != cls) act = false;
        if (act && p.skip && p.skip[i]) act = false;
        if (!__any_sync(kAllLanes, act)) continue;
        bool ok;
        if (SPLIT) {
            ok = groupLoadSplit(m, c, act, w);
            __syncwarp();
            groupSplitFace(m, c, w);
        } else {
            ok = groupLoad(m, c, act, w);
        }
        double d = 0.0;
        d3 ic = mk(0, 0, 0), is = mk(0, 0, 0);
        const double alphaI = act ? p.alpha[c] : 0.0;
        const d3 nI = act ? ld3(p.nrm, i) : mk(0, 0, 0);
        const unsigned box = (act && !SPLIT) ? m.boxCorner[c] : 0u;
        int st = team ? teamSignedDistance(w, act && ok, box, alphaI, nI, d, ic, is, err)
                      : groupSignedDistance(w, act && ok, box, alphaI, nI, d, ic, is, err);
        if (act && !ok) {
            err |= kErrSubFaceOverflow;
            st = 1;
        }
        if (act && w.l == 0 && (!team || w.g == 0)) {
            p.mStatus[i] = int8_t(st);
            p.status[c] = int8_t(st);
            p.dOut[i] = d;
            st3(p.icOut, i, ic);
            st3(p.isOut, i, is);
        }
        __syncwarp();
    }
    if (err) atomicOr(p.err, err);
}

// A grid of exactly the blocks that are resident at once on all SMs, looked
// up once per kernel and device.
template <class Kernel>
int residentGrid(Kernel kernel) {
    struct Entry {
        const void* fn;
        int dev, grid;
    };
    constexpr int kSlots = 32;
    static Entry cache[kSlots] = {};
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    const void* fn = reinterpret_cast<const void*>(kernel);
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < kSlots && cache[i].fn; ++i)
        if (cache[i].fn == fn && cache[i].dev == dev) return cache[i].grid;
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kPlaneThreads, 0);
    const int g = (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
    for (int i = 0; i < kSlots; ++i)
        if (!cache[i].fn) {
            cache[i] = {fn, dev, g};
            break;
        }
    return g;
}

template <class K, int G, bool SPLIT>
void launchClass(const DevMesh& m, const PlaneArgs& p, int cls, cudaStream_t st) {
    kPlaneSolve<K, G, SPLIT><<<residentGrid(kPlaneSolve<K, G, SPLIT>), kPlaneThreads, 0, st>>>(m, p, cls);
}

}  // namespace

int smCount() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

PlaneArgs planeArgs(const StepArgs& a) {
    PlaneArgs p;
    p.alpha = a.aCur;
    p.mixed = a.mixed;
    p.nMixed = a.nMixed;
    p.nrm = a.nrm;
    p.mStatus = a.mStatus;
    p.status = a.status;
    p.dOut = a.dArr;
    p.icOut = a.icArr;
    p.isOut = a.isArr;
    p.err = a.err;
    p.skip = nullptr;
    p.rest = nullptr;
    p.teamMax = kTeamPerSm * smCount();
    return p;
}

static void launchAll(const StepArgs& a, const PlaneArgs& p, cudaStream_t st) {
    // lanes per cell: the faces of the class (6 of hexahedra: five cells a
    // warp; 12 of polyhedra on a half-warp; the whole warp beyond)
    if (a.m.splitClassMask) {
        const int mk = a.m.splitClassMask;
        if (mk & 1) launchClass<CapsHex, 6, true>(a.m, p, 0, st);
        if (mk & 2) launchClass<CapsPoly, 16, true>(a.m, p, 1, st);
        if (mk & 4) launchClass<CapsBig, 32, true>(a.m, p, 2, st);
        return;
    }
    const int mk = a.m.classMask;
    if (mk & 1) launchClass<CapsHex, 6, false>(a.m, p, 0, st);
    if (mk & 2) launchClass<CapsPoly, 16, false>(a.m, p, 1, st);
    if (mk & 4) launchClass<CapsBig, 32, false>(a.m, p, 2, st);
}

void launchPlaneSolve(const StepArgs& a, cudaStream_t st) { launchAll(a, planeArgs(a), st); }

void launchPlaneSolveSkip(const StepArgs& a, const uint8_t* skip, cudaStream_t st) {
    PlaneArgs p = planeArgs(a);
    p.skip = skip;
    launchAll(a, p, st);
}

void launchPlaneSolveRest(const StepArgs& a, const int* rest, const int* nRest, cudaStream_t st) {
    PlaneArgs p = planeArgs(a);
    p.rest = rest;
    p.nMixed = nRest;
    launchAll(a, p, st);
}

}  // namespace simplic
