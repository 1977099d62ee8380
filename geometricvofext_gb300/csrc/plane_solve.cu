// Plane constant of every mixed cell (cutCell::findSignedDistance,
// cutCell.C:611-799), a group of lanes per cell (plane_group.cuh).  Built
// with -fmad=false.
//
// One GB300, kernel time with one thread per cell -> now (deformation field;
// interface cells in brackets):
//   24^3 hex (331) 0.861 -> 0.049 ms, 33^3 (617) 0.880 -> 0.055
//   128^3 hex (30,189) 1.451 -> 0.634, 256^3 (35,452) 1.636 -> 0.720
//   96^3 warped hex (7,146) 0.985 -> 0.348
//   24^3 with 2:1 refinement (755), three solves: 20.8 -> 0.49
// In the middle of the 128^3 run the FP64 pipe is 72% busy in active cycles,
// 64% of the kernel's time (the rest is the tail).
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

// The mixed cells of one class (workspace caps K, G lanes per cell) on the
// blocks first, first + 1 .. of a grid of `blocks`.  With SPLIT the workspace
// is the splitWarpedFace one.
template <class K, int G, bool SPLIT>
__device__ __forceinline__ void solveClass(const DevMesh& m, const PlaneArgs& p, int cls, GroupShared<K, G>* shared,
                                           int block, int blocks) {
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
    const int warps = blocks * (kPlaneThreads / 32);
    const int first = (threadIdx.x >> 5) * blocks + block;
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
        // (of the classes beyond hexahedra any cell may be a box)
        const unsigned box = (act && !SPLIT) ? (K::kFaces == 6 ? m.boxCorner[c] : 1u) : 0u;
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

// Six blocks per SM (168 registers, a few spilled) against four (200
// registers): 0.80 against 0.82 ms at 128^3, 0.35 against 0.44 on the warped
// 96^3 mesh; eight blocks spill more and gain nothing.
template <class K, int G, bool SPLIT>
__global__ void __launch_bounds__(kPlaneThreads, 6) kPlaneSolve(DevMesh m, PlaneArgs p, int cls) {
    __shared__ GroupShared<K, G> shared[kPlaneThreads / 32];
    solveClass<K, G, SPLIT>(m, p, cls, shared, blockIdx.x, gridDim.x);
}

// Meshes with cells of several classes: a set of blocks for each, the largest
// cells (the longest chains) first; the blocks of a class that has few cells
// leave at once and the next take their place.  With one launch per class the
// classes waited for one another: 24^3 of two sizes in a checkerboard (748
// cells) 0.41 -> 0.24 ms, 36^3 (1,755) 0.71 -> 0.44, 48^3 (2,953) 0.69 -> 0.48,
// 32^3 refined in the middle (1,423) 0.30 -> 0.21.
template <bool SPLIT>
__global__ void __launch_bounds__(kPlaneThreads, 5) kPlaneSolveAll(DevMesh m, PlaneArgs p, int mask, int blocks) {
    constexpr int kWarps = kPlaneThreads / 32;
    constexpr size_t kHex = sizeof(GroupShared<CapsHex, 6>), kPoly = sizeof(GroupShared<CapsPoly, 16>),
                     kBig = sizeof(GroupShared<CapsBig, 32>), kMax = kHex > kPoly ? kHex : kPoly;
    __shared__ __align__(16) unsigned char shared[kWarps * (kMax > kBig ? kMax : kBig)];
    int set = blockIdx.x / blocks;
    const int block = blockIdx.x - set * blocks;
    for (int cls = 2; cls >= 0; --cls) {
        if (!((mask >> cls) & 1) || set-- != 0) continue;
        if (cls == 2)
            solveClass<CapsBig, 32, SPLIT>(m, p, 2, reinterpret_cast<GroupShared<CapsBig, 32>*>(shared), block, blocks);
        else if (cls == 1)
            solveClass<CapsPoly, 16, SPLIT>(m, p, 1, reinterpret_cast<GroupShared<CapsPoly, 16>*>(shared), block,
                                            blocks);
        else
            solveClass<CapsHex, 6, SPLIT>(m, p, 0, reinterpret_cast<GroupShared<CapsHex, 6>*>(shared), block, blocks);
    }
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

// lanes per cell: the faces of the class (6 of hexahedra: five cells a warp;
// 12 of polyhedra on a half-warp; the whole warp beyond)
template <bool SPLIT>
static void launchClasses(const DevMesh& m, const PlaneArgs& p, int mask, cudaStream_t st) {
    if (mask & (mask - 1)) {
        const int blocks = residentGrid(kPlaneSolveAll<SPLIT>), sets = (mask & 1) + ((mask >> 1) & 1) + ((mask >> 2) & 1);
        kPlaneSolveAll<SPLIT><<<sets * blocks, kPlaneThreads, 0, st>>>(m, p, mask, blocks);
        return;
    }
    if (mask & 1) launchClass<CapsHex, 6, SPLIT>(m, p, 0, st);
    if (mask & 2) launchClass<CapsPoly, 16, SPLIT>(m, p, 1, st);
    if (mask & 4) launchClass<CapsBig, 32, SPLIT>(m, p, 2, st);
}

static void launchAll(const StepArgs& a, const PlaneArgs& p, cudaStream_t st) {
    if (a.m.splitClassMask) launchClasses<true>(a.m, p, a.m.splitClassMask, st);
    else launchClasses<false>(a.m, p, a.m.classMask, st);
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
