// Launch interface between the C-ABI layer and the kernel translation units.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "simplic_device.cuh"

namespace simplic {

void setCreateError(const std::string& msg);

// Pointers of one reconstruct / advect call (device memory).
struct StepArgs {
    DevMesh m;
    // alpha
    const double* aCur;   // alpha used for classification and upwind fluxes
    const double* aOld;   // alpha.oldTime()
    double* aNew;         // output of advect
    bool handed;          // aCur was handed over again after the interface was found in it
    // per-step inputs
    const double* phi;
    const double* U;
    const double* Ub;
    const double* alphaB;
    const double* Sp;
    const double* Su;
    double dt, rDeltaT;
    double rrDeltaT;      // 1 / rDeltaT (the reciprocal of the update's divisor)
    // controls
    double mixedTol, snapTol;
    int clip, nAlphaBounds;
    // reconstruction state (compact, indexed by position in the mixed list)
    int8_t* status;   // [nc]
    int* mixed;       // [nc]
    int* nMixed;      // [0] mixed cells, [1] those the mixed forms' box planes left to the general solve
    double* nrm;      // [3 nc]
    int8_t* mStatus;  // [nc]
    double* dArr;     // [nc]
    double* icArr;    // [3 nc]
    double* isArr;    // [3 nc]
    // advection state
    double* dvfI;       // [nf] Simpson dVf of faces downwind of cut cells
    double* alphaPhi;   // [nf]
    uint8_t* cutMask;   // [nf] optional record of Simpson faces
    double* un0;        // [nc] interface normal speed of cut cells
    int2* dwList;       // [nf] (mixed index, face) of every downwind face of a cut cell
    int* dwCount;
    int* ovList;        // cells the update left outside [-aTol, 1+aTol]
    int* ovCount;
    int ovCap;
    uint32_t* err;      // device error bits
};

// Polls of the bounding kernel's grid barrier before it gives up: about 1-2 s
// with 64 ns sleeps, far beyond any wait of a working launch.
constexpr long long kBarrierSpins = 20000000;

// Bounding kernel limits and the layout of its per-step control counters.
constexpr int kMaxBoundPasses = 64;   // nAlphaBounds cap
enum : int {
    kCtlCand = 0,     // candidates so far
    kCtlMod = 1,      // faces whose dVf the bounding changed
    kCtlActive0 = 4,  // [pass] overshooting candidates
    kCtlOverDelta0 = kCtlActive0 + kMaxBoundPasses,  // [pass] change of the overshoot count
    kCtlTouched0 = kCtlOverDelta0 + kMaxBoundPasses, // [pass] target cells of the pass
    kCtlFree0 = kCtlTouched0 + kMaxBoundPasses,      // [pass] cells that wait for nobody
    kCtlFreeHead0 = kCtlFree0 + kMaxBoundPasses,     // [pass] of those, taken beyond the first per warp
    kCtlQHead0 = kCtlFreeHead0 + kMaxBoundPasses,    // [pass] released cells taken from the queue
    kCtlQTail0 = kCtlQHead0 + kMaxBoundPasses,       // [pass] released cells written to the queue
    kCtlDone0 = kCtlQTail0 + kMaxBoundPasses,        // [pass] cells run
    kCtlStarts0 = kCtlDone0 + kMaxBoundPasses,       // [pass] chains started
    kCtlSize = kCtlStarts0 + kMaxBoundPasses,
};
// Record of an overshooting candidate: the constants of its loop, then one
// slot per face; whole 128-byte lines.
constexpr int kBoundCellConstBytes = 112;
constexpr int kBoundSlotBytes = 48;
constexpr size_t boundRecordBytes(int maxCellFaces) {
    return (size_t(kBoundCellConstBytes) + size_t(kBoundSlotBytes) * maxCellFaces + 127) / 128 * 128;
}

// Scratch of the bounding kernel (per-candidate arrays have candCap rows).
struct BoundBuffers {
    int* ovList;
    int* ovCount;
    int ovCap;
    int* cand;
    int candCap;
    int* candIdx;      // [nc] position of a candidate cell
    int* candMark;     // [nc] step stamp: cell is a candidate
    int* cellClaim;    // [nc] pass stamp: target already updated
    unsigned* faceKey; // [nf] list position key of a corrected face (cell * 32 + position)
    int* faceStamp;    // [nf] pass stamp of faceKey
    int* touched;
    int touchedCap;
    double* corr;      // [nf], zero outside a pass
    double* dvfMod;    // [nf] dVf of faces the bounding changed
    int* modStamp;     // [nf] step stamp of dvfMod
    int* modList;
    int modCap;
    int* ctl;          // [kCtlSize] counters, zeroed before every launch
    unsigned* barCount;    // zeroed before every launch
    unsigned* barGen;
    long long spinLimit;   // polls before a bounded wait gives up (kBarrierSpins)
    int barrierExtra;      // arrivals a barrier waits for beyond the grid (test setting; 0)
    int stamp;
    int* info;  // [0] passes run, [1] most cells bounded in a pass, [2] most chains started
                // from the ready queue in a pass, [3] overflow code, [4] most cells one warp
                // ran in a row along a chain, [5] cells run in all passes, [6] us in the
                // dependency phases, [7] us of the launch ([6], [7] on block 0's clock)
    // The overshooting candidates of the current pass with everything their
    // loop needs that reads no correction, computed before the dependency
    // phase (per face slot and per cell), the dependency counts and the
    // ready queue.
    int* actList;          // [candCap] overshooting candidates of the pass
    uint8_t* rec;          // [candCap * recBytes] their records (BoundCellConst, BoundSlot per face)
    int recBytes;
    int* candPending;      // [candCap] faces on which the cell waits for an earlier cell that has not started
    unsigned* candPm;      // [candCap] faces that pass in the loop's first iteration
    unsigned long long* readyQ;  // [candCap] (pass stamp << 32) | candidate: from the front the cells
                                 // that wait for nobody, from the back the released ones
};

// arguments of the three plane-solve kernels
struct PlaneArgs {
    const double* alpha;
    const int* mixed;
    const int* nMixed;
    const double* nrm;
    int8_t* mStatus;
    int8_t* status;
    double* dOut;
    double* icOut;
    double* isOut;
    uint32_t* err;
    const uint8_t* skip;  // optional per mixed cell: nonzero keeps the previous plane (isoRDF)
    int teamMax;          // lists up to here: a warp per cell
    const int* rest;      // optional list of mixed positions to solve, *nMixed of them
};

// Buffers of the isoRDF orientation (reconstruction.C:193-405), allocated
// when a handle is created with that method.
struct RdfBuffers {
    double* rdf;        // [nc] reconstructed distance function
    int2* cellMix;      // [nc] (stamp, position in the mixed list) of a mixed cell
    int* bandStamp;     // [nc] stamp: the cell is in the band
    int* bandList;      // [nc] band cells
    int* bandCount;     // [1]
    double* grad;       // [3 nc] per mixed position: the gradient being iterated
    double* res;        // [nc] per mixed position: normal residual
    double* avgA;       // [nc] per mixed position: mean angle to the neighbours' normals
    uint8_t* tooCoarse; // [nc] per mixed position
    int stamp;
};

int smCount();  // of the current device
void launchScanMixed(const StepArgs& a, cudaStream_t st);
// isoRDF: band, cell -> mixed position map, alpha gradient (start); then per
// iteration: normals from the gradient, the plane solve of the cells not
// too coarse, the distance function on the band, its gradient and the
// residuals
void launchRdfStart(const StepArgs& a, const RdfBuffers& r, cudaStream_t st);
void launchRdfNormals(const StepArgs& a, const RdfBuffers& r, cudaStream_t st);
void launchPlaneSolveSkip(const StepArgs& a, const uint8_t* skip, cudaStream_t st);
// the plane solve of the mixed positions rest[0 .. *nRest) only
void launchPlaneSolveRest(const StepArgs& a, const int* rest, const int* nRest, cudaStream_t st);
void launchRdfConstruct(const StepArgs& a, const RdfBuffers& r, cudaStream_t st);
void launchRdfResidual(const StepArgs& a, const RdfBuffers& r, cudaStream_t st);
// PLIC polygon of every mixed cell: up to `stride` points at pts[3 stride i],
// count[i] points (0 where the plane does not cut the cell)
void launchPlicPolygons(const StepArgs& a, int stride, double* pts, int* count, cudaStream_t st);
// alpha = cut volume fraction of the given plane where lower <= alpha <= upper
void launchMapAlpha(const DevMesh& m, double* alpha, const double* normal, const double* distance, double lower,
                    double upper, uint32_t* err, cudaStream_t st);
void launchLsNormal(const StepArgs& a, cudaStream_t st);
PlaneArgs planeArgs(const StepArgs& a);
void launchPlaneSolve(const StepArgs& a, cudaStream_t st);
void launchInterfaceUn0(const StepArgs& a, cudaStream_t st);
void launchInterfaceFaces(const StepArgs& a, cudaStream_t st);
void launchUpdate(const StepArgs& a, cudaStream_t st);
cudaError_t launchBound(const StepArgs& a, const BoundBuffers& b, cudaStream_t st);
void launchBruteForce(const StepArgs& a, cudaStream_t st);
void launchFaceFlatness(const DevMesh& m, const double* Sf, double* flat, cudaStream_t st);
// also the axis codes, and in *warped whether a face is warped (flat is ready)
void launchFaceFull(const DevMesh& m, double* fullC, double* fullA, uint8_t* faceAxis, int* warped, cudaStream_t st);
void launchRecipVolume(const DevMesh& m, double* rV, cudaStream_t st);
// LS stencil rows of all cells: lengths (count) or the rows at off
void launchStencilRows(const DevMesh& m, bool count, int* len, const int* off, int* rows, cudaStream_t st);
// mixed-precision form (FP32 normals and Simpson clipping, FP64 volume matching)
void launchLsNormalMixed(const StepArgs& a, cudaStream_t st);
// boxes: the mesh has axis-aligned box cells
void launchPlaneSolveMixed(const StepArgs& a, bool boxes, cudaStream_t st);
void launchInterfaceUn0Mixed(const StepArgs& a, cudaStream_t st);
void launchInterfaceFacesMixed(const StepArgs& a, cudaStream_t st);
// learned-normal form (the mixed form with the network's normals)
void launchMakeSamples(const DevMesh& m, unsigned long long seed, int count, int spherePct, void* X, float* T,
                       uint32_t* err, cudaStream_t st);
// network inputs of the first maxRows mixed cells, their alphas in FP32
// (A: [row][32], alpha_c then alpha_j - alpha_c per slot), and the FP32
// least-squares normal of every mixed cell (written to a.nrm); the cells
// from maxRows on get no row
void launchGatherFeatures(const StepArgs& a, int maxRows, void* X, float* A, cudaStream_t st);
cudaError_t launchNetwork(const void* X, const int* Mdev, int maxRows, const void* W, const float* bias, float* Y,
                          int ldy, uint32_t* err, cudaStream_t st);
// the learned form's choice per network row: normalise(n_ls + y[0:3]) (n_ls
// from the row's input) unless degenerate or its local volume residual or
// face-flux mismatch exceeds the least-squares normal's by more than
// gateTol; nLearned counts the choices
void launchLearnedGate(const StepArgs& a, int maxRows, const void* X, const float* A, const float* Y, int ldY,
                       float gateTol, int* nLearned, cudaStream_t st);

}  // namespace simplic
