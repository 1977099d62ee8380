// isoRDF orientation of the plain FP64 form (built with -fmad=false):
// reconstruction::calcInterfaceNFromIsoRDF (reconstruction.C:193-405).
//
// The reference iterates: normals from a least-squares gradient, the plane
// solve (cutCell::findSignedDistance) of every mixed cell not marked too
// coarse, a reconstructed distance function (RDF) on the band of cells
// next to the interface, its least-squares gradient as the next normal,
// and a residual per mixed cell whose sums decide whether to stop.  The
// distance function is OpenFOAM v2312's reconstructedDistanceFunction
// (linked into the reference by src/Allwmake:17-19, absent here), restated
// from the published method (Scheufler & Roenby, J. Comput. Phys. 383
// (2019) 1-23) exactly as the CPU oracle restates it:
//   * band: the mixed cells and every cell sharing a point with one;
//   * a mixed cell with a nonzero normal n: RDF = (C_int - C) . n/|n|;
//   * any other band cell: sum_j w_j (C_int,j - C) . n_j / sum_j w_j over
//     its stencil cells j that carry a plane, w_j the squared cosine between
//     n_j and the direction to C_int,j (1 when C_int,j = C); a cell without
//     such a neighbour keeps its value (zero at the start of a reconstruct).
// The per-cell arithmetic is the oracle's, operation for operation, one thread
// per cell or, on lists that leave the FP64 pipes idle (kLsGroup), 16 lanes:
// the gradient as in ls_group.cuh, the terms of the stencil cells a lane each
// and their sums in order.  The residual sums that decide the iteration count
// run on the host over the mixed cells in ascending order.
// The ten launches of 24^3 with 2:1 refinement (755 interface cells, three
// iterations), a thread per cell -> 16 lanes: 1.16 -> 0.20 ms; of 90^3 warped
// hexahedra (6,539, five) 1.34 -> 1.24, of 26^3 x 6 tetrahedra (2,016) 1.95 ->
// 0.46.
#include "ls_group.cuh"
#include "plain_geom.cuh"
#include "simplic_kernels.h"

namespace simplic {

namespace {

// The band has three to four cells per interface cell, each without an
// elimination: its line in cells per SM.  All isoRDF launches of a step with
// the band's kernel by a thread per cell / by 16 lanes, us: hexahedra, band of
// 2,802 cells 316 / 137, 10,731 585 / 437, 19,050 810 / 718, 26,022 815 / 798,
// 37,334 953 / 956; tetrahedra 13,739 1,635 / 1,182; cells of two sizes 4,547
// 607 / 247; warped 15,632 1,124 / 882.  152 SMs: the line is 24,320.
constexpr int kRdfBandGroup = 4 * kLsGroup;

// OpenFOAM Vector::normalise(tol): zero below tol, else divided by |v|.
__device__ __forceinline__ d3 normaliseOF(d3 v, double tol) {
    const double s = mag(v);
    return (s < tol) ? mk(0, 0, 0) : v / s;
}

// The mixed position of cell x this reconstruct, or -1.
__device__ __forceinline__ int mixPos(const RdfBuffers& r, int x) {
    const int2 cm = r.cellMix[x];
    return cm.x == r.stamp ? cm.y : -1;
}

// Band, cell -> mixed position, and the alpha gradient of every mixed cell.
__global__ void __launch_bounds__(128) kRdfStart(DevMesh m, const double* __restrict__ alpha,
                                                 const int* __restrict__ mixed, const int* __restrict__ nMixed,
                                                 RdfBuffers r, int groupMax, uint32_t* __restrict__ errOut) {
    const int nm = *nMixed;
    uint32_t err = 0;
    if (nm <= groupMax) {
        __shared__ LsRows rows[8];
        const int lane = threadIdx.x & 31, l = lane & 15, warps = gridDim.x * (blockDim.x >> 5);
        for (int q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; 2 * q < nm; q += warps) {
            const int i = 2 * q + (lane >> 4);
            const bool act = i < nm;
            const int c = act ? mixed[i] : 0;
            if (act) {
                const int32_t* st;
                const int ns = stencilOf(m, c, st, err);
                for (int s = l - 1; s < ns; s += 16) {
                    const int x = (s < 0) ? c : st[s];
                    if (atomicExch(r.bandStamp + x, r.stamp) != r.stamp) {
                        r.rdf[x] = 0.0;
                        r.bandList[atomicAdd(r.bandCount, 1)] = x;
                    }
                }
            }
            __syncwarp();
            const d3 g = groupLsGradient(m, act, c, alpha, rows[threadIdx.x >> 4], err);
            if (act && l == 0) {
                r.cellMix[c] = make_int2(r.stamp, i);
                st3(r.grad, i, g);
                r.tooCoarse[i] = 0;
            }
        }
        if (err) atomicOr(errOut, err);
        return;
    }
    for (int i = spreadFirst(); i < nm; i += spreadStride()) {
        const int c = mixed[i];
        r.cellMix[c] = make_int2(r.stamp, i);
        const int32_t* st;
        const int ns = stencilOf(m, c, st, err);
        for (int s = -1; s < ns; ++s) {
            const int x = (s < 0) ? c : st[s];
            if (atomicExch(r.bandStamp + x, r.stamp) != r.stamp) {
                r.rdf[x] = 0.0;
                r.bandList[atomicAdd(r.bandCount, 1)] = x;
            }
        }
        st3(r.grad, i, lsGradientField(m, c, alpha, err));
        r.tooCoarse[i] = 0;
    }
    if (err) atomicOr(errOut, err);
}

// interfaceN = -normalise(grad), the gradient normalised in place
// (reconstruction.C:240).
__global__ void __launch_bounds__(128) kRdfNormals(const int* __restrict__ nMixed, RdfBuffers r,
                                                   double* __restrict__ nrm) {
    const int nm = *nMixed;
    for (int i = spreadFirst(); i < nm; i += spreadStride()) {
        const d3 g = normaliseOF(ld3(r.grad, i), kSMALL);
        st3(r.grad, i, g);
        st3(nrm, i, (-1.0) * g);
    }
}

// The sums over a stencil by the 16 lanes of a group: `term` gives the two
// parts of one entry (false: none), which lanes 0 and 1 add up in order.
template <class Term>
__device__ __forceinline__ double2 groupSums(int n, double2* part, const Term& term) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, l = lane & 15, base = lane & 16;
    const int nMax = max(n, __shfl_xor_sync(kAll, n, 16));
    double sum = 0.0;
    for (int e0 = 0; e0 < nMax; e0 += 16) {
        double2 v = make_double2(0.0, 0.0);
        const bool has = e0 + l < n && term(e0 + l, v);
        part[l] = v;
        unsigned mm = (__ballot_sync(kAll, has) >> base) & 0xffffu;
        __syncwarp();
        for (; mm; mm &= mm - 1u) {
            const double2 w = part[__ffs(mm) - 1];
            sum += (l & 1) ? w.y : w.x;
        }
        __syncwarp();
    }
    return make_double2(__shfl_sync(kAll, sum, base), __shfl_sync(kAll, sum, base + 1));
}

// What stencil cell g adds to the distance at p: distance to its plane times
// weight, and weight.
__device__ __forceinline__ bool rdfTerm(const RdfBuffers& r, const double* nrm, const double* icArr, int g, d3 p,
                                        double2& out) {
    const int ig = mixPos(r, g);
    if (ig < 0) return false;  // no plane: a zero normal
    d3 n = (-1.0) * ((-1.0) * ld3(nrm, ig));
    if (!(mag(n) != 0.0)) return false;
    n = n / mag(n);
    d3 toSeg = ld3(icArr, ig) - p;
    const double distToSurf = dot(toSeg, n);
    double weight;
    if (mag(toSeg) != 0.0) {
        toSeg = toSeg / mag(toSeg);
        const double w = fabs(dot(toSeg, n));
        weight = w * w;
    } else {
        weight = 1.0;
    }
    out = make_double2(distToSurf * weight, weight);
    return true;
}

// constructRDF on the band (normals -interfaceN passed in, negated again).
__global__ void __launch_bounds__(128) kRdfConstruct(DevMesh m, RdfBuffers r, const double* __restrict__ nrm,
                                                     const double* __restrict__ icArr, int groupMax,
                                                     uint32_t* __restrict__ errOut) {
    const int nb = *r.bandCount;
    uint32_t err = 0;
    if (nb <= groupMax) {
        __shared__ double2 parts[8][16];
        const int lane = threadIdx.x & 31, l = lane & 15, warps = gridDim.x * (blockDim.x >> 5);
        for (int q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; 2 * q < nb; q += warps) {
            const int k = 2 * q + (lane >> 4);
            const int c = k < nb ? r.bandList[k] : -1;
            const int ic = c >= 0 ? mixPos(r, c) : -1;
            const d3 p = ld3(m.C, max(c, 0));
            bool open = c >= 0;
            if (ic >= 0) {
                const d3 normalC = (-1.0) * ld3(nrm, ic);
                if (mag(normalC) != 0.0) {
                    const d3 n = ((-1.0) * normalC) / mag(normalC);
                    if (l == 0) r.rdf[c] = dot(ld3(icArr, ic) - p, n);
                    open = false;
                }
            }
            const int32_t* st = nullptr;
            const int n = open ? stencilOf(m, c, st, err) + 1 : 0;
            const double2 s = groupSums(n, parts[threadIdx.x >> 4], [&](int e, double2& t) {
                return rdfTerm(r, nrm, icArr, e ? st[e - 1] : c, p, t);
            });
            if (open && l == 0 && s.y != 0.0) r.rdf[c] = s.x / s.y;
        }
        if (err) atomicOr(errOut, err);
        return;
    }
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nb; q += gridDim.x * blockDim.x) {
        const int c = r.bandList[q];
        const int ic = mixPos(r, c);
        if (ic >= 0) {
            const d3 normalC = (-1.0) * ld3(nrm, ic);
            if (mag(normalC) != 0.0) {
                const d3 n = ((-1.0) * normalC) / mag(normalC);
                r.rdf[c] = dot(ld3(icArr, ic) - ld3(m.C, c), n);
                continue;
            }
        }
        double averageDist = 0.0, avgWeight = 0.0;
        const d3 p = ld3(m.C, c);
        const int32_t* st;
        const int ns = stencilOf(m, c, st, err);
        for (int s = -1; s < ns; ++s) {
            const int g = (s < 0) ? c : st[s];
            double2 t;
            if (rdfTerm(r, nrm, icArr, g, p, t)) {
                averageDist += t.x;
                avgWeight += t.y;
            }
        }
        if (avgWeight != 0.0) r.rdf[c] = averageDist / avgWeight;
    }
    if (err) atomicOr(errOut, err);
}

// Angle between n and the normal of stencil cell g, times that one's
// magnitude, and the magnitude.
__device__ __forceinline__ bool angleTerm(const RdfBuffers& r, const double* nrm, int g, d3 n, double2& out) {
    const int ig = mixPos(r, g);
    if (ig < 0) return false;
    const d3 normal = ld3(nrm, ig);
    const double s = mag(normal);
    if (!(s >= kTSMALL)) return false;
    const double cosAngle = fmax(fmin(dot(n, normal / s), 1.0), -1.0);
    out = make_double2(acos(cosAngle) * s, s);
    return true;
}

// The gradient of the distance function and the residual of every mixed
// cell (reconstruction.C:264-332): the mean angle to the neighbours'
// normals (weighted by their magnitudes) and 1 - n . n_new.
__global__ void __launch_bounds__(128) kRdfResidual(DevMesh m, const int* __restrict__ mixed,
                                                    const int* __restrict__ nMixed, RdfBuffers r,
                                                    const double* __restrict__ nrm, int groupMax,
                                                    uint32_t* __restrict__ errOut) {
    const int nm = *nMixed;
    uint32_t err = 0;
    if (nm <= groupMax) {
        __shared__ LsRows rows[8];
        __shared__ double2 parts[8][16];
        const int lane = threadIdx.x & 31, l = lane & 15, warps = gridDim.x * (blockDim.x >> 5);
        for (int q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; 2 * q < nm; q += warps) {
            const int i = 2 * q + (lane >> 4);
            const bool act = i < nm;
            const int c = act ? mixed[i] : 0;
            d3 g = groupLsGradient(m, act, c, r.rdf, rows[threadIdx.x >> 4], err);
            const d3 cellNormal = act ? ld3(nrm, i) : mk(0, 0, 0);
            if (!(mag(cellNormal) < kTSMALL)) g = normaliseOF(g, kSMALL);
            const int32_t* st = nullptr;
            const int n = act ? stencilOf(m, c, st, err) : 0;  // after the cell itself
            const double2 s = groupSums(n, parts[threadIdx.x >> 4], [&](int e, double2& t) {
                return angleTerm(r, nrm, st[e], cellNormal, t);
            });
            g = normaliseOF(g, kSMALL);
            if (act && l == 0) {
                st3(r.grad, i, g);
                r.res[i] = 1.0 - dot(cellNormal, (-1.0) * g);
                r.avgA[i] = (s.y != 0.0) ? s.x / s.y : 0.0;
            }
        }
        if (err) atomicOr(errOut, err);
        return;
    }
    for (int i = spreadFirst(); i < nm; i += spreadStride()) {
        const int c = mixed[i];
        d3 g = lsGradientField(m, c, r.rdf, err);
        const d3 cellNormal = ld3(nrm, i);
        // the reference's zero-normal test normalises the gradient in place
        // when the cell's own normal is not zero
        if (!(mag(cellNormal) < kTSMALL)) g = normaliseOF(g, kSMALL);
        double avgDiff = 0.0, weight = 0.0;
        const int32_t* st;
        const int ns = stencilOf(m, c, st, err);
        for (int s = 0; s < ns; ++s) {  // stencil entries after the cell itself
            double2 t;
            if (angleTerm(r, nrm, st[s], cellNormal, t)) {
                avgDiff += t.x;
                weight += t.y;
            }
        }
        avgDiff = (weight != 0.0) ? avgDiff / weight : 0.0;
        g = normaliseOF(g, kSMALL);
        st3(r.grad, i, g);
        r.res[i] = 1.0 - dot(cellNormal, (-1.0) * g);
        r.avgA[i] = avgDiff;
    }
    if (err) atomicOr(errOut, err);
}

template <class Kernel>
int gridFor(Kernel k, int threads) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, threads, 0);
    return (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
}

}  // namespace

void launchRdfStart(const StepArgs& a, const RdfBuffers& r, cudaStream_t st) {
    kRdfStart<<<gridFor(kRdfStart, 128), 128, 0, st>>>(a.m, a.aCur, a.mixed, a.nMixed, r,
                                                              kLsGroup * smCount(), a.err);
}

void launchRdfNormals(const StepArgs& a, const RdfBuffers& r, cudaStream_t st) {
    kRdfNormals<<<gridFor(kRdfNormals, 128), 128, 0, st>>>(a.nMixed, r, a.nrm);
}

void launchRdfConstruct(const StepArgs& a, const RdfBuffers& r, cudaStream_t st) {
    kRdfConstruct<<<gridFor(kRdfConstruct, 128), 128, 0, st>>>(a.m, r, a.nrm, a.icArr,
                                                                    kRdfBandGroup * smCount(), a.err);
}

void launchRdfResidual(const StepArgs& a, const RdfBuffers& r, cudaStream_t st) {
    kRdfResidual<<<gridFor(kRdfResidual, 128), 128, 0, st>>>(a.m, a.mixed, a.nMixed, r, a.nrm,
                                                                  kLsGroup * smCount(), a.err);
}

}  // namespace simplic
