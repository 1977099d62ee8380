// Plain FP64 SimPLIC kernels (built with -fmad=false: bit-exact to the CPU
// restatement of the reference).
//
//  K1 scanMixed          reconstruction::initialize      reconstruction.C:634-677
//  K2 lsNormal           calcInterfaceNFromIsoAlphaGrad  reconstruction.C:85-141
//  K3 planeSolve         (plane_solve.cu)
//  K4 interfaceFlux      advection::timeIntegratedFlux   advection.C:85-221
//  K5 update             upwind dVf + surfaceIntegrate + alpha update
//                                                        advectionTemplates.C:371,399-406
//  K6 bound              limitFlux / boundFlux           advectionTemplates.C:118-349
//  K7 bruteForce         applyBruteForceBounding         advection.C:291-308
//  faceFlatness          reconstruction::updateFaceFlatness reconstruction.C:408-440
#include "face_group.cuh"
#include "ls_group.cuh"
#include "plain_geom.cuh"
#include "simplic_kernels.h"

#include <cfloat>
#include <climits>
#include <cstring>
#include <mutex>

namespace simplic {

// ---------------------------------------------------------------------------
// K1: mixed-cell list (warp-aggregated append) and per-cell status bytes
// ---------------------------------------------------------------------------
// isAMixedCell (reconstruction.H:281-288): tol < a < 1 - tol.  Evaluated on
// the bit patterns: for 0 <= tol < 0.5 the signed 64-bit order of a double's
// bits matches its numeric order on [+0, +inf], negative values fail the
// first test and NaN fails the second, exactly as the double comparisons do
// -- and it keeps the narrow FP64 pipe out of this memory-bound scan.
__global__ void __launch_bounds__(256) kScanMixed(int nc, const double* __restrict__ alpha, long long tolBits,
                                                  long long oneMinusTolBits, int8_t* __restrict__ status,
                                                  int* __restrict__ mixed, int* __restrict__ nMixed,
                                                  uint32_t* __restrict__ err) {
    // four cells per thread: two 16-byte loads, one 4-byte status store
    const int c0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    unsigned flags = 0;
    bool bad = false;  // a NaN or an infinity (all exponent bits set)
    const auto nonFinite = [](long long v) { return (v & 0x7ff0000000000000LL) == 0x7ff0000000000000LL; };
    if (c0 + 3 < nc) {
        const double2 p = *reinterpret_cast<const double2*>(alpha + c0);
        const double2 q = *reinterpret_cast<const double2*>(alpha + c0 + 2);
        const long long v[4] = {bitsOf(p.x), bitsOf(p.y), bitsOf(q.x), bitsOf(q.y)};
        uint32_t st = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool mx = v[k] > tolBits && v[k] < oneMinusTolBits;
            flags |= unsigned(mx) << k;
            bad = bad || nonFinite(v[k]);
            st |= uint32_t(uint8_t(mx ? kStPending : kStNotMixed)) << (8 * k);
        }
        *reinterpret_cast<uint32_t*>(status + c0) = st;
    } else {
        for (int k = 0; k < 4 && c0 + k < nc; ++k) {
            const long long v = bitsOf(alpha[c0 + k]);
            const bool mx = v > tolBits && v < oneMinusTolBits;
            flags |= unsigned(mx) << k;
            bad = bad || nonFinite(v);
            status[c0 + k] = mx ? kStPending : kStNotMixed;
        }
    }
    // a non-finite alpha is reported (the reference would carry it into
    // every neighbour's flux without notice)
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(err, (uint32_t)kErrNonFinite);
    // the mixed cells in ascending order within each thread, one atomic per warp
    const int lane = threadIdx.x & 31;
    const int cnt = __popc(flags);
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (total == 0) return;
    int base = 0;
    if (lane == 31) base = atomicAdd(nMixed, total);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - cnt;
    for (int k = 0; k < 4; ++k)
        if ((flags >> k) & 1u) mixed[base++] = c0 + k;
}

// ---------------------------------------------------------------------------
// K2: least-squares normal (polyDegree1 fit over the cell-point-cell stencil)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) kLsNormal(DevMesh m, const double* __restrict__ alpha,
                                                 const int* __restrict__ mixed, const int* __restrict__ nMixed,
                                                 double* __restrict__ nrm, int groupMax,
                                                 uint32_t* __restrict__ errOut) {
    const int nm = *nMixed;
    uint32_t err = 0;
    if (nm <= groupMax) {
        __shared__ LsRows rows[8];
        const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
        for (int q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; 2 * q < nm; q += warps) {
            const int i = 2 * q + (lane >> 4);
            const bool act = i < nm;
            const d3 g = groupLsGradient(m, act, act ? mixed[i] : 0, alpha, rows[threadIdx.x >> 4], err);
            const d3 n = (-1.0) * g;
            const int k = lane & 15;
            const double s = mag(n) + kSMALL, v = (k == 0 ? n.x : (k == 1 ? n.y : n.z)) / s;
            if (act && k < 3) nrm[size_t(3) * i + k] = v;
        }
        if (err) atomicOr(errOut, err);
        return;
    }
    for (int i = spreadFirst(); i < nm; i += spreadStride()) {
        const int c = mixed[i];
        const d3 g = lsGradientField(m, c, alpha, err);
        const d3 n = (-1.0) * g;
        st3(nrm, i, n / (mag(n) + kSMALL));
    }
    if (err) atomicOr(errOut, err);
}

// ---------------------------------------------------------------------------
// K4: Simpson time-integrated flux through downwind faces of cut cells
// ---------------------------------------------------------------------------
__device__ __forceinline__ d3 pointValue(const DevMesh& m, int p, const double* U, const double* Ub) {
    const int b0 = m.pbOff[p], b1 = m.pbOff[p + 1];
    d3 r = mk(0, 0, 0);
    if (b1 > b0) {
        for (int k = b0; k < b1; ++k) {
            const int f = m.pbFaces[k];
            const d3 u = Ub ? ld3(Ub, f - m.nfi) : ld3(U, m.own[f]);
            r = r + m.pbW[k] * u;
        }
        return r;
    }
    for (int k = m.pcOff[p]; k < m.pcOff[p + 1]; ++k) r = r + m.pcW[k] * ld3(U, m.pCells[k]);
    return r;
}

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 leadingF3(d3 v) { return {leadingFloat(v.x), leadingFloat(v.y), leadingFloat(v.z)}; }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float maxAbs(F3 a) { return fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z))); }
__device__ __forceinline__ float det3(F3 a, F3 b, F3 c) {
    return a.x * (b.y * c.z - b.z * c.y) + a.y * (b.z * c.x - b.x * c.z) + a.z * (b.x * c.y - b.y * c.x);
}

// Bounds of the least weight of r in the tetrahedron.  The components are
// differences of coordinates up to M cut to 24 bits, so each is within q =
// 2^-21 M + 2^-22 L of the exact one (L the largest of them); a triple
// product's error is below 18 L^2 q from the components and 30 2^-24 L^3 from
// its own roundings, together below E = 32 L^2 q (the apex's, a sum of four: 4
// E).  With |det| > 2 E a quotient w is then within 2 E (4 + |w|) / |det| and
// the division's own error; the double weights are far closer.
__device__ __forceinline__ void leastWeightBounds(F3 r, F3 e1, F3 e2, F3 e3, float M, float& lo, float& hi) {
    const float L = fmaxf(fmaxf(maxAbs(r), maxAbs(e1)), fmaxf(maxAbs(e2), maxAbs(e3)));
    const float E = 32.f * L * L * (0x1p-21f * M + 0x1p-22f * L);
    const float det = det3(e1, e2, e3);
    lo = -FLT_MAX;
    hi = FLT_MAX;
    if (!(E > 1e-30f && L < 1e9f && fabsf(det) > 2.f * E)) return;
    const float y = 1.f / det;
    const float n1 = det3(r, e2, e3), n2 = det3(e1, r, e3), n3 = det3(e1, e2, r);
    const float n0 = ((det - n1) - n2) - n3;
    const float w = fminf(fminf(n0 * y, n1 * y), fminf(n2 * y, n3 * y));
    const float err = 2.f * E * (4.f + fabsf(w)) * fabsf(y) + 1e-6f * fabsf(w);
    lo = w - err;
    hi = w + err;
}

// U(x) in cell c by one thread: the cell-point interpolation (the restatement
// documented in the oracle), the weights in the first of the cell's tetrahedra
// (centre, fan triangle of a face) that holds x up to -1e-10, else in the one
// with the largest least weight.  The search passes over the tetrahedra that
// cannot hold x by their single precision bounds; if none holds it (cells of
// warped faces), over those that cannot have the largest.
__device__ __forceinline__ d3 interpolateU(const DevMesh& m, int c, d3 x, const double* U, const double* Ub) {
    const d3 a = ld3(m.C, c);
    const d3 r = x - a;
    int bp0 = -1, bp1 = -1, bp2 = -1;
    double bw[4] = {0, 0, 0, 0}, bestMin = -1e300;
    const int k1 = m.cOff[c + 1];
    const F3 aF = leadingF3(a), rF = leadingF3(r);
    const float aM = maxAbs(aF);
    float most = -FLT_MAX;  // a lower bound of the largest least weight
    bool found = false;
    for (int trip = 0; trip < 2 && !found; ++trip) {
        bp0 = -1;
        bestMin = -1e300;
        int k = m.cOff[c], i = 0, n = 0, q0 = 0, g0 = 0;
        F3 f1, f3;
        while (!found) {
            bool candidate = false;  // the next tetrahedron x may be in
            while (true) {
                if (i + 1 >= n) {
                    if (k >= k1) break;
                    const int f = m.cFaces[k++];
                    q0 = m.fOff[f];
                    n = m.fOff[f + 1] - q0;
                    if (n < 3) {
                        n = 0;
                        continue;
                    }
                    i = 1;
                    g0 = m.fPts[q0];
                    f1 = leadingF3(ld3(m.pts, g0));
                    f3 = leadingF3(ld3(m.pts, m.fPts[q0 + 1]));
                }
                const F3 f2 = f3;
                f3 = leadingF3(ld3(m.pts, m.fPts[q0 + i + 1]));
                ++i;
                const float M = fmaxf(fmaxf(aM, maxAbs(f1)), fmaxf(maxAbs(f2), maxAbs(f3)));
                float lo, hi;
                leastWeightBounds(rF, f1 - aF, f2 - aF, f3 - aF, M, lo, hi);
                if (trip == 0) most = fmaxf(most, lo);
                candidate = !(hi < (trip == 0 ? -1e-9f : most));
                if (candidate) break;
            }
            if (!candidate) break;
            const int gi = m.fPts[q0 + i - 1], gj = m.fPts[q0 + i];
            const d3 e1 = ld3(m.pts, g0) - a, e2 = ld3(m.pts, gi) - a, e3 = ld3(m.pts, gj) - a;
            const d3 c23 = cross(e2, e3);
            const double det = dot(e1, c23);
            if (!(fabs(det) > kVSMALL)) continue;
            const d3 w = divBy(mk(dot(r, c23), dot(e1, cross(r, e3)), dot(e1, cross(e2, r))), det);
            const double w0 = ((1.0 - w.x) - w.y) - w.z;
            const double mn = fmin(fmin(w0, w.x), fmin(w.y, w.z));
            found = mn >= -1e-10;
            if (found || mn > bestMin) {
                bestMin = mn;
                bp0 = g0;
                bp1 = gi;
                bp2 = gj;
                bw[0] = w0;
                bw[1] = w.x;
                bw[2] = w.y;
                bw[3] = w.z;
            }
        }
    }
    if (bp0 < 0) return ld3(U, c);
    d3 t = bw[0] * ld3(U, c);
    t = t + bw[1] * pointValue(m, bp0, U, Ub);
    t = t + bw[2] * pointValue(m, bp1, U, Ub);
    t = t + bw[3] * pointValue(m, bp2, U, Ub);
    return t;
}

// (a) Interface speed Un0 = U(interface centre) . n of every cut cell, and
//     the list of its downwind faces (advection.C:131-174: phi >= 0 on an
//     owned face, phi < 0 on a neighboured one; boundary faces phi >= 0).
//
// A thread per cell (interpolateU) is a chain of dependent loads and, with 32
// cells a warp, of one or two tetrahedra at 80 FP64 instructions and the
// points' sums at 144 (all twelve tetrahedra of a hexahedron before the single
// precision bounds).  Lists that leave warps idle give a cell eight lanes, four
// cells a warp:
//   * on its faces, naming the first tetrahedron that may hold x;
//   * on that one's determinant and three numerators, the same triple product
//     with one vector each replaced by x;
//   * on the points' cells (velocity times weight), then on the nine sums over
//     them in order; on the faces again for the list.
// That is 70 to 100 FP64 instructions for four cells: more of the pipe per
// cell, which decides beyond kUn0Group cells per SM.
// Kernel time of the walk in double -> a thread per cell with the bounds ->
// eight lanes: 24^3 hexahedra (331 cells) 66 -> 38 -> 20 us, 33^3 (617) 65 -> 44
// -> 29, 112^3 (6,988) - -> 74 -> 54, 128^3 (30,189) 107 -> 81 -> 104, 256^3
// (35,452) 118 -> 95 -> 128, warped 96^3 (7,146) 67 -> 79 -> 51, refined 24^3
// (755) 201 -> 90 -> 43.  The two lines meet near 100 cells per SM.
constexpr int kUn0Group = 96;
constexpr int kUn0Threads = 128;
__global__ void __launch_bounds__(kUn0Threads) kInterfaceUn0(
    DevMesh m, const int* __restrict__ mixed, const int* __restrict__ nMixed, const int8_t* __restrict__ mStatus,
    const double* __restrict__ nrm, const double* __restrict__ icArr, const double* __restrict__ U,
    const double* __restrict__ Ub, const double* __restrict__ phi, double* __restrict__ un0,
    int2* __restrict__ dwList, int* __restrict__ dwCount, int groupMax) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kNone = INT_MAX;
    __shared__ double prodS[kUn0Threads / 32][4][9][9];  // (row padded) [point, component][cell of the chunk]
    const int lane = threadIdx.x & 31, l = lane & 7, g = lane >> 3, base = lane & 24;
    double(*prod)[9] = prodS[threadIdx.x >> 5][g];
    const int nm = *nMixed;
    if (nm > groupMax) {
        // uniform trip count per warp so the list append can use warp shuffles
        const int stride = spreadStride();
        const int nIter = (nm + stride - 1) / stride;
        for (int it = 0; it < nIter; ++it) {
            const int i = it * stride + spreadFirst();
            int nd = 0, k0 = 0;
            unsigned down = 0;  // bit j: the cell's j-th face (cells() order) is downwind
            if (i < nm && mStatus[i] == 0) {
                const int c = mixed[i];
                un0[i] = dot(interpolateU(m, c, ld3(icArr, i), U, Ub), ld3(nrm, i));
                k0 = m.cOff[c];
                down = downwindFaces(m, c, k0, m.cOff[c + 1], phi);
                nd = __popc(down);
            }
            // warp-aggregated append
            int incl = nd;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            int base = 0;
            if (lane == 31 && total) base = atomicAdd(dwCount, total);
            base = __shfl_sync(0xffffffffu, base, 31);
            int q = base + incl - nd;
            for (unsigned mm = down; mm; mm &= mm - 1u) dwList[q++] = make_int2(i, m.cFaces[k0 + __ffs(mm) - 1]);
        }
        return;
    }
    constexpr int kCells = kUn0Threads / 8;  // of a block
    __shared__ int listS[2];  // entries of the block's cells in the list, where they start
    for (int q = blockIdx.x; q * kCells < nm; q += gridDim.x) {
        const int i = q * kCells + 4 * (threadIdx.x >> 5) + g;
        if (threadIdx.x == 0) listS[0] = 0;
        __syncthreads();
        const bool act = i < nm && mStatus[i] == 0;
        const int c = act ? mixed[i] : 0;
        const int k0 = act ? m.cOff[c] : 0, k1 = act ? m.cOff[c + 1] : 0;
        const d3 a = ld3(m.C, c);
        const d3 x = act ? ld3(icArr, i) : a;
        const F3 aF = leadingF3(a), rF = leadingF3(x - a);
        const float aM = maxAbs(aF);
        const int l3 = l < 3 ? l : 0;  // component l on lanes 0-2
        const double uC = U[size_t(3) * c + l3], nI = act ? nrm[size_t(3) * i + l3] : 0.0;
        // the downwind faces: one addition to the list's length per block,
        // whose answer is read at the end
        const auto downwind = [&](int k) {
            if (k >= k1) return false;
            const int f = m.cFaces[k];
            const long long ph = bitsOf(phi[f]);
            const bool owned = f >= m.nfi || m.own[f] == c;
            return owned ? nonNegBits(ph) : (!nonNegBits(ph) && (ph & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL);
        };
        unsigned down = 0;  // bit j: the lane's j-th face, l + 8 j
        for (int j = 0; k0 + l + 8 * j < k1; ++j) down |= unsigned(downwind(k0 + l + 8 * j)) << j;
        int mine = 0;
        if (down) mine = atomicAdd(&listS[0], __popc(down));
        __syncthreads();
        if (threadIdx.x == 0) listS[1] = listS[0] ? atomicAdd(dwCount, listS[0]) : 0;
        // the tetrahedron
        int bp[3] = {-1, -1, -1};
        double bw[4] = {0, 0, 0, 0}, bestMin = -1e300;
        bool open = act, any = false;  // any: the second trip, for the largest weight
        int from = 0;                  // tetrahedra (16 face + triangle) from here on
        float most = -FLT_MAX;         // a lower bound of the largest least weight
        while (__any_sync(kAll, open)) {
            const float least = any ? most : -1e-9f;
            int cand = kNone;
            float low = -FLT_MAX;
            for (int k = k0 + l; open && k < k1; k += 8) {
                const int f = m.cFaces[k];
                const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
                if (n < 3) continue;
                const F3 f1 = leadingF3(ld3(m.pts, m.fPts[q0]));
                F3 f3 = leadingF3(ld3(m.pts, m.fPts[q0 + 1]));
                for (int t = 1; t + 1 < n; ++t) {
                    const F3 f2 = f3;
                    f3 = leadingF3(ld3(m.pts, m.fPts[q0 + t + 1]));
                    const float M = fmaxf(fmaxf(aM, maxAbs(f1)), fmaxf(maxAbs(f2), maxAbs(f3)));
                    float lo, hi;
                    leastWeightBounds(rF, f1 - aF, f2 - aF, f3 - aF, M, lo, hi);
                    low = fmaxf(low, lo);
                    const int id = 16 * (k - k0) + t;
                    if (id >= from && id < cand && !(hi < least)) cand = id;
                }
            }
            for (int o = 4; o; o >>= 1) {
                cand = min(cand, __shfl_xor_sync(kAll, cand, o));
                low = fmaxf(low, __shfl_xor_sync(kAll, low, o));
            }
            if (open) most = low;
            if (cand == kNone) {  // none (left): the second trip, or the end
                open = open && !any;
                if (open) {
                    any = true;
                    from = 0;
                    bp[0] = -1;
                    bestMin = -1e300;
                }
            }
            const bool eval = cand != kNone;
            int gp[3] = {0, 0, 0};
            if (eval) {
                const int q0 = m.fOff[m.cFaces[k0 + (cand >> 4)]], t = cand & 15;
                gp[0] = m.fPts[q0];
                gp[1] = m.fPts[q0 + t];
                gp[2] = m.fPts[q0 + t + 1];
                from = cand + 1;
            }
            const d3 u = ((l & 3) == 1 ? x : ld3(m.pts, gp[0])) - a, v = ((l & 3) == 2 ? x : ld3(m.pts, gp[1])) - a,
                     w = ((l & 3) == 3 ? x : ld3(m.pts, gp[2])) - a;
            const double tri = dot(u, cross(v, w));
            const double det = __shfl_sync(kAll, tri, base);
            const double quot = tri / det;
            const double w1 = __shfl_sync(kAll, quot, base + 1), w2 = __shfl_sync(kAll, quot, base + 2),
                         w3 = __shfl_sync(kAll, quot, base + 3);
            const double w0 = ((1.0 - w1) - w2) - w3;
            const double mn = fmin(fmin(w0, w1), fmin(w2, w3));
            if (eval && fabs(det) > kVSMALL) {
                open = !(mn >= -1e-10);
                if (!open || mn > bestMin) {
                    bestMin = mn;
                    bp[0] = gp[0];
                    bp[1] = gp[1];
                    bp[2] = gp[2];
                    bw[0] = w0;
                    bw[1] = w1;
                    bw[2] = w2;
                    bw[3] = w3;
                }
            }
        }
        // the values at its points: sum k = 3 point + component on lane k, the
        // ninth on lane 0 too
        const bool tet = act && bp[0] >= 0;
        int at[3], end[3];
        bool boundary[3];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const int pt = tet ? bp[p] : 0;
            const int b0 = m.pbOff[pt], b1 = m.pbOff[pt + 1], c0 = m.pcOff[pt], c1 = m.pcOff[pt + 1];
            boundary[p] = b1 > b0;
            at[p] = boundary[p] ? b0 : c0;
            end[p] = tet ? (boundary[p] ? b1 : c1) : at[p];
        }
        double sum = 0.0, sum8 = 0.0;
        while (__any_sync(kAll, at[0] < end[0] || at[1] < end[1] || at[2] < end[2])) {
            int id[3];
            double wt[3];
            bool in[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const int k = at[p] + l;
                in[p] = k < end[p];
                id[p] = in[p] ? (boundary[p] ? m.pbFaces : m.pCells)[k] : 0;
                wt[p] = in[p] ? (boundary[p] ? m.pbW : m.pcW)[k] : 0.0;
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const double* row = U;
                if (in[p]) {
                    if (!boundary[p]) row = U + size_t(3) * id[p];
                    else row = Ub ? Ub + size_t(3) * (id[p] - m.nfi) : U + size_t(3) * m.own[id[p]];
                }
                prod[3 * p][l] = wt[p] * row[0];
                prod[3 * p + 1][l] = wt[p] * row[1];
                prod[3 * p + 2][l] = wt[p] * row[2];
            }
            __syncwarp();
            const int n01 = (l < 3 ? end[0] - at[0] : (l < 6 ? end[1] - at[1] : end[2] - at[2]));
            const int n8 = l == 0 ? end[2] - at[2] : 0;
            for (int j = 0; j < 8; ++j) {
                if (j < n01) sum = sum + prod[l][j];
                if (j < n8) sum8 = sum8 + prod[8][j];
            }
            __syncwarp();
#pragma unroll
            for (int p = 0; p < 3; ++p) at[p] = min(at[p] + 8, end[p]);
        }
        // U(x) by components, and its part of Un0
        double t = uC;
        const double v0 = __shfl_sync(kAll, sum, base + l3), v1 = __shfl_sync(kAll, sum, base + 3 + l3);
        double v2 = __shfl_sync(kAll, sum, base + 6 + (l3 & 1));
        const double v8 = __shfl_sync(kAll, sum8, base);
        if (l3 == 2) v2 = v8;
        if (tet) t = ((bw[0] * t + bw[1] * v0) + bw[2] * v1) + bw[3] * v2;
        const double part = t * nI;
        const double px = __shfl_sync(kAll, part, base), py = __shfl_sync(kAll, part, base + 1),
                     pz = __shfl_sync(kAll, part, base + 2);
        if (act && l == 0) un0[i] = (px + py) + pz;
        __syncthreads();
        int dst = listS[1] + mine;
        for (unsigned mm = down; mm; mm &= mm - 1u)
            dwList[dst++] = make_int2(i, m.cFaces[k0 + l + 8 * (__ffs(mm) - 1)]);
        __syncthreads();
    }
}

// (b) Simpson flux through the downwind faces of cut cells
//     (cutFace::timeIntegratedFaceFlux, cutFace.C:262-389): eight faces a
//     warp (face_group.cuh).  On a mesh with warped faces two: such a face is
//     a fan of triangles about its centre, four at a time (a flat face there
//     takes the first of its four polygons).  One GB300, kernel time with a
//     thread per face -> eight lanes per face -> eight faces a warp with their
//     areas dealt out: 24^3 0.077 -> 0.016 -> 0.016 ms, 128^3 (30,000 interface
//     cells) 0.264 -> 0.233 -> 0.127, 256^3 (35,000) 0.364 -> 0.276 -> 0.152,
//     warped 96^3 0.243 -> 0.286 -> 0.183, refined 24^3 0.105 -> 0.027.
constexpr int kFaceThreads = 64;
template <bool WARPED>
__global__ void __launch_bounds__(kFaceThreads) kInterfaceFaces(DevMesh m, const int2* __restrict__ dwList,
                                                       const int* __restrict__ dwCount,
                                                       const double* __restrict__ nrm, const double* __restrict__ dArr,
                                                       const double* __restrict__ un0, const double* __restrict__ phi,
                                                       double dt, double* __restrict__ dvfI,
                                                       uint8_t* __restrict__ cutMask) {
    __shared__ FaceShared shared[kFaceThreads / 32];
    FaceShared& s = shared[threadIdx.x >> 5];
    constexpr int kPer = WARPED ? 2 : kPolys;  // faces of a warp
    constexpr int kSlots = kPolys / kPer;      // polygons of a face at a time
    const int nItems = *dwCount;
    const int lane = threadIdx.x & 31, g = lane / kPolyLanes, l = lane % kPolyLanes;
    const int face = g / kSlots, slot = g % kSlots;
    const int warps = gridDim.x * (kFaceThreads / 32);
    for (int q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; q * kPer < nItems; q += warps) {
        const int item = q * kPer + face;
        const bool act = item < nItems;
        const int2 it = act ? dwList[item] : make_int2(0, 0);
        const int i = it.x, f = it.y;
        const double ph = phi[f], magSf = m.magSf[f], distance = dArr[i], Un0 = un0[i];
        const d3 n3 = ld3(nrm, i);
        const bool some = act && absOf(ph) > kTSMALL;
        const bool moving = fabs(Un0 * dt) > kTSMALL;
        const bool flat = !WARPED || m.flat[f] > (1.0 - kTSMALL);
        const double rUn0 = 1.0 / Un0;  // the arrival times share the divisor
        const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
        double dVf = 0.0;
        // the rounds of the warp: one, or the triangles of its warped faces
        const int mine = some ? (flat ? 1 : (n + kSlots - 1) / kSlots) : 0;
        const int rounds = WARPED ? __reduce_max_sync(0xffffffffu, mine) : 1;
        for (int r = 0; r < rounds; ++r) {
            const int t = r * kSlots + slot;  // the polygon's triangle
            const bool on = some && r < mine && (flat ? slot == 0 : t < n);
            const int np = !on ? 0 : (flat ? n : 3);
            double magP = magSf;
            unsigned code = 3;
            __syncwarp();
            if (on) {
                if (flat) {
                    code = m.faceAxis[f];
                    // |face::areaNormal| of the whole face
                    const d3 A = ld3(m.fullA, f);
                    const int ax = code & 3;
                    const double Ax = ax == 0 ? A.x : (ax == 1 ? A.y : A.z);
                    const int e = int((bitsOf(Ax) >> 52) & 0x7ff);
                    s.fullMag[g] = ((code & 8) && ax != 3 && e > 543 && e < 1503) ? absOf(Ax) : mag(A);
                } else {
                    const d3 cf = ld3(m.Cf, f), p1 = ld3(m.pts, m.fPts[q0 + t]),
                             p2 = ld3(m.pts, m.fPts[q0 + (t + 1 < n ? t + 1 : 0)]);
                    magP = mag(0.5 * cross(p1 - cf, p2 - cf));
                    s.fullMag[g] = magP;
                }
                for (int k = l; k < np; k += kPolyLanes) {
                    d3 p;
                    if (flat) p = ld3(m.pts, m.fPts[q0 + k]);
                    else if (k == 0) p = ld3(m.Cf, f);
                    else p = ld3(m.pts, m.fPts[q0 + (t + k - 1 < n ? t + k - 1 : 0)]);
                    s.P[g][k][0] = p.x;
                    s.P[g][k][1] = p.y;
                    s.P[g][k][2] = p.z;
                    s.pd[g][k] = dot(p, n3);
                }
                if (l == 0) {
                    s.distance[g] = distance;
                    s.Un0[g] = Un0;
                    s.code[g] = np | int(code << 8);
                }
            }
            __syncwarp();
            const double v = polyTimeArea(s, lane, np, moving, distance, Un0, rUn0, dt, magP);
            if (!on) continue;
            if (flat) {
                dVf = moving ? ph / magSf * v : ph * dt * (v / magSf);
            } else if (l == 0) {
                // phi split by area
                const double phiTri = ph * magP / magSf;
                s.sum[WARPED ? face : 0][t] = moving ? phiTri / magP * v : phiTri * dt * (v / magP);
            }
        }
        if (WARPED) {
            __syncwarp();
            if (some && !flat)
                for (int t = 0; t < n; ++t) dVf += s.sum[WARPED ? face : 0][t];
        }
        if (act && l == 0 && slot == 0) {
            dvfI[f] = dVf;
            if (cutMask) cutMask[f] = 1;
        }
    }
}

// ---------------------------------------------------------------------------
// K5: upwind flux, interface overrides, surfaceIntegrate and alpha update
// ---------------------------------------------------------------------------
struct UpdateArgs {
    const double* phi;
    const double* aCur;
    const double* aOld;
    double* aNew;
    const int8_t* status;
    const double* dvfI;
    const double* alphaB;
    const double* Sp;
    const double* Su;
    double dt, rDeltaT, rrDeltaT;
    double* alphaPhi;
    int* ovList;
    int* ovCount;
    int ovCap;
};

// dVf of face f of cell c (own: c owns it; nb: the cell across, -1 on the
// boundary; ac, stC: c's alpha and status) and, for an owned face, dVf / dt
// in q: the Simpson value when the upwind cell is cut, else the upwind flux.
__device__ __forceinline__ double faceDVf(const DevMesh& m, const UpdateArgs& u, int f, bool own, int nb, double ac,
                                          int8_t stC, double& q) {
    const double ph = u.phi[f];
    const bool pos = nonNegBits(bitsOf(ph));
    double af;
    bool cut;
    if (nb >= 0) {
        const double ax = u.aCur[nb];
        cut = (pos == own ? stC : u.status[nb]) == 0;
        af = cut ? 0.0 : upwindAlpha(ph, own ? ac : ax, own ? ax : ac);
    } else {
        cut = pos && stC == 0;
        af = u.alphaB ? u.alphaB[f - m.nfi] : ac;
    }
    if (cut) {
        const double dv = u.dvfI[f];
        q = own ? divByRecip(dv, u.dt, u.rDeltaT) : 0.0;
        return dv;
    }
    return fluxDtQuot(ph, af, u.dt, u.rDeltaT, q);
}

// The update of one cell.  What bounds it: in the first steps of a run, when
// most cells and their neighbours hold exact zeros, the loads' latency and
// HBM (64 B of traffic per cell); later, when almost every cell holds a small
// remainder, the arithmetic of six upwind fluxes per cell, for which the
// FP64 pipe (16 cycles per warp instruction) is the narrow one.  So:
//   * an empty neighbourhood issues no FP64 at all (below);
//   * the products of the fluxes and alphaPhi are formed on the integer pipe
//     (fluxDtQuot), the FP64 pipe is left the sums, the upwind differences
//     that are not settled on the bits, and the divisions by V and 1/dt;
//   * TILE: on a lattice mesh a block is a tile of TX x TY x TZ cells and
//     each flux inside the tile is formed once, by its owner, and read by the
//     cell across from shared memory; the fluxes through the tile's low sides
//     are one more flux for two thirds of the threads (3.6 fluxes per cell
//     instead of 6).
// An empty cell's three fluxes, for the cells across, are zeros, or NaN where
// phi is not finite.  HANDED: alpha was handed over again after the interface
// was found, so an empty cell or its neighbour may have been cut then: the
// fluxes downwind of a cut cell are its Simpson values all the same (apart
// because the reads of status take the spread case below from 1.00 to 1.06 ms).
// Other meshes take one thread per cell in cell order (TX = TY = TZ = 0).
// One GB300, before -> now: 128^3 in the middle of the deformation run 0.222 ->
// 0.160 ms, 256^3 with alpha spread over the mesh 2.05 -> 1.01 ms (0.28 -> 0.24
// ms in its first steps); 45^3 x 6 tetrahedra (no lattice) 0.048 -> 0.039 ms.
// In that 128^3 step the FP64 pipe is 55% busy, the ALU pipe 61%, the issue
// slots 58%.  Other tiles, 128^3 and spread 256^3 (0.156 and 1.07 ms then): 8 x
// 8 x 4 0.168 and 1.14, 16 x 4 x 4 0.174 and 1.24, 32 x 4 x 2 0.192 and 1.50
// (more sides, or more warps at a barrier); 8 or 12 blocks of 128 per SM
// instead of 10 lose 0.04 ms in the first steps.
template <int TX, int TY, int TZ>
struct UpdateBlock {
    static constexpr int kThreads = TX ? TX * TY * TZ : 256;
};
template <int TX, int TY, int TZ, bool HANDED>
__global__ void __launch_bounds__((UpdateBlock<TX, TY, TZ>::kThreads), (1280 / UpdateBlock<TX, TY, TZ>::kThreads))
    kUpdate(DevMesh m, UpdateArgs u) {
    constexpr bool kTile = TX > 0;
    constexpr int kThreads = UpdateBlock<TX, TY, TZ>::kThreads;
    constexpr int kHz = TX * TY, kHy = TX * TZ, kHx = TY * TZ;  // faces on the tile's low sides
    constexpr int kDx = kTile ? TX : 1, kDy = kTile ? TY : 1;    // (divisors)
    __shared__ double sDv[kTile ? 3 : 1][kTile ? kThreads : 1];  // dVf of each cell's +x, +y, +z face
    __shared__ double sLow[kTile ? kHz + kHy + kHx : 1];         // dVf through the low sides: z, y, x
    __shared__ uint8_t sWork[kTile ? kThreads : 1];              // an interior cell on the arithmetic path
    const int tid = threadIdx.x;
    int c, li = 0, lj = 0, lk = 0, i = 0, j = 0, k = 0;
    bool valid;
    if (kTile) {
        li = tid % kDx;
        lj = tid / kDx % kDy;
        lk = tid / (kDx * kDy);
        i = blockIdx.x * TX + li;
        j = blockIdx.y * TY + lj;
        k = blockIdx.z * TZ + lk;
        valid = i < m.latNx && j < m.latNy && k < m.latNz;
        c = i + m.latNx * (j + m.latNy * k);
    } else {
        c = blockIdx.x * blockDim.x + tid;
        valid = c < m.nc;
    }
    bool ov = false, inSet = false;
    bool work = false, interior = false;
    int k0 = 0, k1 = 0;  // slots in memory; an interior lattice cell: k0 its latticeBase
    double ao = 0.0, ac = 0.0;
    const auto highSide = [&](int nb) { return nb == c + 1 ? 0 : (nb == c + m.latNx ? 1 : 2); };  // an owned face's axis
    if (valid) {
        // The face-slot records: from the lattice formula for the interior
        // cells of a lattice mesh (no addressing read), else the first
        // kBatch from memory, loaded together so they are in flight at once;
        // slots of larger cells follow one by one from k0 + kBatch.  Unused
        // slots hold x = -2.
        constexpr int kBatch = 6;
        int2 sl[kBatch];
        interior = kTile && latticeSlotsAt(c, i, j, k, i + m.latNx * j, m.latNx, m.latNy, m.latNz, sl);
        if (interior) {
            k0 = sl[3].y;
        } else {
            k0 = m.uniformFaces ? c * m.uniformFaces : m.cOff[c];
            k1 = m.uniformFaces ? k0 + m.uniformFaces : m.cOff[c + 1];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) sl[q] = (k0 + q < k1) ? m.cSlot[k0 + q] : make_int2(-2, 0);
        }
        // Every load the common case needs is issued before any is used, so
        // a cell costs one memory round trip: the alpha across each slot
        // (alpha_b on a boundary face when given), phi of the owned faces,
        // the cell's old and current alpha.
        double ax[kBatch];
        double pv[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            ax[q] = 0.0;
            if (sl[q].x >= 0)
                ax[q] = u.aCur[sl[q].x];
            else if (sl[q].x == -1 && u.alphaB)
                ax[q] = u.alphaB[(sl[q].y & 0x7fffffff) - m.nfi];
            pv[q] = (sl[q].x != -2 && sl[q].y >= 0) ? u.phi[sl[q].y] : 0.0;
        }
        ao = u.aOld[c];
        ac = u.aCur[c];
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
            if (sl[q].x == -1 && !u.alphaB) ax[q] = ac;  // zero-gradient boundary value
        // Empty neighbourhood: every dVf is a signed zero, surfaceIntegrate
        // gives +0 and ((ao*r) - 0*r)/r returns ao itself (bit for bit), and
        // alphaPhi = dVf/dt is a zero with the sign of phi.  The zero tests
        // and the sign are integer operations on the bit patterns, so empty
        // cells issue no FP64 instruction.
        const auto isZero = [](double x) { return (bitsOf(x) << 1) == 0; };
        const long long kSign = (long long)0x8000000000000000ULL;
        bool quick = (u.Sp == nullptr) && (u.Su == nullptr) && isZero(ao) && isZero(ac);
        if (quick) {
#pragma unroll
            for (int q = 0; q < kBatch; ++q) quick = quick && isZero(ax[q]);
            for (int q = k0 + kBatch; quick && q < k1; ++q) {
                const int2 s = m.cSlot[q];
                const double x = (s.x >= 0) ? u.aCur[s.x] : (u.alphaB ? u.alphaB[(s.y & 0x7fffffff) - m.nfi] : ac);
                quick = isZero(x);
            }
        }
        if (quick) {
            u.aNew[c] = ao;
            // owned faces only (the owner writes each face); an internal face's
            // alpha_f is +0, a boundary face's zero also carries alpha_b's sign
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                if (sl[q].x == -2 || sl[q].y < 0) continue;
                long long sgnBits = bitsOf(pv[q]) & kSign;
                if (sl[q].x == -1) sgnBits ^= bitsOf(ax[q]) & kSign;
                u.alphaPhi[sl[q].y] = __longlong_as_double(sgnBits);
            }
            for (int q = k0 + kBatch; q < k1; ++q) {
                const int2 s = m.cSlot[q];
                if (s.y < 0) continue;
                long long sgnBits = bitsOf(u.phi[s.y]) & kSign;
                if (s.x < 0) sgnBits ^= bitsOf(u.alphaB ? u.alphaB[s.y - m.nfi] : ac) & kSign;
                u.alphaPhi[s.y] = __longlong_as_double(sgnBits);
            }
        }
        work = !quick;
    }
    double sum = 0.0;  // surfaceIntegrate in ascending face order
    int8_t stC = 0;
    if (work) stC = u.status[c];
    if (kTile) {
        sWork[tid] = interior && work;
        if (!__syncthreads_or(work)) return;
        // each interior cell's +x, +y, +z fluxes, and an empty cell's
        if (interior && work) {
#pragma unroll 1
            for (int d = 0; d < 3; ++d) {
                double q;
                const int f = k0 + d;
                sDv[d][tid] = faceDVf(m, u, f, true, c + m.latNb[3 + d], ac, stC, q);
                u.alphaPhi[f] = q;
            }
        } else if (!work) {
            const auto empty = [&](int f) {  // phi 0
                const bool finite = (bitsOf(u.phi[f]) & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
                return __longlong_as_double(finite ? 0LL : 0x7fffffffffffffffLL);
            };
            if (interior) {
#pragma unroll
                for (int d = 0; d < 3; ++d) sDv[d][tid] = empty(k0 + d);
            }
#pragma unroll 1
            for (int q = k0; q < k1; ++q) {  // (a boundary cell)
                const int2 s = m.cSlot[q];
                if (s.x >= 0 && s.y >= 0) sDv[highSide(s.x)][tid] = empty(s.y);
            }
            if (HANDED && valid) {
                stC = u.status[c];
#pragma unroll 1
                for (int q = 6 * c; q < 6 * c + 6; ++q) {
                    const int2 s = m.cSlot[q];
                    if (s.x < 0 || s.y < 0) continue;
                    if ((nonNegBits(bitsOf(u.phi[s.y])) ? stC : u.status[s.x]) == 0) sDv[highSide(s.x)][tid] = u.dvfI[s.y];
                }
            }
        }
        // the fluxes through the tile's low sides, a thread each
        if (tid < kHz + kHy + kHx) {
            int src, slot;  // the cell of the tile and the slot of its face
            if (tid < kHz) {
                src = tid;
                slot = 0;
            } else if (tid < kHz + kHy) {
                const int t = tid - kHz;
                src = t % kDx + t / kDx * (TX * TY);
                slot = 1;
            } else {
                src = (tid - kHz - kHy) * TX;
                slot = 2;
            }
            if (sWork[src]) {
                const int ci = blockIdx.x * TX + src % kDx, cj = blockIdx.y * TY + src / kDx % kDy,
                          ck = blockIdx.z * TZ + src / (kDx * kDy);
                const int cc = ci + m.latNx * (cj + m.latNy * ck);
                const int f = latticeBase(cc, ci, cj, ck, ci + m.latNx * cj, m.latNx, m.latNy) + m.latFace[slot];
                double q;
                sLow[tid] = faceDVf(m, u, f, false, cc + m.latNb[slot], u.aCur[cc], u.status[cc], q);
            }
        }
    }
    if (work && !interior) {
#pragma unroll 1
        for (int q = k0; q < k1; ++q) {
            const int2 s = m.cSlot[q];
            const bool own = s.y >= 0;
            const int f = s.y & 0x7fffffff;
            double ap;
            const double dv = faceDVf(m, u, f, own, s.x, ac, stC, ap);
            if (own) {
                u.alphaPhi[f] = ap;
                sum += dv;
                if (kTile && s.x >= 0) sDv[highSide(s.x)][tid] = dv;
            } else {
                sum -= dv;
            }
        }
    }
    if (kTile) {
        __syncthreads();
        if (work && interior) {
            sum -= lk == 0 ? sLow[li + TX * lj] : sDv[2][tid - TX * TY];
            sum -= lj == 0 ? sLow[kHz + li + TX * lk] : sDv[1][tid - TX];
            sum -= li == 0 ? sLow[kHz + kHy + lj + TY * lk] : sDv[0][tid - 1];
            sum += sDv[0][tid];
            sum += sDv[1][tid];
            sum += sDv[2][tid];
        }
    }
    if (work) {
        // the divisions through correctly rounded reciprocals (1/V per
        // cell, 1/dt and 1/(1/dt) per step): the same quotients.  One on
        // integers, one on the FP64 pipe: with alpha spread over 256^3 1.07 ->
        // 1.00 ms (both on integers 0.99), 128^3 0.156 -> 0.157 (0.160).
        const double ivf = divByRecip(sum, m.V[c], m.rV[c]);
        double num = ao * u.rDeltaT;
        if (u.Su) num = num + u.Su[c];
        num = num - ivf * u.rDeltaT;
        const double an = u.Sp ? num / (u.rDeltaT - u.Sp[c]) : divByRecip<false>(num, u.rDeltaT, u.rrDeltaT);
        u.aNew[c] = an;
        // cells outside [-aTol, 1 + aTol] are the bounding candidates; the
        // count of them decides limitFlux's loop (advectionTemplates.C:146)
        // (on the bits: an < -aTol or an > 1 + aTol, NaN neither)
        const double aTol = 100.0 * kSMALL;
        const long long ba = bitsOf(an);
        const long long mag = ba & 0x7fffffffffffffffLL;
        ov = mag <= 0x7ff0000000000000LL && (ba < 0 ? mag > bitsOf(aTol) : ba > bitsOf(1.0 + aTol));
        // only cells of the bounding set (mixed cells and their face
        // neighbours, advection.C:54-82) are listed; every overshooting
        // cell is counted
        if (ov) {
            inSet = stC != kStNotMixed;
            const int nf = interior ? 6 : k1 - k0;
            for (int q = 0; q < nf && !inSet; ++q) {
                const int nb = interior ? c + m.latNb[q] : m.cSlot[k0 + q].x;
                inSet = nb >= 0 && u.status[nb] != kStNotMixed;
            }
        }
    }
    const unsigned ball = __ballot_sync(0xffffffffu, ov);
    if (ball) {
        const int lane = threadIdx.x & 31;
        if (lane == 0) atomicAdd(u.ovCount, __popc(ball));  // [0] all overshooting cells
        const unsigned sball = __ballot_sync(0xffffffffu, inSet);
        int base = 0;
        if (lane == 0 && sball) base = atomicAdd(u.ovCount + 1, __popc(sball));  // [1] listed cells
        base = __shfl_sync(0xffffffffu, base, 0);
        const int p = base + __popc(sball & ((1u << lane) - 1u));
        if (inSet && p < u.ovCap) u.ovList[p] = c;
    }
}

// ---------------------------------------------------------------------------
// K7: snapping and clipping
// ---------------------------------------------------------------------------
__global__ void kBruteForce(int nc, double* __restrict__ a, double snap, int clip) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    double x = a[c];
    if (snap > 0.0) x = x * pos0(x - snap) * neg0(x - (1.0 - snap)) + pos0(x - (1.0 - snap));
    if (clip) x = fmin(1.0, fmax(0.0, x));
    a[c] = x;
}

// ---------------------------------------------------------------------------
// face flatness (one-time, reconstruction.C:408-440)
// ---------------------------------------------------------------------------
__global__ void kFaceFlatness(DevMesh m, const double* __restrict__ Sf, double* __restrict__ flat) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= m.nf) return;
    const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
    const double magA = mag(ld3(Sf, f));
    double out = 1.0;
    if (n > 3 && magA > kROOTVSMALL) {
        const d3 fc = ld3(m.Cf, f);
        double sumA = 0.0;
        for (int i = 0; i < n; ++i) {
            const d3 th = ld3(m.pts, m.fPts[q0 + i]);
            const d3 nx = ld3(m.pts, m.fPts[q0 + (i + 1) % n]);
            sumA += mag(0.5 * cross(nx - th, fc - th));
        }
        out = magA / (sumA + kROOTVSMALL);
    }
    flat[f] = out;
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// A grid of exactly the blocks that are resident at once on all SMs (the
// occupancy of `kernel` at `threads` per block), looked up once per kernel
// and device.
template <class Kernel>
static int residentGrid(Kernel kernel, int threads) {
    struct Entry {
        const void* fn;
        int dev, threads, grid;
    };
    constexpr int kSlots = 32;
    static Entry cache[kSlots] = {};
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    const void* fn = reinterpret_cast<const void*>(kernel);
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < kSlots && cache[i].fn; ++i)
        if (cache[i].fn == fn && cache[i].dev == dev && cache[i].threads == threads) return cache[i].grid;
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0);
    const int g = (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
    for (int i = 0; i < kSlots; ++i)
        if (!cache[i].fn) {
            cache[i] = {fn, dev, threads, g};
            break;
        }
    return g;
}

void launchScanMixed(const StepArgs& a, cudaStream_t st) {
    const int nb = ((a.m.nc + 3) / 4 + 255) / 256;
    const double omt = 1.0 - a.mixedTol;
    long long tolBits, omtBits;
    std::memcpy(&tolBits, &a.mixedTol, sizeof(double));
    std::memcpy(&omtBits, &omt, sizeof(double));
    kScanMixed<<<nb, 256, 0, st>>>(a.m.nc, a.aCur, tolBits, omtBits, a.status, a.mixed, a.nMixed, a.err);
}

void launchLsNormal(const StepArgs& a, cudaStream_t st) {
    kLsNormal<<<residentGrid(kLsNormal, 128), 128, 0, st>>>(a.m, a.aCur, a.mixed, a.nMixed, a.nrm,
                                                            kLsGroup * smCount(), a.err);
}

void launchInterfaceUn0(const StepArgs& a, cudaStream_t st) {
    kInterfaceUn0<<<residentGrid(kInterfaceUn0, kUn0Threads), kUn0Threads, 0, st>>>(
        a.m, a.mixed, a.nMixed, a.mStatus, a.nrm, a.icArr, a.U, a.Ub, a.phi, a.un0, a.dwList, a.dwCount,
        kUn0Group * smCount());
}

template <bool WARPED>
static void launchFaces(const StepArgs& a, cudaStream_t st) {
    kInterfaceFaces<WARPED><<<residentGrid(kInterfaceFaces<WARPED>, kFaceThreads), kFaceThreads, 0, st>>>(
        a.m, a.dwList, a.dwCount, a.nrm, a.dArr, a.un0, a.phi, a.dt, a.dvfI, a.cutMask);
}

void launchInterfaceFaces(const StepArgs& a, cudaStream_t st) {
    if (a.m.warped) launchFaces<true>(a, st);
    else launchFaces<false>(a, st);
}

template <int TX, int TY, int TZ>
static void launchUpdateTiles(const StepArgs& a, const UpdateArgs& u, cudaStream_t st) {
    constexpr int kThreads = TX * TY * TZ;
    static_assert(TX * TY + TX * TZ + TY * TZ <= kThreads, "at most one low side per thread");
    const dim3 grid((a.m.latNx + TX - 1) / TX, (a.m.latNy + TY - 1) / TY, (a.m.latNz + TZ - 1) / TZ);
    if (a.handed) kUpdate<TX, TY, TZ, true><<<grid, kThreads, 0, st>>>(a.m, u);
    else kUpdate<TX, TY, TZ, false><<<grid, kThreads, 0, st>>>(a.m, u);
}

void launchUpdate(const StepArgs& a, cudaStream_t st) {
    const UpdateArgs u{a.phi, a.aCur, a.aOld, a.aNew, a.status, a.dvfI, a.alphaB, a.Sp, a.Su, a.dt, a.rDeltaT,
                       a.rrDeltaT, a.alphaPhi, a.ovList, a.ovCount, a.ovCap};
    // every lattice whose tiles fit a grid (the other two dimensions of a
    // grid end at 65,535)
    if (a.m.latNx && (a.m.latNy + 3) / 4 <= 65535 && (a.m.latNz + 3) / 4 <= 65535) {
        launchUpdateTiles<8, 4, 4>(a, u, st);
        return;
    }
    kUpdate<0, 0, 0, false><<<(a.m.nc + 255) / 256, 256, 0, st>>>(a.m, u);
}

void launchBruteForce(const StepArgs& a, cudaStream_t st) {
    if (!(a.snapTol > 0.0) && !a.clip) return;
    const int nb = (a.m.nc + 255) / 256;
    kBruteForce<<<nb, 256, 0, st>>>(a.m.nc, a.aNew, a.snapTol, a.clip);
}

void launchFaceFlatness(const DevMesh& m, const double* Sf, double* flat, cudaStream_t st) {
    kFaceFlatness<<<(m.nf + 255) / 256, 256, 0, st>>>(m, Sf, flat);
}

// face::centre and face::areaNormal of every face (one-time): what
// calcSubFace returns for a fully submerged face (cutFace.C:184-185)
__global__ void kFaceFull(DevMesh m, double* __restrict__ fullC, double* __restrict__ fullA,
                          uint8_t* __restrict__ faceAxis, int* __restrict__ warped) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= m.nf) return;
    const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
    d3 fp[kMaxFacePts];
    for (int i = 0; i < n; ++i) fp[i] = ld3(m.pts, m.fPts[q0 + i]);
    st3(fullC, f, faceCentreOF(fp, n));
    const d3 A = faceAreaNormalOF(fp, n);
    st3(fullA, f, A);
    faceAxis[f] = faceAxisCode(fp, n, A);
    if (!(m.flat[f] > (1.0 - kTSMALL))) *warped = 1;
}

// 1/V of every cell (correctly rounded; the divisor reciprocals of divByRecip)
__global__ void kRecipVolume(int nc, const double* __restrict__ V, double* __restrict__ rV) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < nc) rV[c] = 1.0 / V[c];
}

void launchRecipVolume(const DevMesh& m, double* rV, cudaStream_t st) {
    kRecipVolume<<<(m.nc + 255) / 256, 256, 0, st>>>(m.nc, m.V, rV);
}

void launchFaceFull(const DevMesh& m, double* fullC, double* fullA, uint8_t* faceAxis, int* warped, cudaStream_t st) {
    kFaceFull<<<(m.nf + 255) / 256, 256, 0, st>>>(m, fullC, fullA, faceAxis, warped);
}

// LS stencils of all cells, once per mesh: row lengths (count = true), then
// the rows (count = false).  An overflowing row gets kMaxStencil entries and
// a -1 (the readers report the overflow when they use the row).
__global__ void __launch_bounds__(128) kStencilRows(DevMesh m, bool count, int* __restrict__ len,
                                                    const int* __restrict__ off, int* __restrict__ rows) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < m.nc; c += gridDim.x * blockDim.x) {
        int st[kMaxStencil];
        uint32_t err = 0;
        const int n = buildStencil(m, c, st, err);
        if (count) {
            len[c] = err ? n + 1 : n;
        } else {
            int* row = rows + off[c];
            for (int k = 0; k < n; ++k) row[k] = st[k];
            if (err) row[n] = -1;
        }
    }
}

void launchStencilRows(const DevMesh& m, bool count, int* len, const int* off, int* rows, cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    kStencilRows<<<sms * 16, 128, 0, st>>>(m, count, len, off, rows);
}

}  // namespace simplic
