// Plain-form (FP64, bit-exact) geometry of the SimPLIC step, device side.
//
// Restates, per thread:
//   cutFace::calcSubFace / calcSubFaceCentreAndArea   cutFace.C:37-96, 136-259
//   cutCell::calcSubCell and helpers                  cutCell.C:37-137, 343-542
// with the same floating-point operation order as the reference, so that a
// translation unit built with -fmad=false reproduces the CPU results bit for
// bit.  Work that does not change any result is skipped (sub-cell centres
// that only feed output, face areas of fully submerged faces that depend on
// the face alone and are computed once per cell).
#pragma once

#include "int_math.cuh"
#include "simplic_device.cuh"

namespace simplic {

// v / s for the three components: one division for 1/s, then the
// correctly rounded quotients through it (divByRecip), the same results.
template <bool INTS = true>
__device__ __forceinline__ d3 divBy(d3 v, double s) {
    const double y = 1.0 / s;
    return mk(divByRecip<INTS>(v.x, s, y), divByRecip<INTS>(v.y, s, y), divByRecip<INTS>(v.z, s, y));
}

// OpenFOAM face::centre (triangle direct; otherwise area-weighted fan about
// the point average, centre via sumAc / (3 sumA)).
__device__ __forceinline__ d3 faceCentreOF(const d3* p, int n) {
    if (n == 3) return (1.0 / 3.0) * ((p[0] + p[1]) + p[2]);
    d3 cp = p[0];
    for (int i = 1; i < n; ++i) cp = cp + p[i];
    cp = divCount(cp, n);
    double sumA = 0.0;
    d3 sumAc = mk(0, 0, 0);
    for (int i = 0; i < n; ++i) {
        const d3 nx = p[(i + 1) % n];
        const d3 ttc = (p[i] + nx) + cp;
        const double ta = mag(cross(p[i] - cp, nx - cp));
        sumA += ta;
        sumAc = sumAc + ta * ttc;
    }
    if (sumA > kVSMALL) return sumAc / (3.0 * sumA);
    return cp;
}

// OpenFOAM face::areaNormal (sum of 0.5 (b-a)^(c-a) over (p_i, p_i+1, centre)).
__device__ __forceinline__ d3 faceAreaNormalOF(const d3* p, int n) {
    if (n == 3) return 0.5 * cross(p[1] - p[0], p[2] - p[0]);
    d3 cp = p[0];
    for (int i = 1; i < n; ++i) cp = cp + p[i];
    cp = divCount(cp, n);
    d3 nrm = mk(0, 0, 0);
    for (int i = 0; i < n; ++i) {
        const d3 nx = (i < n - 1) ? p[i + 1] : p[0];
        nrm = nrm + 0.5 * cross(nx - p[i], cp - p[i]);
    }
    return nrm;
}

// calcSubFaceCentreAndArea (cutFace.C:37-96): centre and area of a polygon.
__device__ __forceinline__ void fanCentreArea(const d3* p, int n, d3& cen, d3& area) {
    if (n == 3) {
        cen = (1.0 / 3.0) * ((p[0] + p[1]) + p[2]);
        area = 0.5 * cross(p[1] - p[0], p[2] - p[0]);
        return;
    }
    d3 fc = p[0];
    for (int i = 1; i < n; ++i) fc = fc + p[i];
    fc = divCount(fc, n);
    d3 sumN = mk(0, 0, 0), sumAc = mk(0, 0, 0);
    double sumA = 0.0;
    for (int i = 0; i < n; ++i) {
        const d3 nx = p[(i + 1) % n];
        const d3 c = (p[i] + nx) + fc;
        const d3 nv = cross(nx - p[i], fc - p[i]);
        const double a = mag(nv);
        sumN = sumN + nv;
        sumA += a;
        sumAc = sumAc + a * c;
    }
    if (sumA < kROOTVSMALL) {
        cen = fc;
        area = mk(0, 0, 0);
    } else {
        cen = divBy((1.0 / 3.0) * sumAc, sumA);
        area = 0.5 * sumN;
    }
}

// Area vector only.  sumA < ROOTVSMALL is decided without the square roots
// when any fan triangle has |n|^2 >= 1e-299 (then sumA >= 1e-150 for sure);
// otherwise sumA is summed exactly as the reference does.
__device__ __forceinline__ d3 fanArea(const d3* p, int n) {
    if (n == 3) return 0.5 * cross(p[1] - p[0], p[2] - p[0]);
    d3 fc = p[0];
    for (int i = 1; i < n; ++i) fc = fc + p[i];
    fc = divCount(fc, n);
    d3 sumN = mk(0, 0, 0);
    double s2max = 0.0;
    for (int i = 0; i < n; ++i) {
        const d3 nx = p[(i + 1) % n];
        const d3 nv = cross(nx - p[i], fc - p[i]);
        sumN = sumN + nv;
        s2max = fmax(s2max, dot(nv, nv));
    }
    if (!(s2max >= 1e-299)) {
        double sumA = 0.0;
        for (int i = 0; i < n; ++i) {
            const d3 nx = p[(i + 1) % n];
            sumA += mag(cross(nx - p[i], fc - p[i]));
        }
        if (sumA < kROOTVSMALL) return mk(0, 0, 0);
    }
    return 0.5 * sumN;
}

// The TSMALL lift of cutFace.C:159-165: |di| < TSMALL and sgn(di) (+1 for
// -0) decided on the bits; the lift adds the same +-TSMALL.
__device__ __forceinline__ double liftedDistance(d3 p, d3 n, double d) {
    double di = dot(p, n) + d;
    const long long b = bitsOf(di);
    if ((b & 0x7fffffffffffffffLL) < bitsOf(kTSMALL)) {
        const bool pos = b >= 0 || (b << 1) == 0;  // di >= 0, -0 included
        di += pos ? kTSMALL : -kTSMALL;
    }
    return di;
}
// A lifted distance is below the plane (d < 0): at least TSMALL in
// magnitude, so the sign bit decides (NaN never).
__device__ __forceinline__ bool belowBits(double x) {
    const long long b = bitsOf(x);
    return b < 0 && (b & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL && (b << 1) != 0;
}
// dc * dn < 0 for two lifted distances: the product of two numbers of at
// least TSMALL in magnitude is not zero, so it is negative exactly when the
// signs differ (NaN never).
__device__ __forceinline__ bool crossesBits(double a, double b) {
    const long long ba = bitsOf(a), bb = bitsOf(b);
    const long long kMag = 0x7fffffffffffffffLL, kInf = 0x7ff0000000000000LL;
    return (ba ^ bb) < 0 && (ba & kMag) <= kInf && (bb & kMag) <= kInf && (ba << 1) != 0 && (bb << 1) != 0;
}

// One cut face of a cell clipped against the plane (the cut branch of
// calcSubFace, cutFace.C:198-257).  P: cell points, idx: the face's local
// point indices in stored order, dist: lifted distances of the cell points,
// subMask: bit i set when dist[i] < 0.  Returns 0 with the sub-face centre /
// area and the cut points appended to edge[], or -1 when fewer than three
// points remain (then the face counts as fully submerged).
template <class K>
__device__ __forceinline__ int clipCutFace(const d3* P, const uint8_t* idx, int n, const double* dist,
                                           unsigned subMask, d3& cen, d3& area, d3* edge, int& nEdge,
                                           uint32_t& err) {
    int first = 0;
    while (first < n - 1 && !((subMask >> idx[first]) & 1u)) ++first;
    // The edges the plane cuts, by position j in the walk from `first` (edge
    // first + j).  A convex face has two: their cut points are computed
    // first, on every lane of the warp at once (cells cut their faces at
    // different positions of the walk, which would otherwise serialise the
    // divisions); further cut points (warped faces) follow in the walk.
    unsigned cutE = 0;
    for (int j = 0; j < n; ++j) {
        const int cur = (first + j) % n, nxt = (first + j + 1) % n;
        if (crossesBits(dist[idx[cur]], dist[idx[nxt]])) cutE |= 1u << j;
    }
    const auto cutPoint = [&](int j) {
        const int cur = (first + j) % n, nxt = (first + j + 1) % n;
        const double dc = dist[idx[cur]], dn = dist[idx[nxt]];
        const double w = dc / (dc - dn);
        return P[idx[cur]] + w * (P[idx[nxt]] - P[idx[cur]]);
    };
    const int j1 = cutE ? __ffs(cutE) - 1 : 0;
    const unsigned rest = cutE & (cutE - 1u);
    const int j2 = rest ? __ffs(rest) - 1 : j1;
    const d3 c1 = cutPoint(j1), c2 = cutPoint(j2);
    d3 sp[K::kSub];
    int ns = 0;
    const int e0 = nEdge;
    for (int j = 0; j < n; ++j) {
        const int cur = (first + j) % n;
        if ((subMask >> idx[cur]) & 1u) sp[ns++] = P[idx[cur]];
        if ((cutE >> j) & 1u) {
            const d3 cp = (j == j1) ? c1 : (j == j2 ? c2 : cutPoint(j));
            sp[ns++] = cp;
            if (nEdge < K::kEdge) edge[nEdge++] = cp;
            else err |= kErrEdgeOverflow;
        }
    }
    if (ns >= 3) {
        fanCentreArea(sp, ns, cen, area);
        return 0;
    }
    nEdge = e0;  // fewer than 3 points: treated as fully submerged (cutFace.C:249-255)
    return -1;
}

// Per-thread copy of one cell (points ascending by id, faces in cells()
// order as local point indices), plus the face::centre / areaNormal of each
// face, which calcSubFace returns for fully submerged faces.  Sized by the
// caps K of the cell's class.
template <class K>
struct CellWS {
    int np, nf, cell;
    double V, rV;  // volume, 1 / V
    d3 C;
    d3 P[K::kPts];
    uint8_t fsz[K::kFaces];
    uint8_t fidx[K::kFaces][K::kFacePts];
    d3 fullC[K::kFaces], fullA[K::kFaces];
};

template <class K>
__device__ __forceinline__ bool loadCell(const DevMesh& m, int c, CellWS<K>& w) {
    w.cell = c;
    w.V = m.V[c];
    w.rV = m.rV[c];
    w.C = ld3(m.C, c);
    const int p0 = m.cpOff[c], np = m.cpOff[c + 1] - p0;
    const int f0 = m.cOff[c], nf = m.cOff[c + 1] - f0;
    if (np > K::kPts || nf > K::kFaces) return false;
    w.np = np;
    w.nf = nf;
    int gid[K::kPts];
    for (int i = 0; i < np; ++i) {
        gid[i] = m.cPts[p0 + i];
        w.P[i] = ld3(m.pts, gid[i]);
    }
    for (int k = 0; k < nf; ++k) {
        const int f = m.cFaces[f0 + k];
        const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
        if (n > K::kFacePts) return false;
        w.fsz[k] = uint8_t(n);
        for (int i = 0; i < n; ++i) {
            const int g = m.fPts[q0 + i];
            int loc = 0;
            while (loc < np - 1 && gid[loc] != g) ++loc;
            w.fidx[k][i] = uint8_t(loc);
        }
        w.fullC[k] = ld3(m.fullC, f);
        w.fullA[k] = ld3(m.fullA, f);
    }
    return true;
}

// The bracket the bisection over vertex levels ends with (cutCell.C:682-719):
// plane constants and VOF of the two levels that enclose alpha.
struct Bracket {
    double lowD, upD, lowA, upA;
};

__device__ __forceinline__ bool absBelow(double x, double t) {  // fabs(x) < t, t > 0 (false for NaN)
    return (bitsOf(x) & 0x7fffffffffffffffLL) < bitsOf(t);
}

// a double's leading 24 bits as a float (truncated), on the integer pipe;
// zero below the float range, infinite above it
__device__ __forceinline__ float leadingFloat(double x) {
    const long long b = bitsOf(x);
    const int e = int((b >> 52) & 0x7ff) - 896;
    const unsigned s = unsigned(b >> 32) & 0x80000000u;
    if (e <= 0) return __uint_as_float(s);
    if (e >= 255) return __uint_as_float(s | 0x7f800000u);
    return __uint_as_float(s | (unsigned(e) << 23) | (unsigned(b >> 29) & 0x7fffffu));
}

// Newton on the cubic through the bracket (cutCell.C:743-789); returns the
// plane constant.
__device__ __forceinline__ double cubicDistance(const Bracket& br, double v13, double v23, double alphaI) {
    const double alphaPrismatoid = br.upA - br.lowA;
    const double a13 = v13 - br.lowA;
    const double a23 = v23 - br.lowA;
    const double a = 13.5 * a13 - 13.5 * a23 + 4.5 * alphaPrismatoid;
    const double b = -22.5 * a13 + 18.0 * a23 - 4.5 * alphaPrismatoid;
    const double c = 9.0 * a13 - 4.5 * a23 + 1.0 * alphaPrismatoid;
    const double dd = br.lowA - alphaI;
    double lambda = 0.5;
    // Where the change never falls below TSMALL (one cell in a few hundred:
    // the round-off of the cubic moves lambda further) the iterates go round a
    // cycle, mostly of two, until the hundredth.  A cycle is found by keeping
    // an iterate and comparing (Brent 1980), and only what is left of the
    // hundred modulo its length is run: the same lambda.
    double kept = lambda;
    int keptAt = 0, limit = 100;
    bool cycle = false;
    for (int iter = 0; iter < limit; ++iter) {
        const double l2 = lambda * lambda;
        const double func = a * (lambda * l2) + b * l2 + c * lambda + dd;
        const double funcPrime = 3.0 * a * l2 + 2.0 * b * lambda + c;
        const double lambdaNew = lambda - (func / funcPrime);
        if (absBelow(lambdaNew - lambda, kTSMALL)) break;
        lambda = lambdaNew;
        if (!cycle) {
            const int done = iter + 1;
            if (bitsOf(lambda) == bitsOf(kept)) {
                cycle = true;
                limit = done + (100 - done) % (done - keptAt);
            } else if ((done & (done - 1)) == 0) {
                kept = lambda;
                keptAt = done;
            }
        }
    }
    return br.lowD - lambda * (br.lowD - br.upD);
}

struct SubCell {
    int status;
    double vof;
    d3 ic, is;  // interface centre / area vector
};

// cutCell::calcSubCell (cutCell.C:343-542) without the sub-cell centre,
// which no caller of this routine uses.
template <class K>
static __device__ __noinline__ void calcSubCell(const CellWS<K>& w, d3 n, double d, SubCell& out, uint32_t& err) {
    double dist[K::kPts];
    unsigned subMask = 0;  // bit i: cell point i lies below the plane
    for (int i = 0; i < w.np; ++i) {
        dist[i] = liftedDistance(w.P[i], n, d);
        if (belowBits(dist[i])) subMask |= 1u << i;
    }
    // face classification from the point mask (calcSubFace's counting)
    int8_t fst[K::kFaces];
    int cutK[K::kFaces], nCut = 0;
    for (int k = 0; k < w.nf; ++k) {
        int cnt = 0;
        for (int i = 0; i < w.fsz[k]; ++i) cnt += (subMask >> w.fidx[k][i]) & 1u;
        fst[k] = int8_t(cnt == w.fsz[k] ? -1 : (cnt == 0 ? 1 : 0));
        if (cnt != 0 && cnt != w.fsz[k]) cutK[nCut++] = k;
    }
    // The cut faces are clipped as a compact list: the lanes of a warp (one
    // cell each) run their j-th cut face together instead of idling on the
    // faces other cells leave uncut.  Face order is kept for the sums below.
    d3 cenK[K::kFaces], areaK[K::kFaces];
    d3 edge[K::kEdge];
    int eStartK[K::kFaces], eCntK[K::kFaces], nEdge = 0;
    for (int j = 0; j < nCut; ++j) {
        const int k = cutK[j];
        const int e0 = nEdge;
        if (clipCutFace<K>(w.P, w.fidx[k], w.fsz[k], dist, subMask, cenK[k], areaK[k], edge, nEdge, err) == 0) {
            eStartK[k] = e0;
            eCntK[k] = nEdge - e0;
        } else {
            fst[k] = -1;
        }
    }
    // the sub-cell's faces in face order: the cut faces' sub-faces (fst 0)
    // and the fully submerged faces (fst -1), then the interface
    int ncut = 0;
    bool fullySub = true, fullyEmpty = true;
    int nSubFaces = 0;
    for (int k = 0; k < w.nf; ++k) {
        if (fst[k] == 0) {
            ++ncut;
            fullySub = false;
            fullyEmpty = false;
        } else if (fst[k] == -1) {
            ++ncut;
            fullyEmpty = false;
            ++nSubFaces;
        } else {
            fullySub = false;
        }
    }
    out.ic = mk(0, 0, 0);
    out.is = mk(0, 0, 0);
    if (!fullySub && !fullyEmpty) {
        // calcInterfaceCentreAndArea (cutCell.C:37-100)
        d3 fc = mk(0, 0, 0);
        for (int i = 0; i < nEdge; ++i) fc = fc + edge[i];
        if (nEdge > 0) fc = divCount(fc, nEdge);
        d3 sumN = mk(0, 0, 0), sumAc = mk(0, 0, 0);
        double sumA = 0.0;
        for (int k = 0; k < w.nf; ++k) {
            if (fst[k] != 0) continue;
            const d3* ep = edge + eStartK[k];
            for (int i = 0; i < eCntK[k] - 1; ++i) {
                const d3 nx = ep[i + 1];
                const d3 c = (ep[i] + nx) + fc;
                const d3 nv = cross(nx - ep[i], fc - ep[i]);
                const double a = mag(nv);
                sumN = sumN + sgn(dot(nv, sumN)) * nv;
                sumA += a;
                sumAc = sumAc + a * c;
            }
        }
        d3 ic, is;
        if (sumA < kROOTVSMALL) {
            ic = fc;
            is = mk(0, 0, 0);
        } else {
            ic = divBy((1.0 / 3.0) * sumAc, sumA);
            is = 0.5 * sumN;
        }
        // the sub-cell centre is still zero at this point in the reference
        if (dot(is, ic) < 0.0) is = (-1.0) * is;
        out.ic = ic;
        out.is = is;
        if (mag(is) < kTSMALL) {
            if (nSubFaces == 0) {
                out.status = 1;
                out.vof = 0.0;
            } else {
                out.status = -1;
                out.vof = 1.0;
            }
            return;
        }
        ++ncut;  // the interface closes the sub-cell
        // calcSubCellCentreAndVolume (cutCell.C:103-137), volume only
        d3 cEst = mk(0, 0, 0);
        for (int k = 0; k < w.nf; ++k) {
            if (fst[k] == 0) cEst = cEst + cenK[k];
            else if (fst[k] == -1) cEst = cEst + w.fullC[k];
        }
        cEst = cEst + ic;
        cEst = divCount(cEst, ncut);
        double vol = 0.0;
        for (int k = 0; k < w.nf; ++k) {
            if (fst[k] == 0) vol += fmax(fabs(dot(areaK[k], cenK[k] - cEst)), kVSMALL);
            else if (fst[k] == -1) vol += fmax(fabs(dot(w.fullA[k], w.fullC[k] - cEst)), kVSMALL);
        }
        vol += fmax(fabs(dot(is, ic - cEst)), kVSMALL);
        vol /= 3.0;
        out.status = 0;
        out.vof = divByRecip(vol, w.V, w.rV);  // vol / V
    } else if (fullyEmpty) {
        out.status = 1;
        out.vof = 0.0;
    } else {
        out.status = -1;
        out.vof = 1.0;
    }
}

// What is known of a face whose points share a coordinate bit for bit: the
// axis in bits 0-1 (3: none), bit 2 set when the rounded average of five such
// coordinates is that coordinate, bit 3 when the whole face's area vector has
// that component only.
__device__ __forceinline__ uint8_t faceAxisCode(const d3* p, int n, d3 fullA) {
    const auto comp = [](d3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); };
    for (int k = 0; k < 3; ++k) {
        const double x0 = comp(p[0], k);
        bool same = true;
        for (int i = 1; i < n; ++i) same = same && bitsOf(comp(p[i], k)) == bitsOf(x0);
        if (!same) continue;
        const double five = ((((x0 + x0) + x0) + x0) + x0) / 5.0;
        bool only = true;
        for (int q = 0; q < 3; ++q) only = only && (q == k || (bitsOf(comp(fullA, q)) << 1) == 0);
        return uint8_t(k | (bitsOf(five) == bitsOf(x0) ? 4 : 0) | (only ? 8 : 0));
    }
    return 3;
}

// The downwind faces of cell c (advection.C:131-174: phi >= 0 on an owned
// face, phi < 0 on a neighboured one; boundary faces phi >= 0) as a mask of
// its cells() slots k0 .. k1 - 1 (at most 32).
__device__ __forceinline__ unsigned downwindFaces(const DevMesh& m, int c, int k0, int k1, const double* phi) {
    unsigned down = 0;
    for (int k = k0; k < k1; ++k) {
        const int f = m.cFaces[k];
        const double ph = phi[f];
        bool dn;
        if (f < m.nfi)
            dn = (c == m.own[f]) ? (ph >= 0.0) : (ph < 0.0);
        else
            dn = ph >= 0.0;
        if (dn) down |= 1u << (k - k0);
    }
    return down;
}

// x >= 0 on the bits of x (true for -0, false for NaN)
__device__ __forceinline__ bool nonNegBits(long long b) {
    return b >= 0 ? b <= 0x7ff0000000000000LL : (b << 1) == 0;
}

// The upwind face value w (aP - aN) + aN with w = pos0(phi) (the linear
// interpolation form of OpenFOAM's upwind scheme), without the multiply:
// w = 1 gives 1 x = x exactly; w = 0 gives 0 x + aN = aN exactly when aN is
// a nonzero finite number and x is finite, and +0 when aN is +0.  For w = 1,
// (aP - aN) + aN is aP itself when aN is +0 (aP not -0), when aP is +0 (the
// sum cancels to +0), when aP and aN share sign and binade (Sterbenz: the
// difference is exact), or where upwindSettled shows it on the bits.  Other
// cases (a zero or non-finite value where the sign of a zero decides, an aN
// above aP or of the other sign) take the reference's arithmetic.  The tests
// are integer operations on the bits.
__device__ __forceinline__ double upwindAlpha(double ph, double aP, double aN) {
    const long long bp = bitsOf(ph), bP = bitsOf(aP), bN = bitsOf(aN);
    const long long kExp = 0x7ff0000000000000LL, kSign = (long long)0x8000000000000000ULL;
    const bool finite = (bP & kExp) != kExp && (bN & kExp) != kExp;
    if (nonNegBits(bp)) {
        if (finite && ((bN == 0 && bP != kSign) || bP == 0 ||
                       (((bP ^ bN) & (kSign | kExp)) == 0 && (bP & kExp) != 0)))
            return aP;
        const int settled = upwindSettled(uint64_t(bP), uint64_t(bN));
        if (settled) return settled > 0 ? aP : 0.0;
        return (aP - aN) + aN;
    }
    if (finite && (bN << 1) != 0) return aN;
    if (finite && bN == 0) return 0.0;  // (+0 or -0) + +0
    const double w = 0.0;
    return w * (aP - aN) + aN;
}

// (phi * alpha_f) * dt: a zero carrying the signs of phi and dt when alpha_f
// is +0 (phi and dt finite), one multiply less when alpha_f is 1.  x gets the
// product phi * alpha_f when the result is that product times dt (so that
// divOfProduct can give dVf / dt), and prod says so.
__device__ __forceinline__ double fluxDt(double ph, double af, double dt, double& x, bool& prod) {
    const long long ba = bitsOf(af), bp = bitsOf(ph), bd = bitsOf(dt);
    const long long kExp = 0x7ff0000000000000LL, kSign = (long long)0x8000000000000000ULL;
    if (ba == 0 && (bp & kExp) != kExp && (bd & kExp) != kExp) {
        prod = false;
        return __longlong_as_double((bp ^ bd) & kSign);
    }
    x = (ba == 0x3ff0000000000000LL) ? ph : ph * af;
    prod = true;
    return x * dt;
}

// (phi * alpha_f) * dt and, in q, that over dt (alphaPhi of the face): both
// products and the quotient on the integer pipe where every value is a normal
// number, else by fluxDt and a division through y = RN(1/dt).
__device__ __forceinline__ double fluxDtQuot(double ph, double af, double dt, double y, double& q) {
    uint64_t x = uint64_t(bitsOf(ph)), dv, qb;
    const uint64_t ba = uint64_t(bitsOf(af)), bt = uint64_t(bitsOf(dt));
    bool ok = true;
    if (ba != 0x3ff0000000000000ull) ok = mulOnInts(x, ba, x);
    if (ok && mulQuotOnInts(x, bt, dv, qb)) {
        q = __longlong_as_double((long long)qb);
        return __longlong_as_double((long long)dv);
    }
    double p;
    bool prod;
    const double v = fluxDt(ph, af, dt, p, prod);
    q = prod ? divOfProduct(v, dt, y, p) : divByRecip(v, dt, y);
    return v;
}

// dVf of one face before bounding: the Simpson value when the upwind cell is
// cut, else (phi * alpha_f) * dt with alpha_f = w (aP - aN) + aN, w = pos0(phi)
// (upwind weights through the linear interpolation formula); boundary faces
// use the boundary value of alpha.
__device__ __forceinline__ double baseDVf(const DevMesh& m, int f, double ph, const double* aCur,
                                          const int8_t* status, const double* dvfI, const double* alphaB, double dt) {
    const bool pos = nonNegBits(bitsOf(ph));
    double x;
    bool prod;
    if (f < m.nfi) {
        const int o = m.own[f], nb = m.nei[f];
        const int up = pos ? o : nb;
        if (status[up] == 0) return dvfI[f];
        return fluxDt(ph, upwindAlpha(ph, aCur[o], aCur[nb]), dt, x, prod);
    }
    const int o = m.own[f];
    if (pos && status[o] == 0) return dvfI[f];
    const double ab = alphaB ? alphaB[f - m.nfi] : aCur[o];
    return fluxDt(ph, ab, dt, x, prod);
}

}  // namespace simplic
