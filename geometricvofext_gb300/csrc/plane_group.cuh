// Plane solve with one lane per face: cutCell::findSignedDistance
// (cutCell.C:611-799) and cutCell::calcSubCell (cutCell.C:343-542) of a cell
// by a group of G lanes of one warp, lane k of the group on the cell's k-th
// face and, where a sum runs over faces or edges, on one component of it.
// Built with -fmad=false: every operation is the one the serial restatement
// (plain_geom.cuh) makes, in its order, so planes, statuses, centres and
// areas are the same bits.
//
// What bounds it: the FP64 pipe takes a warp instruction every 16 cycles per
// SM, 64 per warp, whatever the number of its active lanes (a division or a
// square root is about nine of them).  So a kernel's time is its count of
// FP64 warp instructions, for one warp as for a full chip.  One thread per
// cell took some 20,000 per warp (0.86 ms, however few cells there were) and,
// with the cells of a warp cutting different faces into polygons of
// different sizes, kept 14 of 32 lanes busy.  One lane per face takes about
// 2,700 per warp of five hexahedra; what does not change a bit is then left
// out (1,400 to 1,700):
//   * on axis-aligned faces the operations whose results are known
//     (setFaceAxis);
//   * the cuts of the bisection that a single precision estimate decides
//     (levelEstimate): the two ends of the bracket are the only levels cut;
//   * the sub-faces in the final cut, whose volume nobody reads;
//   * Newton iterations that repeat (cubicDistance);
//   * comparisons, halvings, signs and magnitudes on the bits, and sums over
//     faces or edges on one lane per component.
#pragma once

#include "cube_fraction_f32.cuh"
#include "plain_geom.cuh"

namespace simplic {

// Shared memory of one warp: NC cells, and per-lane (per-face) columns.
template <class K, int G>
struct GroupShared {
    static constexpr int kCells = 32 / G;
    static constexpr int kSegRows = (K::kFacePts - 1) * 7;
    static constexpr int kBufRows = 3 * K::kSub > kSegRows ? 3 * K::kSub : kSegRows;
    double P[kCells][K::kPts][3];
    double pd[kCells][K::kPts];    // n.P of the cell points
    double dist[kCells][K::kPts];  // lifted distances of the current plane
    double sv[kCells][K::kPts];    // vertex levels -n.P, descending
    double edge[3 * K::kFacePts][32];  // cut points of the lane's face: row 3 e + component
    double cen[3][32];                 // centre of the lane's sub-face
    double term[32];                   // its part of the volume
    float segN[3][32];                 // normal of the lane's only interface segment
    double buf[kBufRows][32];  // polygon of the lane's sub-face (row 3 q + component), then its
                               // interface segments (row 7 s: nx ny nz |n| |n|cx |n|cy |n|cz)
    int gid[kCells][K::kPts];
    int faceOf[kCells][K::kFaces];  // splitWarpedFace: original face | triangle << 8
};

// Local point indices of a face, a byte each.
template <bool WIDE>
struct FaceIndices {
    using type = uint32_t;
};
template <>
struct FaceIndices<true> {
    using type = uint64_t;
};

// The lane's place in the group and the cell it works on.
template <class K, int G>
struct GroupCell {
    GroupShared<K, G>* sh;
    int lane, base, l, g;  // lane of the warp, first lane of the group, lane of the group, group
    int np, nf;            // 0 for an idle group
    double V, rV;
    int fsz;               // the lane's face: points, their local indices (a byte each)
    using Indices = typename FaceIndices<(K::kFacePts > 4)>::type;
    Indices fidx;
    d3 fullC, fullA;       // face::centre / areaNormal of the whole face
    int axis;              // the axis the face is constant on (-1: none), see setFaceAxis
    bool five, fullFlat;   // a pentagon's average keeps the constant; fullA has that component only
    double x0, x3;         // the constant coordinate, (x0 + x0) + x0
    __device__ __forceinline__ unsigned groupBits(unsigned ballot) const {
        return G == 32 ? ballot : ((ballot >> base) & ((1u << (G & 31)) - 1u));
    }
    __device__ __forceinline__ int vertex(int i) const { return int((fidx >> (8 * i)) & 0xff); }
    __device__ __forceinline__ d3 point(int i) const {
        const double* p = sh->P[g][i];
        return mk(p[0], p[1], p[2]);
    }
};

constexpr unsigned kAllLanes = 0xffffffffu;

__device__ __forceinline__ d3 shflD3(d3 v, int src) {
    return mk(__shfl_sync(kAllLanes, v.x, src), __shfl_sync(kAllLanes, v.y, src), __shfl_sync(kAllLanes, v.z, src));
}

// x / 2 on the bits (exact; the pipe only for a subnormal result)
__device__ __forceinline__ double halfOf(double x) {
    const long long b = bitsOf(x);
    const int e = int((b >> 52) & 0x7ff);
    if ((b << 1) == 0) return x;
    if (e >= 2 && e < 0x7ff) return __longlong_as_double(b - (1ll << 52));
    return 0.5 * x;
}

// dot(a, b) >= 0 for the double-precision dot: the sign of a single
// precision estimate where it is certain (each product is within 2^-21 of
// the exact one, the estimate's sums within 2^-22 of the terms' magnitudes,
// and the double sums are far closer), else the double operations.
__device__ __forceinline__ bool dotNonNegative(d3 a, d3 b) {
    const float tx = leadingFloat(a.x) * leadingFloat(b.x), ty = leadingFloat(a.y) * leadingFloat(b.y),
                tz = leadingFloat(a.z) * leadingFloat(b.z);
    const float s = (tx + ty) + tz, t = (fabsf(tx) + fabsf(ty)) + fabsf(tz);
    if (t > 1e-30f && t < 1e30f && fabsf(s) > 1e-5f * t) return s > 0.f;
    return dot(a, b) >= 0.0;
}

// Quotients on the integer pipe for hexahedra, whose warps fill the FP64 pipe;
// the larger classes have few cells and long chains (divByRecip).
template <class K>
constexpr bool kIntDiv = K::kFaces == 6;

// x / n for a small count n: exact scaling for powers of two, else the
// correctly rounded quotient through 1 / n (5 operations instead of a
// division's 9).
__constant__ double kInvCount[33] = {
    0.0,      1.0 / 1,  1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,  1.0 / 7,  1.0 / 8,  1.0 / 9,  1.0 / 10,
    1.0 / 11, 1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15, 1.0 / 16, 1.0 / 17, 1.0 / 18, 1.0 / 19, 1.0 / 20, 1.0 / 21,
    1.0 / 22, 1.0 / 23, 1.0 / 24, 1.0 / 25, 1.0 / 26, 1.0 / 27, 1.0 / 28, 1.0 / 29, 1.0 / 30, 1.0 / 31, 1.0 / 32};
template <bool INTS>
__device__ __forceinline__ double divCount1(double x, int n) {
    if (n > 32) return x / double(n);
    const double y = kInvCount[n];
    return (n & (n - 1)) == 0 ? x * y : divByRecip<INTS>(x, double(n), y);
}
template <bool INTS>
__device__ __forceinline__ d3 divCount3(d3 v, int n) {
    return mk(divCount1<INTS>(v.x, n), divCount1<INTS>(v.y, n), divCount1<INTS>(v.z, n));
}

// fmax(fabs(x), VSMALL) on the bits
__device__ __forceinline__ double absAtLeastVSmall(double x) {
    const long long b = bitsOf(x) & 0x7fffffffffffffffLL;
    return (b > bitsOf(kVSMALL) && b <= 0x7ff0000000000000LL) ? __longlong_as_double(b) : kVSMALL;
}

// Axis-aligned flat faces.  When all points of a face have the same
// coordinate x0 on one axis (the same double: boxes, refined boxes), the
// reference's operations on that component are known without doing them:
//   * a cut point P + w (P' - P) keeps it: x0 + w 0 = x0;
//   * the point average of a sub-face keeps it: the sum of four x0 rounds to
//     4 x0 (2 x0 is exact; 3 x0 is off by at most 2 units of x0's last place,
//     and 4 x0 plus that rounds to 4 x0, a tie going to the even 4 x0), and
//     of five when five x0 / 5 does, which is tested once per face;
//   * so edge vectors and p - centre have a zero there, the fan's cross
//     products have only that component, and |n| = sqrt(RN(n^2)) = |n|
//     (Boldo 2015: exact barring underflow and overflow, which is tested);
//   * products with a zero component are zeros, and adding a zero changes
//     nothing but the sign of a zero, which no result shows.
// A fan triangle then takes 18 operations instead of about 45.  u, v are the
// two axes after the constant one in cyclic order.
// code: faceAxisCode of the lane's face.
template <class K, int G>
__device__ __forceinline__ void setFaceAxis(GroupCell<K, G>& w, unsigned code) {
    w.axis = (code & 3) == 3 ? -1 : int(code & 3);
    w.five = code & 4;
    w.fullFlat = code & 8;
    w.x0 = w.x3 = 0.0;
    if (w.axis >= 0) {
        w.x0 = w.sh->P[w.g][w.vertex(0)][w.axis];
        w.x3 = (w.x0 + w.x0) + w.x0;
    }
}

// The cell's points, and the lane's face in cells() order as local point
// indices (loadCell of the serial form).  False beyond the caps.
template <class K, int G>
__device__ __forceinline__ bool groupLoad(const DevMesh& m, int c, bool act, GroupCell<K, G>& w) {
    GroupShared<K, G>& s = *w.sh;
    w.np = w.nf = 0;
    w.fsz = 0;
    w.fidx = 0;
    w.fullC = w.fullA = mk(0, 0, 0);
    bool ok = true;
    int f0 = 0;
    if (act) {
        const int p0 = m.cpOff[c], np = m.cpOff[c + 1] - p0;
        f0 = m.cOff[c];
        const int nf = m.cOff[c + 1] - f0;
        w.V = m.V[c];
        w.rV = m.rV[c];
        ok = np <= K::kPts && nf <= K::kFaces;
        if (ok) {
            w.np = np;
            w.nf = nf;
            for (int i = w.l; i < np && w.l < G; i += G) {
                const int gp = m.cPts[p0 + i];
                s.gid[w.g][i] = gp;
                const d3 q = ld3(m.pts, gp);
                s.P[w.g][i][0] = q.x;
                s.P[w.g][i][1] = q.y;
                s.P[w.g][i][2] = q.z;
            }
        }
    }
    __syncwarp();
    unsigned code = 3;  // (no face)
    if (w.l < w.nf) {
        const int f = m.cFaces[f0 + w.l];
        const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
        if (n > K::kFacePts) {
            ok = false;
        } else {
            w.fsz = n;
            for (int i = 0; i < n; ++i) {
                const int gp = m.fPts[q0 + i];
                int lo = 0, hi = w.np - 1;  // ascending ids
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s.gid[w.g][mid] < gp) lo = mid + 1;
                    else hi = mid;
                }
                w.fidx |= typename GroupCell<K, G>::Indices(lo) << (8 * i);
            }
            w.fullC = ld3(m.fullC, f);
            w.fullA = ld3(m.fullA, f);
            code = m.faceAxis[f];
        }
    }
    // all lanes of the group agree
    const bool good = w.groupBits(__ballot_sync(kAllLanes, !ok)) == 0;
    if (!good) {
        w.np = w.nf = w.fsz = 0;
        code = 3;
    }
    setFaceAxis(w, code);
    return good;
}

// The workspace of a cell with splitWarpedFace (getLocalPointFieldAndFaceList,
// cutCell.C:140-236): the cell points, then the centre (mesh Cf) of every
// warped face (flatness <= 1 - 1e-14) in face order; flat faces keep their
// points, warped faces become the triangles (centre, p_i, p_i+1); on the
// neighbour side every local face is reversed with its first point kept
// (face::reverseFace).  The whole-face centre and area of each local face
// (calcSubFace's result for a fully submerged face) are face::centre /
// areaNormal of the local point list.  False when the split cell exceeds
// the caps K.
template <class K, int G>
__device__ __forceinline__ bool groupLoadSplit(const DevMesh& m, int c, bool act, GroupCell<K, G>& w) {
    GroupShared<K, G>& s = *w.sh;
    w.np = w.nf = 0;
    w.fsz = 0;
    w.fidx = 0;
    w.fullC = w.fullA = mk(0, 0, 0);
    bool ok = true;
    int p0 = 0, np = 0, f0 = 0, nfc = 0;
    if (act) {
        p0 = m.cpOff[c];
        np = m.cpOff[c + 1] - p0;
        f0 = m.cOff[c];
        nfc = m.cOff[c + 1] - f0;
        w.V = m.V[c];
        w.rV = m.rV[c];
        ok = np <= K::kPts && nfc <= G;
        for (int i = w.l; ok && i < np && w.l < G; i += G) {
            const int gp = m.cPts[p0 + i];
            s.gid[w.g][i] = gp;
            const d3 q = ld3(m.pts, gp);
            s.P[w.g][i][0] = q.x;
            s.P[w.g][i][1] = q.y;
            s.P[w.g][i][2] = q.z;
        }
    }
    // local faces and centres of the original face on this lane
    int cnt = 0;
    bool warped = false;
    int f = 0, n = 0;
    if (ok && w.l < nfc) {
        f = m.cFaces[f0 + w.l];
        n = m.fOff[f + 1] - m.fOff[f];
        warped = !(m.flat[f] > (1.0 - kTSMALL));
        cnt = warped ? n : 1;
        ok = n <= kMaxFacePts && (warped ? K::kFacePts >= 3 : n <= K::kFacePts);
    }
    int incl = cnt;
    for (int o = 1; o < G; o <<= 1) {
        const int v = __shfl_up_sync(kAllLanes, incl, o);
        if (w.l >= o && w.l < G) incl += v;
    }
    const unsigned wm = w.groupBits(__ballot_sync(kAllLanes, warped));
    const int nf = __shfl_sync(kAllLanes, incl, w.base + G - 1);
    const int npl = np + __popc(wm);
    ok = ok && nf <= K::kFaces && nf <= G && npl <= K::kPts;
    const bool good = w.groupBits(__ballot_sync(kAllLanes, !ok)) == 0;
    if (!act || !good) return good;
    // (groups that leave here take no further part: the lanes below only
    // synchronise through the caller's __syncwarp)
    if (w.l < nfc) {
        for (int t = 0; t < cnt; ++t) s.faceOf[w.g][incl - cnt + t] = w.l | ((warped ? t + 1 : 0) << 8);
        if (warped) {
            const d3 q = ld3(m.Cf, f);
            const int ctr = np + __popc(wm & ((1u << w.l) - 1u));
            s.P[w.g][ctr][0] = q.x;
            s.P[w.g][ctr][1] = q.y;
            s.P[w.g][ctr][2] = q.z;
        }
    }
    w.np = npl;
    w.nf = nf;
    return true;
}
// second half of groupLoadSplit, after a __syncwarp: the lane's local face
template <class K, int G>
__device__ __forceinline__ void groupSplitFace(const DevMesh& m, int c, GroupCell<K, G>& w) {
    GroupShared<K, G>& s = *w.sh;
    setFaceAxis(w, 3);  // (no face yet)
    if (!(w.l < w.nf)) return;
    const int code = s.faceOf[w.g][w.l];
    const int k = code & 0xff, t = (code >> 8) - 1;
    const int f0 = m.cOff[c], np = m.cpOff[c + 1] - m.cpOff[c];
    const int f = m.cFaces[f0 + k];
    const int q0 = m.fOff[f], n = m.fOff[f + 1] - q0;
    const bool owner = m.own[f] == c;
    const auto local = [&](int i) {
        const int gp = m.fPts[q0 + i];
        int lo = 0, hi = np - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s.gid[w.g][mid] < gp) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    d3 fp[kMaxFacePts];
    if (t < 0) {
        for (int i = 0; i < n; ++i) {
            const int src = (owner || i == 0) ? i : n - i;  // reverseFace keeps the first point
            const int v = local(src);
            w.fidx |= typename GroupCell<K, G>::Indices(v) << (8 * i);
            fp[i] = w.point(v);
        }
        w.fsz = n;
    } else {
        int ctr = np;
        for (int j = 0; j < k; ++j) ctr += !(m.flat[m.cFaces[f0 + j]] > (1.0 - kTSMALL));
        const int a = local(t), b = local((t + 1) % n);
        const int v1 = owner ? a : b, v2 = owner ? b : a;
        w.fidx = uint32_t(ctr) | (uint32_t(v1) << 8) | (uint32_t(v2) << 16);
        w.fsz = 3;
        fp[0] = w.point(ctr);
        fp[1] = w.point(v1);
        fp[2] = w.point(v2);
    }
    w.fullC = faceCentreOF(fp, w.fsz);
    w.fullA = faceAreaNormalOF(fp, w.fsz);
    setFaceAxis(w, faceAxisCode(fp, w.fsz, w.fullA));
}

// calcSubFaceCentreAndArea (fanCentreArea of the serial form) of the polygon
// in the lane's column of buf.
template <class K, int G>
__device__ __forceinline__ void groupFan(const GroupShared<K, G>& s, int lane, int n, d3& cen, d3& area) {
    const auto at = [&](int q) { return mk(s.buf[3 * q][lane], s.buf[3 * q + 1][lane], s.buf[3 * q + 2][lane]); };
    const d3 p0 = at(0);
    if (n == 3) {
        const d3 p1 = at(1), p2 = at(2);
        cen = (1.0 / 3.0) * ((p0 + p1) + p2);
        const d3 x = cross(p1 - p0, p2 - p0);
        area = mk(halfOf(x.x), halfOf(x.y), halfOf(x.z));
        return;
    }
    d3 fc = p0;
    for (int i = 1; i < n; ++i) fc = fc + at(i);
    fc = divCount3<kIntDiv<K>>(fc, n);
    d3 sumN = mk(0, 0, 0), sumAc = mk(0, 0, 0);
    double sumA = 0.0;
    d3 p = p0;
    for (int i = 0; i < n; ++i) {
        const d3 nx = (i + 1 < n) ? at(i + 1) : p0;
        const d3 c = (p + nx) + fc;
        const d3 nv = cross(nx - p, fc - p);
        const double a = mag(nv);
        sumN = sumN + nv;
        sumA += a;
        sumAc = sumAc + a * c;
        p = nx;
    }
    if (sumA < kROOTVSMALL) {
        cen = fc;
        area = mk(0, 0, 0);
    } else {
        cen = divBy<kIntDiv<K>>((1.0 / 3.0) * sumAc, sumA);
        area = mk(halfOf(sumN.x), halfOf(sumN.y), halfOf(sumN.z));
    }
}

// The same on an axis-aligned face (setFaceAxis): centre as (constant axis, u,
// v) in cen and the area's one component.  False where a condition of the
// shortcut does not hold (more than five points, areas too small or of both
// signs); the general fan decides then.
template <class K, int G>
__device__ __forceinline__ bool groupFanFlat(const GroupShared<K, G>& s, const GroupCell<K, G>& w, int n, d3& cen,
                                             double& area) {
    if (n > 5 || (n == 5 && !w.five)) return false;
    const int iu = w.axis == 2 ? 0 : w.axis + 1, iv = iu == 2 ? 0 : iu + 1;
    const int lane = w.lane;
    const auto pu = [&](int q) { return s.buf[3 * q + iu][lane]; };
    const auto pv = [&](int q) { return s.buf[3 * q + iv][lane]; };
    const double u0 = pu(0), v0 = pv(0);
    if (n == 3) {
        const double u1 = pu(1), v1 = pv(1), u2 = pu(2), v2 = pv(2);
        cen = (1.0 / 3.0) * mk(w.x3, (u0 + u1) + u2, (v0 + v1) + v2);
        area = halfOf((u1 - u0) * (v2 - v0) - (v1 - v0) * (u2 - u0));
        return true;
    }
    double fu = u0, fv = v0;
    for (int i = 1; i < n; ++i) {
        fu = fu + pu(i);
        fv = fv + pv(i);
    }
    fu = divCount1<kIntDiv<K>>(fu, n);
    fv = divCount1<kIntDiv<K>>(fv, n);
    double sumN = 0.0;
    d3 sumAc = mk(0, 0, 0);
    bool neg = false, pos = false, range = true;
    double qu = u0, qv = v0;
    for (int i = 0; i < n; ++i) {
        const double nu = (i + 1 < n) ? pu(i + 1) : u0, nv = (i + 1 < n) ? pv(i + 1) : v0;
        const double x = (nu - qu) * (fv - qv) - (nv - qv) * (fu - qu);
        const long long b = bitsOf(x), ab = b & 0x7fffffffffffffffLL;
        const int e = int(ab >> 52);
        range = range && (ab == 0 || (e > 543 && e < 1503));  // the square and its root neither under- nor overflow
        neg = neg || (b < 0 && ab != 0);
        pos = pos || (b >= 0 && ab != 0);
        const double a = __longlong_as_double(ab);
        sumN = sumN + x;
        sumAc = sumAc + a * mk(w.x3, (qu + nu) + fu, (qv + nv) + fv);
        qu = nu;
        qv = nv;
    }
    // of one sign, the magnitudes add up to the sum's magnitude, rounding by rounding
    const double sumA = fabs(sumN);
    if (!range || (neg && pos) || bitsOf(sumA) < bitsOf(kROOTVSMALL)) return false;
    cen = divBy<kIntDiv<K>>((1.0 / 3.0) * sumAc, sumA);
    area = halfOf(sumN);
    return true;
}

// cutCell::calcSubCell for the cells of a warp, each with its plane constant
// d (n enters through pd).  Groups with act false take part in the shuffles
// only.  Status, volume fraction and the interface centre / area vector are
// the same on every lane of the group.  Without wantVof (the same on the
// whole warp) the sub-faces' centres and areas, which only the volume needs,
// are left out and vof is not set for a cut cell.
template <class K, int G>
__device__ __forceinline__ void groupSubCell(GroupCell<K, G>& w, bool act, bool wantVof, double d, SubCell& out,
                                             uint32_t& err) {
    GroupShared<K, G>& s = *w.sh;
    const int np = act ? w.np : 0, nf = act ? w.nf : 0;
    const int l = w.l, lane = w.lane;
    // lifted distances, the mask of the points below the plane
    unsigned subMask = 0;
#pragma unroll
    for (int r = 0; r * G < K::kPts; ++r) {
        const int i = r * G + l;
        bool below = false;
        if (l < G && i < np) {
            double di = s.pd[w.g][i] + d;
            const long long b = bitsOf(di);
            if ((b & 0x7fffffffffffffffLL) < bitsOf(kTSMALL)) {
                const bool pos = b >= 0 || (b << 1) == 0;
                di += pos ? kTSMALL : -kTSMALL;
            }
            s.dist[w.g][i] = di;
            below = belowBits(di);
        }
        subMask |= w.groupBits(__ballot_sync(kAllLanes, below)) << ((r * G) & 31);
    }
    __syncwarp();
    // the lane's face: -1 submerged, 1 empty, 0 cut
    int fst = 1, eCnt = 0;
    d3 area = w.fullA;
    double areaFlat = w.axis == 0 ? area.x : (w.axis == 1 ? area.y : area.z);
    bool flatArea = w.fullFlat;
    const int iu = w.axis == 2 ? 0 : w.axis + 1, iv = iu == 2 ? 0 : iu + 1;
    if (l < nf) {
        const int n = w.fsz;
        unsigned fm = 0;  // bit i: the face's i-th point lies below
        for (int i = 0; i < n; ++i) fm |= ((subMask >> w.vertex(i)) & 1u) << i;
        fst = fm == 0 ? 1 : (fm == (1u << n) - 1u ? -1 : 0);
        if (fst == 0) {
            // clipCutFace: the walk from the first point below the plane.
            // Lifted distances are at least TSMALL in magnitude, so an edge
            // crosses where one of its points lies below and the other not.
            const int first = __ffs(fm) - 1;
            const unsigned walk = ((fm >> first) | (fm << (n - first))) & ((1u << n) - 1u);
            const unsigned cutE = walk ^ ((walk >> 1) | ((walk & 1u) << (n - 1)));
            const double* dist = s.dist[w.g];
            const auto vertexAt = [&](int j) {  // j-th vertex of the walk, j <= n
                int i = first + j;
                if (i >= n) i -= n;
                return w.vertex(i);
            };
            const auto cutPoint = [&](int j) {
                const int vc = vertexAt(j), vn = vertexAt(j + 1 < n ? j + 1 : 0);
                const double dc = dist[vc], dn = dist[vn];
                const double wgt = dc / (dc - dn);
                if (w.axis >= 0) {  // (x0, u, v) on an axis-aligned face
                    const double *pc = s.P[w.g][vc], *pn = s.P[w.g][vn];
                    return mk(w.x0, pc[iu] + wgt * (pn[iu] - pc[iu]), pc[iv] + wgt * (pn[iv] - pc[iv]));
                }
                const d3 a = w.point(vc);
                return a + wgt * (w.point(vn) - a);
            };
            const int j1 = cutE ? __ffs(cutE) - 1 : 0;
            const unsigned rest = cutE & (cutE - 1u);
            const int j2 = rest ? __ffs(rest) - 1 : j1;
            const d3 c1 = cutPoint(j1), c2 = cutPoint(j2);
            // rows of the components of a cut point
            const int r0 = w.axis >= 0 ? w.axis : 0, r1 = w.axis >= 0 ? iu : 1, r2 = w.axis >= 0 ? iv : 2;
            int ns = 0;
            for (int j = 0; j < n; ++j) {
                if ((walk >> j) & 1u) {
                    if (wantVof) {
                        const double* p = s.P[w.g][vertexAt(j)];
                        s.buf[3 * ns][lane] = p[0];
                        s.buf[3 * ns + 1][lane] = p[1];
                        s.buf[3 * ns + 2][lane] = p[2];
                    }
                    ++ns;
                }
                if ((cutE >> j) & 1u) {
                    const d3 cp = (j == j1) ? c1 : (j == j2 ? c2 : cutPoint(j));
                    if (wantVof) {
                        s.buf[3 * ns + r0][lane] = cp.x;
                        s.buf[3 * ns + r1][lane] = cp.y;
                        s.buf[3 * ns + r2][lane] = cp.z;
                    }
                    ++ns;
                    s.edge[3 * eCnt + r0][lane] = cp.x;
                    s.edge[3 * eCnt + r1][lane] = cp.y;
                    s.edge[3 * eCnt + r2][lane] = cp.z;
                    ++eCnt;
                }
            }
            if (ns >= 3) {
                if (wantVof) {
                    d3 cen;
                    flatArea = w.axis >= 0 && groupFanFlat(s, w, ns, cen, areaFlat);
                    if (!flatArea) groupFan(s, lane, ns, cen, area);
                    s.cen[flatArea ? r0 : 0][lane] = cen.x;
                    s.cen[flatArea ? r1 : 1][lane] = cen.y;
                    s.cen[flatArea ? r2 : 2][lane] = cen.z;
                }
            } else {
                fst = -1;  // fewer than 3 points: fully submerged (cutFace.C:249-255)
                eCnt = 0;
            }
        }
        if (fst == -1) {
            s.cen[0][lane] = w.fullC.x;
            s.cen[1][lane] = w.fullC.y;
            s.cen[2][lane] = w.fullC.z;
        }
    }
    const unsigned cutF = w.groupBits(__ballot_sync(kAllLanes, l < nf && fst == 0));
    const unsigned subF = w.groupBits(__ballot_sync(kAllLanes, l < nf && fst == -1));
    const unsigned allF = G == 32 ? (nf == 32 ? kAllLanes : ((1u << (nf & 31)) - 1u)) : ((1u << nf) - 1u);
    const bool fullySub = subF == allF, fullyEmpty = (cutF | subF) == 0;
    out.ic = mk(0, 0, 0);
    out.is = mk(0, 0, 0);
    out.status = fullyEmpty ? 1 : -1;
    out.vof = fullyEmpty ? 0.0 : 1.0;
    const bool cut = act && !fullySub && !fullyEmpty;
    const bool anyCut = __any_sync(kAllLanes, cut);
    __syncwarp();  // (also before the next call writes dist)
    if (!anyCut) return;
    // calcInterfaceCentreAndArea (cutCell.C:37-100).  A face the plane cuts
    // has two edge points, one segment (plain: all of the warp's do); warped
    // or concave faces may have more.
    const bool plain = !__any_sync(kAllLanes, cut && l < nf && fst == 0 && eCnt != 2);
    const int q3 = l < 3 ? l : 0;
    const unsigned listF = cut ? cutF : 0u;
    // the average of all edge points, faces in order: lanes 0-2 of the group
    // on one component
    double fcq = 0.0;
    int nEdge = 0;
    if (plain) {
        for (unsigned mm = listF; mm; mm &= mm - 1u) {
            const int src = w.base + __ffs(mm) - 1;
            fcq = (fcq + s.edge[q3][src]) + s.edge[3 + q3][src];
        }
        nEdge = 2 * __popc(listF);
    } else {
#pragma unroll 1
        for (int k = 0; k < G; ++k) {
            const int ne = __shfl_sync(kAllLanes, eCnt, w.base + k);
            if ((listF >> k) & 1u) {
                for (int e = 0; e < ne; ++e) fcq = fcq + s.edge[3 * e + q3][w.base + k];
                nEdge += ne;
            }
        }
    }
    if (nEdge > K::kEdge) err |= kErrEdgeOverflow;
    if (nEdge > 0) fcq = divCount1<kIntDiv<K>>(fcq, nEdge);
    const d3 fc = mk(__shfl_sync(kAllLanes, fcq, w.base), __shfl_sync(kAllLanes, fcq, w.base + 1),
                     __shfl_sync(kAllLanes, fcq, w.base + 2));
    // the lane's segments
    if (cut && l < nf && fst == 0) {
        if (plain && w.axis >= 0) {
            // (axis, u, v): the segment has no component along the axis
            const double fA = w.axis == 0 ? fc.x : (w.axis == 1 ? fc.y : fc.z);
            const double fU = iu == 0 ? fc.x : (iu == 1 ? fc.y : fc.z), fV = iv == 0 ? fc.x : (iv == 1 ? fc.y : fc.z);
            const double pu = s.edge[iu][lane], pv = s.edge[iv][lane];
            const double nu = s.edge[3 + iu][lane], nv = s.edge[3 + iv][lane];
            const double eu = nu - pu, ev = nv - pv, tA = fA - w.x0, tU = fU - pu, tV = fV - pv;
            const double nA = eu * tV - ev * tU, nU = ev * tA, nV = -(eu * tA);
            const double sA = nA * nA, sU = nU * nU, sV = nV * nV;
            // (x^2 + y^2) + z^2 with the squares in x, y, z order
            const double sx = w.axis == 0 ? sA : (w.axis == 1 ? sV : sU),
                         sy = w.axis == 1 ? sA : (w.axis == 2 ? sV : sU),
                         sz = w.axis == 2 ? sA : (w.axis == 0 ? sV : sU);
            const double a = sqrt((sx + sy) + sz);
            s.buf[w.axis][lane] = nA;
            s.buf[iu][lane] = nU;
            s.buf[iv][lane] = nV;
            s.buf[3][lane] = a;
            s.buf[4 + w.axis][lane] = a * ((w.x0 + w.x0) + fA);
            s.buf[4 + iu][lane] = a * ((pu + nu) + fU);
            s.buf[4 + iv][lane] = a * ((pv + nv) + fV);
            s.segN[w.axis][lane] = leadingFloat(nA);
            s.segN[iu][lane] = leadingFloat(nU);
            s.segN[iv][lane] = leadingFloat(nV);
        } else {
            d3 p = mk(s.edge[0][lane], s.edge[1][lane], s.edge[2][lane]);
            for (int i = 0; i < eCnt - 1; ++i) {
                const d3 nx = mk(s.edge[3 * i + 3][lane], s.edge[3 * i + 4][lane], s.edge[3 * i + 5][lane]);
                const d3 c = (p + nx) + fc;
                const d3 nv = cross(nx - p, fc - p);
                const double a = mag(nv);
                double(*r)[32] = s.buf + 7 * i;
                r[0][lane] = nv.x;
                r[1][lane] = nv.y;
                r[2][lane] = nv.z;
                r[3][lane] = a;
                r[4][lane] = a * c.x;
                r[5][lane] = a * c.y;
                r[6][lane] = a * c.z;
                p = nx;
                s.segN[0][lane] = leadingFloat(nv.x);
                s.segN[1][lane] = leadingFloat(nv.y);
                s.segN[2][lane] = leadingFloat(nv.z);
            }
        }
    }
    __syncwarp();
    // The sums over the segments in order.  Plain: the signs sgn(nv . sumN)
    // first, from single precision sums of the leading bits (at most 32 terms:
    // within 2^-17 of the sum of the products of magnitudes; where the dot is
    // clear of that its sign is settled), then lanes 0-2 of the group on a component of sumN
    // and of sumAc each and lane 3 on sumA.
    d3 sumN = mk(0, 0, 0);
    double sumQ = 0.0, sumA = 0.0;  // sumQ: sumAc's component on lanes 0-2
    unsigned minus = 0;
    bool signs = plain;
    if (plain) {
        float nx = 0.f, ny = 0.f, nz = 0.f, mx = 0.f, my = 0.f, mz = 0.f;
        for (unsigned mm = listF; mm; mm &= mm - 1u) {
            const int src = w.base + __ffs(mm) - 1;
            const float ax = s.segN[0][src], ay = s.segN[1][src], az = s.segN[2][src];
            float sg = 1.f;
            if (mm != listF) {
                const float dt = (ax * nx + ay * ny) + az * nz;
                const float mg = (fabsf(ax) * mx + fabsf(ay) * my) + fabsf(az) * mz;
                signs = signs && mg > 1e-30f && mg < 1e30f && fabsf(dt) > 1e-5f * mg;
                if (dt < 0.f) {
                    sg = -1.f;
                    minus |= mm & (0u - mm);
                }
            }
            nx += sg * ax;
            ny += sg * ay;
            nz += sg * az;
            mx += fabsf(ax);
            my += fabsf(ay);
            mz += fabsf(az);
        }
    }
    if (!__any_sync(kAllLanes, !signs)) {
        const int q4 = l < 4 ? l : 0;
        double sq = 0.0;  // sumN's component on lanes 0-2, sumA on lane 3
        for (unsigned mm = listF; mm; mm &= mm - 1u) {
            const int src = w.base + __ffs(mm) - 1;
            const long long flip = (q4 < 3 && (minus & mm & (0u - mm))) ? (long long)0x8000000000000000ULL : 0ll;
            sq += __longlong_as_double(bitsOf(s.buf[q4][src]) ^ flip);
            sumQ += s.buf[4 + q3][src];
        }
        sumN = mk(__shfl_sync(kAllLanes, sq, w.base), __shfl_sync(kAllLanes, sq, w.base + 1),
                  __shfl_sync(kAllLanes, sq, w.base + 2));
        sumA = __shfl_sync(kAllLanes, sq, w.base + 3);
    } else {
        bool firstSeg = true;
#pragma unroll 1
        for (int k = 0; k < G; ++k) {
            const int ne = __shfl_sync(kAllLanes, eCnt, w.base + k);
            if ((listF >> k) & 1u) {
                for (int i = 0; i < ne - 1; ++i) {
                    const double(*r)[32] = s.buf + 7 * i;
                    const int src = w.base + k;
                    const d3 nv = mk(r[0][src], r[1][src], r[2][src]);
                    const bool plus = firstSeg || dotNonNegative(nv, sumN);  // a zero sumN counts as >= 0
                    sumN = plus ? sumN + nv : sumN - nv;  // sgn(...) * nv exactly
                    sumA += r[3][src];
                    sumQ += r[4 + q3][src];
                    firstSeg = false;
                }
            }
        }
    }
    const bool tiny = sumA < kROOTVSMALL;
    const double icq = (1.0 / 3.0) * sumQ / sumA;
    d3 ic = mk(__shfl_sync(kAllLanes, icq, w.base), __shfl_sync(kAllLanes, icq, w.base + 1),
               __shfl_sync(kAllLanes, icq, w.base + 2));
    d3 is = mk(halfOf(sumN.x), halfOf(sumN.y), halfOf(sumN.z));
    if (tiny) {
        ic = fc;
        is = mk(0, 0, 0);
    }
    // the sub-cell centre is still zero at this point in the reference
    if (cut && !dotNonNegative(is, ic)) is = mk(-is.x, -is.y, -is.z);
    bool vanishing = false;
    if (cut) {
        out.ic = ic;
        out.is = is;
        // mag(is) < TSMALL, without the root where one component alone decides
        vanishing = absBelow(is.x, 2.0 * kTSMALL) && absBelow(is.y, 2.0 * kTSMALL) && absBelow(is.z, 2.0 * kTSMALL) &&
                    mag(is) < kTSMALL;
        if (vanishing) {
            out.status = subF == 0 ? 1 : -1;
            out.vof = subF == 0 ? 0.0 : 1.0;
        }
    }
    const bool vol = cut && !vanishing;
    if (!wantVof) {
        if (vol) out.status = 0;
        __syncwarp();
        return;
    }
    // calcSubCellCentreAndVolume (cutCell.C:103-137), volume only
    const unsigned inF = vol ? (cutF | subF) : 0u;
    double ceq = 0.0;
    for (unsigned mm = inF; mm; mm &= mm - 1u) ceq = ceq + s.cen[q3][w.base + __ffs(mm) - 1];
    ceq = ceq + (q3 == 0 ? ic.x : (q3 == 1 ? ic.y : ic.z));
    ceq = divCount1<kIntDiv<K>>(ceq, __popc(inF) + 1);
    const d3 cEst = mk(__shfl_sync(kAllLanes, ceq, w.base), __shfl_sync(kAllLanes, ceq, w.base + 1),
                       __shfl_sync(kAllLanes, ceq, w.base + 2));
    double pyr = 0.0;
    if (l < nf && fst != 1) {
        if (flatArea) {  // area x (centre - cEst) on the one axis
            const double cx = s.cen[w.axis][lane];
            pyr = areaFlat * (cx - (w.axis == 0 ? cEst.x : (w.axis == 1 ? cEst.y : cEst.z)));
        } else {
            pyr = dot(area, mk(s.cen[0][lane], s.cen[1][lane], s.cen[2][lane]) - cEst);
        }
    }
    s.term[lane] = absAtLeastVSmall(pyr);
    __syncwarp();
    double v = 0.0;
    for (unsigned mm = inF; mm; mm &= mm - 1u) v += s.term[w.base + __ffs(mm) - 1];
    if (vol) {
        v += absAtLeastVSmall(dot(is, ic - cEst));
        v = divByRecip<kIntDiv<K>>(v, 3.0, 1.0 / 3.0);
        out.status = 0;
        out.vof = divByRecip<kIntDiv<K>>(v, w.V, w.rV);  // volume / V
    }
    __syncwarp();
}

// Whether the level at distance a (of the box's extent M along n) cuts clearly
// more (up) or less (dn) of a box with edges Lx, Ly, Lz than alpha (beta = 1 -
// alpha).  The single precision fraction of the box below the level, or above
// it where that is the smaller one, is within a relative 2e-5 of the exact one
// unless cubeCoefficientsF raised a coefficient (then within 2e-4), and the
// double cut volume is within 1e-6 of the exact one, so the margins below
// settle the bisection's test (midAlpha > alphaI, and its exit at TSMALL)
// without the cut.  A section whose area comes near TSMALL counts as none in
// calcSubCell; the test on the edges keeps that to fractions below 1e-5, inside
// the margin.  Nearly axis-aligned planes, whose levels coincide, and (the
// caller's test) boxes so far from the origin that their edges lose half their
// digits are left to the cut.
__device__ __forceinline__ void levelEstimate(d3 n, float Lx, float Ly, float Lz, float M, float a, float alpha,
                                              float beta, bool& up, bool& dn) {
    const float mx = leadingFloat(n.x) * Lx, my = leadingFloat(n.y) * Ly, mz = leadingFloat(n.z) * Lz;
    const float least = fminf(fabsf(mx), fminf(fabsf(my), fabsf(mz)));
    // section area >= fraction x volume / diagonal
    const float diag = Lx + Ly + Lz;
    if (!(M > 1e-20f) || !(least > 1e-6f * M) || !(Lx * Ly * Lz > 1e-8f * diag)) return;
    CubeCoef c;
    float3 p;
    if (!cubeCoefficientsF(mx, my, mz, c, p)) return;
    const float r = a / M;
    const bool flip = r > 0.5f;
    float dF;
    const float F = cubeFractionF(flip ? 1.f - r : r, c, dF), f = flip ? beta : alpha;
    // (1 - r loses digits where r is near 1: F is then below the 1e-5 floor)
    const float margin = least > 2.f * kCubeMinM * M ? 1e-3f * fmaxf(F, f) + 1e-5f : 1e-3f;
    const bool more = F > f + margin, less = F < f - margin;
    up = flip ? less : more;
    dn = flip ? more : less;
}

// The vertex levels of the group's cell in descending order (sv), and which
// of them cut clearly more (above) or less (under) than alpha.  False for an
// idle group and for a cell without a normal (status in st).
template <class K, int G>
__device__ __forceinline__ bool groupLevels(GroupCell<K, G>& w, bool act, unsigned box, double alphaI, d3 nI, int& st,
                                            unsigned& above, unsigned& under) {
    GroupShared<K, G>& s = *w.sh;
    // mag(nI) < TSMALL, without the root where one component alone decides
    if (act && absBelow(nI.x, 2.0 * kTSMALL) && absBelow(nI.y, 2.0 * kTSMALL) && absBelow(nI.z, 2.0 * kTSMALL) &&
        mag(nI) < kTSMALL) {
        st = int(sgn(0.5 - alphaI));
        act = false;
    }
    const int np = act ? w.np : 0;
    const int l = w.l;
    for (int i = l; i < np && l < G; i += G) {
        const double* p = s.P[w.g][i];
        s.pd[w.g][i] = dot(nI, mk(p[0], p[1], p[2]));
    }
    __syncwarp();
    // vertex levels -n.P in stable descending order: a point's place is the
    // number of points before it (orders on the bits, -0 as +0)
    const auto key = [&](int i) {
        const long long b = bitsOf(-s.pd[w.g][i]);
        if ((b << 1) == 0) return 0ll;
        return b >= 0 ? b : (long long)(0x8000000000000000ULL - (unsigned long long)b);
    };
    for (int i = l; i < np && l < G; i += G) {
        const long long ki = key(i);
        int rank = 0;
        for (int j = 0; j < np; ++j) {
            const long long kj = key(j);
            rank += (kj > ki || (kj == ki && j < i)) ? 1 : 0;
        }
        s.sv[w.g][rank] = -s.pd[w.g][i];
    }
    __syncwarp();
    // Box cells: which levels cut clearly more or less than alpha, from the
    // volume fraction of the box below each level in single precision
    // (lane l on level l + 1).
    above = under = 0;
    const double* sv = s.sv[w.g];
    bool up = false, dn = false;
    float Lx = 0.f, Ly = 0.f, Lz = 0.f, far = 0.f;
    const float V = act ? leadingFloat(w.V) : 0.f;
    if (K::kFaces == 6) {
        if (act && box && l < 6) {
            const double *pl = s.P[w.g][(box >> 3) & 7], *ph = s.P[w.g][box & 7];
            Lx = leadingFloat(ph[0] - pl[0]);
            Ly = leadingFloat(ph[1] - pl[1]);
            Lz = leadingFloat(ph[2] - pl[2]);
            for (int k = 0; k < 3; ++k) far = fmaxf(far, fabsf(leadingFloat(pl[k])) + fabsf(leadingFloat(ph[k])));
        }
    } else if (__any_sync(kAllLanes, act && box)) {
        // A cell that fills its bounding box (refined boxes, faces and edges
        // split) cuts like the box, inside the margins:
        // kernel on a 24^3 checkerboard 0.24 -> 0.165 ms, 56^3 0.73 -> 0.49.
        static_assert(K::kFaces == 6 || K::kPts <= G, "a lane per point");
        float lo[3], hi[3];
        for (int k = 0; k < 3; ++k) {
            const double p0 = act ? s.P[w.g][0][k] : 0.0, p = l < np ? s.P[w.g][l][k] : p0;
            lo[k] = hi[k] = leadingFloat(p - p0);
            far = fmaxf(far, 2.f * fabsf(leadingFloat(p)));
        }
        for (int o = G / 2; o; o >>= 1) {
            for (int k = 0; k < 3; ++k) {
                lo[k] = fminf(lo[k], __shfl_xor_sync(kAllLanes, lo[k], o));
                hi[k] = fmaxf(hi[k], __shfl_xor_sync(kAllLanes, hi[k], o));
            }
            far = fmaxf(far, __shfl_xor_sync(kAllLanes, far, o));
        }
        if (act && box) {
            Lx = hi[0] - lo[0];
            Ly = hi[1] - lo[1];
            Lz = hi[2] - lo[2];
        }
    }
    // (alpha is compared with cut volume / V, V as the mesh gives it: the
    // fraction of the box stands for that only where V is the box's volume, here
    // up to 1e-6 of it)
    const bool boxVolume = fabsf(Lx * Ly * Lz - V) <= 1e-6f * V;
    if (act && boxVolume && l < np - 2 && fminf(Lx, fminf(Ly, Lz)) > 1e-8f * far)
        levelEstimate(nI, Lx, Ly, Lz, leadingFloat(sv[0] - sv[np - 1]), leadingFloat(sv[0] - sv[l + 1]),
                      leadingFloat(alphaI), leadingFloat(1.0 - alphaI), up, dn);
    above = w.groupBits(__ballot_sync(kAllLanes, up)) << 1;
    under = w.groupBits(__ballot_sync(kAllLanes, dn)) << 1;
    return act;
}

// cutCell::findSignedDistance (cutCell.C:611-799): the bracket of two vertex
// levels by bisection, the cuts at 1/3 and 2/3, Newton on the cubic, the
// final cut.  d / ic / is are set where the reference writes interfaceD/C/S.
template <class K, int G>
__device__ __forceinline__ int groupSignedDistance(GroupCell<K, G>& w, bool act, unsigned box, double alphaI, d3 nI,
                                                   double& dOut, d3& icOut, d3& isOut, uint32_t& err) {
    GroupShared<K, G>& s = *w.sh;
    int st = 0;
    unsigned above, under;
    act = groupLevels(w, act, box, alphaI, nI, st, above, under);
    const int np = act ? w.np : 0;
    const double* sv = s.sv[w.g];
    Bracket br;
    br.lowA = 0.0;
    br.upA = 1.0;
    int lowLabel = 0, upLabel = np - 1;
    bool lowKnown = true, upKnown = true;  // lowA / upA are the cut volumes of the levels
    // the bisection as far as the clear levels decide it
    const auto settle = [&] {
        while (upLabel - lowLabel > 1) {
            const int mid = (upLabel + lowLabel + 1) >> 1;
            if ((above >> mid) & 1u) {
                upLabel = mid;
                upKnown = false;
            } else if ((under >> mid) & 1u) {
                lowLabel = mid;
                lowKnown = false;
            } else {
                return true;
            }
        }
        return false;
    };
    // The warp's cells go through the phases together (one call site, so the
    // sub-cell routine is inlined once): the bisections until no cell of the
    // warp has one left, the ends of the brackets that are not known yet, the
    // cuts at 1/3 and 2/3, the final cut.
    enum { kBisect, kEnds, kEnds2, kThird, kTwoThirds, kFinal };
    int phase = kBisect;
    bool busy = act && settle();  // a bisection left
    bool done = !act, cubic = false;
    double v13 = 0.0, deltaDistance = 0.0, distance = 0.0;
    SubCell sc;
    for (;;) {
        if (phase == kBisect && !__any_sync(kAllLanes, busy)) {
            if (!__any_sync(kAllLanes, !done)) break;
            br.lowD = done ? 0.0 : sv[lowLabel];
            br.upD = done ? 1.0 : sv[upLabel];
            // levels that coincide take the cut at their middle, the others the cubic
            cubic = !done && !absBelow(br.lowD - br.upD, kTSMALL);
            if (!done && !cubic) distance = 0.5 * (br.lowD + br.upD);
            deltaDistance = divByRecip<kIntDiv<K>>(br.upD - br.lowD, 3.0, 1.0 / 3.0);
            phase = kEnds;
        }
        // (every group takes its first unknown end in kEnds, a second one in kEnds2)
        const bool endLow = cubic && !lowKnown, endUp = cubic && !upKnown;
        if ((phase == kEnds || phase == kEnds2) && !__any_sync(kAllLanes, endLow || endUp)) phase = kThird;
        if (phase == kThird && !__any_sync(kAllLanes, cubic)) phase = kFinal;
        bool want;
        double d = 0.0;
        if (phase == kBisect) {
            want = busy;
            if (want) d = sv[(upLabel + lowLabel + 1) >> 1];
        } else if (phase <= kEnds2) {
            want = endLow || endUp;
            d = endLow ? br.lowD : br.upD;
        } else if (phase == kFinal) {
            want = !done;
            d = distance;
        } else {
            want = cubic;
            d = br.lowD + (phase == kThird ? deltaDistance : 2.0 * deltaDistance);
        }
        groupSubCell(w, want, phase != kFinal, d, sc, err);
        if (phase == kBisect) {
            if (busy) {
                const int midLabel = (upLabel + lowLabel + 1) >> 1;
                const double midAlpha = sc.vof;
                if (absBelow(midAlpha - alphaI, kTSMALL)) {
                    dOut = d;
                    icOut = sc.ic;
                    isOut = sc.is;
                    st = sc.status;
                    done = true;
                    busy = false;
                } else {
                    if (midAlpha > alphaI) {
                        upLabel = midLabel;
                        br.upA = midAlpha;
                        upKnown = true;
                    } else {
                        lowLabel = midLabel;
                        br.lowA = midAlpha;
                        lowKnown = true;
                    }
                    busy = settle();
                }
            }
        } else if (phase <= kEnds2) {
            if (endLow) {
                br.lowA = sc.vof;
                lowKnown = true;
            } else if (endUp) {
                br.upA = sc.vof;
                upKnown = true;
            }
            phase = kEnds2;
        } else if (phase == kThird) {
            v13 = sc.vof;
            phase = kTwoThirds;
        } else if (phase == kTwoThirds) {
            if (cubic) distance = cubicDistance(br, v13, sc.vof, alphaI);
            phase = kFinal;
        } else {
            if (!done) {
                dOut = d;
                icOut = sc.ic;
                isOut = sc.is;
                st = sc.status;
            }
            break;
        }
    }
    return st;
}

// The same for one cell on all groups of the warp, every group with the cell
// loaded: cuts that do not wait for one another run at once, a group each.
// A bisection cuts its next level and those that may follow it (group g the
// g-th node, breadth first, of the tree of levels below the bracket) and then
// takes the serial decisions as far as the volumes are there; the unknown ends
// of the bracket and its thirds go together.  The planes are the same: a
// level's volume does not depend on when it is cut, and one that is never
// asked for is not looked at.  For lists that leave warps idle: a box cell
// waits for two cuts in a row instead of five, any hexahedron for four instead
// of seven.
template <class K, int G>
__device__ __forceinline__ int teamSignedDistance(GroupCell<K, G>& w, bool act, unsigned box, double alphaI, d3 nI,
                                                  double& dOut, d3& icOut, d3& isOut, uint32_t& err) {
    constexpr int kGroups = 32 / G;
    int st = 0;
    unsigned above, under;
    if (!groupLevels(w, act, box, alphaI, nI, st, above, under)) return st;  // (the whole warp)
    const double* sv = w.sh->sv[w.g];
    int lowLabel = 0, upLabel = w.np - 1;
    unsigned known = 0;  // levels whose volume is known,
    double vol = 0.0;    // that of level j on lane j
    // moves (lo, up) past the clear levels; whether that ends the bisection
    const auto fixed = [&](int& lo, int& up) {
        while (up - lo > 1) {
            const int mid = (up + lo + 1) >> 1;
            if ((above >> mid) & 1u) up = mid;
            else if ((under >> mid) & 1u) lo = mid;
            else return false;
        }
        return true;
    };
    enum { kBisect, kCubic, kFinal };
    int phase = kBisect;
    unsigned tasks = 0;  // kCubic: 1, 2 the ends of the bracket, 4, 8 its thirds
    Bracket br;
    br.lowA = 0.0;
    br.upA = 1.0;
    br.lowD = br.upD = 0.0;
    double v13 = 0.0, v23 = 0.0, deltaDistance = 0.0, distance = 0.0;
    SubCell sc;
    for (;;) {
        bool want = false;
        double d = 0.0;
        int mine = -1;  // the group's level or task
        if (phase == kBisect) {
            bool found = false;
            while (upLabel - lowLabel > 1) {
                const int mid = (upLabel + lowLabel + 1) >> 1;
                bool more;
                if ((known >> mid) & 1u) {
                    const double a = __shfl_sync(kAllLanes, vol, mid);
                    if (absBelow(a - alphaI, kTSMALL)) {
                        found = true;
                        distance = sv[mid];
                        break;
                    }
                    more = a > alphaI;
                } else if ((above >> mid) & 1u) {
                    more = true;
                } else if ((under >> mid) & 1u) {
                    more = false;
                } else {
                    break;
                }
                (more ? upLabel : lowLabel) = mid;
            }
            if (found) {
                phase = kFinal;
            } else if (upLabel - lowLabel > 1) {
                // node g of the tree of levels that may be asked for
                int lo = lowLabel, up = upLabel;
                int bit = 31 - __clz(w.g + 1);
                bool open = !fixed(lo, up);
                for (--bit; bit >= 0 && open; --bit) {
                    const int mid = (up + lo + 1) >> 1;
                    (((w.g + 1) >> bit) & 1 ? lo : up) = mid;
                    open = !fixed(lo, up);
                }
                want = open;
                if (want) {
                    mine = (up + lo + 1) >> 1;
                    d = sv[mine];
                }
            } else {
                br.lowD = sv[lowLabel];
                br.upD = sv[upLabel];
                deltaDistance = divByRecip<kIntDiv<K>>(br.upD - br.lowD, 3.0, 1.0 / 3.0);
                if (absBelow(br.lowD - br.upD, kTSMALL)) {  // levels that coincide: their middle
                    distance = 0.5 * (br.lowD + br.upD);
                    phase = kFinal;
                } else {
                    phase = kCubic;
                    tasks = 12u;
                    const double a = __shfl_sync(kAllLanes, vol, lowLabel), b = __shfl_sync(kAllLanes, vol, upLabel);
                    if ((known >> lowLabel) & 1u) br.lowA = a;
                    else if (lowLabel != 0) tasks |= 1u;
                    if ((known >> upLabel) & 1u) br.upA = b;
                    else if (upLabel != w.np - 1) tasks |= 2u;
                }
            }
        }
        if (phase == kCubic) {
            unsigned t = tasks;
            for (int k = 0; k < w.g; ++k) t &= t - 1u;
            want = t != 0;
            mine = want ? __ffs(t) - 1 : -1;
            d = mine == 0 ? br.lowD : (mine == 1 ? br.upD : br.lowD + (mine == 2 ? deltaDistance : 2.0 * deltaDistance));
        } else if (phase == kFinal) {
            want = true;
            d = distance;
        }
        groupSubCell(w, want, phase != kFinal, d, sc, err);
        if (phase == kFinal) {
            dOut = d;
            icOut = sc.ic;
            isOut = sc.is;
            return sc.status;
        }
#pragma unroll
        for (int k = 0; k < kGroups; ++k) {
            const int q = __shfl_sync(kAllLanes, mine, k * G);
            const double v = __shfl_sync(kAllLanes, sc.vof, k * G);
            if (q < 0) continue;
            if (phase == kBisect) {
                known |= 1u << q;
                if (w.lane == q) vol = v;
            } else {
                tasks &= ~(1u << q);
                if (q == 0) br.lowA = v;
                else if (q == 1) br.upA = v;
                else if (q == 2) v13 = v;
                else v23 = v;
            }
        }
        if (phase == kCubic && tasks == 0) {
            distance = cubicDistance(br, v13, v23, alphaI);
            phase = kFinal;
        }
    }
}

}  // namespace simplic
