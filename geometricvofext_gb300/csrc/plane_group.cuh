// Plane solve with one lane per face: cutCell::findSignedDistance
// (cutCell.C:611-799) and cutCell::calcSubCell (cutCell.C:343-542) of a cell
// by a group of G lanes of one warp, lane k of the group on the cell's k-th
// face and, where a sum runs over faces or edges, on one component of it.
// Built with -fmad=false: every operation is the one the serial restatement
// (plain_geom.cuh) makes, in its order, so planes, statuses, centres and
// areas are the same bits.
//
// What bounds it: the FP64 pipe issues a warp instruction every 16 cycles
// whatever the number of its active lanes, and returns it 64 cycles later
// (a division or a square root is a chain of about nine).  One thread per
// cell makes a cell's solve one chain of some 20,000 operations (0.86 ms,
// however few cells there are) and, with the cells of a warp cutting
// different faces into polygons of different sizes, keeps 14 of 32 lanes
// busy.  One lane per face takes the same number of warp instructions per
// cell (the faces of a cell run together instead of the cells of a warp) and
// a sixth of the chain.
#pragma once

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
    double buf[kBufRows][32];  // polygon of the lane's sub-face (row 3 q + component), then its
                               // interface segments (row 7 s: nx ny nz |n| |n|cx |n|cy |n|cz)
    int gid[kCells][K::kPts];
    int faceOf[kCells][K::kFaces];  // splitWarpedFace: original face | triangle << 8
};

// The lane's place in the group and the cell it works on.
template <class K, int G>
struct GroupCell {
    GroupShared<K, G>* sh;
    int lane, base, l, g;  // lane of the warp, first lane of the group, lane of the group, group
    int np, nf;            // 0 for an idle group
    double V, rV;
    int fsz;               // the lane's face: points, their local indices (a byte each)
    uint64_t fidx;
    d3 fullC, fullA;       // face::centre / areaNormal of the whole face
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

// One component of divCount: x / n for a small count n.
__device__ __forceinline__ double divCount1(double x, int n) {
    if (n == 4) return 0.25 * x;
    if (n == 8) return 0.125 * x;
    if (n == 2) return 0.5 * x;
    if (n == 1) return x;
    return x / double(n);
}

// fmax(fabs(x), VSMALL) on the bits
__device__ __forceinline__ double absAtLeastVSmall(double x) {
    const long long b = bitsOf(x) & 0x7fffffffffffffffLL;
    return (b > bitsOf(kVSMALL) && b <= 0x7ff0000000000000LL) ? __longlong_as_double(b) : kVSMALL;
}
__device__ __forceinline__ bool absBelow(double x, double t) {  // fabs(x) < t, t > 0 (false for NaN)
    return (bitsOf(x) & 0x7fffffffffffffffLL) < bitsOf(t);
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
                w.fidx |= uint64_t(lo) << (8 * i);
            }
            w.fullC = ld3(m.fullC, f);
            w.fullA = ld3(m.fullA, f);
        }
    }
    // all lanes of the group agree
    const bool good = w.groupBits(__ballot_sync(kAllLanes, !ok)) == 0;
    if (!good) w.np = w.nf = 0;
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
            w.fidx |= uint64_t(v) << (8 * i);
            fp[i] = w.point(v);
        }
        w.fsz = n;
    } else {
        int ctr = np;
        for (int j = 0; j < k; ++j) ctr += !(m.flat[m.cFaces[f0 + j]] > (1.0 - kTSMALL));
        const int a = local(t), b = local((t + 1) % n);
        const int v1 = owner ? a : b, v2 = owner ? b : a;
        w.fidx = uint64_t(ctr) | (uint64_t(v1) << 8) | (uint64_t(v2) << 16);
        w.fsz = 3;
        fp[0] = w.point(ctr);
        fp[1] = w.point(v1);
        fp[2] = w.point(v2);
    }
    w.fullC = faceCentreOF(fp, w.fsz);
    w.fullA = faceAreaNormalOF(fp, w.fsz);
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
        area = 0.5 * cross(p1 - p0, p2 - p0);
        return;
    }
    d3 fc = p0;
    for (int i = 1; i < n; ++i) fc = fc + at(i);
    fc = divCount(fc, n);
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
        cen = divBy((1.0 / 3.0) * sumAc, sumA);
        area = mk(halfOf(sumN.x), halfOf(sumN.y), halfOf(sumN.z));
    }
}

// cutCell::calcSubCell for the cells of a warp, each with its plane constant
// d (n enters through pd).  Groups with act false take part in the shuffles
// only.  Status, volume fraction and the interface centre / area vector are
// the same on every lane of the group.
template <class K, int G>
__device__ __forceinline__ void groupSubCell(GroupCell<K, G>& w, bool act, double d, SubCell& out, uint32_t& err) {
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
    d3 cen = w.fullC, area = w.fullA;
    if (l < nf) {
        int cnt = 0;
        for (int i = 0; i < w.fsz; ++i) cnt += (subMask >> w.vertex(i)) & 1u;
        fst = cnt == w.fsz ? -1 : (cnt == 0 ? 1 : 0);
        if (fst == 0) {
            // clipCutFace: the walk from the first point below the plane
            const int n = w.fsz;
            int first = 0;
            while (first < n - 1 && !((subMask >> w.vertex(first)) & 1u)) ++first;
            const double* dist = s.dist[w.g];
            unsigned cutE = 0;
            for (int j = 0; j < n; ++j) {
                int cur = first + j, nxt = cur + 1;
                if (cur >= n) cur -= n;
                if (nxt >= n) nxt -= n;
                if (crossesBits(dist[w.vertex(cur)], dist[w.vertex(nxt)])) cutE |= 1u << j;
            }
            const auto cutPoint = [&](int j) {
                int cur = first + j, nxt = cur + 1;
                if (cur >= n) cur -= n;
                if (nxt >= n) nxt -= n;
                const int vc = w.vertex(cur), vn = w.vertex(nxt);
                const double dc = dist[vc], dn = dist[vn];
                const double wgt = dc / (dc - dn);
                const d3 a = w.point(vc);
                return a + wgt * (w.point(vn) - a);
            };
            const int j1 = cutE ? __ffs(cutE) - 1 : 0;
            const unsigned rest = cutE & (cutE - 1u);
            const int j2 = rest ? __ffs(rest) - 1 : j1;
            const d3 c1 = cutPoint(j1), c2 = cutPoint(j2);
            int ns = 0;
            const auto put = [&](d3 p) {
                s.buf[3 * ns][lane] = p.x;
                s.buf[3 * ns + 1][lane] = p.y;
                s.buf[3 * ns + 2][lane] = p.z;
                ++ns;
            };
            for (int j = 0; j < n; ++j) {
                int cur = first + j;
                if (cur >= n) cur -= n;
                const int vc = w.vertex(cur);
                if ((subMask >> vc) & 1u) put(w.point(vc));
                if ((cutE >> j) & 1u) {
                    const d3 cp = (j == j1) ? c1 : (j == j2 ? c2 : cutPoint(j));
                    put(cp);
                    s.edge[3 * eCnt][lane] = cp.x;
                    s.edge[3 * eCnt + 1][lane] = cp.y;
                    s.edge[3 * eCnt + 2][lane] = cp.z;
                    ++eCnt;
                }
            }
            if (ns >= 3) {
                groupFan(s, lane, ns, cen, area);
            } else {
                fst = -1;  // fewer than 3 points: fully submerged (cutFace.C:249-255)
                eCnt = 0;
            }
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
    if (!__any_sync(kAllLanes, cut)) return;
    __syncwarp();
    // calcInterfaceCentreAndArea (cutCell.C:37-100).  The average of all
    // edge points, faces in order: lanes 0-2 of the group on one component.
    const int q3 = l < 3 ? l : 0;
    const unsigned listF = cut ? cutF : 0u;
    double fcq = 0.0;
    int nEdge = 0;
#pragma unroll 1
    for (int k = 0; k < G; ++k) {
        const int ne = __shfl_sync(kAllLanes, eCnt, w.base + k);
        if ((listF >> k) & 1u) {
            for (int e = 0; e < ne; ++e) fcq = fcq + s.edge[3 * e + q3][w.base + k];
            nEdge += ne;
        }
    }
    if (nEdge > K::kEdge) err |= kErrEdgeOverflow;
    if (nEdge > 0) fcq = divCount1(fcq, nEdge);
    const d3 fc = mk(__shfl_sync(kAllLanes, fcq, w.base), __shfl_sync(kAllLanes, fcq, w.base + 1),
                     __shfl_sync(kAllLanes, fcq, w.base + 2));
    // the lane's segments
    if (cut && l < nf && fst == 0) {
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
        }
    }
    __syncwarp();
    // the sums over the segments in order: sumN on every lane, sumA on lane
    // 0 and sumAc on lanes 1-3 of the group
    const int q4 = l < 4 ? l : 0;
    d3 sumN = mk(0, 0, 0);
    double sumQ = 0.0;
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
                sumQ += r[3 + q4][src];
                firstSeg = false;
            }
        }
    }
    const double sumA = __shfl_sync(kAllLanes, sumQ, w.base);
    double icq;
    d3 is;
    const bool tiny = sumA < kROOTVSMALL;
    {
        const double y = 1.0 / sumA;
        icq = divByRecip((1.0 / 3.0) * sumQ, sumA, y);
    }
    d3 ic = mk(__shfl_sync(kAllLanes, icq, w.base + 1), __shfl_sync(kAllLanes, icq, w.base + 2),
               __shfl_sync(kAllLanes, icq, w.base + 3));
    is = mk(halfOf(sumN.x), halfOf(sumN.y), halfOf(sumN.z));
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
    // calcSubCellCentreAndVolume (cutCell.C:103-137), volume only
    const bool vol = cut && !vanishing;
    const unsigned inF = vol ? (cutF | subF) : 0u;
    s.cen[0][lane] = cen.x;
    s.cen[1][lane] = cen.y;
    s.cen[2][lane] = cen.z;
    __syncwarp();
    double ceq = 0.0;
#pragma unroll 1
    for (int k = 0; k < G; ++k)
        if ((inF >> k) & 1u) ceq = ceq + s.cen[q3][w.base + k];
    ceq = ceq + (q3 == 0 ? ic.x : (q3 == 1 ? ic.y : ic.z));
    ceq = divCount1(ceq, __popc(inF) + 1);
    const d3 cEst = mk(__shfl_sync(kAllLanes, ceq, w.base), __shfl_sync(kAllLanes, ceq, w.base + 1),
                       __shfl_sync(kAllLanes, ceq, w.base + 2));
    const double term = absAtLeastVSmall(dot(area, cen - cEst));
    double v = 0.0;
#pragma unroll 1
    for (int k = 0; k < G; ++k) {
        const double t = __shfl_sync(kAllLanes, term, w.base + k);
        if ((inF >> k) & 1u) v += t;
    }
    if (vol) {
        v += absAtLeastVSmall(dot(is, ic - cEst));
        v = divByRecip(v, 3.0, 1.0 / 3.0);
        out.status = 0;
        out.vof = divByRecip(v, w.V, w.rV);  // volume / V
    }
    __syncwarp();
}

// cutCell::findSignedDistance (cutCell.C:611-799): the bracket of two vertex
// levels by bisection, the cuts at 1/3 and 2/3, Newton on the cubic, the
// final cut.  d / ic / is are set where the reference writes interfaceD/C/S.
template <class K, int G>
__device__ __forceinline__ int groupSignedDistance(GroupCell<K, G>& w, bool act, double alphaI, d3 nI, double& dOut,
                                                   d3& icOut, d3& isOut, uint32_t& err) {
    GroupShared<K, G>& s = *w.sh;
    int st = 0;
    if (act && mag(nI) < kTSMALL) {
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
    const double* sv = s.sv[w.g];
    Bracket br;
    br.lowD = act ? sv[0] : 0.0;
    br.upD = act ? sv[np - 1] : 1.0;
    br.lowA = 0.0;
    br.upA = 1.0;
    int lowLabel = 0, upLabel = np - 1;
    // The warp's cells go through the phases together (one call site, so the
    // sub-cell routine is inlined once): the bisections until no cell of the
    // warp has one left, the cuts at 1/3 and 2/3, the final cut.
    enum { kBisect, kThird, kTwoThirds, kFinal };
    int phase = kBisect;
    bool busy = act && (upLabel - lowLabel) > 1;  // a bisection left
    bool done = !act, cubic = false;
    double v13 = 0.0, deltaDistance = 0.0, distance = 0.0;
    SubCell sc;
    for (;;) {
        if (phase == kBisect && !__any_sync(kAllLanes, busy)) {
            // levels that coincide take the cut at their middle, the others the cubic
            cubic = !done && !absBelow(br.lowD - br.upD, kTSMALL);
            if (!done && !cubic) distance = 0.5 * (br.lowD + br.upD);
            deltaDistance = divByRecip(br.upD - br.lowD, 3.0, 1.0 / 3.0);
            phase = __any_sync(kAllLanes, cubic) ? kThird : kFinal;
            if (!__any_sync(kAllLanes, !done)) break;
        }
        const int midLabel = (upLabel + lowLabel + 1) >> 1;
        const bool want = phase == kBisect ? busy : (phase == kFinal ? !done : cubic);
        double d = 0.0;
        if (want)
            d = phase == kBisect ? sv[midLabel]
                                 : (phase == kFinal ? distance
                                                    : br.lowD + (phase == kThird ? deltaDistance : 2.0 * deltaDistance));
        groupSubCell(w, want, d, sc, err);
        if (phase == kBisect) {
            if (busy) {
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
                        br.upD = d;
                        br.upA = midAlpha;
                    } else {
                        lowLabel = midLabel;
                        br.lowD = d;
                        br.lowA = midAlpha;
                    }
                    busy = (upLabel - lowLabel) > 1;
                }
            }
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

}  // namespace simplic
