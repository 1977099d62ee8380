// Simpson time-integrated face areas (cutFace::timeIntegratedArea,
// cutFace.C:392-506), eight polygons to a warp.  Built with -fmad=false: the
// operations and their order are those of the serial restatement, so the
// fluxes are the same bits.
//
// What bounds it: FP64 warp instructions, 16 cycles each per SM and 64 per
// warp whatever the lanes (see plane_group.cuh).  One thread per face went
// through up to eleven clipped areas one after the other, some 230 operations
// each, with 13 of 32 lanes busy.  Here four lanes prepare a polygon (arrival
// times, their order, the intervals), the clipped areas of the warp's
// polygons -- which depend on nothing but a polygon and a time -- are dealt
// out over all lanes, and the four lanes add up.  A point's n.P is formed once
// (its distance at a time is one addition), and on axis-aligned faces the
// area has one component and its magnitude no root (faceAxisCode).
#pragma once

#include "plain_geom.cuh"

namespace simplic {

constexpr int kPolyLanes = 4;
constexpr int kPolys = 32 / kPolyLanes;
constexpr int kMaxTimes = kMaxFacePts + 2;
constexpr int kMaxAreas = 2 * kMaxTimes;  // areas at the first time, the middles and the ends

// Shared memory of one warp.
struct FaceShared {
    double P[kPolys][kMaxFacePts][3];
    double pd[kPolys][kMaxFacePts];    // n.P
    double t[kPolys][kMaxFacePts];     // arrival times, ascending
    double tau[kPolys][kMaxTimes];     // the times between which the area is integrated
    double area[kPolys][kMaxAreas];    // 0: at the first time; 1 + 2k, 2 + 2k: middle and end of interval k
    double term[kPolys][kMaxTimes];    // arrival times as they come, then the intervals' terms
    double distance[kPolys], Un0[kPolys], fullMag[kPolys];
    int code[kPolys];                  // points, then the face's axis code << 8, bit 16: no area at time 0 to form
    int first[kPolys + 1];             // the polygon's first area among the warp's
    double buf[3 * kMaxSubPts][32];    // the lane's clipped polygon (row 3 q + component)
    double sum[2][kMaxFacePts];        // warped faces: the triangles' parts
};

// A polygon and its plane.
struct PolyView {
    int g, lane;      // polygon of the warp, lane of the warp
    int n;            // points
    int axis;         // the axis it is constant on, -1: none
    bool five;        // a pentagon's average keeps the constant
    double fullMag;   // |area| of the whole polygon
};

__device__ __forceinline__ double absOf(double x) { return __longlong_as_double(bitsOf(x) & 0x7fffffffffffffffLL); }
// a total order of doubles as integers (-0 as +0)
__device__ __forceinline__ long long orderOf(double x) {
    const long long b = bitsOf(x);
    if ((b << 1) == 0) return 0ll;
    return b >= 0 ? b : (long long)(0x8000000000000000ULL - (unsigned long long)b);
}

// |area| of the part of the polygon with n.x + d < 0 (clippedFaceArea of the
// serial form), by one lane.
__device__ __forceinline__ double laneClippedArea(FaceShared& s, const PolyView& w, double d) {
    const int n = w.n;
    const double* pd = s.pd[w.g];
    const auto dist = [&](int i) {
        double di = pd[i] + d;
        const long long b = bitsOf(di);
        if ((b & 0x7fffffffffffffffLL) < bitsOf(kTSMALL)) {
            const bool pos = b >= 0 || (b << 1) == 0;
            di += pos ? kTSMALL : -kTSMALL;
        }
        return di;
    };
    unsigned fm = 0;
    double dd[kMaxFacePts];
#pragma unroll
    for (int i = 0; i < kMaxFacePts; ++i) {
        dd[i] = i < n ? dist(i) : 0.0;
        if (i < n && belowBits(dd[i])) fm |= 1u << i;
    }
    if (fm == (1u << n) - 1u) return w.fullMag;
    if (fm == 0) return 0.0;
    const auto pick = [&](int i) {  // dd[i] without a memory index
        double x = dd[0];
#pragma unroll
        for (int k = 1; k < kMaxFacePts; ++k) x = i == k ? dd[k] : x;
        return x;
    };
    const int first = __ffs(fm) - 1;
    const unsigned walk = ((fm >> first) | (fm << (n - first))) & ((1u << n) - 1u);
    const unsigned cutE = walk ^ ((walk >> 1) | ((walk & 1u) << (n - 1)));
    const auto at = [&](int j) {
        const int i = first + j;
        return i >= n ? i - n : i;
    };
    const bool flat = w.axis >= 0;
    const int r0 = flat ? w.axis : 0, r1 = flat ? (w.axis == 2 ? 0 : w.axis + 1) : 1,
              r2 = flat ? (r1 == 2 ? 0 : r1 + 1) : 2;
    const auto cutPoint = [&](int j) {  // components in the order r0, r1, r2
        const int c = at(j), x = at(j + 1 < n ? j + 1 : 0);
        const double dc = pick(c), dn = pick(x);
        const double wgt = dc / (dc - dn);
        const double *pc = s.P[w.g][c], *pn = s.P[w.g][x];
        const double a1 = pc[r1] + wgt * (pn[r1] - pc[r1]), a2 = pc[r2] + wgt * (pn[r2] - pc[r2]);
        return mk(flat ? pc[r0] : pc[r0] + wgt * (pn[r0] - pc[r0]), a1, a2);
    };
    const int j1 = cutE ? __ffs(cutE) - 1 : 0;
    const unsigned rest = cutE & (cutE - 1u);
    const int j2 = rest ? __ffs(rest) - 1 : j1;
    const d3 c1 = cutPoint(j1), c2 = cutPoint(j2);
    int ns = 0;
    const int lane = w.lane;
    for (int j = 0; j < n; ++j) {
        if ((walk >> j) & 1u) {
            const double* p = s.P[w.g][at(j)];
            s.buf[3 * ns][lane] = p[0];
            s.buf[3 * ns + 1][lane] = p[1];
            s.buf[3 * ns + 2][lane] = p[2];
            ++ns;
        }
        if ((cutE >> j) & 1u) {
            const d3 cp = (j == j1) ? c1 : (j == j2 ? c2 : cutPoint(j));
            s.buf[3 * ns + r0][lane] = cp.x;
            s.buf[3 * ns + r1][lane] = cp.y;
            s.buf[3 * ns + r2][lane] = cp.z;
            ++ns;
        }
    }
    if (ns < 3) return w.fullMag;
    // mag(fanArea(polygon))
    if (flat && ns <= 5 && (ns < 5 || w.five)) {
        const auto pu = [&](int q) { return s.buf[3 * q + r1][lane]; };
        const auto pv = [&](int q) { return s.buf[3 * q + r2][lane]; };
        const double u0 = pu(0), v0 = pv(0);
        double sum;
        bool range = true;
        if (ns == 3) {
            const double u1 = pu(1), v1 = pv(1), u2 = pu(2), v2 = pv(2);
            sum = (u1 - u0) * (v2 - v0) - (v1 - v0) * (u2 - u0);
        } else {
            double fu = u0, fv = v0;
            for (int i = 1; i < ns; ++i) {
                fu = fu + pu(i);
                fv = fv + pv(i);
            }
            if (ns == 4) {
                fu = 0.25 * fu;
                fv = 0.25 * fv;
            } else {
                fu = divByRecip(fu, 5.0, 1.0 / 5.0);
                fv = divByRecip(fv, 5.0, 1.0 / 5.0);
            }
            sum = 0.0;
            bool any = false;
            double qu = u0, qv = v0;
            for (int i = 0; i < ns; ++i) {
                const double nu = (i + 1 < ns) ? pu(i + 1) : u0, nv = (i + 1 < ns) ? pv(i + 1) : v0;
                const double x = (nu - qu) * (fv - qv) - (nv - qv) * (fu - qu);
                any = any || int((bitsOf(x) >> 52) & 0x7ff) > 527;  // its square is above 1e-299
                sum = sum + x;
                qu = nu;
                qv = nv;
            }
            range = any;
        }
        const double h = 0.5 * sum;
        const int e = int((bitsOf(h) >> 52) & 0x7ff);
        // |h| = sqrt(RN(h^2)) unless the square leaves the range
        if (range && ((bitsOf(h) << 1) == 0 || (e > 543 && e < 1503))) return absOf(h);
    }
    const auto pt = [&](int q) { return mk(s.buf[3 * q][lane], s.buf[3 * q + 1][lane], s.buf[3 * q + 2][lane]); };
    if (ns == 3) return mag(0.5 * cross(pt(1) - pt(0), pt(2) - pt(0)));
    d3 fc = pt(0);
    for (int i = 1; i < ns; ++i) fc = fc + pt(i);
    fc = divCount(fc, ns);
    d3 sumN = mk(0, 0, 0);
    bool any = false;
    d3 p = pt(0);
    for (int i = 0; i < ns; ++i) {
        const d3 nx = pt(i + 1 < ns ? i + 1 : 0);
        const d3 nv = cross(nx - p, fc - p);
        sumN = sumN + nv;
        // |nv|^2 >= 1e-299 for certain where a component alone makes it so
        any = any || int((bitsOf(nv.x) >> 52) & 0x7ff) > 527 || int((bitsOf(nv.y) >> 52) & 0x7ff) > 527 ||
              int((bitsOf(nv.z) >> 52) & 0x7ff) > 527;
        p = nx;
    }
    if (!any) {
        double sumA = 0.0;
        p = pt(0);
        for (int i = 0; i < ns; ++i) {
            const d3 nx = pt(i + 1 < ns ? i + 1 : 0);
            sumA += mag(cross(nx - p, fc - p));
            p = nx;
        }
        if (sumA < kROOTVSMALL) return 0.0;
    }
    return mag(0.5 * sumN);
}

// The areas of all polygons of the warp, dealt out over its lanes: count is
// the polygon's (on each of its lanes), area e of a polygon is at its first
// time (e = 0) or at the middle / end of an interval.
__device__ __forceinline__ void warpAreas(FaceShared& s, int lane, int count) {
    int off = 0, total = 0;
#pragma unroll
    for (int q = 0; q < kPolys; ++q) {
        const int c = __shfl_sync(0xffffffffu, count, q * kPolyLanes);
        if (q == lane / kPolyLanes) off = total;
        total += c;
    }
    if (lane % kPolyLanes == 0) s.first[lane / kPolyLanes] = off;
    __syncwarp();
    for (int j = lane; j < total; j += 32) {
        int g = 0;
#pragma unroll
        for (int q = 1; q < kPolys; ++q) g = j >= s.first[q] ? q : g;
        const int code = s.code[g];
        const int e = j - s.first[g] + (code >> 16);
        PolyView w;
        w.g = g;
        w.lane = lane;
        w.n = code & 0xff;
        const int ax = (code >> 8) & 3;
        w.axis = ax == 3 ? -1 : ax;
        w.five = (code >> 8) & 4;
        w.fullMag = s.fullMag[g];
        double d = s.distance[g];
        if (e > 0) {
            const int k = (e - 1) >> 1;
            const double tauOld = s.tau[g][k], tauNew = s.tau[g][k + 1];
            d = d - ((e & 1) ? tauOld + 0.5 * (tauNew - tauOld) : tauNew) * s.Un0[g];
        }
        s.area[g][e] = laneClippedArea(s, w, d);
    }
    __syncwarp();
}

// The polygon of a group of lanes: where P, pd, distance, Un0, fullMag and
// code are filled in shared memory.  Returns timeIntegratedArea, or with
// moving false (Un0 dt too small to move the plane) the clipped area, the
// same on the group's lanes; n = 0: no polygon.  The whole warp takes part.
__device__ __forceinline__ double polyTimeArea(FaceShared& s, int lane, int n, bool moving, double distance, double Un0,
                                               double rUn0, double dt, double magSf) {
    const int g = lane / kPolyLanes, l = lane % kPolyLanes;
    // arrival times in stable ascending order: a point's place is the number
    // of points before it
    if (moving)
        for (int i = l; i < n; i += kPolyLanes) {
            const double t = divByRecip(s.pd[g][i] + distance, Un0, rUn0);
            s.term[g][i] = (bitsOf(t) & 0x7fffffffffffffffLL) < bitsOf(kTSMALL) ? 0.0 : t;
        }
    __syncwarp();
    if (moving)
        for (int i = l; i < n; i += kPolyLanes) {
            const double t = s.term[g][i];
            const long long k = orderOf(t);
            int rank = 0;
            for (int j = 0; j < n; ++j) {
                const long long kj = orderOf(s.term[g][j]);
                rank += (kj < k || (kj == k && j < i)) ? 1 : 0;
            }
            s.t[g][rank] = t;
        }
    __syncwarp();
    const long long kDt = orderOf(dt);
    const bool toward = nonNegBits(bitsOf(Un0));  // pos0(Un0)
    double result = 0.0, tInt = 0.0;
    bool open = moving && n > 0;
    int nT = 0, count = !moving && n > 0 ? 1 : 0;
    if (open) {
        const double firstTime = s.t[g][0], lastTime = s.t[g][n - 1];
        if (!(orderOf(lastTime) > 0)) {
            result = toward ? magSf * dt : 0.0;
            open = false;
        } else if (orderOf(firstTime) >= kDt) {
            result = toward ? 0.0 : magSf * dt;
            open = false;
        } else {
            const bool later = orderOf(firstTime) > 0;  // whole or empty until the first time
            double prev = 0.0;
            if (later) {
                prev = firstTime;
                if (!toward) tInt = magSf * firstTime;
                if (l == 0) {
                    s.area[g][0] = toward ? 0.0 : magSf;
                    s.code[g] |= 1 << 16;
                }
            }
            if (l == 0) s.tau[g][0] = prev;
            nT = 1;
            double smallTime = divByRecip(kTSMALL, absOf(Un0), absOf(rUn0));
            if (orderOf(smallTime) < orderOf(kTSMALL)) smallTime = kTSMALL;
            for (int i = 0; i < n; ++i) {
                const double ti = s.t[g][i];
                if (orderOf(ti) < kDt && orderOf(ti) > orderOf(prev + smallTime)) {
                    if (l == 0) s.tau[g][nT] = ti;
                    ++nT;
                    prev = ti;
                }
            }
            if (orderOf(lastTime) > kDt) {
                if (l == 0) s.tau[g][nT] = dt;
                ++nT;
            } else if (toward) {
                tInt += magSf * (dt - lastTime);
            }
            count = 2 * (nT - 1) + (later ? 0 : 1);
        }
    }
    warpAreas(s, lane, count);
    if (!moving) return s.area[g][0];
    for (int k = l; k < nT - 1; k += kPolyLanes) {
        const double deltaTau = 0.5 * (s.tau[g][k + 1] - s.tau[g][k]);
        s.term[g][k] = divByRecip(deltaTau, 3.0, 1.0 / 3.0) *
                       (s.area[g][2 * k] + 4.0 * s.area[g][2 * k + 1] + s.area[g][2 * k + 2]);
    }
    __syncwarp(0xfu << (lane & ~3));
    if (open) {
        for (int k = 0; k < nT - 1; ++k) tInt += s.term[g][k];
        result = tInt;
    }
    return result;
}

}  // namespace simplic
