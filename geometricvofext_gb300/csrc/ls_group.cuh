// The least-squares gradient of ls_fp64.cuh by 16 lanes per cell, two cells a
// warp, the same operations in the same order (-fmad=false), for lists that
// leave the FP64 pipes idle: one thread takes some 870 FP64 instructions per
// cell one after another (a 27-cell stencil's 13 sums and the elimination, 64
// cycles each), the 16 lanes about 150.  Lane 4 r + q holds the sum A[r][q] of
// the normal equations (b on the lanes below the diagonal) and its element in
// the elimination.
#pragma once

#include "ls_fp64.cuh"

namespace simplic {

// Up to this many cells per SM 16 lanes take a cell.  Kernel time of the
// normals, a thread per cell against 16 lanes: hexahedra 365 cells 41 / 17 us,
// 3,593 41 / 29, 5,103 43 / 40, 6,988 46 / 51; warped 6,539 42 / 43;
// tetrahedra 560 78 / 20, 3,252 80 / 39, 7,172 82 / 66.
constexpr int kLsGroup = 40;

using LsRows = double[16][5];  // of a cell: 1, x, y, z, field of 16 stencil cells

// All lanes of the warp call it; groups without a cell pass act = false (and
// any valid c).  The gradient comes back on every lane of the group.
__device__ __forceinline__ d3 groupLsGradient(const DevMesh& m, bool act, int c, const double* __restrict__ field,
                                              LsRows& ent, uint32_t& err) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, l = lane & 15, base = lane & 16, r = l >> 2, q = l & 3;
    const int32_t* st = nullptr;
    const int n = act ? stencilOf(m, c, st, err) + 1 : 0;  // the cell itself first
    const int nMax = max(n, __shfl_xor_sync(kAll, n, 16));
    // the two factors of the lane's sum: A[r][q] on and above the diagonal,
    // b[0..3] on lanes 4, 8, 12, 9
    const bool upper = r <= q;
    const int ia = upper ? r : (l == 9 ? 3 : r - 1), ib = upper ? q : 4;
    const d3 Cc = ld3(m.C, c);
    double acc = 0.0;
    for (int e0 = 0; e0 < nMax; e0 += 16) {
        const int e = e0 + l;
        if (e < n) {
            const int x = e ? st[e - 1] : c;
            const d3 dx = ld3(m.C, x) - Cc;
            ent[l][0] = 1.0;
            ent[l][1] = dx.x;
            ent[l][2] = dx.y;
            ent[l][3] = dx.z;
            ent[l][4] = field[x];
        }
        __syncwarp();
        const int top = min(16, nMax - e0);
#pragma unroll 4
        for (int j = 0; j < top; ++j)
            if (e0 + j < n) acc = acc + ent[j][ia] * ent[j][ib];
        __syncwarp();
    }
    double A = __shfl_sync(kAll, acc, base + (upper ? l : 4 * q + r));
    double b = __shfl_sync(kAll, acc, base + (r < 3 ? 4 * (r + 1) : 9));  // (the same along a row)
    bool singular = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int p = k;
        double best = fabs(__shfl_sync(kAll, A, base + 5 * k));
#pragma unroll
        for (int i = k + 1; i < 4; ++i) {
            const double v = fabs(__shfl_sync(kAll, A, base + 4 * i + k));
            if (v > best) {
                best = v;
                p = i;
            }
        }
        if (!(best > kVSMALL)) singular = true;
        if (k == 3) break;
        const int row = r == k ? p : (r == p ? k : r);
        A = __shfl_sync(kAll, A, base + 4 * row + q);
        b = __shfl_sync(kAll, b, base + 4 * row);
        const double f = __shfl_sync(kAll, A, base + 4 * r + k) / __shfl_sync(kAll, A, base + 5 * k);
        const double pivA = __shfl_sync(kAll, A, base + 4 * k + q), pivB = __shfl_sync(kAll, b, base + 4 * k);
        if (r > k) {
            A = A - f * pivA;
            b = b - f * pivB;
        }
    }
    const auto el = [&](int i, int j) { return __shfl_sync(kAll, A, base + 4 * i + j); };
    const auto rhs = [&](int i) { return __shfl_sync(kAll, b, base + 4 * i); };
    const double x3 = rhs(3) / el(3, 3);
    const double x2 = (rhs(2) - el(2, 3) * x3) / el(2, 2);
    const double x1 = ((rhs(1) - el(1, 2) * x2) - el(1, 3) * x3) / el(1, 1);
    return singular ? mk(0, 0, 0) : mk(x1, x2, x3);
}

}  // namespace simplic
