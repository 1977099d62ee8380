// Training of the learned-normal network: one gradient evaluation in four
// kernels, all matrix products on the 5th-generation tensor cores.
//
//   kTrainForward   the four layers on a 128-row tile per CTA: weights and
//                   activations stay in shared memory, the accumulator in
//                   TMEM; writes the pre-activations Z, the transposed
//                   activations H^T (the weight gradients' operand) and Y
//   kLoss           loss and its gradient for the four outputs, a warp per row
//   kTrainBackward  the chain dZ = (dZ W) gelu'(Z) on a 128-row tile per CTA;
//                   writes X^T and dZ^T of all layers
//   kWeightGrad     gW = dZ^T H of the four layers, K split over CTAs, and the
//                   bias gradients as row sums of dZ^T
//
// What bounds it: the work is 2.9 GFLOP and 50 MB a batch of 8192 (a few tens
// of microseconds on this part), but spread over 11 matrix products and
// some sixty elementwise launches of a Python loop it took 1.4 ms of launches
// and host work.  The layers of a row tile depend on nothing outside it, so
// they are fused, and the rest are four launches: 1.37 -> 0.12 ms for
// forward, loss (whose value the host reads) and backward on one GB300.
// Every mbarrier wait is bounded, as in mlp_kernels.cu.
#include "../../include/simplic_mlp.h"
#include "mlp_tc.cuh"

namespace simplic {
namespace {

constexpr int kTileBytes = kNetWidth * kNetWidth * 2;  // a 128 x 128 BF16 operand
constexpr int kFuseThreads = 256;  // two warps per 32 accumulator rows, half the columns each

// rows x 128 columns from memory (row stride ld elements) into the core-matrix
// layout, asynchronously; rows from validRows and columns from validCols on
// are zero.
__device__ __forceinline__ void stageTile(uint8_t* dst, const __nv_bfloat16* src, size_t ld, int validRows,
                                          int validCols, int tid, int threads) {
    for (int v = tid; v < kNetWidth * (kNetWidth / 8); v += threads) {
        const int r = v / (kNetWidth / 8), kc = (v % (kNetWidth / 8)) * 8;
        const bool ok = r < validRows && kc < validCols;
        const __nv_bfloat16* g = ok ? src + size_t(r) * ld + kc : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smemAddr(dst + coreOffset128(r, kc))),
                     "l"(g), "r"(ok ? 16u : 0u)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void stageWait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Barrier, TMEM and failure flag of a CTA.
struct TcState {
    uint64_t* bar;
    uint32_t tmem;
    int* failed;
    uint32_t phase;
};
__device__ __forceinline__ uint32_t tcBegin(uint64_t* bar, uint32_t* tmemBase, int* failed, int tid) {
    if (tid == 0) {
        mbarInit(bar, 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemBase)),
                     "r"(uint32_t(kNetWidth))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return *tmemBase;
}
__device__ __forceinline__ void tcEnd(TcState& t, unsigned* err, int tid) {
    if (*t.failed) {
        // give the MMAs still in flight a second bounded wait before the
        // tensor memory they write is released
        mbarWait(t.bar, t.phase ^ 1u);
        if (tid == 0) atomicOr(err, 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t.tmem), "r"(uint32_t(kNetWidth))
                     : "memory");
}
// Operands staged by all threads -> accumulator ready on all threads; false
// when the wait ran out.
__device__ __forceinline__ bool tcMultiply(TcState& t, const uint8_t* A, const uint8_t* B, bool accumulate, int tid) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        mma128(t.tmem, smemAddr(A), smemAddr(B), kNetWidth, accumulate, t.bar);
    }
    if (!mbarWait(t.bar, t.phase)) *t.failed = 1;
    t.phase ^= 1u;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return !*t.failed;
}

__global__ void __launch_bounds__(kFuseThreads) kTrainForward(const __nv_bfloat16* __restrict__ X, int M, int ld,
                                                              const __nv_bfloat16* __restrict__ W,
                                                              const float* __restrict__ bias, float* __restrict__ Z,
                                                              __nv_bfloat16* __restrict__ HT, float* __restrict__ Y,
                                                              unsigned* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sW = smem;  // four layers
    uint8_t* sA = smem + 4 * kTileBytes;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmemBase;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kTileM;
    stageTile(sA, X + size_t(m0) * kNetWidth, kNetWidth, M - m0, kNetWidth, tid, kFuseThreads);
    for (int l = 0; l < 4; ++l)
        stageTile(sW + l * kTileBytes, W + size_t(l) * kNetWidth * kNetWidth, kNetWidth, kNetWidth, kNetWidth, tid,
                  kFuseThreads);
    TcState t{&bar, tcBegin(&bar, &tmemBase, &failed, tid), &failed, 0};
    const int rloc = (warp & 3) * 32 + lane, row = m0 + rloc, half = (warp >> 2) * 64;
    for (int l = 0; l < 4; ++l) {
        if (l == 0) stageWait<3>();  // the tile and the first layer; the others come meanwhile
        else if (l == 1) stageWait<2>();
        else if (l == 2) stageWait<1>();
        else stageWait<0>();
        if (!tcMultiply(t, sA, sW + l * kTileBytes, false, tid)) break;
        const float* bl = bias + l * kNetWidth;
#pragma unroll 1
        for (int c0 = half; c0 < half + 64; c0 += 32) {
            uint32_t r[32];
            tmemLoad32(t.tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(c0), r);
            float* out = (l < 3 ? Z + (size_t(l) * ld + row) * kNetWidth : Y + size_t(row) * kNetWidth) + c0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float z[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) z[j] = __uint_as_float(r[8 * q + j]) + bl[c0 + 8 * q + j];
                if (row < M) {
                    *reinterpret_cast<float4*>(out + 8 * q) = make_float4(z[0], z[1], z[2], z[3]);
                    *reinterpret_cast<float4*>(out + 8 * q + 4) = make_float4(z[4], z[5], z[6], z[7]);
                }
                if (l < 3) {
                    // the next layer's input, in place (this layer's MMAs are complete)
                    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        h[j] = __float2bfloat16_rn(geluF(z[j]));
                        if (row < M) HT[(size_t(l) * kNetWidth + c0 + 8 * q + j) * ld + row] = h[j];
                    }
                    *reinterpret_cast<uint4*>(sA + coreOffset128(rloc, c0 + 8 * q)) = *reinterpret_cast<const uint4*>(h);
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    stageWait<0>();
    tcEnd(t, err, tid);
}

// scratch: X^T, then dZ^T of layers 0 .. 3 ([128][ld] each)
__global__ void __launch_bounds__(kFuseThreads) kTrainBackward(const __nv_bfloat16* __restrict__ X,
                                                               const float* __restrict__ dY, int M, int ld,
                                                               const __nv_bfloat16* __restrict__ WT,
                                                               const float* __restrict__ Z,
                                                               __nv_bfloat16* __restrict__ scratch,
                                                               float* __restrict__ gb, unsigned* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sW = smem;  // W^T of layers 3, 2, 1
    uint8_t* sA = smem + 3 * kTileBytes;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmemBase;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kTileM;
    for (int k = 0; k < 3; ++k)
        stageTile(sW + k * kTileBytes, WT + size_t(3 - k) * kNetWidth * kNetWidth, kNetWidth, kNetWidth, kNetWidth,
                  tid, kFuseThreads);
    const size_t plane = size_t(kNetWidth) * ld;
    const int rloc = (warp & 3) * 32 + lane, row = m0 + rloc, half = (warp >> 2) * 64;
    // dY as the first operand and, transposed, for the output layer's weight
    // gradient; X transposed for the first layer's
    for (int c = half; c < half + 64; c += 8) {
        __align__(16) __nv_bfloat16 h[8], x[8];
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (row < M) {
            const float4 p = *reinterpret_cast<const float4*>(dY + size_t(row) * kNetWidth + c);
            const float4 q = *reinterpret_cast<const float4*>(dY + size_t(row) * kNetWidth + c + 4);
            v[0] = p.x, v[1] = p.y, v[2] = p.z, v[3] = p.w, v[4] = q.x, v[5] = q.y, v[6] = q.z, v[7] = q.w;
            *reinterpret_cast<uint4*>(x) = *reinterpret_cast<const uint4*>(X + size_t(row) * kNetWidth + c);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            h[j] = __float2bfloat16_rn(v[j]);
            if (row < M) {
                scratch[size_t(c + j) * ld + row] = x[j];
                scratch[4 * plane + size_t(c + j) * ld + row] = h[j];
            }
        }
        *reinterpret_cast<uint4*>(sA + coreOffset128(rloc, c)) = *reinterpret_cast<const uint4*>(h);
    }
    // the output layer's bias gradient from the FP32 rows
    if (tid < kNetWidth) {
        float s = 0.f;
        const int end = min(M, m0 + kTileM);
        for (int r = m0; r < end; ++r) s += dY[size_t(r) * kNetWidth + tid];
        atomicAdd(gb + 3 * kNetWidth + tid, s);
    }
    TcState t{&bar, tcBegin(&bar, &tmemBase, &failed, tid), &failed, 0};
    for (int l = 2; l >= 0; --l) {
        if (l == 2) stageWait<2>();
        else if (l == 1) stageWait<1>();
        else stageWait<0>();
        if (!tcMultiply(t, sA, sW + (2 - l) * kTileBytes, false, tid)) break;
#pragma unroll 1
        for (int c0 = half; c0 < half + 64; c0 += 32) {
            uint32_t r[32];
            tmemLoad32(t.tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(c0), r);
            const float* z = Z + (size_t(l) * ld + row) * kNetWidth + c0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                __align__(16) __nv_bfloat16 h[8];
                float zz[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (row < M) {
                    const float4 p = *reinterpret_cast<const float4*>(z + 8 * q);
                    const float4 u = *reinterpret_cast<const float4*>(z + 8 * q + 4);
                    zz[0] = p.x, zz[1] = p.y, zz[2] = p.z, zz[3] = p.w, zz[4] = u.x, zz[5] = u.y, zz[6] = u.z, zz[7] = u.w;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    h[j] = __float2bfloat16_rn(__uint_as_float(r[8 * q + j]) * geluGradF(zz[j]));
                    if (row < M) scratch[size_t(1 + l) * plane + size_t(c0 + 8 * q + j) * ld + row] = h[j];
                }
                if (l > 0)
                    *reinterpret_cast<uint4*>(sA + coreOffset128(rloc, c0 + 8 * q)) = *reinterpret_cast<const uint4*>(h);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    stageWait<0>();
    tcEnd(t, err, tid);
}

// gW[l] += dZ_l^T H_(l-1) over a range of rows (H_(-1) = X), gb[l] += row sums
// of dZ_l^T (l < 3); blockIdx.y = l.  K in 128-wide stages, the next one in
// flight while one is multiplied.
__global__ void __launch_bounds__(kThreads) kWeightGrad(const __nv_bfloat16* __restrict__ scratch,
                                                        const __nv_bfloat16* __restrict__ HT, int M, int ld,
                                                        float* __restrict__ gW, float* __restrict__ gb,
                                                        unsigned* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];  // two stages of A, B
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmemBase;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = blockIdx.y;
    const size_t plane = size_t(kNetWidth) * ld;
    const __nv_bfloat16* A = scratch + size_t(1 + l) * plane;
    const __nv_bfloat16* B = l == 0 ? scratch : HT + size_t(l - 1) * plane;
    const int stages = (M + kNetWidth - 1) / kNetWidth;
    const int per = (stages + gridDim.x - 1) / gridDim.x;
    const int s0 = blockIdx.x * per, s1 = min(stages, s0 + per);
    if (s0 >= s1) return;
    const auto stage = [&](int s) {
        uint8_t* d = smem + ((s - s0) & 1) * 2 * kTileBytes;
        const int k0 = s * kNetWidth;
        stageTile(d, A + k0, ld, kNetWidth, M - k0, tid, kThreads);
        stageTile(d + kTileBytes, B + k0, ld, kNetWidth, M - k0, tid, kThreads);
    };
    stage(s0);
    TcState t{&bar, tcBegin(&bar, &tmemBase, &failed, tid), &failed, 0};
    float rowSum = 0.f;
    for (int s = s0; s < s1; ++s) {
        if (s + 1 < s1) {
            stage(s + 1);
            stageWait<2>();
        } else {
            stageWait<0>();
        }
        const uint8_t* a = smem + ((s - s0) & 1) * 2 * kTileBytes;
        const bool ok = tcMultiply(t, a, a + kTileBytes, s > s0, tid);
        if (!ok) break;
        if (l < 3) {
            for (int kc = 0; kc < kNetWidth; kc += 8) {
                const uint4 v = *reinterpret_cast<const uint4*>(a + coreOffset128(tid, kc));
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    rowSum += __uint_as_float(w[j] << 16) + __uint_as_float(w[j] & 0xffff0000u);
            }
        }
        __syncthreads();  // the stage is read before it is filled again
    }
    stageWait<0>();
    if (!failed) {
        if (l < 3) atomicAdd(gb + l * kNetWidth + tid, rowSum);
        float* g = gW + (size_t(l) * kNetWidth + warp * 32 + lane) * kNetWidth;
#pragma unroll 1
        for (int c0 = 0; c0 < kNetWidth; c0 += 32) {
            uint32_t r[32];
            tmemLoad32(t.tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0), r);
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g + c0 + j),
                             "f"(__uint_as_float(r[j])), "f"(__uint_as_float(r[j + 1])), "f"(__uint_as_float(r[j + 2])),
                             "f"(__uint_as_float(r[j + 3]))
                             : "memory");
        }
    }
    tcEnd(t, err, tid);
}

// loss = mean(1 - nn . T[0:3]) + dWeight mean((y3 - T3)^2) with nn = n / max(|n|,
// 1e-6), n = n_ls + y[0:3] (n_ls: features 124 .. 126), and dY = its gradient
// (zero beyond the four outputs).  A warp per row.
__global__ void __launch_bounds__(256) kLoss(const float* __restrict__ Y, const __nv_bfloat16* __restrict__ X,
                                             const float* __restrict__ T, int n, float dWeight,
                                             float* __restrict__ dY, double* __restrict__ loss) {
    __shared__ double part[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float inv = 1.f / float(n);
    double sum = 0.0;
    for (int r = blockIdx.x * 8 + warp; r < n; r += gridDim.x * 8) {
        const float4 y = *reinterpret_cast<const float4*>(Y + size_t(r) * kNetWidth);
        const float4 t = *reinterpret_cast<const float4*>(T + 4 * size_t(r));
        const uint2 q = *reinterpret_cast<const uint2*>(X + size_t(r) * kNetWidth + 124);
        const float vx = __uint_as_float(q.x << 16) + y.x, vy = __uint_as_float(q.x & 0xffff0000u) + y.y,
                    vz = __uint_as_float(q.y << 16) + y.z;
        const float len = sqrtf(vx * vx + vy * vy + vz * vz);
        const bool clamped = len < 1e-6f;
        const float c = 1.f / fmaxf(len, 1e-6f);
        const float nx = vx * c, ny = vy * c, nz = vz * c;
        const float cosA = nx * t.x + ny * t.y + nz * t.z, off = y.w - t.w;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane == 0) {
            // d(-nn . T) = -(T - (nn . T) nn) / |n|; below the clamp nn is linear in n
            const float s = clamped ? 0.f : cosA, k = -inv * c;
            g = make_float4(k * (t.x - s * nx), k * (t.y - s * ny), k * (t.z - s * nz), 2.f * dWeight * inv * off);
            sum += double(1.f - cosA) + double(dWeight) * double(off * off);
        }
        reinterpret_cast<float4*>(dY + size_t(r) * kNetWidth)[lane] = g;
    }
    if (lane == 0) part[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += part[w];
        atomicAdd(loss, s / double(n));
    }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace simplic

using namespace simplic;

extern "C" int simplic_mlp_train_forward(const void* X, int32_t M, int32_t ld, const void* W, const float* b, float* Z,
                                         void* HT, float* Y, uint32_t* err, void* stream) {
    if (!X || !W || !b || !Z || !HT || !Y || !err || M <= 0 || ld < M) return 1;
    if (!aligned16(X) || !aligned16(W) || !aligned16(Z) || !aligned16(Y)) return 1;
    constexpr int kBytes = 5 * kTileBytes;
    if (cudaFuncSetAttribute(kTrainForward, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) != cudaSuccess)
        return 2;
    kTrainForward<<<(M + kTileM - 1) / kTileM, kFuseThreads, kBytes, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(X), M, ld, static_cast<const __nv_bfloat16*>(W), b, Z,
        static_cast<__nv_bfloat16*>(HT), Y, err);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int simplic_mlp_train_backward(const void* X, const float* dY, int32_t M, int32_t ld, const void* WT,
                                          const float* Z, const void* HT, void* scratch, float* gW, float* gb,
                                          int32_t splitK, uint32_t* err, void* stream) {
    if (!X || !dY || !WT || !Z || !HT || !scratch || !gW || !gb || !err || M <= 0 || M % 64 != 0 || ld < M ||
        ld % 8 != 0)
        return 1;
    if (!aligned16(X) || !aligned16(dY) || !aligned16(WT) || !aligned16(Z) || !aligned16(HT) || !aligned16(scratch) ||
        !aligned16(gW))
        return 1;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    constexpr int kBytes = 4 * kTileBytes;
    if (cudaFuncSetAttribute(kTrainBackward, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) != cudaSuccess ||
        cudaFuncSetAttribute(kWeightGrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) != cudaSuccess)
        return 2;
    if (cudaMemsetAsync(gW, 0, sizeof(float) * 4 * kNetWidth * kNetWidth, st) != cudaSuccess ||
        cudaMemsetAsync(gb, 0, sizeof(float) * 4 * kNetWidth, st) != cudaSuccess)
        return 2;
    kTrainBackward<<<(M + kTileM - 1) / kTileM, kFuseThreads, kBytes, st>>>(
        static_cast<const __nv_bfloat16*>(X), dY, M, ld, static_cast<const __nv_bfloat16*>(WT), Z,
        static_cast<__nv_bfloat16*>(scratch), gb, err);
    // two stages or more per CTA where the batch allows it, at most 32 splits
    const int stages = (M + kNetWidth - 1) / kNetWidth;
    int splits = stages / 2 < 32 ? stages / 2 : 32;
    if (splits < splitK) splits = splitK;
    if (splits > stages) splits = stages;
    if (splits < 1) splits = 1;
    kWeightGrad<<<dim3(splits, 4), kThreads, kBytes, st>>>(static_cast<const __nv_bfloat16*>(scratch),
                                                           static_cast<const __nv_bfloat16*>(HT), M, ld, gW, gb, err);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int simplic_mlp_loss(const float* Y, const void* X, const float* T, int32_t n, float dWeight, float* dY,
                                double* loss, void* stream) {
    if (!Y || !X || !T || !dY || !loss || n <= 0) return 1;
    if (!aligned16(Y) || !aligned16(X) || !aligned16(T) || !aligned16(dY)) return 1;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(loss, 0, sizeof(double), st) != cudaSuccess) return 2;
    const int blocks = (n + 7) / 8;
    kLoss<<<blocks < 608 ? blocks : 608, 256, 0, st>>>(Y, static_cast<const __nv_bfloat16*>(X), T, n, dWeight, dY,
                                                       loss);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
