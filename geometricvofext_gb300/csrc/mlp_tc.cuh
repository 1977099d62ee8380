// Tensor-core building blocks of the network kernels: shared-memory and
// instruction descriptors of tcgen05.mma kind::f16 (BF16 operands, FP32
// accumulator), bounded mbarrier waits, the activation function.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace simplic {

constexpr int kTileM = 128;
constexpr int kTileK = 64;
constexpr int kThreads = 128;
constexpr long long kWaitLimit = 1ll << 22;  // try_wait polls (a few seconds at most)

__device__ __forceinline__ uint32_t smemAddr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Byte offset of element (r, k) of a K-major tile with kTileK columns in the
// no-swizzle canonical layout.
__device__ __forceinline__ uint32_t coreOffset(int r, int k) {
    return uint32_t((r >> 3) * 1024 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// tcgen05 shared-memory matrix descriptor: start address, leading (K) and
// stride (row) byte offsets, version bits 46-48 = 0b001, no swizzle.
__device__ __forceinline__ uint64_t smemDesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= uint64_t((addr >> 4) & 0x3FFF);
    d |= uint64_t((lbo >> 4) & 0x3FFF) << 16;
    d |= uint64_t((sbo >> 4) & 0x3FFF) << 32;
    d |= uint64_t(1) << 46;
    return d;
}

// Instruction descriptor of kind::f16: D = F32, A = B = BF16, both K-major,
// M = 128, N = n.
__host__ __device__ constexpr uint32_t instrDesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(kTileM >> 4) << 24);
}

__device__ __forceinline__ void mbarInit(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
}

// Bounded wait for the completion of the phase with the given parity.
__device__ __forceinline__ bool mbarWait(uint64_t* bar, uint32_t parity) {
    const uint32_t a = smemAddr(bar);
    for (long long i = 0; i < kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// tanh form of GELU with the hardware tanh (tanh.approx.f32, relative error
// about 2^-11, far below the BF16 rounding of the activations); training
// and inference use the same function
__device__ __forceinline__ float tanhHw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float geluF(float z) {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    return 0.5f * z * (1.f + tanhHw(k0 * (z + k1 * z * z * z)));
}
__device__ __forceinline__ float geluGradF(float z) {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    const float u = k0 * (z + k1 * z * z * z);
    const float t = tanhHw(u);
    const float du = k0 * (1.f + 3.f * k1 * z * z);
    return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * du;
}

constexpr int kNetWidth = 128;
constexpr int kNetOut = 16;  // rows of the output layer evaluated (4 used)
constexpr uint32_t kNetSbo = (kNetWidth / 8) * 128;  // row-adjacent core matrices for K = 128

__device__ __forceinline__ uint32_t coreOffset128(int r, int k) {
    return uint32_t((r >> 3) * kNetSbo + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// D[128 x N] (+)= A[128 x 128] B[N x 128]^T at TMEM address tmem: A and B in the
// core-matrix layout of coreOffset128; one thread issues, the commit arrives
// at bar.
__device__ __forceinline__ void mma128(uint32_t tmem, uint32_t aAddr, uint32_t bAddr, int N, bool accumulate,
                                       uint64_t* bar) {
    const uint32_t idesc = instrDesc(N);
#pragma unroll
    for (int s = 0; s < kNetWidth / 16; ++s) {
        const uint64_t ad = smemDesc(aAddr + s * 256, 128, kNetSbo);
        const uint64_t bd = smemDesc(bAddr + s * 256, 128, kNetSbo);
        const uint32_t acc = s > 0 || accumulate ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smemAddr(bar))
                 : "memory");
}

// 32 accumulator columns of the warp's 32 rows
__device__ __forceinline__ void tmemLoad32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
        "%30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace simplic
