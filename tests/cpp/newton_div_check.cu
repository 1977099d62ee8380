// Both forms of divByRecip against the division, host or device instantiation:
//   newton_div_check host|gpu N SEED -> mismatches of quotNewton, of
//   divByRecip<false> and of divByRecip<true> over N random pairs (significands
//   of several kinds, exponents to the ends of the range).
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "simplic_device.cuh"

using namespace simplic;

using u64 = unsigned long long;

__host__ __device__ u64 mix(u64 x) {  // splitmix64's finaliser
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
__host__ __device__ double fromBits(u64 b) {
    double x;
    memcpy(&x, &b, 8);
    return x;
}
__host__ __device__ u64 significand(u64 r) {
    const u64 f = (r >> 12) & 0xfffffffffffffull;
    switch (r & 7) {
        case 0: return f % 8;
        case 1: return 0xfffffffffffffull - f % 8;
        case 2: return (f & 0xff) << ((f >> 8) % 45);
        case 3: return 0xfffffffffffffull ^ ((f & 0xff) << ((f >> 8) % 45));
        default: return f;
    }
}
__host__ __device__ bool differ(double a, double b) { return memcmp(&a, &b, 8) != 0 && !(a != a && b != b); }

// counts of the three forms for pair i
__host__ __device__ void check(u64 i, u64 seed, u64* bad) {
    const u64 r = mix(seed + 4 * i), ra = mix(seed + 4 * i + 1), rb = mix(seed + 4 * i + 2);
    int ea = 1 + int((r >> 8) % 2046), eb = 1 + int((r >> 20) % 2046);
    switch (r & 7) {
        case 0: case 1: case 2: ea = 993 + int((r >> 8) % 60), eb = 993 + int((r >> 20) % 60); break;
        case 3: ea = 64 + int((r >> 8) % 8); break;                                // the ends of the range of a,
        case 4: ea = 1973 + int((r >> 8) % 8); break;
        case 5: eb = 64 + int((r >> 20) % 900), ea = eb + 950 + int((r >> 8) % 8); break;  // of the quotient
        case 6: eb = 1030 + int((r >> 20) % 900), ea = eb - 959 + int((r >> 8) % 8); break;
        default: break;
    }
    const double a = fromBits(significand(ra) | (u64(ea) << 52) | (r & (1ull << 63)));
    const double b = fromBits(significand(rb) | (u64(eb) << 52) | ((r << 1) & (1ull << 63)));
    const double want = a / b, y = 1.0 / b;
    if (ea >= 64 && ea <= 1980 && eb >= 64 && eb <= 1980 && ea - eb >= 64 - 1023 && ea - eb <= 1980 - 1023)
        bad[0] += differ(quotNewton(a, b, y), want);
    bad[1] += differ(divByRecip<false>(a, b, y), want);
    bad[2] += differ(divByRecip<true>(a, b, y), want);
}

__global__ void kCheck(long long n, u64 seed, u64* bad) {
    u64 mine[3] = {0, 0, 0};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        check(u64(i), seed, mine);
    for (int k = 0; k < 3; ++k)
        if (mine[k]) atomicAdd(bad + k, mine[k]);
}

int main(int argc, char** argv) {
    if (argc < 4) return 2;
    const long long n = std::atoll(argv[2]);
    const u64 seed = mix(std::strtoull(argv[3], nullptr, 10) + 1);
    u64 bad[3] = {0, 0, 0};
    if (argv[1][0] == 'g') {
        u64* d = nullptr;
        if (cudaMalloc(&d, sizeof bad) != cudaSuccess || cudaMemset(d, 0, sizeof bad) != cudaSuccess) return 3;
        kCheck<<<1024, 256>>>(n, seed, d);
        if (cudaMemcpy(bad, d, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess) return 4;
        cudaFree(d);
    } else {
        for (long long i = 0; i < n; ++i) check(u64(i), seed, bad);
    }
    std::printf("%llu %llu %llu\n", bad[0], bad[1], bad[2]);
}
