// Test helper: the FP64 engine's operations as multiply-adds (Fp) and its shared-denominator division
// (Divisor) against the plain IEEE operators, bit for bit, on pseudo-random operands generated on the
// device.  mode: 0 any significand, 1 near all ones, 2 near a power of two, 3 a signed zero.
#include <cstdint>
#include "fv2d_kernels.cuh"

namespace {
__device__ uint64_t mix(uint64_t z) {   // splitmix64 finaliser
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__device__ double operand(uint64_t r, int elo, int ehi, int mode) {
    const uint64_t s = mix(r), sign = (s >> 40) & 1ULL;
    uint64_t man = r & 0xFFFFFFFFFFFFFULL;
    if (mode == 1) man |= 0xFFFFFFFFFFF00ULL;
    if (mode == 2) man &= 0xFFULL;
    const uint64_t e = (uint64_t)(elo + (int)(s % (uint64_t)(ehi - elo + 1)) + 1023);
    return __longlong_as_double((long long)(mode == 3 ? sign << 63 : (sign << 63) | (e << 52) | man));
}
__device__ bool differ(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }

__global__ void k_check(uint64_t n, uint64_t seed, int elo, int ehi, int ma, int mb, unsigned long long* bad) {
    const fv2d::Fp f;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const double a = operand(mix(seed ^ (2 * i)), elo, ehi, ma), b = operand(mix(seed ^ (2 * i + 1)), elo, ehi, mb);
        if (differ(f.add(a, b), a + b) || differ(f.sub(a, b), a - b) || differ(f.sub(a, a), a - a)) atomicAdd(bad, 1ULL);
        if (differ(f.mul(a, b), a * b)) atomicAdd(bad + 1, 1ULL);
        if (mb != 3) {
            const fv2d::Divisor d(b, f);
            if (differ(d.div(a, f), a / b)) atomicAdd(bad + 2, 1ULL);
        }
    }
}
}  // namespace

extern "C" int arith_check(unsigned long long n, unsigned long long seed, int elo, int ehi, int ma, int mb,
                           unsigned long long* bad_out) {
    unsigned long long* bad;
    if (cudaMalloc(&bad, 24) != cudaSuccess) return 1;
    cudaMemset(bad, 0, 24);
    k_check<<<152 * 8, 256>>>(n, seed, elo, ehi, ma, mb, bad);
    const bool ok = cudaDeviceSynchronize() == cudaSuccess;
    cudaMemcpy(bad_out, bad, 24, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return ok ? 0 : 2;
}
