// fvconv::quotient (fpconv.cuh) against the IEEE division on pseudo-random
// numerators and divisors: mantissas of all kinds (random, near 1, near 2, few
// bits set), exponents in and out of the multiply-add path's range, zeros,
// infinities and NaN.  Prints "checked N mismatch M" (bit patterns; a NaN for
// a NaN counts as equal).
#include <cstdint>
#include <cstdio>

#include "fpconv.cuh"

__device__ unsigned long long g_bad;

__device__ __forceinline__ uint64_t mix(uint64_t x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull;
    return x ^ (x >> 33);
}
__device__ __forceinline__ double make(uint64_t r, int kind, unsigned e) {
    uint64_t m = r & 0x000fffffffffffffull;
    if (kind == 1) m &= 0xfull;                                   // just above a power of two
    if (kind == 2) m = 0x000fffffffffffffull - (m & 0xfull);      // just below the next
    if (kind == 3) m &= 0x000f0000f000f000ull;
    return __longlong_as_double((long long)(((uint64_t)e << 52) | m | (r & 0x8000000000000000ull)));
}

__global__ void check(uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = mix(2 * i + 1), b = mix(2 * i + 2), c = mix(a ^ b);
        const unsigned ex = (i & 7) ? 1023 - 40 + (unsigned)(c % 80) : (unsigned)(c % 2048);
        const double x = make(a, (int)(c >> 20) & 3, ex);
        const double d = fabs(make(b, (int)(c >> 24) & 3, 1023 - 60 + (unsigned)((c >> 32) % 120)));
        const double q = fvconv::quotient(x, make_double2(d, d > 1e-100 && d < 1e100 ? 1.0 / d : 0.0)), r = x / d;
        if (__double_as_longlong(q) != __double_as_longlong(r) && !(q != q && r != r)) atomicAdd(&g_bad, 1ull);
    }
}

int main() {
    const uint64_t n = 1ull << 28;
    check<<<152 * 8, 256>>>(n);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    unsigned long long bad;
    cudaMemcpyFromSymbol(&bad, g_bad, sizeof(bad));
    printf("checked %llu mismatch %llu\n", (unsigned long long)n, bad);
    return 0;
}
