// inv_root6 (rans.cu, the default build): z^(-1/6) against long double over its
// whole range of exponents and just outside.  Each line: "exponent E worst W",
// the largest relative error of 2,000 mantissas times 2^E.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "rans_fast.cu"

__global__ void k_root(const double* z, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = ransk_fast::inv_root6(z[i]);
}

int main() {
    printf("long_double_digits %d\n", (int)__LDBL_MANT_DIG__);
    std::mt19937_64 rng(1);
    std::uniform_real_distribution<double> U(1.0, 2.0);
    const int per = 2000, lo = -64, hi = 112, n = per * (hi - lo);
    std::vector<double> z(n), y(n);
    for (int i = 0; i < n; ++i) z[i] = std::ldexp(i % per == 0 ? 1.0 : i % per == 1 ? std::nextafter(2.0, 0.0) : U(rng), lo + i / per);
    double *dz, *dy;
    cudaMalloc(&dz, n * sizeof(double));
    cudaMalloc(&dy, n * sizeof(double));
    cudaMemcpy(dz, z.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    k_root<<<(n + 255) / 256, 256>>>(dz, n, dy);
    cudaMemcpy(y.data(), dy, n * sizeof(double), cudaMemcpyDeviceToHost);
    for (int e = lo; e < hi; ++e) {
        long double worst = 0;
        for (int i = (e - lo) * per; i < (e - lo + 1) * per; ++i) {
            const long double x = powl(z[i], -1.0L / 6);
            worst = fmaxl(worst, fabsl(y[i] - x) / x);
        }
        printf("exponent %d worst %.4Le\n", e, worst);
    }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("cuda_error %s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
