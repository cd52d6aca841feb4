// block_min_step (euler_o1.cuh): the smallest cfl * len / lam of a block's faces,
// against the FP64 minimum over all of them.  Kinds: like sizes; speeds and
// lengths across FP32's range and beyond, small lengths with small speeds beside
// them; ties within 2^-20; zeros, infinities and NaN among them; dead threads.
// Each line: "kind K blocks B worst W" with W the largest relative difference.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#define FV_KNS fast
#include "euler_o1.cuh"

__global__ void k_min(const double* lam, const double* len, const int* live, double cfl, unsigned long long* slot) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    fast::block_min_step(live[i] != 0, lam[i], len[i], cfl, slot + blockIdx.x);
}

template <typename T> static T* up(const std::vector<T>& v) {
    T* p;
    cudaMalloc(&p, sizeof(T) * v.size());
    cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    return p;
}

int main() {
    for (int bs : {128, 256})
        for (int kind = 0; kind < 5; ++kind) {
            const int nb = 2000, n = nb * bs;
            std::mt19937_64 rng(3 + kind);
            std::uniform_real_distribution<double> U(0.0, 1.0);
            std::vector<double> lam(n), len(n), want(nb, DBL_MAX);
            std::vector<int> live(n, 1);
            const double cfl = 0.7, big = DBL_MAX;
            unsigned long long big_bits;
            std::memcpy(&big_bits, &big, 8);
            std::vector<unsigned long long> slot(nb, big_bits);
            for (int i = 0; i < n; ++i) {
                lam[i] = 0.5 + U(rng);
                len[i] = 0.01 * (0.5 + U(rng));
                if (kind == 1) {
                    // lengths from 2^-134 to 2^-120 of speeds that make the longer ones' rates the larger; every
                    // third block a wide spread of both
                    const double e = -134 + 14 * U(rng);
                    len[i] = std::exp2(e);
                    lam[i] = std::exp2(1.5 * (e + 120) + U(rng));
                    if (i / bs % 3 == 0) { lam[i] = std::exp2(400 * U(rng) - 200); len[i] = std::exp2(400 * U(rng) - 200); }
                }
                if (kind == 2) { lam[i] = 1.0 + std::ldexp(U(rng), -20); len[i] = 0.01 * (1.0 + std::ldexp(U(rng), -20)); }
                if (kind == 3) {
                    const double odd[5] = {INFINITY, NAN, 0.0, 1e-310, DBL_MAX};
                    const int r = (int)(rng() % 400);
                    if (r < 5) lam[i] = odd[r];
                    else if (r < 10 && r != 5 && r != 6) len[i] = odd[r - 5];
                }
                if (kind == 4) live[i] = (int)(rng() % 16 == 0);
                if (!live[i]) continue;
                const double dt = cfl * len[i] / lam[i];
                if (dt >= 0.0) want[i / bs] = std::fmin(want[i / bs], dt);
            }
            unsigned long long* d = up(slot);
            k_min<<<nb, bs>>>(up(lam), up(len), up(live), cfl, d);
            cudaMemcpy(slot.data(), d, sizeof(slot[0]) * nb, cudaMemcpyDeviceToHost);
            double worst = 0.0;
            for (int b = 0; b < nb; ++b) {
                double x;
                std::memcpy(&x, &slot[b], 8);
                if (x == want[b]) continue;
                worst = std::fmax(worst, std::fabs(x - want[b]) / std::fmax(want[b], DBL_MIN));
            }
            printf("kind %d blocks %d worst %.3e\n", kind, nb, worst);
        }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("cuda_error %s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
