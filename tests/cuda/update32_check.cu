// The FP32-flux mode's Runge-Kutta stages 1 and 2 (euler_o2.cuh, k_update)
// against their operations in order on the host, bit for bit:
//   e = fma(dtv, R, u)
//   stage 1: fma(1/4, e, 3/4 u0)    stage 2: fma(2/3, e, 1/3 u0)
// with the product of u0 rounded first.  The face fluxes are multiples of
// 2^-20 below 2^10, so that their sum R is exact.  Kinds: any state, states
// with mantissas about the ties of 3/4 u0, zeros and states at the ends of the
// exponent range.  Each line: "stage S kind K n N differ D".
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#define FV_KNS fast
#include "euler_o2.cuh"

using namespace fast;

template <typename T> static T* up(const std::vector<T>& v) {
    T* p;
    cudaMalloc(&p, sizeof(T) * v.size());
    cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    return p;
}

template <int STAGE> static void check(int kind) {
    const int n = 40000, F = 4 * n;
    std::mt19937_64 rng(11 + kind);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::vector<int> off(n + 1), cf(F);
    std::vector<float4> ff(F);
    std::vector<St> u(n), u0(n);
    std::vector<double> dtv(n);
    auto flux = [&] { return (float)std::ldexp(std::nearbyint(std::ldexp(U(rng), 22)), -20); };
    auto state = [&] {
        const double x = U(rng);
        if (kind == 0) return x * std::exp2(4 * U(rng));
        if (kind == 1) {
            const int low = (int)(rng() % 8);  // 3/4 of these is a tie or next to one
            return std::ldexp(x < 0 ? -1.0 : 1.0, (int)(rng() % 9) - 4) * (1.0 + std::ldexp((double)(((rng() % (1u << 20)) << 3) + low), -52));
        }
        const double end[8] = {0.0, -0.0, 4.9e-324, 1e-310, -2.3e-308, 2.3e-308, 1.7e308, -8.9e307};
        return end[rng() % 8];
    };
    auto fill = [&](St& s) { s.r = state(); s.ru = state(); s.rv = state(); s.E = state(); };
    for (int c = 0; c <= n; ++c) off[c] = 4 * c;
    for (int f = 0; f < F; ++f) {
        cf[f] = 2 * f + (int)(rng() & 1);
        ff[f] = make_float4(flux(), flux(), flux(), flux());
    }
    for (int c = 0; c < n; ++c) {
        fill(u[c]);
        fill(u0[c]);
        dtv[c] = std::exp2(-4 + 2 * U(rng));
    }
    fvgb::O2Args a{};
    a.m.n_cells = n;
    a.m.cf_off = up(off);
    a.m.cf = up(cf);
    a.ff = up(ff);
    a.U = up(u);
    a.U0 = up(u0);
    a.dtv = up(dtv);
    a.W = up(std::vector<float4>(n));
    a.cs = up(std::vector<float>(n));
    a.gamma = 1.4;
    a.gamma32 = 1.4f;
    a.ctl = up(std::vector<fvgb::StepCtl>(1));
    a.partials = up(std::vector<double>(4 * (n / 128 + 1)));
    a.hist = up(std::vector<double>(4));
    a.hist_cap = 1;
    // stage 1's first block folds the norms
    k_update<float, STAGE, 3, 2><<<(n + 127) / 128 + (STAGE == 1), 128>>>(a);
    std::vector<St> out(n);
    cudaMemcpy(out.data(), a.U, sizeof(St) * n, cudaMemcpyDeviceToHost);
    long differ = 0;
    for (int c = 0; c < n; ++c) {
        double R[4] = {0, 0, 0, 0};
        for (int e = off[c]; e < off[c + 1]; ++e) {
            const float* q = &ff[cf[e] >> 1].x;
            for (int k = 0; k < 4; ++k) R[k] += cf[e] & 1 ? -(double)q[k] : (double)q[k];
        }
        for (int k = 0; k < 4; ++k) {
            const double e = std::fma(dtv[c], R[k], (&u[c].r)[k]), x0 = (&u0[c].r)[k];
            const volatile double third = 1.0 / 3.0, p = STAGE == 1 ? 0.75 * x0 : third * x0;
            const double w = STAGE == 1 ? std::fma(0.25, e, p) : std::fma(2.0 / 3.0, e, p);
            differ += std::memcmp(&w, &(&out[c].r)[k], sizeof(double)) != 0;
        }
    }
    printf("stage %d kind %d n %d differ %ld\n", STAGE, kind, 4 * n, differ);
}

int main() {
    for (int kind = 0; kind < 3; ++kind) {
        check<1>(kind);
        check<2>(kind);
    }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("cuda_error %s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
