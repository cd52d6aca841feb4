// The fixed-point fluxes (fixed.cuh) and their FP64 forms, component by
// component, against long double on the host: errors relative to the face's
// scale (r q for the mass, r q^2 for the momenta, r q^3 for the energy, q the
// larger of speed and sound speed) and relative to the component itself.  Kinds:
//   smooth   any direction, Mach numbers up to 1.5
//   aligned  normals within 2^-20 of an axis, one velocity 2^-20 of the other
//   shear    the same normals, equal states but for that small velocity
// Each line: "<flux> <kind> component K n N taken T scale_fixed A scale_fp64 B self_fixed C self_fp64 D",
// root mean squares.
#include <cmath>
#include <cstdio>
#include <random>
#include <utility>
#include <vector>

#define FV_KNS fast
#include "euler_o2_fixed.cuh"

using namespace fast;
using LD = long double;
using V = V4<double>;

template <int FLUX>
__global__ void k_flux(const V* L, const V* R, const double4_32a* g, int n, fvfix::FluxConst k, double gam, V* fx, V* f64,
                       int* took) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V F = {0, 0, 0, 0};
    double lam;
    took[i] = fvfix::flux<FLUX, false, false>(L[i], R[i], 0.0, 0.0, fvfix::NoCons{}, fvfix::NoCons{}, g[i].x, g[i].y,
                                              g[i].z, k, F, true, lam);
    fx[i] = F;
    const V q = num_flux_p<double, FLUX>(L[i], R[i], g[i].x, g[i].y, gam, 1.0 / (gam - 1.0), 0.0, 0);
    f64[i] = {g[i].z * q.r, g[i].z * q.u, g[i].z * q.v, g[i].z * q.p};
}

static void flux_ld(int flux, const V& L, const V& R, const double4_32a& q, LD g, LD F[4]) {
    const V* w[2] = {&L, &R};
    const LD nx = q.x, ny = q.y;
    LD vn[2], c[2], E[2], U[2][4], f[2][4];
    for (int s = 0; s < 2; ++s) {
        const LD r = w[s]->r, u = w[s]->u, v = w[s]->v, p = w[s]->p;
        vn[s] = u * nx + v * ny;
        c[s] = sqrtl(g * p / r);
        E[s] = p / (g - 1) + r * (u * u + v * v) / 2;
        const LD a[4] = {r, r * u, r * v, E[s]}, b[4] = {r * vn[s], r * u * vn[s] + p * nx, r * v * vn[s] + p * ny, (E[s] + p) * vn[s]};
        for (int k = 0; k < 4; ++k) { U[s][k] = a[k]; f[s][k] = b[k]; }
    }
    if (flux == 0) {
        const LD S = fmaxl(fabsl(vn[0]) + c[0], fabsl(vn[1]) + c[1]);
        for (int k = 0; k < 4; ++k) F[k] = q.z * ((f[0][k] + f[1][k]) / 2 - S / 2 * (U[1][k] - U[0][k]));
        return;
    }
    const LD SL = fminl(vn[0] - c[0], vn[1] - c[1]), SR = fmaxl(vn[0] + c[0], vn[1] + c[1]);
    const LD mL = (LD)L.r * (SL - vn[0]), mR = (LD)R.r * (SR - vn[1]);
    const LD Ss = ((LD)R.p - L.p + mL * vn[0] - mR * vn[1]) / (mL - mR);
    const int s = SL >= 0 ? 0 : (SR <= 0 ? 1 : (Ss >= 0 ? 0 : 1));
    if (SL >= 0 || SR <= 0) {
        for (int k = 0; k < 4; ++k) F[k] = q.z * f[s][k];
        return;
    }
    // star state: the tangential velocity stays, the normal one becomes S*
    const LD S = s ? SR : SL, r = w[s]->r, d = S - vn[s], fac = r * d / (S - Ss), dv = Ss - vn[s];
    const LD Us[4] = {fac, fac * (w[s]->u + dv * nx), fac * (w[s]->v + dv * ny), fac * (E[s] / r + dv * (Ss + w[s]->p / (r * d)))};
    for (int k = 0; k < 4; ++k) F[k] = q.z * (f[s][k] + S * (Us[k] - U[s][k]));
}

template <typename T> static T* up(const std::vector<T>& v) {
    T* p;
    cudaMalloc(&p, sizeof(T) * v.size());
    cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    return p;
}

template <int FLUX> static void check(const char* name, int kind) {
    const char* kinds[3] = {"smooth", "aligned", "shear"};
    const int n = 1 << 15;
    const double gam = 1.4;
    std::mt19937_64 rng(29 + kind);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::vector<V> L(n), R(n);
    std::vector<double4_32a> g(n);
    for (int i = 0; i < n; ++i) {
        const double M = 1.5 * U(rng), al = 6.2831853 * U(rng), th = 6.2831853 * U(rng), e = 0.02, small = std::ldexp(1.0, -20);
        L[i] = {1 + 0.5 * U(rng), M * cos(al), M * sin(al), (1 + 0.5 * U(rng)) / gam};
        R[i] = {L[i].r * (1 + e * (U(rng) - 0.5)), L[i].u + e * (U(rng) - 0.5), L[i].v + e * (U(rng) - 0.5),
                L[i].p * (1 + e * (U(rng) - 0.5))};
        double nx = cos(th), ny = sin(th);
        if (kind > 0) {
            if (kind == 2) R[i] = L[i];
            L[i].v = L[i].u * small * (U(rng) - 0.5);
            R[i].v = R[i].u * small * (U(rng) - 0.5);
            nx = small * (U(rng) - 0.5);
            ny = sqrt(1 - nx * nx);
            if (kind == 1 && (i & 1)) std::swap(nx, ny);
        }
        g[i].x = nx; g[i].y = ny; g[i].z = exp2(10 * U(rng) - 8); g[i].w = 0;
    }
    fvfix::FluxConst k{llrint(ldexp(gam, 60)), llrint(ldexp(0.25 / (gam - 1.0), 60)), (float)gam};
    V *fx, *f64;
    int* tk;
    cudaMalloc(&fx, sizeof(V) * n); cudaMalloc(&f64, sizeof(V) * n); cudaMalloc(&tk, sizeof(int) * n);
    k_flux<FLUX><<<n / 256, 256>>>(up(L), up(R), up(g), n, k, gam, fx, f64, tk);
    std::vector<V> a(n), b(n);
    std::vector<int> took(n);
    cudaMemcpy(a.data(), fx, sizeof(V) * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(b.data(), f64, sizeof(V) * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(took.data(), tk, sizeof(int) * n, cudaMemcpyDeviceToHost);
    LD s[4][4] = {};
    long t = 0;
    for (int i = 0; i < n; ++i) {
        if (!took[i]) continue;
        ++t;
        LD F[4];
        flux_ld(FLUX, L[i], R[i], g[i], gam, F);
        const LD r = fmax(L[i].r, R[i].r), c = sqrtl(gam * fmax(L[i].p / L[i].r, R[i].p / R[i].r));
        const LD q = fmaxl(c, hypotl(L[i].u, L[i].v)), sc[4] = {r * q, r * q * q, r * q * q, r * q * q * q};
        for (int j = 0; j < 4; ++j) {
            const LD e0 = (&a[i].r)[j] - F[j], e1 = (&b[i].r)[j] - F[j], x = sc[j] * g[i].z;
            s[j][0] += e0 * e0 / (x * x); s[j][1] += e1 * e1 / (x * x);
            s[j][2] += e0 * e0 / (F[j] * F[j]); s[j][3] += e1 * e1 / (F[j] * F[j]);
        }
    }
    for (int j = 0; j < 4; ++j)
        printf("%s %s component %d n %d taken %ld scale_fixed %.3Le scale_fp64 %.3Le self_fixed %.3Le self_fp64 %.3Le\n", name,
               kinds[kind], j, n, t, sqrtl(s[j][0] / t), sqrtl(s[j][1] / t), sqrtl(s[j][2] / t), sqrtl(s[j][3] / t));
}

int main() {
    printf("long_double_digits %d\n", (int)__LDBL_MANT_DIG__);
    for (int kind = 0; kind < 3; ++kind) {
        check<0>("rusanov", kind);
        check<1>("hllc", kind);
    }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("cuda_error %s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
