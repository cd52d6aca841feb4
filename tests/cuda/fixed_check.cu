// Checks the fixed-point passes of the second-order path (fixed.cuh,
// euler_o2_fixed.cuh) and their FP64 forms against long double on the host
// (128-bit on the Arm machines that carry the GPU).
//
//   flux: random face states of several kinds, Rusanov and HLLC
//   first: the same states as the first-order kernel's faces, conserved
//   grad: random "cells" of 3 to 18 faces (18 takes the FP64 form), random weights,
//         offsets and neighbours, both limiters
// Each line: "<what> n N taken T rms_fixed A rms_fp64 B max_fixed C max_fp64 D",
// errors relative to the face's (cell's) own scale; T counts those that the
// fixed-point form took.  "refused" lines count states it must refuse and did not.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#define FV_KNS fast
#include "euler_o1p.cuh"
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

// the first-order kernel's face, from conserved states
template <int FLUX>
__global__ void k_first(const St* L, const St* R, const double4_32a* g, int n, fvfix::FluxConst k, double gam, V* fx, V* f64,
                        int* took) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Prim PL = prim_of(L[i], gam), PR = prim_of(R[i], gam);
    V F;
    double lam;
    took[i] = fvfix::flux<FLUX, true, false>(fvfix::State{L[i].r, PL.u, PL.v, PL.p}, fvfix::State{R[i].r, PR.u, PR.v, PR.p},
                                             PL.c, PR.c, L[i], R[i], g[i].x, g[i].y, g[i].z, k,
                                             reinterpret_cast<fvfix::State&>(F), true, lam);
    fx[i] = F;
    const St q = g[i].z * num_flux_p<FLUX>(L[i], PL, R[i], PR, g[i].x, g[i].y, gam, 0.0, 0);
    f64[i] = {q.r, q.ru, q.rv, q.E};
}

struct VL { LD r, u, v, p; };
static VL wide(const V& w) { return {w.r, w.u, w.v, w.p}; }
static VL wide(const St& s, LD g) {
    const LD r = s.r, u = s.ru / r, v = s.rv / r;
    return {r, u, v, (g - 1) * (s.E - r * (u * u + v * v) / 2)};
}

static void flux_ld(int flux, const VL& L, const VL& R, LD nx, LD ny, LD ar, LD g, LD F[4]) {
    const VL* w[2] = {&L, &R};
    LD vn[2], vt[2], c[2], E[2], U[2][4], f[2][4];
    for (int s = 0; s < 2; ++s) {
        const LD r = w[s]->r, u = w[s]->u, v = w[s]->v, p = w[s]->p;
        vn[s] = u * nx + v * ny; vt[s] = v * nx - u * ny;
        c[s] = sqrtl(g * p / r);
        E[s] = p / (g - 1) + r * (u * u + v * v) / 2;
        const LD a[4] = {r, r * u, r * v, E[s]}, b[4] = {r * vn[s], r * u * vn[s] + p * nx, r * v * vn[s] + p * ny, (E[s] + p) * vn[s]};
        memcpy(U[s], a, sizeof(a)); memcpy(f[s], b, sizeof(b));
    }
    if (flux == 0) {
        const LD S = fmaxl(fabsl(vn[0]) + c[0], fabsl(vn[1]) + c[1]);
        for (int k = 0; k < 4; ++k) F[k] = ar * ((f[0][k] + f[1][k]) / 2 - S / 2 * (U[1][k] - U[0][k]));
        return;
    }
    const LD SL = fminl(vn[0] - c[0], vn[1] - c[1]), SR = fmaxl(vn[0] + c[0], vn[1] + c[1]);
    const LD mL = L.r * (SL - vn[0]), mR = R.r * (SR - vn[1]);
    const LD Ss = (R.p - L.p + mL * vn[0] - mR * vn[1]) / (mL - mR);
    const int s = SL >= 0 ? 0 : (SR <= 0 ? 1 : (Ss >= 0 ? 0 : 1));
    if (SL >= 0 || SR <= 0) {
        for (int k = 0; k < 4; ++k) F[k] = ar * f[s][k];
        return;
    }
    const LD S = s ? SR : SL, r = w[s]->r, p = w[s]->p, fac = r * (S - vn[s]) / (S - Ss);
    const LD Us[4] = {fac, fac * (Ss * nx - vt[s] * ny), fac * (Ss * ny + vt[s] * nx),
                      fac * (E[s] / r + (Ss - vn[s]) * (Ss + p / (r * (S - vn[s]))))};
    for (int k = 0; k < 4; ++k) F[k] = ar * (f[s][k] + S * (Us[k] - U[s][k]));
}

struct Err {
    LD s[2] = {0, 0}, m[2] = {0, 0};
    long n = 0;
    void add(int i, LD e) { s[i] += e * e; m[i] = fmaxl(m[i], e); }
    void print(const char* what, long total, long took) const {
        printf("%s n %ld taken %ld rms_fixed %.4Le rms_fp64 %.4Le max_fixed %.4Le max_fp64 %.4Le\n", what, total, took,
               sqrtl(s[0] / (n ? n : 1)), sqrtl(s[1] / (n ? n : 1)), m[0], m[1]);
    }
};

template <typename T> static T* up(const std::vector<T>& v) {
    T* p;
    cudaMalloc(&p, sizeof(T) * v.size());
    cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    return p;
}
template <typename T> static std::vector<T> down(const T* p, size_t n) {
    std::vector<T> v(n);
    cudaMemcpy(v.data(), p, sizeof(T) * n, cudaMemcpyDeviceToHost);
    return v;
}

template <int FLUX> static void check_flux(const char* name, int kind, double gam, bool first) {
    const int n = 1 << 15;
    std::mt19937_64 rng(17 + kind);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::vector<V> L(n), R(n);
    std::vector<double4_32a> g(n);
    for (int i = 0; i < n; ++i) {
        // kind 0 smooth, any Mach number up to 3; 1 jumps; 2 low Mach; 3 aligned with the axes, one velocity zero;
        // 4 states that have to be refused
        const double sr = kind == 0 ? ldexp(1.0, (int)(60 * U(rng)) - 30) : 1.0, sp = kind == 0 ? ldexp(1.0, (int)(60 * U(rng)) - 30) : 1.0;
        const double c = sqrt(gam * sp / sr), M = kind == 2 ? 0.02 : 3.0 * U(rng), al = 6.2831853 * U(rng), th = 6.2831853 * U(rng);
        const double e = kind == 1 ? 1.0 : 0.02;
        L[i] = {sr * (1 + 0.5 * U(rng)), M * c * cos(al), M * c * sin(al), sp * (1 + 0.5 * U(rng))};
        R[i] = {L[i].r * (1 + e * (U(rng) - 0.5)), L[i].u + e * c * (U(rng) - 0.5), L[i].v + e * c * (U(rng) - 0.5),
                L[i].p * (1 + e * (U(rng) - 0.5))};
        if (kind == 1) { R[i].r *= exp2(4 * U(rng) - 2); R[i].p *= exp2(4 * U(rng) - 2); }
        double nx = cos(th), ny = sin(th);
        if (kind == 3) {
            nx = i & 1; ny = 1 - nx;
            if (i & 2) L[i].u = R[i].u = 0.0; else L[i].v = R[i].v = 0.0;
        }
        if (kind == 4) {
            const double bad[8] = {0.0, -1.0, INFINITY, NAN, 1e-310, -0.0, 1e300, 1e-300};
            const double x = bad[i & 7];
            switch ((i >> 3) % 4) {
                case 0: L[i].r = x; break;
                case 1: R[i].p = x; break;
                case 2: if (std::isfinite(x) && fabs(x) < 1e100) L[i].p = x; else L[i].u = x; break;
                default: R[i].r = x;
            }
        }
        g[i].x = nx; g[i].y = ny; g[i].z = exp2(10 * U(rng) - 8); g[i].w = 0;
    }
    fvfix::FluxConst k{llrint(ldexp(gam, 60)), llrint(ldexp(0.25 / (gam - 1.0), 60)), (float)gam};
    V *fx, *f64;
    int* tk;
    cudaMalloc(&fx, sizeof(V) * n); cudaMalloc(&f64, sizeof(V) * n); cudaMalloc(&tk, sizeof(int) * n);
    std::vector<St> UL(n), UR(n);
    for (int i = 0; i < n; ++i)
        for (int q = 0; q < 2; ++q) {
            const V& w = q ? R[i] : L[i];
            St& u = q ? UR[i] : UL[i];
            u.r = w.r; u.ru = w.r * w.u; u.rv = w.r * w.v;
            u.E = w.p / (gam - 1.0) + 0.5 * w.r * (w.u * w.u + w.v * w.v);
        }
    if (first) k_first<FLUX><<<n / 256, 256>>>(up(UL), up(UR), up(g), n, k, gam, fx, f64, tk);
    else k_flux<FLUX><<<n / 256, 256>>>(up(L), up(R), up(g), n, k, gam, fx, f64, tk);
    auto a = down(fx, n), b = down(f64, n);
    auto took = down(tk, n);
    Err err;
    long t = 0;
    for (int i = 0; i < n; ++i) t += took[i];
    if (kind == 4) {
        printf("%s refused %d accepted %ld\n", name, n, t);
        return;
    }
    for (int i = 0; i < n; ++i) {
        if (!took[i]) continue;
        LD F[4];
        flux_ld(FLUX, first ? wide(UL[i], gam) : wide(L[i]), first ? wide(UR[i], gam) : wide(R[i]), g[i].x, g[i].y,
                g[i].z, gam, F);
        const LD r = fmax(L[i].r, R[i].r), c = sqrt(gam * fmax(L[i].p / L[i].r, R[i].p / R[i].r));
        const LD q = fmaxl(c, hypot(L[i].u, L[i].v)), sc[4] = {r * q, r * q * q, r * q * q, r * q * q * q};
        const double *x = &a[i].r, *y = &b[i].r;
        LD e0 = 0, e1 = 0;
        for (int j = 0; j < 4; ++j) {
            e0 = fmaxl(e0, fabsl(x[j] - F[j]) / (sc[j] * (LD)g[i].z));
            e1 = fmaxl(e1, fabsl(y[j] - F[j]) / (sc[j] * (LD)g[i].z));
        }
        err.add(0, e0); err.add(1, e1);
        ++err.n;
    }
    err.print(name, n, t);
}

template <int LIM> static void check_grad(const char* name, int kind) {
    const int n = 1 << 13;
    std::mt19937_64 rng(5 + kind);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::vector<int> off(n + 1, 0), nb;
    std::vector<double2> w, r;
    std::vector<St> W(n);
    std::vector<double> eps(n);
    // kind 0 smooth, 1 jumps, 2 stretched cells, 3 velocities of either sign about zero, scales 2^-40 .. 2^40
    for (int i = 0; i < n; ++i) {
        const double d = kind == 1 ? 1.0 : 0.01;
        W[i].r = 1 + d * U(rng);
        W[i].ru = 0.5 + d * U(rng);
        W[i].rv = (kind == 3 ? 1.0 : 0.1) * (U(rng) - 0.5);
        W[i].E = 0.7 * (1 + d * U(rng));
        if (kind == 3) { W[i].ru = 1e-3 * (U(rng) - 0.5); W[i].r *= 1099511627776.0; W[i].E *= 9.094947017729282e-13; }
    }
    for (int i = 0; i < n; ++i) {
        const int f = i % 16 == 15 ? 18 : 3 + i % 16;
        const double h = exp2(-10 * U(rng)), as = kind == 2 ? exp2(10 * U(rng)) : 1.0, al = 6.2831853 * U(rng);
        eps[i] = pow(5 * h * sqrt(as), 3) * (kind == 1 ? 1e-6 : 1.0);
        LD m00 = 0, m01 = 0, m11 = 0;
        std::vector<double2> dx(f);
        for (int j = 0; j < f; ++j) {
            const double t = 6.2831853 * (j + 0.3 * U(rng)) / f, x = as * h * cos(t), y = h * sin(t);
            dx[j] = make_double2(x * cos(al) - y * sin(al), x * sin(al) + y * cos(al));
            const LD q = 1 / ((LD)dx[j].x * dx[j].x + (LD)dx[j].y * dx[j].y);
            m00 += q * dx[j].x * dx[j].x; m01 += q * dx[j].x * dx[j].y; m11 += q * dx[j].y * dx[j].y;
        }
        const LD det = m00 * m11 - m01 * m01;
        for (int j = 0; j < f; ++j) {
            const LD q = 1 / ((LD)dx[j].x * dx[j].x + (LD)dx[j].y * dx[j].y);
            w.push_back(make_double2((double)(q * (m11 * dx[j].x - m01 * dx[j].y) / det), (double)(q * (m00 * dx[j].y - m01 * dx[j].x) / det)));
            r.push_back(make_double2(0.5 * dx[j].x, 0.5 * dx[j].y));
            nb.push_back((int)(U(rng) * n) % n);
        }
        off[i + 1] = (int)nb.size();
    }
    const int E = (int)nb.size();
    std::vector<double2> sum(n);
    for (int i = 0; i < n; ++i) {
        sum[i] = make_double2(0, 0);
        for (int e = off[i]; e < off[i + 1]; ++e) { sum[i].x += w[e].x; sum[i].y += w[e].y; }
    }
    fvgb::O2Args a{};
    a.m.n_cells = n;
    a.m.cf_off = up(off);
    a.cnb = up(nb);
    a.lsq = up(w); a.lsq_sum = up(sum); a.erf = up(r); a.eps2 = up(eps);
    a.W = up(W);
    a.gamma = 1.4;
    int4 *xa, *xr;
    int* xs;
    cudaMalloc(&xa, sizeof(int4) * E); cudaMalloc(&xr, sizeof(int4) * E); cudaMalloc(&xs, sizeof(int) * n);
    k_fix_geom<<<(n + 255) / 256, 256>>>(a, xa, xr, xs);
    a.fxa = xa; a.fxr = xr; a.fxs = xs;
    St *fx, *f64;
    cudaMalloc(&fx, sizeof(St) * E); cudaMalloc(&f64, sizeof(St) * E);
    a.wf = fx;
    k_grad_fx<LIM><<<4 * n / 256, 256>>>(a);
    a.wf = f64;
    k_grad<double, 0, LIM><<<n / 256, 256>>>(a);
    auto A = down(fx, E), B = down(f64, E);
    auto S = down(xs, n);
    Err err;
    long t = 0;
    for (int i = 0; i < n; ++i) {
        if (S[i] < 0) continue;
        ++t;
        const double* wc = &W[i].r;
        LD e0 = 0, e1 = 0;
        std::vector<LD> out(4 * (off[i + 1] - off[i]));
        for (int k = 0; k < 4; ++k) {
            LD gx = 0, gy = 0, hi = 0, lo = 0, amp = 0, psi = 1, big = fabsl(wc[k]);
            for (int e = off[i]; e < off[i + 1]; ++e) {
                const LD v = (&W[nb[e]].r)[k], d = v - wc[k];
                gx += w[e].x * d; gy += w[e].y * d;
                hi = fmaxl(hi, d); lo = fminl(lo, d); big = fmaxl(big, fabsl(v));
            }
            for (int e = off[i]; e < off[i + 1]; ++e) {
                const LD y = gx * r[e].x + gy * r[e].y, d1 = y > 0 ? hi : -lo, ay = fabsl(y), ep = eps[i];
                LD sx = 0, sy = 0;
                for (int q = off[i]; q < off[i + 1]; ++q) { sx += fabs(w[q].x); sy += fabs(w[q].y); }
                amp = fmaxl(amp, sx * fabs(r[e].x) + sy * fabs(r[e].y));
                if (ay > 0) psi = fminl(psi, LIM == 1 ? d1 / ay : (d1 * d1 + ep + 2 * d1 * ay) / (d1 * d1 + 2 * ay * ay + d1 * ay + ep));
            }
            for (int e = off[i]; e < off[i + 1]; ++e) out[4 * (e - off[i]) + k] = wc[k] + psi * (gx * r[e].x + gy * r[e].y);
            for (int e = off[i]; e < off[i + 1]; ++e) {
                const LD x = out[4 * (e - off[i]) + k];
                // relative to the largest value, and to how much the weights amplify its rounding
                const LD sc = big * fmaxl(1, amp);
                e0 = fmaxl(e0, fabsl((&A[e].r)[k] - x) / sc);
                e1 = fmaxl(e1, fabsl((&B[e].r)[k] - x) / sc);
            }
        }
        bool positive = true;
        for (int e = 0; e < off[i + 1] - off[i]; ++e) positive = positive && out[4 * e] > 0 && out[4 * e + 3] > 0;
        if (!positive) continue;
        err.add(0, e0); err.add(1, e1);
        ++err.n;
    }
    err.print(name, n, t);
}

int main() {
    for (double g : {1.2, 1.4, 5.0 / 3.0, 3.0}) {
        char s[64];
        const char* kinds[5] = {"smooth", "jumps", "lowmach", "aligned", "outside"};
        for (int k = 0; k < 5; ++k) {
            for (int first = 0; first < 2; ++first) {
                snprintf(s, sizeof(s), "%s_rusanov_%s_%.2f", first ? "first" : "flux", kinds[k], g);
                check_flux<0>(s, k, g, first);
                snprintf(s, sizeof(s), "%s_hllc_%s_%.2f", first ? "first" : "flux", kinds[k], g);
                check_flux<1>(s, k, g, first);
            }
        }
    }
    const char* kinds[4] = {"smooth", "jumps", "stretched", "scaled"};
    for (int k = 0; k < 4; ++k) {
        char s[64];
        snprintf(s, sizeof(s), "grad_barth_%s", kinds[k]);
        check_grad<1>(s, k);
        snprintf(s, sizeof(s), "grad_venkat_%s", kinds[k]);
        check_grad<2>(s, k);
    }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        printf("cuda_error %s\n", cudaGetErrorString(e));
        return 2;
    }
    printf("long_double_digits %d\n", __LDBL_MANT_DIG__);
    return 0;
}
