// Which cells the fixed-point gradient pass (euler_o2_fixed.cuh) serves itself,
// and what it gives beside boundaries and where reconstructed states are not
// positive, against long double on the host.
//
// Cells of 3 to 18 faces with none, one, two or three boundary faces (slip and
// no-slip walls, outflow, fixed and characteristic farfield), both limiters,
// evaluated (live) and frozen at one (open: states overshoot, many fall back to
// the cell's).  A live run captures the limiter values, too.  A second run has NaN in place of the FP64 weights and offsets,
// which only cells that the FP64 pass takes read: those without NaN were served.
// Each line: "<run> faces F boundary B n N served S fallback P wrong Q rms_fixed A
// rms_fp64 C max_fixed D max_fp64 E", errors relative to the largest value (for
// velocities: speed or sound speed) and to how much the weights amplify its
// rounding; wrong: fallbacks that are not the cell's state.  Live runs then:
// "<run>_psi faces F boundary B n N small M rms_fixed A rms_fp64 C", the limiter
// values' errors relative to themselves or 2^-7, and how many are below 2^-4.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#define FV_KNS fast
#include "euler_o2_fixed.cuh"

using namespace fast;
using LD = long double;

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

constexpr double kG = 1.4;
static const double kFar[4] = {1.05, 0.45, 0.2, 0.75};  // r, u, v, p

static void ghost(int type, const LD w[4], LD nx, LD ny, LD o[4]) {
    const LD g = kG, vn = w[1] * nx + w[2] * ny;
    for (int k = 0; k < 4; ++k) o[k] = w[k];
    if (type == BC_WALL) {
        o[1] -= 2 * vn * nx;
        o[2] -= 2 * vn * ny;
    } else if (type == BC_NOSLIP) {
        o[1] = 2 * (LD)0.1 - w[1];
        o[2] = -w[2];
    } else if (type == BC_FARFIELD) {
        for (int k = 0; k < 4; ++k) o[k] = kFar[k];
    } else if (type == BC_CHAR) {
        const LD c = sqrtl(g * w[3] / w[0]), cf = sqrtl(g * kFar[3] / kFar[0]), vf = kFar[1] * nx + kFar[2] * ny;
        if (vf <= -cf) {
            for (int k = 0; k < 4; ++k) o[k] = kFar[k];
        } else if (vn < c) {
            const LD k = 2 / (g - 1), vb = (vn + k * c + vf - k * cf) / 2, cb = (g - 1) / 4 * (vn + k * c - vf + k * cf);
            const bool out = vb > 0;
            o[0] = out ? w[0] * powl(fabsl(cb) / c, k) : kFar[0] * powl(fabsl(cb) / cf, k);
            o[1] = (out ? w[1] - vn * nx : kFar[1] - vf * nx) + vb * nx;
            o[2] = (out ? w[2] - vn * ny : kFar[2] - vf * ny) + vb * ny;
            o[3] = o[0] * cb * cb / g;
        }
    }
}

template <int LIM> static void check(const char* run, int faces, int bnd, bool open) {
    const int n = 1 << 11;
    std::mt19937_64 rng(100 * faces + 10 * bnd + LIM);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::vector<int> off(n + 1, 0), cnb, fpatch;
    std::vector<double2> w, r;
    std::vector<St> W(n);
    std::vector<double> eps(n);
    std::vector<double4_32a> geo;
    const double d = open ? 1.6 : 0.6;
    for (St& q : W) {
        q.r = 1.0 + d * (U(rng) - 0.5);
        q.ru = 0.4 + d * 0.5 * (U(rng) - 0.5);
        q.rv = 0.2 + d * 0.5 * (U(rng) - 0.5);
        q.E = 0.7 * (1.0 + d * (U(rng) - 0.5));
    }
    for (int i = 0; i < n; ++i) {
        const double h = exp2(-10 * U(rng)), al = 6.2831853 * U(rng);
        eps[i] = pow(5 * h, 3) * 1e-3;
        LD m00 = 0, m01 = 0, m11 = 0;
        std::vector<double2> dx(faces);
        for (int j = 0; j < faces; ++j) {
            const double t = al + 6.2831853 * (j + 0.3 * U(rng)) / faces;
            dx[j] = make_double2(h * cos(t), h * sin(t));
            const LD q = 1 / ((LD)dx[j].x * dx[j].x + (LD)dx[j].y * dx[j].y);
            m00 += q * dx[j].x * dx[j].x; m01 += q * dx[j].x * dx[j].y; m11 += q * dx[j].y * dx[j].y;
        }
        const LD det = m00 * m11 - m01 * m01;
        const int first = (int)(rng() % faces);
        for (int j = 0; j < faces; ++j) {
            const LD q = 1 / ((LD)dx[j].x * dx[j].x + (LD)dx[j].y * dx[j].y);
            w.push_back(make_double2((double)(q * (m11 * dx[j].x - m01 * dx[j].y) / det), (double)(q * (m00 * dx[j].y - m01 * dx[j].x) / det)));
            r.push_back(make_double2(0.5 * dx[j].x, 0.5 * dx[j].y));
            if ((j - first + faces) % faces < bnd) {
                const double l = hypot(dx[j].x, dx[j].y);
                double4_32a q4;
                q4.x = dx[j].x / l; q4.y = dx[j].y / l; q4.z = h; q4.w = h;
                cnb.push_back(-1 - (int)geo.size());
                geo.push_back(q4);
                fpatch.push_back((int)(rng() % 5));
            } else {
                cnb.push_back((int)(rng() % n));
            }
        }
        off[i + 1] = (int)cnb.size();
    }
    if (geo.empty()) { geo.resize(1); fpatch.resize(1); }
    const int E = (int)cnb.size();
    std::vector<double2> sum(n);
    for (int i = 0; i < n; ++i) {
        sum[i] = make_double2(0, 0);
        for (int e = off[i]; e < off[i + 1]; ++e) { sum[i].x += w[e].x; sum[i].y += w[e].y; }
    }
    fvgb::O2Args a{};
    a.m.n_cells = n;
    a.m.cf_off = up(off);
    a.m.fpatch = up(fpatch);
    a.m.fgeom = up(geo);
    a.cnb = up(cnb);
    a.lsq = up(w); a.lsq_sum = up(sum); a.erf = up(r); a.eps2 = up(eps);
    a.W = up(W);
    a.gamma = kG;
    a.igm1 = 1.0 / (kG - 1.0);
    a.bc.n = 5;
    std::vector<double> fsp;
    for (int p = 0; p < 5; ++p) {
        a.bc.type[p] = p;
        a.bc.wall_u[p] = 0.1;
        const double q = kFar[0], u = kFar[1], v = kFar[2], pr = kFar[3], c = std::sqrt(kG * pr / q);
        const double st[4] = {q, q * u, q * v, pr / (kG - 1.0) + 0.5 * q * (u * u + v * v)};
        for (int k = 0; k < 4; ++k) a.bc.st[p][k] = st[k];
        for (double x : {q, u, v, pr, c, 1.0 / c, 1.0 / kG, 0.0}) fsp.push_back(x);
    }
    a.fsp = up(fsp);
    if (open) {
        a.psi_buf = up(std::vector<double>(4 * n, 1.0));
        a.psi_mode = 2;
    }
    double *p0 = nullptr, *p1 = nullptr;
    if (!open) {
        p0 = up(std::vector<double>(4 * n));
        p1 = up(std::vector<double>(4 * n));
        a.psi_mode = 1;
    }
    int4 *xa, *xr;
    int *xs, *dec;
    cudaMalloc(&xa, sizeof(int4) * E); cudaMalloc(&xr, sizeof(int4) * E); cudaMalloc(&xs, sizeof(int) * n);
    dec = up(std::vector<int>(1, 0));
    k_fix_geom<<<(n + 255) / 256, 256>>>(a, xa, xr, xs, dec);
    a.fxa = xa; a.fxr = xr; a.fxs = xs;
    const int declined = down(dec, 1)[0];
    St *fx, *f64, *fn;
    cudaMalloc(&fx, sizeof(St) * E); cudaMalloc(&f64, sizeof(St) * E); cudaMalloc(&fn, sizeof(St) * E);
    a.wf = fx;
    if (!open) a.psi_buf = p0;
    k_grad_fx<LIM><<<4 * n / 256, 256>>>(a);
    a.wf = f64;
    if (!open) a.psi_buf = p1;
    k_grad<double, 0, LIM><<<n / 256, 256>>>(a);
    a.wf = fn;
    if (!open) a.psi_mode = 0;
    a.lsq = a.erf = up(std::vector<double2>(E, make_double2(NAN, NAN)));
    k_grad_fx<LIM><<<4 * n / 256, 256>>>(a);
    auto A = down(fx, E), B = down(f64, E), C = down(fn, E);
    std::vector<double> P0, P1;
    if (!open) {
        P0 = down(p0, 4 * n);
        P1 = down(p1, 4 * n);
        cudaFree(p0);
        cudaFree(p1);
    }
    LD q0 = 0, q1 = 0;
    long small = 0;
    LD s0 = 0, s1 = 0, mx0 = 0, mx1 = 0;
    long served = 0, fallback = 0, wrong = 0, count = 0;
    for (int i = 0; i < n; ++i) {
        bool own = true;
        for (int e = off[i]; e < off[i + 1]; ++e)
            for (int k = 0; k < 4; ++k) own = own && !std::isnan((&C[e].r)[k]);
        served += own;
        const LD wc[4] = {W[i].r, W[i].ru, W[i].rv, W[i].E}, c = sqrtl(kG * wc[3] / wc[0]);
        std::vector<LD> out(4 * faces);
        LD sc[4];
        for (int k = 0; k < 4; ++k) {
            LD gx = 0, gy = 0, hi = 0, lo = 0, amp = 0, psi = 1, big = fabsl(wc[k]), sx = 0, sy = 0;
            if (k == 1 || k == 2) big = fmaxl(c, hypotl(wc[1], wc[2]));
            for (int e = off[i]; e < off[i + 1]; ++e) {
                LD v;
                if (cnb[e] >= 0) v = (&W[cnb[e]].r)[k];
                else {
                    LD o[4];
                    const int f = -1 - cnb[e];
                    ghost(fpatch[f], wc, geo[f].x, geo[f].y, o);
                    v = (wc[k] + o[k]) / 2;
                }
                const LD dv = v - wc[k];
                gx += w[e].x * dv; gy += w[e].y * dv;
                hi = fmaxl(hi, dv); lo = fminl(lo, dv); big = fmaxl(big, fabsl(v));
                sx += fabs(w[e].x); sy += fabs(w[e].y);
            }
            for (int e = off[i]; e < off[i + 1]; ++e) {
                const LD y = gx * r[e].x + gy * r[e].y, d1 = y > 0 ? hi : -lo, ay = fabsl(y), ep = eps[i];
                amp = fmaxl(amp, sx * fabs(r[e].x) + sy * fabs(r[e].y));
                if (ay > 0) psi = fminl(psi, LIM == 1 ? d1 / ay : (d1 * d1 + ep + 2 * d1 * ay) / (d1 * d1 + 2 * ay * ay + d1 * ay + ep));
            }
            if (open) psi = 1;
            else {
                const LD s = fmaxl(psi, 1.0L / 128), e0 = (P0[4 * i + k] - psi) / s, e1 = (P1[4 * i + k] - psi) / s;
                q0 += e0 * e0; q1 += e1 * e1;
                small += psi < 1.0L / 16;
            }
            for (int e = off[i]; e < off[i + 1]; ++e) out[4 * (e - off[i]) + k] = wc[k] + psi * (gx * r[e].x + gy * r[e].y);
            sc[k] = big * fmaxl(1, amp);
        }
        for (int e = off[i]; e < off[i + 1]; ++e) {
            LD* x = &out[4 * (e - off[i])];
            if (fabsl(x[0]) < 1e-9L || fabsl(x[3]) < 1e-9L) continue;  // rounding decides
            const bool fall = x[0] < 0 || x[3] < 0;
            fallback += fall;
            LD e0 = 0, e1 = 0;
            for (int k = 0; k < 4; ++k) {
                const double p = (&A[e].r)[k], q = (&B[e].r)[k];
                if (fall) {
                    wrong += p != (double)wc[k] || q != (double)wc[k];
                    continue;
                }
                e0 = fmaxl(e0, fabsl(p - x[k]) / sc[k]);
                e1 = fmaxl(e1, fabsl(q - x[k]) / sc[k]);
            }
            if (fall) continue;
            s0 += e0 * e0; s1 += e1 * e1;
            mx0 = fmaxl(mx0, e0); mx1 = fmaxl(mx1, e1);
            ++count;
        }
    }
    printf("%s faces %d boundary %d n %d declined %d served %ld fallback %ld wrong %ld rms_fixed %.4Le rms_fp64 %.4Le max_fixed %.4Le max_fp64 %.4Le\n",
           run, faces, bnd, n, declined, served, fallback, wrong, sqrtl(s0 / (count ? count : 1)), sqrtl(s1 / (count ? count : 1)), mx0, mx1);
    if (!open)
        printf("%s_psi faces %d boundary %d n %d small %ld rms_fixed %.4Le rms_fp64 %.4Le\n", run, faces, bnd, 4 * n, small,
               sqrtl(q0 / (4 * n)), sqrtl(q1 / (4 * n)));
    for (const void* p : {(const void*)a.m.cf_off, (const void*)a.m.fpatch, (const void*)a.m.fgeom, (const void*)a.cnb, a.lsq,
                          (const void*)a.lsq_sum, (const void*)a.eps2, (const void*)a.W, (const void*)fx, (const void*)f64,
                          (const void*)fn, (const void*)xa, (const void*)xr, (const void*)xs})
        cudaFree(const_cast<void*>(p));
}

int main() {
    printf("long_double_digits %d\n", (int)__LDBL_MANT_DIG__);
    for (int faces : {3, 4, 5, 7, 16, 18})
        for (int bnd = 0; bnd < 4; ++bnd) {
            check<1>("barth_live", faces, bnd, false);
            check<2>("venkat_live", faces, bnd, false);
            check<1>("barth_open", faces, bnd, true);
            check<2>("venkat_open", faces, bnd, true);
        }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("cuda_error %s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
