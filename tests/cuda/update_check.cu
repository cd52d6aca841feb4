// Checks the fixed-point pieces of the second-order update (fixed.cuh) and
// their FP64 forms against long double on the host (128-bit on the Arm
// machines that carry the GPU).
//
//   stage: Runge-Kutta stages 1 and 2 of a signed sum of face fluxes; kinds: any, step factors
//          with all mantissa bits set, fluxes with all of them set, sums that
//          cancel, step factors and states of very different sizes
//   sound: sound speeds (kind 0)
//   dt: a step factor over a sum of wave speeds (kind 0)
//   squares: a warp's sums of squares; kinds: like sizes, sizes 2^30 apart,
//            one value far above the others, mantissas of all ones, one zero column
// Each line: "<what> kind K n N taken T rms_fixed A rms_fp64 B max_fixed C max_fp64 D",
// errors relative to the largest term.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#define FV_KNS fast
#include "euler_o2.cuh"

using namespace fast;
using LD = long double;

struct In { double x[4], u, u0, dtv; int neg[4]; };
struct Out { double fx, f64; int took; };

template <int STAGE>
__global__ void k_stage(const In* in, int n, Out* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x[4], s = 0.0, un = 0.0;
    int neg[4];
    for (int k = 0; k < 4; ++k) { x[k] = in[i].x[k]; neg[k] = in[i].neg[k]; }
    for (int k = 0; k < 4; ++k) s += neg[k] & 1 ? -x[k] : x[k];
    fvfix::Fixed R;
    bool ok = fvfix::fixed_sum<4>(x, neg, R);
    ok = ok && fvfix::rk_stage<STAGE>(in[i].u, in[i].u0, R, in[i].dtv, un);
    const double e = in[i].u + in[i].dtv * s;
    out[i].took = ok;
    out[i].fx = un;
    out[i].f64 = STAGE == 1 ? 0.75 * in[i].u0 + 0.25 * e : (1.0 / 3.0) * in[i].u0 + (2.0 / 3.0) * e;
}

__global__ void k_sound(const In* in, int n, Out* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double r = fabs(in[i].x[0]), p = fabs(in[i].x[1]), g = in[i].u;
    double c = 0.0;
    out[i].took = fvfix::sound_speed(r, p, g, c);
    out[i].fx = c;
    out[i].f64 = sqrt(g * p / r);
}

__global__ void k_dt(const In* in, int n, Out* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x[4], s = 0.0, q = 0.0;
    int none[4] = {0, 0, 0, 0};
    for (int k = 0; k < 4; ++k) s += x[k] = fabs(in[i].x[k]);
    fvfix::Fixed R;
    const bool ok = fvfix::fixed_sum<4>(x, none, R) && fvfix::quotient(in[i].dtv, R, q);
    out[i].took = ok;
    out[i].fx = q;
    out[i].f64 = in[i].dtv / s;
}

// n lanes, whole warps; the sum of value k of a warp in its lanes 8 k to 8 k + 7
__global__ void k_squares(const In* in, int n, Out* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x[4], s = 0.0;
    for (int k = 0; k < 4; ++k) x[k] = in[i].x[k];
    out[i].took = fvfix::warp_squares4(x, s);
    out[i].fx = s;
    out[i].f64 = warp_sum4(x[0] * x[0], x[1] * x[1], x[2] * x[2], x[3] * x[3]);
}

template <class K, class Ref>
static void run(const char* what, int kind, const std::vector<In>& in, K kernel, Ref ref) {
    const int n = (int)in.size();
    In* d;
    Out* o;
    cudaMalloc(&d, n * sizeof(In));
    cudaMalloc(&o, n * sizeof(Out));
    cudaMemcpy(d, in.data(), n * sizeof(In), cudaMemcpyHostToDevice);
    kernel<<<(n + 255) / 256, 256>>>(d, n, o);
    std::vector<Out> h(n);
    cudaMemcpy(h.data(), o, n * sizeof(Out), cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(o);
    LD a = 0, b = 0, ma = 0, mb = 0;
    int took = 0;
    for (int i = 0; i < n; ++i) {
        if (!h[i].took) continue;
        ++took;
        LD scale;
        const LD x = ref(in[i], scale);
        const LD e = fabsl(h[i].fx - x) / scale, f = fabsl(h[i].f64 - x) / scale;
        a += e * e; b += f * f;
        ma = fmaxl(ma, e); mb = fmaxl(mb, f);
    }
    printf("%s kind %d n %d taken %d rms_fixed %.4Le rms_fp64 %.4Le max_fixed %.4Le max_fp64 %.4Le\n", what, kind, n, took,
           sqrtl(a / (took ? took : 1)), sqrtl(b / (took ? took : 1)), ma, mb);
}

int main() {
    printf("long_double_digits %d\n", (int)__LDBL_MANT_DIG__);
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    auto full = [](double x) { return std::nextafter(std::ldexp(x < 0 ? -1.0 : 1.0, std::ilogb(x) + 1), 0.0); };
    auto sum = [](const In& q, LD& big) {
        LD s = 0;
        for (int k = 0; k < 4; ++k) { s += q.neg[k] & 1 ? -(LD)q.x[k] : (LD)q.x[k]; big = fmaxl(big, fabsl(q.x[k])); }
        return s;
    };
    for (int kind = 0; kind < 5; ++kind) {
        std::vector<In> in(100000);
        for (In& q : in) {
            for (int k = 0; k < 4; ++k) { q.x[k] = U(rng) * std::exp2(4 * U(rng)); q.neg[k] = (int)(rng() & 1023); }
            q.u = U(rng); q.u0 = q.u * (1.0 + 0.01 * U(rng));
            q.dtv = std::exp2(-4 + 2 * U(rng));
            if (kind == 1) q.dtv = full(q.dtv);
            if (kind == 2) for (double& x : q.x) x = full(x);
            if (kind == 3) { q.x[1] = q.x[0]; q.neg[1] = q.neg[0] ^ 1; q.x[3] = q.x[2] * (1.0 + 1e-9 * U(rng)); q.neg[3] = q.neg[2] ^ 1; }
            if (kind == 4) { q.dtv *= std::exp2(30 * U(rng)); q.u0 = U(rng) * std::exp2(10 * U(rng)); }
        }
        for (int st = 1; st <= 2; ++st) {
            auto ref = [&](const In& q, LD& s) {
                LD big = 0;
                const LD dr = (LD)q.dtv * sum(q, big);
                s = fmaxl(fmaxl(fabsl(q.u), fabsl(q.u0)), q.dtv * big);
                const LD e = q.u + dr;
                return st == 1 ? (3 * (LD)q.u0 + e) / 4 : ((LD)q.u0 + 2 * e) / 3;
            };
            if (st == 1) run("stage1", kind, in, k_stage<1>, ref);
            else run("stage2", kind, in, k_stage<2>, ref);
        }
        std::vector<In> sq(32 * 4000);
        for (size_t i = 0; i < sq.size(); ++i) {
            for (int k = 0; k < 4; ++k) {
                double& x = sq[i].x[k];
                x = U(rng) * (kind == 1 ? std::exp2(15 * U(rng)) : kind == 2 && i % 32 == 5 ? 1e6 : 1.0);
                if (kind == 3) x = full(x);
                if (kind == 4 && k == 2) x = 0.0;
            }
        }
        run("squares", kind, sq, k_squares, [&](const In& q, LD& s) {
            const size_t i = &q - sq.data(), w = i & ~(size_t)31;
            s = 0;
            for (int l = 0; l < 32; ++l) { const LD x = sq[w + l].x[i / 8 % 4]; s += x * x; }
            const LD sum = s;
            if (s == 0) s = 1;
            return sum;
        });
        if (kind != 0) continue;
        run("dt", kind, in, k_dt, [&](const In& q, LD& s) {
            LD t = 0;
            for (double x : q.x) t += fabsl(x);
            return s = q.dtv / t;
        });
        for (In& q : in) q.u = 1.2 + 0.9 * (1.0 + U(rng));
        run("sound", kind, in, k_sound, [&](const In& q, LD& s) {
            return s = sqrtl((LD)q.u * fabsl(q.x[1]) / fabsl(q.x[0]));
        });
    }
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("cuda_error %s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
