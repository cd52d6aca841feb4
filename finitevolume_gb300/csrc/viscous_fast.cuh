// Shared parts of the default (contracted) builds of the Navier-Stokes and
// RANS-SA steps, arranged for the FP64 pipe, which bounds them: divisions by
// geometry are prepared (GradDev::gg, lsq_w, fgrad in their fast layouts), one
// reciprocal per cell gives all of its primitives, the inviscid flux and the
// wave speed come from the integer pipe (fixed.cuh), and of the corrected face
// gradients only the parts that the fluxes use are formed.  Included by ns.cu
// and rans.cu under FV_NS_FAST, after euler_o1.cuh and gradients.cuh.
#pragma once

#include "fixed.cuh"
#include "fpconv.cuh"

namespace FV_KNS {

using fvgb::GradDev;
using fvgb::NSArgs;

// u, v, T and 1/rho of a conserved state, and its pressure
__device__ __forceinline__ double4_32a prim_visc(const St& s, double g, double inv_R, double& p) {
    const double ir = fvconv::rcp_nr3(s.r);
    double4_32a w;
    w.x = s.ru * ir;
    w.y = s.rv * ir;
    p = (g - 1.0) * (s.E - 0.5 * (s.ru * w.x + s.rv * w.y));
    w.z = p * (ir * inv_R);
    w.w = ir;
    return w;
}

__device__ __forceinline__ double comp(const double4_32a& w, int k) {
    return k == 0 ? w.x : (k == 1 ? w.y : (k == 2 ? w.z : w.w));
}

// The larger of two values that are not negative, by their bit patterns
__device__ __forceinline__ double max_pos(double a, double b) {
    return __double_as_longlong(a) < __double_as_longlong(b) ? b : a;
}

// Gradients of the first NV components of prim; bvec(face): the boundary
// values.  Fast layouts: gg = (outward n * length / V, owner weight, 0),
// lsq_w the weights folded with the inverse normal matrix.
template <int NV, class BVec>
__device__ __forceinline__ void cell_gradient_fast(const GradDev& g, const double4_32a* prim, int c, const BVec& bvec,
                                                   double gx[NV], double gy[NV]) {
    const int e0 = g.cf_off[c], e1 = g.cf_off[c + 1];
    const double4_32a wc = prim[c];
#pragma unroll
    for (int k = 0; k < NV; ++k) gx[k] = gy[k] = 0.0;
    for (int e = e0; e < e1; ++e) {
        const int nb = g.nb[e];
        const double4_32a wn = nb >= 0 ? prim[nb] : bvec(-1 - nb, wc);
        if (g.scheme == 0) {
            const double2 a = g.lsq_w[e];
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const double d = comp(wn, k) - comp(wc, k);
                gx[k] += a.x * d;
                gy[k] += a.y * d;
            }
        } else {
            const double4_32a q = g.gg[e];
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const double pf = comp(wn, k) + q.z * (comp(wc, k) - comp(wn, k));
                gx[k] += q.x * pf;
                gy[k] += q.y * pf;
            }
        }
    }
}

// Interpolated face gradient and the corrected normal derivative (fast fgrad:
// 1/nd, length, kx, ky, w_L, nd, nx, ny).
__device__ __forceinline__ void face_normal_gradient(const double* fg, bool bnd, double d, double2 gL, double2 gR,
                                                     double& gx, double& gy, double& dn) {
    gx = gL.x;
    gy = gL.y;
    if (!bnd) {
        gx = gR.x + fg[4] * (gL.x - gR.x);
        gy = gR.y + fg[4] * (gL.y - gR.y);
    }
    dn = d * fg[0] + gx * fg[2] + gy * fg[3];
}

// Inviscid flux times length and the largest wave speed in FP64: the exact
// Riemann flux, boundary kinds of the Euler solvers, and what the
// fixed-point form refuses.
template <int FLUX>
__device__ __noinline__ double inviscid_f64(const NSArgs& n, int f, int cl, int cr, St* F) {
    const double4_32a geo = n.fgeom[f];
    const St UL = ld_state(n.U, cl);
    const St UR = cr < 0 ? ghost_state(n.bc, n.fpatch[f], UL, geo.x, geo.y, n.gamma) : ld_state(n.U, cr);
    *F = geo.z * num_flux<FLUX>(UL, UR, geo.x, geo.y, n.gamma, n.exact_tol, n.exact_max_iter);
    return face_smax(UL, UR, cr >= 0, geo.x, geo.y, n.gamma);
}

// qL, qR: the cells' densities and pressures (qR unused on a boundary face);
// fg: the fast fgrad row.  uR, vR: the velocity of the right state (a boundary face's
// ghost).
template <int FLUX>
__device__ __forceinline__ double inviscid(const NSArgs& n, int f, int cl, int cr, const double* fg,
                                           const double2& qL, const double4_32a& wl, const double2& qR,
                                           const double4_32a& wr, St& F, double& uR, double& vR) {
    fvfix::State L = {qL.x, wl.x, wl.y, qL.y}, R;
    bool ok = FLUX != FLUX_EXACT && n.fixed;
    if (cr >= 0) {
        R = {qR.x, wr.x, wr.y, qR.y};
    } else {
        const int p = n.fpatch[f], t = n.bc.type[p];
        R = L;
        if (t == BC_NOSLIP) {
            R.u = 2.0 * n.bc.wall_u[p] - L.u;
            R.v = 2.0 * n.bc.wall_v[p] - L.v;
        } else if (t == BC_FARFIELD) {
            const double* q = n.bc.st[p];
            R = {q[0], q[1] / q[0], q[2] / q[0], 0.0};
            R.p = (n.gamma - 1.0) * (q[3] - 0.5 * (q[1] * R.u + q[2] * R.v));
        } else if (t != BC_OUTFLOW) {
            ok = false;
            const St g = ghost_state(n.bc, p, ld_state(n.U, cl), fg[6], fg[7], n.gamma);
            R.u = g.ru / g.r;
            R.v = g.rv / g.r;
        }
    }
    uR = R.u;
    vR = R.v;
    double smax;
    fvfix::State q;
    if (ok && fvfix::flux<FLUX == FLUX_HLLC ? 1 : 0, false, true>(L, R, 0.0, 0.0, fvfix::NoCons{}, fvfix::NoCons{},
                                                                  fg[6], fg[7], fg[1], n.fxc, q, cr >= 0,
                                                                  smax)) {
        F = st_make(q.r, q.u, q.v, q.p);
        // Equal densities: the Rusanov mass flux has no dissipation and is the
        // mean of rho Vn, in FP64 as the strict build forms it, so that a
        // uniform flow's density residual keeps that rounding.
        if (FLUX == FLUX_RUSANOV && L.r == R.r) {
            const double VnL = L.u * fg[6] + L.v * fg[7], VnR = R.u * fg[6] + R.v * fg[7];
            F.r = fg[1] * (0.5 * (L.r * VnL + R.r * VnR));
        }
        return smax;
    }
    return inviscid_f64<FLUX>(n, f, cl, cr, &F);
}

// Traction of mu (grad v + grad v^T - 2/3 div v) on the face normal, per unit
// mu, from the interpolated gradients and corrected normal derivatives of u
// and v.
__device__ __forceinline__ void traction(const double* fg, double ux, double uy, double dnu, double vx, double vy,
                                         double dnv, double& tx, double& ty) {
    const double nx = fg[6], ny = fg[7];
    const double du = dnu - (ux * nx + uy * ny), dv = dnv - (vx * nx + vy * ny);
    ux += du * nx; uy += du * ny;
    vx += dv * nx; vy += dv * ny;
    const double div = (2.0 / 3.0) * (ux + vy), xy = uy + vx;
    tx = (2.0 * ux - div) * nx + xy * ny;
    ty = xy * nx + (2.0 * vy - div) * ny;
}

// The block's largest wave rate (a face's wave speed over its length scale,
// not negative; NaN does not count), as the time step cfl / rate, into the
// step's slot: one reciprocal a block instead of one a face.
__device__ __forceinline__ void max_rate(double rate, fvgb::StepCtl* ctl) {
    __shared__ unsigned long long smax[fvgb::kFaceBlock / 32];
    unsigned long long b = (unsigned long long)__double_as_longlong(rate);
    if (b > 0x7ff0000000000000ull) b = 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) b = max(b, smax[w]);
        if (b == 0) return;
        const double dt = ctl->cfl * fvconv::rcp_nr3(__longlong_as_double((long long)b));
        atomicMin(&ctl->dt_bits, (unsigned long long)__double_as_longlong(dt));
    }
}

// The signed sum of a cell's N face fluxes: momentum and energy on the
// integer pipe, the mass in FP64 in the reference's order, which leaves the
// density residual of a uniform flow its rounding.
template <int N>
__device__ __forceinline__ St gather_visc(const St* ff, const int* cf) {
    double x[3][N], m = 0.0;
    int neg[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int ent = __ldg(cf + i);
        const St F = flip_if(ld_state(ff, ent >> 1), ent);
        m += F.r;
        x[0][i] = F.ru; x[1][i] = F.rv; x[2][i] = F.E;
        neg[i] = 0;
    }
    return st_make(m, fvfix::signed_sum<N>(x[0], neg), fvfix::signed_sum<N>(x[1], neg), fvfix::signed_sum<N>(x[2], neg));
}
__device__ __forceinline__ St gather_any(const St* ff, const int* cf, int e0, int e1) {
    if (e1 - e0 == 4) return gather_visc<4>(ff, cf + e0);
    if (e1 - e0 == 3) return gather_visc<3>(ff, cf + e0);
    St R = st_make(0.0, 0.0, 0.0, 0.0);
    for (int e = e0; e < e1; ++e) {
        const int ent = cf[e];
        R += flip_if(ld_state(ff, ent >> 1), ent);
    }
    return R;
}

}  // namespace FV_KNS
