// The FP64 gradient, limiter and face passes of the second-order path on the
// integer pipe (fixed.cuh).  Same scheme and interfaces as k_grad and k_face
// (euler_o2.cuh), whose FP64 forms take every cell and face outside the
// ranges of the fixed-point one.
//
// Measured on the GB300 (1.05M-cell O-grid, Venkatakrishnan, HLLC, time per
// launch): gradients and limiter 417 us in FP64 (the FP64 pipe 86% busy), 143
// here; face fluxes 387 us in FP64 (88% busy), 80 here.  On 2k cells, where a
// launch is one wave and the length of a thread's dependent chain counts
// (FP64 64 clocks an operation, integers 5 to 13), 32 and 21 us became 10
// and 8.5.  Errors against 128-bit arithmetic, relative to the face's or cell's
// own scale, are no larger than the FP64 forms' (tests/cuda/fixed_check.cu,
// flux_components_check.cu, grad_cells_check.cu); a component far below that
// scale keeps fewer bits of its own.
#pragma once

#include "euler_o2.cuh"

namespace FV_KNS {

using fvfix::i64;
using fvfix::Sp;
using fvfix::split;
using fvfix::u64;

// Per cell and entry the least-squares weights and face offsets of the
// fixed-point pass, from the FP64 ones: weights in units of 2^(e_x - 62) and
// 2^(e_y - 62), with 2^e above the cell's sum of |weights| of that axis;
// offsets in units of 2^(S - e_x - 61) and 2^(S - e_y - 61), S >= 0 the larger of
// e + (exponent above the largest |offset|) over the two axes.  So weighted
// differences of at most d stay below d in the weights' units, an increment
// below 2^S d.  fxs[c] = S, or -1 where the cell takes the FP64 pass: more
// than 16 faces, S above 16, or a weight or offset that is not finite or out of
// range; *declined counts those.
static __global__ void __launch_bounds__(256) k_fix_geom(const fvgb::O2Args a, int4* __restrict__ fxa,
                                                         int4* __restrict__ fxr, int* __restrict__ fxs,
                                                         int* __restrict__ declined = nullptr) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.m.n_cells) return;
    const double2* w = static_cast<const double2*>(a.lsq);
    const double2* r = static_cast<const double2*>(a.erf);
    const int e0 = a.m.cf_off[c], e1 = a.m.cf_off[c + 1];
    double sx = 0.0, sy = 0.0, rx = 0.0, ry = 0.0;
    for (int e = e0; e < e1; ++e) {
        sx += fabs(w[e].x);
        sy += fabs(w[e].y);
        rx = fmax(rx, fabs(r[e].x));
        ry = fmax(ry, fabs(r[e].y));
    }
    // frexp's exponent: |x| < 2^e; one more keeps the rounded sum below
    int ex, ey, px, py;
    frexp(sx * 1.0000001, &ex);
    frexp(sy * 1.0000001, &ey);
    frexp(rx, &px);
    frexp(ry, &py);
    const int S = max(0, max(ex + px, ey + py));
    bool ok = e1 - e0 <= 16 && S <= 16 && isfinite(sx) && isfinite(sy) && isfinite(rx) && isfinite(ry);
    ok = ok && abs(ex) < 300 && abs(ey) < 300 && abs(px) < 300 && abs(py) < 300;
    fxs[c] = ok ? S : -1;
    if (!ok && declined) atomicAdd(declined, 1);
    for (int e = e0; e < e1; ++e) {
        const Sp ax = split(ok ? llrint(ldexp(w[e].x, 62 - ex)) : 0), ay = split(ok ? llrint(ldexp(w[e].y, 62 - ey)) : 0);
        const Sp bx = split(ok ? llrint(ldexp(r[e].x, 61 - (S - ex))) : 0);
        const Sp by = split(ok ? llrint(ldexp(r[e].y, 61 - (S - ey))) : 0);
        fxa[e] = make_int4(ax.h, ax.l, ay.h, ay.l);
        fxr[e] = make_int4(bx.h, bx.l, by.h, by.l);
    }
}

// The FP64 pass for one cell, out of line: rare, and its registers should
// not count for the others.
template <int LIM> __device__ __noinline__ void grad_cell_f64(const O2Args& a, int c, const double* fs) {
    grad_cell<double, 0, LIM>(a, c, fs);
}

// Numerator and denominator of phi(d1, y) of one side: d1 >= 0 the neighbour
// extreme, y >= 0 the face extreme, both in the unit 2^(E - 1080); equal
// where the side does not limit.  eps2 in FP64.
template <int LIM>
__device__ __forceinline__ void limiter_side(i64 d1, i64 y, double eps2, int E, i64& num, i64& den) {
    using namespace fvfix;
    const i64 m = LIM == 1 ? y : 2 * y;
    if (d1 >= m) {
        num = den = (i64)1 << 59;
        return;
    }
    int s = __clzll(m) - 4;  // the larger of d1 and m, m, into [1/2, 1) of Q60
    if constexpr (LIM == 1) {
        num = d1 << s;
        den = y << s;
    } else {
        // ... or less, so that eps2 stays below 1 in the square of that unit
        const int hi = hi_word(eps2), ee = biased(hi);
        s = min(s, hi >= 0x100000 ? ((1022 - ee) >> 1) + E - 1020 : 64);
        const i64 en = hi >= 0x100000 ? (i64)shr(top_bits(eps2), 1026 - ee - 2 * (s + 1020 - E)) : 0;
        const Sp ds = split(s >= 0 ? d1 << s : (i64)shr(d1, -s)), ys = split(s >= 0 ? y << s : (i64)shr(y, -s));
        const i64 p = mul<4>(ds, ys), q = mul<4>(ds, ds) + en;
        num = q + 2 * p;
        den = q + p + 2 * mul<4>(ys, ys);
    }
}

// Ghost state of a boundary face in FP64 (ghost_core's states up to
// rounding) with short dependent chains: the freestream's primitives, sound
// speed and its reciprocal are prepared (O2Args::fsp: r, u, v, p, c, 1/c per
// patch, or per instance of a batch), and the characteristic farfield takes
// one power (pow_near1) of |cb / c| of its upwind side; see
// char_farfield_p of the first-order kernel.
__device__ __forceinline__ V4<double> ghost_fast(const O2Args& a, int f, int cell, const V4<double>& w, double nx,
                                                 double ny) {
    const int patch = a.m.fpatch[f], t = a.bc.type[patch];
    if (t == BC_OUTFLOW) return w;
    const double Vn = w.u * nx + w.v * ny;
    if (t == BC_FARFIELD || t == BC_CHAR) {
        const double* q = a.fsp + 8 * (a.cell_inst ? a.cell_inst[cell] : patch);
        const V4<double> fs = {q[0], q[1], q[2], q[3]};
        if (t == BC_FARFIELD) return fs;
        const double g = a.gamma, cf = q[4], vnf = fs.u * nx + fs.v * ny;
        const double gp = g * w.p, y = rsqrt(gp * w.r), ci = gp * y;
        if (vnf <= -cf) return fs;  // supersonic inflow
        if (Vn >= ci) return w;     // supersonic outflow
        const double k = 2.0 * a.igm1;
        const double Rp = Vn + k * ci, Rm = vnf - k * cf;
        const double vnb = 0.5 * (Rp + Rm), cb = 0.25 * (g - 1.0) * (Rp - Rm);
        const bool out = vnb > 0.0;
        const double rs = out ? w.r : fs.r, ics = out ? w.r * y : q[5];
        const double ut = out ? w.u - Vn * nx : fs.u - vnf * nx, vt = out ? w.v - Vn * ny : fs.v - vnf * ny;
        const double rb = rs * fvconv::pow_near1(fabs(cb) * ics, k);
        return {rb, ut + vnb * nx, vt + vnb * ny, rb * cb * cb * q[6]};
    }
    if (t == BC_NOSLIP) return {w.r, 2.0 * a.bc.wall_u[patch] - w.u, 2.0 * a.bc.wall_v[patch] - w.v, w.p};
    return {w.r, w.u - 2.0 * Vn * nx, w.v - 2.0 * Vn * ny, w.p};
}

// A third boundary face of one cell: rare, out of line
static __device__ __noinline__ V4<double> ghost_more(const O2Args& a, int f, int c) {
    const double4_32a q = a.m.fgeom[f];
    return ghost_fast(a, f, c, WStore<double>::ld(static_cast<const St*>(a.W), c), q.x, q.y);
}

// Bitwise or over a quad, by two shuffles: a warp-wide reduction with a mask of
// its own per quad runs once for each of the warp's eight quads (1.05M cells:
// eight steps 7.35 -> 7.25 ms).
__device__ __forceinline__ unsigned quad_or(unsigned quad, unsigned x) {
    x |= __shfl_xor_sync(quad, x, 1, 4);
    return x | __shfl_xor_sync(quad, x, 2, 4);
}

// One variable k of one cell.  The four lanes of a cell meet at the votes:
// an FP64 cell is one for all its variables, and a face state that is not
// positive falls back to the cell's.  N: the cell's face count (3 or 4, its
// values then stay in registers), or 0 for any.
template <int LIM, int N>
__device__ __forceinline__ void grad_lane(const O2Args& a, int c, int k, int e0, int e1, const double* fs) {
    using namespace fvfix;
    const unsigned quad = 0xfu << (threadIdx.x & 28);
    const double* W = static_cast<const double*>(a.W);
    const int n = N ? N : e1 - e0;
    const double wc = __ldg(W + 4 * (size_t)c + k);
    // Values across the faces; a boundary face's is the mean of the cell's and
    // the ghost's.  A ghost is a long FP64 chain (2 to 3 us) and a warp's cells
    // have their boundary faces at different places: each lane forms the ghost
    // of one face, all at once, and the quad shares them.
    auto ghost = [&](int f) -> V4<double> {
        const double4_32a q = a.m.fgeom[f];
        return ghost_fast(a, f, c, WStore<double>::ld(static_cast<const St*>(a.W), c), q.x, q.y);
    };
    auto mean = [&](double r, double u, double v, double p) {
        return 0.5 * (wc + (k == 0 ? r : (k == 1 ? u : (k == 2 ? v : p))));
    };
    auto share = [&](const V4<double>& g, int lane) {
        return mean(__shfl_sync(quad, g.r, lane, 4), __shfl_sync(quad, g.u, lane, 4), __shfl_sync(quad, g.v, lane, 4),
                    __shfl_sync(quad, g.p, lane, 4));
    };
    double wn[N ? N : 1], wb0 = 0.0, wb1 = 0.0;
    int b0 = -1, b1 = -1;
    auto across = [&](int e) -> double {  // N = 0 only
        const int nb = a.cnb[e];
        if (nb >= 0) return __ldg(W + 4 * (size_t)nb + k);
        if (e == b0) return wb0;
        if (e == b1) return wb1;
        const V4<double> g = ghost_more(a, -1 - nb, c);
        return mean(g.r, g.u, g.v, g.p);
    };
    int E = biased(hi_word(wc));
    if constexpr (N != 0) {
        // all loads first; the rare boundary values replace theirs afterwards
        int nb[N], any = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) any |= nb[i] = a.cnb[e0 + i];
#pragma unroll
        for (int i = 0; i < N; ++i) wn[i] = __ldg(W + 4 * (size_t)(nb[i] < 0 ? c : nb[i]) + k);
        if (any < 0) {
            V4<double> g = {0.0, 0.0, 0.0, 0.0};
            const int mine = k < N ? a.cnb[e0 + k] : 0;
            if (mine < 0) g = ghost(-1 - mine);
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (nb[i] < 0) wn[i] = share(g, i);
        }
#pragma unroll
        for (int i = 0; i < N; ++i) E = max(E, biased(hi_word(wn[i])));
    } else {
        for (int e = e0; e < e1; ++e) {
            if (a.cnb[e] >= 0) continue;
            if (b0 < 0) b0 = e;
            else if (b1 < 0) b1 = e;
        }
        if (b0 >= 0) {
            V4<double> g = {0.0, 0.0, 0.0, 0.0};
            const int mine = k == 0 ? b0 : (k == 1 ? b1 : -1);
            if (mine >= 0) g = ghost(-1 - a.cnb[mine]);
            wb0 = share(g, 0);
            wb1 = share(g, 1);
        }
        for (int e = e0; e < e1; ++e) E = max(E, biased(hi_word(across(e))));
    }
    const int S = a.fxs[c];
    // out of range: the arithmetic below still runs, its result is not used
    unsigned bad = S < 0 || E > 1900 || (unsigned)(E - 1) < 149u;
    E = max(E, 150);  // an all-zero variable
    const i64 w0 = to_fixed<57>(wc, E);
    i64 dmax = 0, dmin = 0, hx = 0, hy = 0, lx = 0, ly = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const i64 d = to_fixed<57>(N ? wn[N ? i : 0] : across(e0 + i), E) - w0;
        const int4 q = __ldg(a.fxa + e0 + i);
        dmax = max(dmax, d);
        dmin = min(dmin, d);
        const Sp s = split(d);
        hx = madw(q.x, s.h, hx);
        lx = madw(q.x, s.l, madw(q.y, s.h, lx));
        hy = madw(q.z, s.h, hy);
        ly = madw(q.z, s.l, madw(q.w, s.h, ly));
    }
    const Sp gx = split(funnel(hx + (lx >> 32), (unsigned)lx, 5)), gy = split(funnel(hy + (ly >> 32), (unsigned)ly, 5));
    int over = 0;
    auto increment = [&](int e) -> i64 {
        const int4 r = __ldg(a.fxr + e);
        const i64 mid = madw(gx.h, r.y, madw(gx.l, r.x, madw(gy.h, r.w, (i64)gy.l * r.z)));
        const i64 acc = madw(gx.h, r.x, madw(gy.h, r.z, mid >> 32));
        over |= (int)(acc >> 32) ^ (int)(acc >> 63);  // the bits above the shift by S
        return (i64)(((u64)__funnelshift_l((unsigned)acc, (unsigned)(acc >> 32), S) << 32) |
                     __funnelshift_l((unsigned)mid, (unsigned)acc, S));
    };
    i64 inc[N ? N : 1], up = 0, dn = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const i64 d = increment(e0 + i);
        if (N) inc[N ? i : 0] = d;
        up = max(up, d);
        dn = min(dn, d);
    }
    bad |= (over >> (27 - max(S, 0))) != 0;  // an increment of 2^59 units or more
    i64 psi;  // Q60
    if (a.psi_mode == 2) {
        psi = to_fixed<60>(static_cast<const double*>(a.psi_buf)[4 * (size_t)c + k], 1023);
    } else {
        const double eps2 = LIM == 2 ? __ldg(static_cast<const double*>(a.eps2) + c) : 0.0;
        i64 nu, du, nd, dd;
        limiter_side<LIM>(dmax, up, eps2, E, nu, du);
        limiter_side<LIM>(-dmin, -dn, eps2, E, nd, dd);
        // the smaller quotient, to 53 bits or 2^-60: exact as a double, which
        // limiter freezing stores
        const bool lower = mul<3>(nd, du) < mul<3>(nu, dd);  // both below 16
        const i64 num = lower ? nd : nu, den = lower ? dd : du;
        psi = num < den ? ratio60(num, den) : (i64)1 << 60;
    }
    const Sp p = split(psi);
    // Captured once the quad has taken the cell: a declined cell's four values
    // are all lane 0's, from the FP64 pass, and nothing orders another lane's
    // store before them.
    auto capture = [&]() {
        if (a.psi_mode == 1) static_cast<double*>(a.psi_buf)[4 * (size_t)c + k] = to_double(psi, -60);
    };
    const bool any_sign = k == 1 || k == 2;  // velocities; density and pressure must stay positive
    double* out = reinterpret_cast<double*>(a.wf) + 4 * (size_t)e0 + k;
    if constexpr (N != 0) {
        unsigned flags = bad << 31;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            inc[i] = w0 + mul<4>(split(inc[i]), p);
            if (!any_sign && inc[i] <= 0) flags |= 1u << i;
        }
        flags = quad_or(quad, flags);
        if (flags >> 31) {
            if (k == 0) grad_cell_f64<LIM>(a, c, fs);
            return;
        }
        capture();
#pragma unroll
        for (int i = 0; i < N; ++i) out[4 * i] = flags >> i & 1 ? wc : to_double(inc[i], E - 1080);
    } else {
        if (quad_or(quad, bad)) {
            if (k == 0) grad_cell_f64<LIM>(a, c, fs);
            return;
        }
        capture();
        for (int i = 0; i < n; ++i) {
            const i64 w = w0 + mul<4>(split(increment(e0 + i)), p);
            const unsigned low = quad_or(quad, (unsigned)(!any_sign && w <= 0));
            out[4 * i] = low ? wc : to_double(w, E - 1080);
        }
    }
}

// Gradients, limiter and reconstructed face states: four lanes per cell, one
// primitive variable each.  Per variable the differences to the neighbours
// are integers in units of 2^-57 of the largest value's binade; weights and
// offsets are prepared (k_fix_geom), so a gradient component is a sum of
// three-product terms and an increment two of them.  Bound by latency and the
// integer pipes (ALU 55%, wide multiply-adds 39%, DRAM 22% busy): four lanes
// a cell keep a lane's state within 64 registers, 32 warps per SM (a thread
// a cell at 128 registers measured 296 us, 72 to 128 registers a lane 175 to 260).
template <int LIM>
__global__ void __launch_bounds__(fvgb::kMaxBlock, 2) k_grad_fx(const O2Args a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t >> 7) * 32 >= a.m.n_cells) return;
    const int c = (a.tile_order ? a.tile_order[t >> 7] * 32 : (t >> 7) * 32) + ((t & 127) >> 2), k = t & 3;
    if (c >= a.m.n_cells) return;
    // The geometry is read behind the neighbours' values and between long
    // stretches of arithmetic, with no registers to hold it earlier: the lanes
    // ask for its lines here (162 -> 155 us at 1.05M cells).
    prefetch(LIM == 2 && k ? static_cast<const void*>(static_cast<const double*>(a.eps2) + c) : a.fxs + c);
    const double* fs;
    if (!live_cell(a, c, fs)) return;
    const int e0 = a.m.cf_off[c], e1 = a.m.cf_off[c + 1];
    prefetch((k < 2 ? a.fxa : a.fxr) + e0 + 2 * (k & 1));
    if (e1 - e0 == 4) grad_lane<LIM, 4>(a, c, k, e0, e1, fs);
    else if (e1 - e0 == 3) grad_lane<LIM, 3>(a, c, k, e0, e1, fs);
    else grad_lane<LIM, 0>(a, c, k, e0, e1, fs);
}

template <int FLUX>
__device__ __noinline__ V4<double> face_flux_f64(const V4<double>& L, const V4<double>& R, double nx, double ny,
                                                 double ar, double g, double igm1) {
    const V4<double> F = num_flux_p<double, FLUX>(L, R, nx, ny, g, igm1, 0.0, 0);
    return {ar * F.r, ar * F.u, ar * F.v, ar * F.p};
}

// Face fluxes, one thread per face; blocks take the faces from the last one
// down, so that the boundary faces (FP64 ghost states, the longest chains)
// start first.  Bound by integer issue and latency (ALU 70%, issue 60%): 64
// registers for 32 warps an SM (72 registers, 24 warps: 84 us for 81, with
// the local time step 111 for 92).
template <int FLUX, int ORDER, int DT>
__global__ void __launch_bounds__(fvgb::kMaxBlock, 2) k_face_fx(const O2Args a) {
    const int f = (gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x;
    double cand = DBL_MAX;
    const bool live = f < a.m.n_faces && (!a.active || a.active[a.cell_inst[a.m.fl[f]]]);
    if (live) {
        const St* W = static_cast<const St*>(a.W);
        const double4_32a q = a.m.fgeom[f];
        const double nx = q.x, ny = q.y, ar = q.z;
        V4<double> wl, wr;
        int L = 0, R;
        if (ORDER == 2) {
            const int2 ee = __ldg(a.fe + f);
            wl = WStore<double>::ld(a.wf, ee.x);
            R = ee.y;
            if (R >= 0) wr = WStore<double>::ld(a.wf, ee.y);
        } else {
            L = a.m.fl[f];
            R = a.m.fr[f];
            wl = WStore<double>::ld(W, L);
            if (R >= 0) wr = WStore<double>::ld(W, R);
        }
        if (R < 0) wr = ghost_fast(a, f, a.m.fl[f], wl, nx, ny);
        V4<double> F;
        double unused;
        if (!fvfix::flux<FLUX == FLUX_HLLC ? 1 : 0, false, false>(wl, wr, 0.0, 0.0, fvfix::NoCons{}, fvfix::NoCons{}, nx,
                                                                         ny, ar, a.fxc, F, true, unused))
            F = face_flux_f64<FLUX>(wl, wr, nx, ny, ar, a.gamma, a.igm1);
        st_flux(static_cast<St*>(a.ff), f, F);
        if (DT != 0) {
            // compute_dt's per-face candidate from cell-centred states, as in
            // k_face: in FP64, beside the integer work
            const double* cs = static_cast<const double*>(a.cs);
            if (ORDER == 2) {
                L = a.m.fl[f];
                R = a.m.fr[f];
            }
            const V4<double> wlc = WStore<double>::ld(W, L);
            double Smax = fabs(wlc.u * nx + wlc.v * ny) + cs[L];
            if (R >= 0) {
                const V4<double> wrc = WStore<double>::ld(W, R);
                Smax = rmax(Smax, fabs(wrc.u * nx + wrc.v * ny) + cs[R]);
            }
            if (DT == 2) a.dtf[f] = Smax * ar;
            else cand = (a.ctl->cfl * q.w) * fvconv::rcp_nr3(Smax);
        }
    }
    if (DT == 1) block_min_dt(cand, a.ctl);
}

}  // namespace FV_KNS
