// FP64-class arithmetic on the integer pipe, in block fixed point.
//
// GB300 issues 1.7 FP64 thread instructions per SM-clock (add, multiply and
// fused multiply-add alike, 64 clocks from one dependent instruction to the
// next), but 64 32-bit integer ones and 24 32 x 32 + 64 -> 64 multiply-adds
// (5 and 13 clocks).  A sum of products whose terms share a power-of-two
// scale therefore costs a fraction of its FP64 price as 64-bit integers:
// an addition is two instructions, a product three multiply-adds and a
// funnel shift.
//
// Format "Qn": the integer i stands for i * 2^-n times a scale 2^k that the
// caller keeps per quantity (density, velocity, pressure of one face; one
// primitive variable of one cell).  Scales come from the operands' own
// exponents, so the largest operand of a block has its leading bit at a
// fixed place and keeps all its 53 bits with 4 to 7 bits below them; a
// smaller operand loses only bits below 2^-58 of the largest.  That is the
// absolute size of every error here, against 2^-53 of the result for each
// FP64 operation: a component far below its block's scale keeps fewer bits of its
// own (normals within 2^-20 of an axis beside a velocity 2^-20 of the other: the
// small momentum flux to 3e-7 of itself, 3e-17 of the face's scale; FP64 3e-14 and
// 5e-17).  Inputs outside the ranges that rule out overflow (checked
// from the exponents and from the intermediate values) are reported, and the
// caller evaluates them in FP64: zeros, subnormals, infinities, NaN,
// non-positive densities and pressures, density ratios above 16, pressure
// ratios above 32 or Mach numbers above about 8 across one face, and the
// rest of what a solver meets only while it diverges.
#pragma once

#include <cstdint>

#include "fixed_types.h"

namespace fvfix {

using i64 = long long;
using u64 = unsigned long long;

// v = h * 2^32 + l with l signed, so that all partial products are
// signed 32 x 32; v below 2^63 - 2^31, as h rounds up.
struct Sp { int h, l; };
__device__ __forceinline__ Sp split(i64 v) {
    const int l = (int)v;
    return {(int)(v >> 32) + (int)((unsigned)l >> 31), l};
}
__device__ __forceinline__ i64 madw(int a, int b, i64 c) {
    i64 r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 madwu(unsigned a, unsigned b, u64 c) {
    u64 r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// 64 bits of hi * 2^32 + lo (lo the low word) shifted left by S (0 < S < 32)
__device__ __forceinline__ i64 funnel(i64 hi, unsigned lo, int S) {
    const unsigned h1 = (unsigned)((u64)hi >> 32), h0 = (unsigned)hi;
    const unsigned r1 = __funnelshift_l(h0, h1, S), r0 = __funnelshift_l(lo, h0, S);
    return (i64)(((u64)r1 << 32) | r0);
}
// a * b >> (64 - S), without the product of the low halves (an error below
// 2^(S-2) units of the result).  The middle sum must stay below 2^63:
// |a| + |b| < 2^64, i.e. below 16 in Q60.
template <int S>
__device__ __forceinline__ i64 mul(const Sp& a, const Sp& b) {
    const i64 mid = madw(a.h, b.l, (i64)a.l * b.h);
    if (S == 0) return madw(a.h, b.h, (i64)(int)(mid >> 32));
    return funnel(madw(a.h, b.h, (i64)(int)(mid >> 32)), (unsigned)mid, S);
}
template <int S> __device__ __forceinline__ i64 mul(i64 a, i64 b) { return mul<S>(split(a), split(b)); }
// v * m >> (32 - S) for v >= 0 and a 32-bit m >= 0
template <int S>
__device__ __forceinline__ i64 mul_u32(i64 v, unsigned m) {
    const u64 t = madwu((unsigned)v, m, 0);
    return funnel((i64)madwu((unsigned)((u64)v >> 32), m, t >> 32), (unsigned)t, S);
}

__device__ __forceinline__ i64 iabs(i64 x) { return x < 0 ? -x : x; }

__device__ __forceinline__ int hi_word(double x) { return __double2hiint(x); }
__device__ __forceinline__ int biased(int hi) { return (hi >> 20) & 0x7ff; }

// |x| * 2^63 / 2^(e+1) for a normal x of biased exponent e: the 53
// significant bits at the top of 64.
__device__ __forceinline__ u64 top_bits(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    return ((u64)(__funnelshift_l(lo, hi, 11) | 0x80000000u) << 32) | (lo << 11);
}
// top_bits >> n for 0 < n < 32
__device__ __forceinline__ i64 shr_short(u64 t, int n) {
    const unsigned h = (unsigned)(t >> 32);
    return (i64)(((u64)(h >> n) << 32) | __funnelshift_r((unsigned)t, h, n));
}
// t >> n, 0 for n >= 64
__device__ __forceinline__ u64 shr(u64 t, int n) {
    u64 r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(t), "r"(n));
    return r;
}
// x as an integer in units of 2^(E - 1023 - Q): E a biased exponent not
// below x's own (x < 2^(E - 1023 + 1)) and at least 64, Q <= 62.  Zeros and
// subnormals give 0; bits below the unit are dropped.
// With neg (0 or -1) the value changes sign.
template <int Q>
__device__ __forceinline__ i64 to_fixed(double x, int E, int neg = 0) {
    const int hi = __double2hiint(x);
    const i64 s = (i64)((hi >> 31) ^ neg);
    return ((i64)shr(top_bits(x), E - biased(hi) + (63 - Q)) ^ s) - s;
}
// i * 2^k by the exponent field (i converted by the FP64 pipe; the result
// is normal or i is 0)
__device__ __forceinline__ double to_double(i64 i, int k) {
    const double d = __ll2double_rn(i);
    const int hi = __double2hiint(d);
    return i == 0 ? 0.0 : __hiloint2double(hi + (k << 20), __double2loint(d));
}
__device__ __forceinline__ double scale2(double x, int k) {
    return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
}

// ---------------------------------------------------------------------------
// Numerical fluxes of one face
// ---------------------------------------------------------------------------
// Units of a face: density 2^(er+1) above the larger density, velocity 2^ev
// above every velocity component and both sound speeds, pressure their
// product r v^2, energy four times that.  In these units densities, speeds
// and sound speeds are below 1, pressures below 1/gamma, everything else
// below 8, the range of Q60.
struct State { double r, u, v, p; };
struct NoCons {};  // no conserved states given

__device__ __forceinline__ float mant_float(double x, int k) {
    // mantissa of x (in [1, 2)) times 2^k, truncated to 24 bits
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    return __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) + ((unsigned)(127 + k) << 23));
}
__device__ __forceinline__ float rcp_f(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_f(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// sqrt(gp / r) in Q60 from gp = gamma p and x = gp r (both Q60), Y = the
// Q24 approximation of 1/sqrt(x) within 2^-21: with e = 1 - x Y^2 (below
// 2^-20, formed exactly to 2^-60) gp Y (1 + e/2 + 3 e^2/8) leaves 5 e^3/16 <
// 2^-62.
__device__ __forceinline__ i64 sound(i64 gp, i64 x, unsigned Y) {
    const i64 h = mul_u32<8>(gp, Y);
    const i64 z = mul_u32<8>(mul_u32<10>(x, Y), Y);  // x Y^2 in Q62
    const i64 e = ((i64)1 << 62) - z;
    const int e42 = (int)(e >> 20);
    const i64 w = (e >> 1) + (((i64)e42 * e42 * 3) >> 25);
    return h + mul<2>(split(h), split(w));
}
// 1 / D in Q58 for D (Q60) in [2^-4, 4)
__device__ __forceinline__ i64 recip(i64 D) {
    const float rf = rcp_f((float)(int)(D >> 32));  // 2^-28 / D
    const int R0 = __float2int_rn(rf * 18014398509481984.0f);  // 2^54: Q26
    const i64 z = mul_u32<8>(D, (unsigned)R0);  // D R0 in Q62
    const i64 e = ((i64)1 << 62) - z;
    const int e42 = (int)(e >> 20);
    const i64 g = e + (((i64)e42 * e42) >> 22);
    const Sp q = split(g);
    const i64 t = (i64)q.l * R0;
    return ((i64)R0 << 32) + funnel(madw(q.h, R0, (i64)(int)(t >> 32)), (unsigned)t, 2);
}

// Flux times the face length: FLUX 0 Rusanov, 1 HLLC, on primitive inputs
// (r, u, v, p) and, with C, the sound speeds and the conserved states, whose
// energies (and momenta, for Rusanov's dissipation) are taken instead of
// formed.  False where the ranges do not hold (F is not set then).  With LAM, lam is the face's largest wave speed
// max(|Vn| + c) over both sides, or the left one's (`both` false).
//
// Bound: the integer pipes (about 620 32-bit and 120 wide multiply-add
// instructions for HLLC, next to the 8 FP64 ones that convert and scale the
// result; the FP64 form takes 94 FP64 instructions a face).
template <int FLUX, bool C, bool LAM, typename W, typename Cons>
__device__ __forceinline__ bool flux(const W& L, const W& R, double cLd, double cRd, const Cons& UL, const Cons& UR,
                                     double nx, double ny, double ar, const FluxConst& k, W& F, bool both,
                                     double& lam) {
    const int rLh = hi_word(L.r), rRh = hi_word(R.r), pLh = hi_word(L.p), pRh = hi_word(R.p);
    const int erL = (int)((unsigned)rLh >> 20), erR = (int)((unsigned)rRh >> 20);  // sign included: must be clear
    const int epL = (int)((unsigned)pLh >> 20), epR = (int)((unsigned)pRh >> 20);
    const int er = max(erL, erR), ep = max(epL, epR);
    const int eu = max(max(biased(hi_word(L.u)), biased(hi_word(L.v))), max(biased(hi_word(R.u)), biased(hi_word(R.v))));
    const int ea = (int)((unsigned)hi_word(ar) >> 20);
    // exponents within 2^+-100, ratios across the face within 2^4 and 2^5
    bool bad = (unsigned)(er - 923) > 200u || (unsigned)(ep - 923) > 200u || eu > 1123 || (unsigned)(ea - 723) > 600u;
    bad |= er - min(erL, erR) > 4 || ep - min(epL, epR) > 5;
    if (bad) return false;
    int ev;
    unsigned YL = 0, YR = 0;
    if constexpr (C) {
        const int ecL = (int)((unsigned)hi_word(cLd) >> 20), ecR = (int)((unsigned)hi_word(cRd) >> 20);
        if ((unsigned)(ecL - 823) > 400u || (unsigned)(ecR - 823) > 400u) return false;
        ev = max(eu, max(ecL, ecR)) - 1022;
        if (ev + 1022 - min(ecL, ecR) > 5) return false;
    } else {
        // sound speeds to 2^-21: c = c^ 2^kc
        const int d = ep - er, kc = d >> 1, odd = d & 1;
        const float gpL = k.gammaf * mant_float(L.p, epL - ep + odd), gpR = k.gammaf * mant_float(R.p, epR - ep + odd);
        const float yL = rsqrt_f(gpL * mant_float(L.r, erL - er)), yR = rsqrt_f(gpR * mant_float(R.r, erR - er));
        const float cmax = fmaxf(gpL * yL, gpR * yR);
        ev = max(eu - 1023, kc + (int)(__float_as_uint(cmax) >> 23) - 127) + 1;
        if (ev - kc > 4) return false;
        const float ysc = __uint_as_float((unsigned)(127 + 25 + ev - kc) << 23);
        const float YfL = yL * ysc, YfR = yR * ysc;
        if (fmaxf(YfL, YfR) >= 1073741824.0f) return false;  // Q24 below 2^30
        YL = (unsigned)__float2int_rn(YfL);
        YR = (unsigned)__float2int_rn(YfR);
    }
    // fixed point
    const int ep1 = er + 1 + 2 * ev;
    if (ep1 - min(epL, epR) > 9) return false;
    const Sp rL = split(shr_short(top_bits(L.r), er + 4 - erL)), rR = split(shr_short(top_bits(R.r), er + 4 - erR));
    const i64 pLq = shr_short(top_bits(L.p), ep1 + 3 - epL), pRq = shr_short(top_bits(R.p), ep1 + 3 - epR);
    const Sp pL = split(pLq), pR = split(pRq);
    const int evb = ev + 1023;  // above 1023 - 105
    const int emb = er + 1 + ev, eeb = er + 3 + 2 * ev;  // units of momentum and of energy / 4
    if constexpr (C) {
        if (max(biased(hi_word(UL.E)), biased(hi_word(UR.E))) > eeb) return false;
    }
    const Sp uL = split(to_fixed<60>(L.u, evb)), vL = split(to_fixed<60>(L.v, evb));
    const Sp uR = split(to_fixed<60>(R.u, evb)), vR = split(to_fixed<60>(R.v, evb));
    const Sp nX = split(to_fixed<60>(nx, 1023)), nY = split(to_fixed<60>(ny, 1023));
    i64 cL, cR;
    if constexpr (C) {
        cL = shr_short(top_bits(cLd), evb + 3 - biased(hi_word(cLd)));
        cR = shr_short(top_bits(cRd), evb + 3 - biased(hi_word(cRd)));
    } else {
        const Sp gam = split(k.gamma);
        const i64 gL = mul<4>(gam, pL), gR = mul<4>(gam, pR);  // gamma p
        cL = sound(gL, mul<4>(split(gL), rL), YL);
        cR = sound(gR, mul<4>(split(gR), rR), YR);
    }
    const i64 VL = mul<4>(uL, nX) + mul<4>(vL, nY), VR = mul<4>(uR, nX) + mul<4>(vR, nY);
    // mass in Q60, momentum and energy / 4 in Q60 (Rusanov: below 5) or Q58
    constexpr int Qm = FLUX == 0 ? 60 : 58;
    i64 f0, f1, f2, f3;
    if constexpr (FLUX == 0) {
        const i64 S = max(iabs(VL) + cL, iabs(VR) + cR);
        const Sp S2 = split(S >> 1), vnL = split(VL), vnR = split(VR);
        const Sp mL = split(mul<4>(rL, vnL) >> 1), mR = split(mul<4>(rR, vnR) >> 1);  // half the mass fluxes
        i64 EL, ER, du, dv;
        if constexpr (C) {
            EL = to_fixed<60>(UL.E, eeb);
            ER = to_fixed<60>(UR.E, eeb);
            du = to_fixed<60>(UR.ru, emb) - to_fixed<60>(UL.ru, emb);
            dv = to_fixed<60>(UR.rv, emb) - to_fixed<60>(UL.rv, emb);
        } else {
            const Sp ig = split(k.igm1_4);
            const i64 qL = mul<4>(uL, uL) + mul<4>(vL, vL), qR = mul<4>(uR, uR) + mul<4>(vR, vR);
            EL = mul<4>(pL, ig) + (mul<4>(rL, split(qL)) >> 3);
            ER = mul<4>(pR, ig) + (mul<4>(rR, split(qR)) >> 3);
            du = mul<4>(rR, uR) - mul<4>(rL, uL);
            dv = mul<4>(rR, vR) - mul<4>(rL, vL);
        }
        const Sp ps = split((pLq >> 1) + (pRq >> 1));
        const i64 rLq = ((i64)rL.h << 32) + rL.l, rRq = ((i64)rR.h << 32) + rR.l;
        f0 = (mul<4>(rL, vnL) >> 1) + (mul<4>(rR, vnR) >> 1) - mul<4>(S2, split(rRq - rLq));
        f1 = mul<4>(mL, uL) + mul<4>(mR, uR) + mul<4>(ps, nX) - mul<4>(S2, split(du));
        f2 = mul<4>(mL, vL) + mul<4>(mR, vR) + mul<4>(ps, nY) - mul<4>(S2, split(dv));
        f3 = (mul<4>(split(EL + (pLq >> 2)), vnL) >> 1) + (mul<4>(split(ER + (pRq >> 2)), vnR) >> 1) -
             mul<4>(S2, split(ER - EL));
    } else {
        const i64 SL = min(VL - cL, VR - cR), SR = max(VL + cL, VR + cR);
        const i64 dL = SL - VL, dR = SR - VR;  // dL < 0 < dR
        const i64 mL = mul<4>(rL, split(dL)), mR = mul<4>(rR, split(dR));
        const i64 num = pRq - pLq + mul<4>(split(mL), split(VL)) - mul<4>(split(mR), split(VR));
        const i64 D = mR - mL;  // S* = -num / D
        constexpr i64 one = (i64)1 << 60;
        bad = max(-dL, dR) >= 2 * one || D < one / 16;
        const bool supL = SL >= 0, supR = !supL && SR <= 0, sup = supL || supR;
        const bool left = supL || (!supR && num <= 0);
        const Sp rK = left ? rL : rR, uK = left ? uL : uR, vK = left ? vL : vR, pK = left ? pL : pR;
        const i64 VK = left ? VL : VR, pKq = left ? pLq : pRq, SK = left ? SL : SR, mK = left ? mL : mR;
        const i64 dK = left ? dL : dR;
        i64 EK;  // E / 4
        if constexpr (C) EK = to_fixed<60>(left ? UL.E : UR.E, eeb);
        else EK = mul<4>(pK, split(k.igm1_4)) + (mul<4>(rK, split(mul<4>(uK, uK) + mul<4>(vK, vK))) >> 3);
        i64 Ss, fac, Es, ps, w = 0;
        if (sup) {
            Ss = VK;
            fac = ((i64)rK.h << 32) + rK.l;
            Es = EK;
            ps = pKq;
        } else {
            // |S*| < 2, |S* - Vn| < 2 and |S_K - S*| >= 1/16 keep what
            // follows in range; S* itself is checked in float first
            const i64 Dc = D < one / 16 ? one : D;
            const float s_f = (float)(int)(num >> 32) * rcp_f((float)(int)(Dc >> 32));
            if (!(fabsf(s_f) < 1.99f)) return false;
            Ss = -mul<6>(split(num), split(recip(Dc)));
            w = Ss - VK;
            const i64 gap = left ? Ss - SK : SK - Ss;  // > 0
            bad |= gap < one / 16 || gap >= 4 * one - 1 || iabs(w) >= 2 * one;
            if (bad) return false;
            const i64 Rq = recip(gap);
            const Sp Rs = split(left ? -Rq : Rq);  // 1 / (S_K - S*) in Q58
            const float fac_f = (float)(int)(mK >> 32) * (float)Rs.h;  // Q28 * Q26
            if (!(fabsf(fac_f) < 1.99f * 18014398509481984.0f)) return false;
            fac = mul<6>(split(mK), Rs);
            ps = pKq + mul<4>(split(mK), split(w));
            const i64 A = mul<4>(split(dK), split(EK)) - (mul<4>(pK, split(VK)) >> 2) + (mul<4>(split(ps), split(Ss)) >> 2);
            const float es_f = (float)(int)(A >> 32) * (float)Rs.h;
            if (!(fabsf(es_f) < 3.99f * 18014398509481984.0f)) return false;
            Es = mul<6>(split(A), Rs);
        }
        if (bad && !sup) return false;
        const Sp sS = split(Ss);
        f0 = mul<4>(split(fac), sS);
        const Sp M = split(f0);
        const Sp T = split((ps >> 2) + mul<2>(M, split(w)));  // momentum along n, less M Vn, Q58
        f1 = mul<2>(M, uK) + mul<4>(T, nX);
        f2 = mul<2>(M, vK) + mul<4>(T, nY);
        f3 = mul<2>(sS, split(Es + (ps >> 2)));
    }
    if constexpr (LAM) {
        const i64 sL = iabs(VL) + cL;
        lam = scale2(__ll2double_rn(both ? max(sL, iabs(VR) + cR) : sL), ev - 60);
    }
    const int k0 = er - 1023 + 1 + ev;
    const double s0 = scale2(ar, k0 - 60), s1 = scale2(ar, k0 + ev - Qm), s2 = scale2(ar, k0 + 2 * ev + 2 - Qm);
    F.r = __ll2double_rn(f0) * s0;
    F.u = __ll2double_rn(f1) * s1;
    F.v = __ll2double_rn(f2) * s1;
    F.p = __ll2double_rn(f3) * s2;
    return true;
}

// a * b >> 60 to one unit: mul<4> with the low halves' product
__device__ __forceinline__ i64 mul_low(const Sp& a, const Sp& b) {
    const i64 mid = madw(a.h, b.l, madw(a.l, b.h, (i64)a.l * b.l >> 32));
    return funnel(madw(a.h, b.h, (i64)(int)(mid >> 32)), (unsigned)mid, 4);
}
// Sound speed sqrt(g p / r) rounded once but for 2^-56 of it, with one FP64
// instruction (the FP64 form takes ten); false outside the ranges.
__device__ __forceinline__ bool sound_speed(double r, double p, double g, double& c) {
    const int er = (int)((unsigned)hi_word(r) >> 20), ep = (int)((unsigned)hi_word(p) >> 20);
    const int eg = (int)((unsigned)hi_word(g) >> 20) - 1023;  // 0 or 1: gamma in [1, 4)
    if ((unsigned)(er - 723) > 600u || (unsigned)(ep - 723) > 600u || (unsigned)eg > 1u) return false;
    // r = m 2^er, p = q 2^(er + 2 kc) with q in [1, 4): c = sqrt(g q / m) 2^kc
    const int kc = (ep - er) >> 1, odd = (ep - er) & 1;
    const float y = rsqrt_f((float)g * mant_float(p, odd) * mant_float(r, 0));
    const i64 m4 = shr_short(top_bits(r), 5), g2 = shr_short(top_bits(g), 4 - eg), q2 = shr_short(top_bits(p), 4 - odd);
    const i64 gq = mul_low(split(g2), split(q2));  // g q / 4, below 4
    const i64 x = mul_low(split(gq), split(m4));   // g q m / 16, below 2
    c = scale2(__ll2double_rn(sound(gq, x, (unsigned)__float2int_rn(y * 67108864.0f))), kc - 60);  // Q24 of 4 y
    return true;
}

// m * 2^k
struct Fixed { i64 m; int k; };
__device__ __forceinline__ double value(const Fixed& x) { return to_double(x.m, x.k); }

// The signed sum of N FP64 values (bit 0 of neg[i] flips the sign of x[i]) in
// fixed point: exact but for bits below 2^-59 of the largest.  False where a
// value is not finite, or all are zero or below 2^-873.
template <int N>
__device__ __forceinline__ bool fixed_sum(const double (&x)[N], const int (&neg)[N], Fixed& s) {
    int E = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) E = max(E, biased(hi_word(x[i])));
    s.m = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) s.m += to_fixed<59>(x[i], E, -(neg[i] & 1));
    s.k = E - 1023 - 59;
    return (unsigned)(E - 150) <= 1750u;
}
template <int N>
__device__ __forceinline__ double signed_sum(const double (&x)[N], const int (&neg)[N]) {
    Fixed q;
    if (fixed_sum<N>(x, neg, q)) return value(q);
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) s += neg[i] & 1 ? -x[i] : x[i];
    return s;
}
// One component of a Shu-Osher stage, with e = u + dtv R: stage 1 (3 u0 + e) / 4,
// stage 2 (u0 + 2 e) / 3, as integers in units of 2^-59 of the largest term's
// binade (an FP64 form rounds three or four times at 2^-53).  False out of
// range.
template <int STAGE>
__device__ __forceinline__ bool rk_stage(double u, double u0, const Fixed& R, double dtv, double& un) {
    const int ed = (int)((unsigned)hi_word(dtv) >> 20);  // sign included: must be clear
    const i64 mag = iabs(R.m);
    const int lz = mag ? __clzll(mag) : 63;
    const int er = R.k + 64 - lz + ed;  // above the biased exponent of dtv R
    const int E = max(max(biased(hi_word(u)), biased(hi_word(u0))), er);
    // dtv R: R's leading bit at 2^61 times dtv's at 2^61 (one place higher,
    // a mantissa of ones would overflow split's high half), >> 62: below 2^62
    // in units of 2^(er - 1023 - 62)
    const i64 p = mul<2>(split(R.m << (lz - 2)), split((i64)(top_bits(dtv) >> 2)));
    i64 q;
    asm("shr.s64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(E - er + 1));
    const i64 a = to_fixed<59>(u0, E), e = to_fixed<59>(u, E) + ((q + 1) >> 1);
    // rounded, not floored: a floor's bias would add up over the steps
    const i64 s = STAGE == 1 ? (a + a + a + e + 2) >> 2 : mul<2>(split(a + e + e + 1), split(0x1555555555555555ll));
    un = to_double(s, E - 1023 - 59);
    return (unsigned)(E - 150) <= 1750u && (unsigned)(ed - 123) < 1800u && lz > 1;
}

// a / s for a > 0 and a sum s > 0 of the above, rounded once but for 2^-55 of
// it; false out of range.
__device__ __forceinline__ bool quotient(double a, const Fixed& s, double& q) {
    const int ea = (int)((unsigned)hi_word(a) >> 20);  // sign included: must be clear
    if ((unsigned)(ea - 123) >= 1800u || s.m <= 0) return false;
    const int lz = __clzll(s.m);  // at least 2
    const i64 D = lz >= 3 ? s.m << (lz - 3) : s.m >> 1;  // in [1, 2) of Q60, times 2^(s.k + 63 - lz)
    const i64 x = mul_low(split((i64)(top_bits(a) >> 3)), split(recip(D)));  // Q58
    q = to_double(x, ea - 1023 - (s.k + 63 - lz) - 58);
    return abs(ea - 1023 - (s.k + 63 - lz)) < 900;
}
// x^2 in units of 2^(2 (E - 1023) - 57), E the warp's largest biased exponent:
// rounded, below 2^59, so that 32 of them add up exactly in 64 bits.  All 32
// lanes call it; false (on all) where a value is not finite or its square out
// of range.
__device__ __forceinline__ bool warp_square(double x, u64& v, int& E) {
    const int e = biased(hi_word(x));
    E = __reduce_max_sync(0xffffffffu, e);
    const Sp m = split((i64)(top_bits(x) >> 3));  // Q60, in [1, 2)
    v = e == 0 ? 0 : (shr((u64)mul<1>(m, m) << 1, 2 * (E - e)) + 1) >> 1;
    return E <= 1500 && (E == 0 || E >= 550);
}
// The sum of x^2 over a warp, in every lane; as above.
__device__ __forceinline__ bool warp_squares(double x, double& sum) {
    u64 s;
    int E;
    const bool ok = warp_square(x, s, E);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    sum = s == 0 ? 0.0 : scale2(__ull2double_rn(s), 2 * (E - 1023) - 57);
    return ok;
}
// The sums over a warp of x^2 for four values a lane (all 32 lanes call it):
// the k-th in the lanes 8 k to 8 k + 7, as warp_sum4's; one FP64 instruction
// instead of ten.
__device__ __forceinline__ bool warp_squares4(const double (&x)[4], double& sum) {
    u64 v[4];
    int E[4];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) ok &= warp_square(x[k], v[k], E[k]);
    const int lane = threadIdx.x & 31;
    const bool h16 = lane & 16, h8 = lane & 8;
    u64 a = h16 ? v[2] : v[0], b = h16 ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[2], 16);
    b += __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[3], 16);
    u64 s = h8 ? b : a;
    s += __shfl_xor_sync(0xffffffffu, h8 ? a : b, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    const int e = h16 ? (h8 ? E[3] : E[2]) : (h8 ? E[1] : E[0]);
    sum = s == 0 ? 0.0 : scale2(__ull2double_rn(s), 2 * (e - 1023) - 57);
    return ok;
}

// num / den * 2^60 for 0 < num <= den, den in [2^56, 2^62): three quotient
// digits of 20 bits, each from the float quotient of the exact remainder (within
// 3/4 of a unit), rounded to 53 significant bits: exact as a double.
__device__ __forceinline__ i64 ratio60(i64 num, i64 den) {
    const float rf = rcp_f((float)(unsigned)((u64)den >> 32));
    const int q1 = __float2int_rn((float)(int)(num >> 32) * rf * 1048576.0f);
    i64 t = (num << 20) - (i64)q1 * den;
    const int q2 = __float2int_rn((float)(int)(t >> 32) * rf * 1048576.0f);
    t = (t << 20) - (i64)q2 * den;
    const int q3 = __float2int_rn((float)(int)(t >> 32) * rf * 1048576.0f);
    const i64 q = ((i64)q1 << 40) + ((i64)q2 << 20) + q3;
    const unsigned one = 1u << max(11 - __clz((int)(q >> 32)), 0);  // the last of 53 bits, if above bit 0
    const i64 r = q + (one >> 1);
    return min((i64)((u64)r & ~(u64)(one - 1u)), (i64)1 << 60);
}

}  // namespace fvfix
