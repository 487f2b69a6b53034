// Hand-written reverse mode of the sweep's face function for the adjoint
// (isothermal EOS, the configuration the adjoint covers).
//
// Each function replays the FP64 building block of pg_hydro.cuh with the
// same expressions, keeping the intermediates it needs on a small tape (a
// struct), and then propagates adjoints backwards through the branch the
// replay took: limiter selections, clamps of the swept fraction, floors,
// HLLC wave signs.  The result equals the dual-number derivative of the
// same blocks (pg_dual.cuh) contracted with the output adjoint; the dual
// kernels check it.  Adjoints accumulate into the caller's variables (+=).
#pragma once

#include <cmath>

#include "pg_hydro.cuh"

namespace pg {
namespace rev {

// ------------------------------------------------------------- HLLC (EOS 0)
// Adjoint of hllc(0, ie, gam, L, R) for the flux components r, u, v, w and pres
// (the energy fluxes vanish for EOS 0).  bF: {r, u, v, w, pres}.  The reciprocals of the
// replay serve the reverse as well, which has no division of its own.
__device__ __forceinline__ void hllc_rev(double gam, const Half& L, const Half& R, const double* bF, Half& bL,
                                         Half& bR) {
    const double sL = rsq(gam * L.p * L.r), sR = rsq(gam * R.p * R.r);  // c = gam p s, 1 / c = r s
    const double cl = __dmul_rn(gam * L.p, sL), cr = __dmul_rn(gam * R.p, sR);
    const double ic = inv(cl + cr);
    const double p_ = 0.5 * (R.p + L.p);
    const double xe = gam * (L.u - R.u) * ic;
    const double el = exp_lim(xe);
    const double pm = p_ * el;
    const double w = rsq(L.r * R.r), q = R.r * w, iq = inv(1.0 + q);
    const double K = L.u + q * R.u, u_ = K * iq;
    const double du = R.u - L.u;
    const double H = cl * cl + cr * cr * q;
    const double n2 = 0.5 * q * (iq * iq);
    const double c2 = H * iq + n2 * (du * du);
    const double icc = rsq(c2), cc = c2 * icc;
    const double sl = u_ - cc, sr = u_ + cc;
    const double ml = L.r * cl, mr = R.r * cr;
    const double num = ml * L.u + mr * R.u, id = inv(ml + mr);
    const double iS = inv(L.r + R.r), dp = L.p - R.p;
    const double q1 = num * id, q2 = 2.0 * dp * (iS * ic);
    const double sm = q1 + q2;
    const bool left = (std::signbit(sl) == 0) || (std::signbit(sr) == 0 && std::signbit(sm) == 0);
    const Half& S = left ? L : R;
    Half& bS = left ? bL : bR;
    const bool super = (std::signbit(sl) == 0 || std::signbit(sr) != 0);
    double Fr;
    double b_sl = 0.0, b_sr = 0.0, b_sm = 0.0, b_pm = 0.0;
    double s_ = 0.0, is = 0.0, A = 0.0, B = 0.0;
    if (super) {
        Fr = S.u * S.r;
    } else {
        s_ = left ? sl : sr;
        is = inv(s_ - sm);
        A = sm * S.r * (s_ - S.u);
        B = s_ * pm - sm * S.p;
        Fr = A * is;
    }
    // F.u = S.u F.r, F.v = S.v F.r, F.w = S.w F.r
    const double bFr = bF[0] + bF[1] * S.u + bF[2] * S.v + bF[3] * S.w;
    bS.u += bF[1] * Fr;
    bS.v += bF[2] * Fr;
    bS.w += bF[3] * Fr;
    if (super) {
        bS.u += bFr * S.r;
        bS.r += bFr * S.u;
        bS.p += bF[4];
    } else {
        const double b_is = (bFr * A + bF[4] * B) * (is * is);
        const double bA = bFr * is, bB = bF[4] * is;
        double b_s = -b_is;
        b_sm += b_is + bA * S.r * (s_ - S.u) - bB * S.p;
        bS.r += bA * sm * (s_ - S.u);
        b_s += bA * sm * S.r + bB * pm;
        bS.u -= bA * sm * S.r;
        b_pm += bB * s_;
        bS.p -= bB * sm;
        if (left) b_sl += b_s;
        else b_sr += b_s;
    }
    // sl = u_ - cc, sr = u_ + cc
    const double b_u = b_sl + b_sr;
    const double b_c2 = 0.5 * (b_sr - b_sl) * icc;
    double b_cl, b_cr, b_q, b_iq, b_ic;
    // sm = num id + 2 dp iS ic
    {
        const double b_num = b_sm * id, b_den = -b_num * q1;
        const double b_ml = b_num * L.u + b_den, b_mr = b_num * R.u + b_den;
        bL.u += b_num * ml;
        bR.u += b_num * mr;
        bL.r += b_ml * cl;
        b_cl = b_ml * L.r;
        bR.r += b_mr * cr;
        b_cr = b_mr * R.r;
        const double b_dp = 2.0 * b_sm * (iS * ic);
        bL.p += b_dp;
        bR.p -= b_dp;
        const double b_S = -b_sm * q2 * iS;
        bL.r += b_S;
        bR.r += b_S;
        b_ic = 2.0 * b_sm * dp * iS;
    }
    // c2 = H iq + n2 du^2, H = cl^2 + cr^2 q, n2 = q iq^2 / 2; u_ = (L.u + q R.u) iq
    {
        const double b_H = b_c2 * iq;
        b_iq = b_c2 * H;
        b_cl += 2.0 * b_H * cl;
        b_cr += 2.0 * b_H * cr * q;
        b_q = b_H * cr * cr;
        const double b_n2 = b_c2 * (du * du), b_du = 2.0 * b_c2 * n2 * du;
        bR.u += b_du;
        bL.u -= b_du;
        b_q += 0.5 * b_n2 * (iq * iq);
        b_iq += b_n2 * q * iq;
        const double b_K = b_u * iq;
        b_iq += b_u * K;
        bL.u += b_K;
        bR.u += b_K * q;
        b_q += b_K * R.u;
        b_q -= b_iq * (iq * iq);
        // q = sqrt(R.r / L.r): dq = q / 2 (dR.r / R.r - dL.r / L.r), and 1 / R.r = w q / (...)
        // taken from w = (L.r R.r)^-1/2: 1 / R.r = L.r w^2, 1 / L.r = R.r w^2
        const double hq = 0.5 * b_q * q * (w * w);
        bR.r += hq * L.r;
        bL.r -= hq * R.r;
    }
    // pm = p_ exp_lim(xe), xe = gam (L.u - R.u) ic, ic = 1 / (cl + cr)
    {
        const double b_p = 0.5 * b_pm * el;
        const double b_xe = (1.0e-6 > 1.0 + xe) ? 0.0 : b_pm * p_;
        const double g = b_xe * gam * ic;
        bL.u += g;
        bR.u -= g;
        b_ic += b_xe * gam * (L.u - R.u);
        bR.p += b_p;
        bL.p += b_p;
        const double b_c = -b_ic * (ic * ic);
        b_cl += b_c;
        b_cr += b_c;
    }
    // c = sqrt(gam p / r): dc = c / 2 (dp / p - dr / r) = gam s / 2 (dp - p s^2 gam p dr)
    {
        const double a = 0.5 * gam * b_cl * sL, b = 0.5 * gam * b_cr * sR;
        bL.p += a;
        bL.r -= a * L.p * (cl * sL);
        bR.p += b;
        bR.r -= b * R.p * (cr * sR);
    }
}

// ---------------------------------------------------------- reconstruction
// Tape of recon(): the slope selections, the zeroing and monotonicity branches.
struct ReconTape {
    double sL2, sR2;   // slopes after the extremum zeroing, before flattening
    signed char selL, selR;  // fmin picked |d1| / |d2| (1) or the 4th-order slope (0)
    signed char cfL, cfR;    // copysign factor
    signed char fsL, fsR;    // fabs factor of the chosen operand
    signed char zero, mono;  // extremum zeroing; monotonicity branch (0 none, 1 sL = 2 sR, 2 sR = 2 sL)
};

__device__ __forceinline__ double fabs_factor(double x) { return std::signbit(x) ? -1.0 : 1.0; }

__device__ __forceinline__ Par recon_tape(const double* __restrict__ w, double am2, double am1, double a0, double ap1,
                                          double ap2, double flat, ReconTape& t) {
    const double d0 = am1 - am2, d1 = a0 - am1, d2 = ap1 - a0, d3 = ap2 - ap1;
    const double sL0 = w[0] * d0 + w[1] * d1 + w[2] * d2;
    const double sR0 = w[3] * d1 + w[4] * d2 + w[5] * d3;
    const double aL = fabs(sL0), bL = fabs(d1);
    const double mL = (bL < aL) ? bL : aL;
    t.selL = (bL < aL) ? 1 : 0;
    t.fsL = (signed char)fabs_factor(t.selL ? d1 : sL0);
    double sL = copysign(mL, d1);
    t.cfL = (std::signbit(sL) == std::signbit(mL)) ? 1 : -1;
    const double aR = fabs(sR0), bR = fabs(d2);
    const double mR = (bR < aR) ? bR : aR;
    t.selR = (bR < aR) ? 1 : 0;
    t.fsR = (signed char)fabs_factor(t.selR ? d2 : sR0);
    double sR = copysign(mR, d2);
    t.cfR = (std::signbit(sR) == std::signbit(mR)) ? 1 : -1;
    t.zero = (sR * sL <= 0.0) ? 1 : 0;
    if (t.zero) {
        sL = 0.0;
        sR = 0.0;
    }
    t.sL2 = sL;
    t.sR2 = sR;
    sR *= (1.0 - flat);
    sL *= (1.0 - flat);
    // slopes of one sign: each at most twice the other in size (recon, pg_hydro.cuh)
    t.mono = 0;
    if (fabs(sL) > 2.0 * fabs(sR)) {
        sL = 2.0 * sR;
        t.mono = 1;
    } else if (fabs(sR) > 2.0 * fabs(sL)) {
        sR = 2.0 * sL;
        t.mono = 2;
    }
    return {sL, a0, sR};
}

// bP: adjoint of {sL, a, sR}; accumulates into ba[5] (am2..ap2) and bflat
__device__ __forceinline__ void recon_rev(const double* __restrict__ w, const ReconTape& t, double flat,
                                          const Par& bP, double* ba, double& bflat) {
    double bsL3 = bP.sL, bsR3 = bP.sR;
    if (t.mono == 1) {
        bsR3 += 2.0 * bsL3;
        bsL3 = 0.0;
    } else if (t.mono == 2) {
        bsL3 += 2.0 * bsR3;
        bsR3 = 0.0;
    }
    bflat -= bsR3 * t.sR2 + bsL3 * t.sL2;
    double bsL = bsL3 * (1.0 - flat), bsR = bsR3 * (1.0 - flat);
    if (t.zero) {
        bsL = 0.0;
        bsR = 0.0;
    }
    double bd0 = 0.0, bd1 = 0.0, bd2 = 0.0, bd3 = 0.0;
    const double gL = bsL * t.cfL * t.fsL;
    if (t.selL) {
        bd1 += gL;
    } else {
        bd0 += w[0] * gL;
        bd1 += w[1] * gL;
        bd2 += w[2] * gL;
    }
    const double gR = bsR * t.cfR * t.fsR;
    if (t.selR) {
        bd2 += gR;
    } else {
        bd1 += w[3] * gR;
        bd2 += w[4] * gR;
        bd3 += w[5] * gR;
    }
    // d0 = am1 - am2, d1 = a0 - am1, d2 = ap1 - a0, d3 = ap2 - ap1
    ba[0] -= bd0;
    ba[1] += bd0 - bd1;
    ba[2] += bd1 - bd2 + bP.a;
    ba[3] += bd2 - bd3;
    ba[4] += bd3;
}

// ---------------------------------------------------------------- flattening
// Tape of flatten() (pg_hydro.cuh): f = 10 num big / (den p0) of the steeper side.
struct FlatTape {
    double p0, num, den, big, iD, f;
    signed char live, back, bigb;    // the coefficient is not constant; side; which |dp1| is the larger
    signed char s1, s2, sb;          // signs of dp1 - dp2 / 2, of dp2 and of the larger dp1
};

__device__ __forceinline__ double flatten_tape(double p0, double pm2, double pm1, double pp1, double pp2, double um1,
                                               double u0, double up1, FlatTape& t) {
    const double dp1f = pp1 - p0, dp2f = pp2 - pm1;
    const double dp1b = p0 - pm1, dp2b = pp1 - pm2;
    const double wf = fabs(dp2f), wb = fabs(dp2b);
    const double ef = dp1f - 0.5 * dp2f, eb = dp1b - 0.5 * dp2b;
    const double nf = fabs(ef) - 0.25 * wf;
    const double nb = fabs(eb) - 0.25 * wb;
    t.live = 0;
    if (!((u0 > up1 || um1 > u0) && wf > 0.0 && wb > 0.0 && (nf > 0.0 || nb > 0.0))) return 0.0;
    const bool back = nb * wf > nf * wb;
    const bool bigb = fabs(dp1b) > fabs(dp1f);
    t.p0 = p0;
    t.num = back ? nb : nf;
    t.den = back ? wb : wf;
    t.big = bigb ? fabs(dp1b) : fabs(dp1f);
    t.iD = inv(t.den * p0);
    t.back = back;
    t.bigb = bigb;
    t.s1 = (signed char)fabs_factor(back ? eb : ef);
    t.s2 = (signed char)fabs_factor(back ? dp2b : dp2f);
    t.sb = (signed char)fabs_factor(bigb ? dp1b : dp1f);
    t.f = 10.0 * t.num * t.big * t.iD;
    if (!(t.f < 0.5)) return 0.5;
    t.live = 1;
    return t.f;
}

// accumulates into bp[5] = (pm2, pm1, p0, pp1, pp2)
__device__ __forceinline__ void flatten_rev(const FlatTape& t, double bf, double* bp) {
    if (!t.live) return;
    const double g = 10.0 * bf * t.iD;
    const double b_num = g * t.big, b_big = g * t.num;
    const double b_D = -bf * t.f * t.iD;  // f = 10 num big / D, D = den p0
    bp[2] += b_D * t.den;
    const double b_den = b_D * t.p0 - 0.25 * b_num;  // num = |dp1 - dp2 / 2| - |dp2| / 4, den = |dp2|
    const double b_e = b_num * t.s1;
    const double b1 = b_e, b2 = b_den * t.s2 - 0.5 * b_e;
    double b_dp1f = 0.0, b_dp1b = 0.0, b_dp2f = 0.0, b_dp2b = 0.0;
    if (t.back) {
        b_dp1b = b1;
        b_dp2b = b2;
    } else {
        b_dp1f = b1;
        b_dp2f = b2;
    }
    if (t.bigb) b_dp1b += b_big * t.sb;
    else b_dp1f += b_big * t.sb;
    // dp1f = pp1 - p0, dp2f = pp2 - pm1, dp1b = p0 - pm1, dp2b = pp1 - pm2
    bp[3] += b_dp1f + b_dp2b;
    bp[2] += b_dp1b - b_dp1f;
    bp[4] += b_dp2f;
    bp[1] -= b_dp2f + b_dp1b;
    bp[0] -= b_dp2b;
}

// --------------------------------------------------- parabola averages
// Adjoints of aveL / aveR at the swept fraction x (frac): accumulate the Par adjoint and
// return the adjoint of x.
__device__ __forceinline__ double aveL_rev(double x, const Par& p, double b, Par& bp) {
    const double h = 0.5 * x, g = 1.0 - x * (2.0 / 3.0);
    const double a6 = 3.0 * (p.sL - p.sR);
    const double S = p.sR + p.sL;
    // aL + h (S + g a6), aL = a - sL
    const double bh = b * h;
    bp.a += b;
    bp.sL += bh * (1.0 + 3.0 * g) - b;
    bp.sR += bh * (1.0 - 3.0 * g);
    return b * (0.5 * (S + g * a6) - h * a6 * (2.0 / 3.0));
}
__device__ __forceinline__ double aveR_rev(double x, const Par& p, double b, Par& bp) {
    const double h = 0.5 * x, g = 1.0 - x * (2.0 / 3.0);
    const double a6 = 3.0 * (p.sL - p.sR);
    const double S = p.sR + p.sL;
    // aR - h (S - g a6), aR = a + sR
    const double bh = b * h;
    bp.a += b;
    bp.sL -= bh * (1.0 - 3.0 * g);
    bp.sR += b - bh * (1.0 + 3.0 * g);
    return -b * (0.5 * (S - g * a6) + h * a6 * (2.0 / 3.0));
}

// ------------------------------------------------------- interface states
// Adjoint of state_at_left_edge (SIDE 0) or state_at_right_edge (SIDE 1)
// (states.cu:151-264) given bs, the adjoint of the returned state: the forward's
// expressions (pg_hydro.cuh), then back through the branches they took.  V is the one
// transported field (v or w, adjoint bt).  Accumulates into bcs0, br0c, bp0c, bu0c and the
// Par adjoints.
template <int SIDE>
__device__ __forceinline__ double ave(double x, const Par& p) {
    return SIDE == 0 ? aveL(frac(x), p) : aveR(frac(x), p);
}
template <int SIDE>
__device__ __forceinline__ double ave_rev(double x, const Par& p, double b, Par& bp) {
    return SIDE == 0 ? aveL_rev(x, p, b, bp) : aveR_rev(x, p, b, bp);
}
template <int SIDE>
__device__ __forceinline__ void state_rev(double gam, double sx, double cs0, double r0c, double p0c, double u0c,
                                          const Par& R, const Par& Pp, const Par& U, const Par& V, const Half& bs,
                                          double bt, double& bcs0, double& br0c, double& bp0c, double& bu0c, Par& bR,
                                          Par& bP, Par& bU, Par& bV) {
    constexpr double sg = SIDE == 0 ? -1.0 : 1.0;  // the speed towards the edge is sg u
    // forward replay
    const bool t0pass = !(0.0 > sg * u0c);
    const double x1r = (cs0 + (t0pass ? sg * u0c : 0.0)) * sx;
    const bool pass1 = !(1.0 < x1r);
    const double x1 = pass1 ? x1r : 1.0;
    const double ue = ave<SIDE>(x1, U);
    const bool dpass = !(0.0 > sg * ue);
    const double m = dpass ? sg * ue : 0.0;  // >= 0
    const double x2r = m * sx;
    const bool pass2 = !(1.0 < x2r);
    const double x2 = pass2 ? x2r : 1.0;
    const double rmin = r0c * 1.0e-10, pmin = p0c * 1.0e-10;
    const double r0r = ave<SIDE>(x2, R), p0r = ave<SIDE>(x2, Pp), u0 = ave<SIDE>(x2, U);
    const bool rsel = rmin > r0r, psel = pmin > p0r;
    const double r0 = rsel ? rmin : r0r, p0 = psel ? pmin : p0r;
    const double g = gam * p0;
    const double s = rsq(g * r0);
    const double x3r = (g * s + m) * sx;
    const bool pass3 = !(1.0 < x3r);
    const double x3 = pass3 ? x3r : 1.0;
    const double uA = ave<SIDE>(x3, U), pA = ave<SIDE>(x3, Pp);
    const double ics = r0 * s;                        // 1 / cs
    const double eu = sg * (uA - u0), du = eu * ics;  // u0 - uA on the left, uA - u0 on the right
    const double dp = sg * (p0 - pA);
    const double E1 = exp_lim(du), E2 = exp_lim(gam * du);
    // reverse: r = r0 E1, p = p0 E2, u = u0 - dp s
    double bx3 = ave_rev<SIDE>(x3, V, bt, bV);
    double b_u0 = bs.u;
    const double b_dp = -bs.u * s;
    double b_s = -bs.u * dp;
    double b_p0 = bs.p * E2 + sg * b_dp, b_r0 = bs.r * E1;
    double b_du = 0.0;
    if (!(1.0e-6 > 1.0 + gam * du)) b_du += bs.p * p0 * gam;
    if (!(1.0e-6 > 1.0 + du)) b_du += bs.r * r0;
    const double b_eu = b_du * ics * sg;
    b_u0 -= b_eu;
    b_r0 += b_du * eu * s;
    b_s += b_du * eu * r0;
    bx3 += ave_rev<SIDE>(x3, U, b_eu, bU) + ave_rev<SIDE>(x3, Pp, -sg * b_dp, bP);
    double b_m = 0.0, b_g = 0.0;
    if (pass3) {
        const double b = bx3 * sx;
        b_g = b * s;
        b_s += b * g;
        b_m = b;
    }
    // s = (g r0)^-1/2
    const double b_gr = -0.5 * b_s * s * (s * s);
    b_g += b_gr * r0;
    b_r0 += b_gr * g;
    b_p0 += b_g * gam;
    double b_r0r = 0.0, b_p0r = 0.0;
    if (rsel) br0c += b_r0 * 1.0e-10;
    else b_r0r = b_r0;
    if (psel) bp0c += b_p0 * 1.0e-10;
    else b_p0r = b_p0;
    const double bx2 =
        ave_rev<SIDE>(x2, R, b_r0r, bR) + ave_rev<SIDE>(x2, Pp, b_p0r, bP) + ave_rev<SIDE>(x2, U, b_u0, bU);
    if (pass2) b_m += bx2 * sx;
    const double bx1 = ave_rev<SIDE>(x1, U, dpass ? sg * b_m : 0.0, bU);
    if (pass1) {
        const double b = bx1 * sx;
        if (t0pass) bu0c += sg * b;
        bcs0 += b;
    }
}

// reverse of viscous(): the force is linear in the second derivatives and bilinear in
// nr = Sigma nu and the first ones, so with (a, b) the adjoint of the force its stencil adjoints
// are fixed by eleven numbers: those of the six first derivatives, p = a nr and q = b nr (every
// second derivative's is p, 2 p, q or 2 q) and the middle cell's own.  Eleven planes from
// the cells to their gather instead of the 27 adjoints of the stencil: 128 registers instead
// of 254, kick1's and kick2's cells 29.7 and 29.7 -> 20.1 and 19.4 us at 256x768
struct StressAdj {
    double nx, ny, ux, uy, vx, vy;  // of d nr/dx, d nr/dy, du/dx, ...
    double p, q;
    double n, u, v;  // the middle cell's, through every path
};
__device__ __forceinline__ StressAdj viscous_rev(const double* __restrict__ X, const double* __restrict__ Y,
                                                 const double* u, const double* v, const double* nr, double a,
                                                 double b) {
    const double i_r20 = X[0], i_r21 = X[1], i_r10 = X[2], i_hr20 = X[3], i_r1 = X[4];
    const double i_t20 = Y[0], i_t21 = Y[1], i_t10 = Y[2], i_ht20 = Y[3];
    const double dudx = (u[2] - u[0]) * i_r20;
    const double d2udx2 = ((u[2] - u[1]) * i_r21 - (u[1] - u[0]) * i_r10) * i_hr20;
    const double dndx = (nr[2] - nr[0]) * i_r20;
    const double dvdx = (v[2] - v[0]) * i_r20;
    const double d2vdx2 = ((v[2] - v[1]) * i_r21 - (v[1] - v[0]) * i_r10) * i_hr20;
    const double dvdy = (v[7] - v[4]) * i_t20 * i_r1;
    const double d2vdy2 = ((v[7] - v[1]) * i_t21 - (v[1] - v[4]) * i_t10) * i_ht20 * i_r1 * i_r1;
    const double d2vdxy = (v[8] - v[6] - v[5] + v[3]) * i_r20 * i_t20 * i_r1;
    const double dudy = (u[7] - u[4]) * i_t20 * i_r1;
    const double d2udy2 = ((u[7] - u[1]) * i_t21 - (u[1] - u[4]) * i_t10) * i_ht20 * i_r1 * i_r1;
    const double d2udxy = (u[8] - u[6] - u[5] + u[3]) * i_r20 * i_t20 * i_r1;
    const double dndy = (nr[7] - nr[4]) * i_t20 * i_r1;
    const double n1 = nr[1], u1 = u[1], v1 = v[1];
    StressAdj o;
    o.p = a * n1;
    o.q = b * n1;
    o.nx = a * 2.0 * dudx + b * ((dudy + dvdx) - v1 * i_r1);
    o.ny = a * ((dudy + dvdx) - v1 * i_r1) + b * (2.0 * dvdy + 2.0 * u1 * i_r1);
    o.ux = a * (2.0 * dndx + 2.0 * n1 * i_r1);
    o.uy = a * dndy + b * (dndx + 4.0 * n1 * i_r1);
    o.vx = a * dndy + b * (dndx + n1 * i_r1);
    o.vy = -3.0 * a * n1 * i_r1 + 2.0 * b * dndy;
    o.n = a * (2.0 * d2udx2 + 2.0 * dudx * i_r1 + (d2udy2 + d2vdxy) - dvdy * i_r1 - 2.0 * (dvdy + u1 * i_r1) * i_r1) +
          b * (2.0 * d2vdy2 + 2.0 * dudy * i_r1 + (d2udxy + d2vdx2) - dvdx * i_r1 + v1 * i_r1 * i_r1 +
               2.0 * (dudy + dvdx - v1 * i_r1) * i_r1);
    const double D = (i_r21 + i_r10) * i_hr20, K = (i_t21 + i_t10) * i_ht20 * i_r1 * i_r1;
    o.u = -a * 2.0 * n1 * i_r1 * i_r1 + b * 2.0 * dndy * i_r1 - 2.0 * o.p * D - o.p * K;
    o.v = -a * dndy * i_r1 + b * (-dndx * i_r1 - n1 * i_r1 * i_r1) - o.q * D - 2.0 * o.q * K;
    return o;
}

}  // namespace rev
}  // namespace pg
