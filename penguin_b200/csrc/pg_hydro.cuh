// FP64 hydrodynamics building blocks of the Godunov sweep: 4th-order PPM
// reconstruction, characteristic interface states, HLLC flux, conservative
// update.  They compute what the cited lines of the reference compute and differ
// from it at the rounding level, but not in its order: the 4th-order edge slopes
// use per-index linear weights built once on the host instead of re-deriving 15
// grid moments and 56 divisions per call, the slopes are limited by their sizes,
// swept fractions come from the speeds, and quotients and roots are products of
// inv and rsq (2 ulp).
//
// Range: a cell's density times its pressure and the densities of neighbours are
// multiplied where the reference divides them, so the products have to be normal
// doubles, 2^-1022 to 2^1024.  Every update floors density and pressure at 1e-10:
// only a state the caller sets can leave that range, and gives a NaN that the error
// word reports.  Roots taken factor by factor outside it, behind a test of the
// product's exponent, cost 6.5 % of a step at 1024x3072 (532 -> 567 us).
//
// The functions are templates on the scalar type T: the sweeps instantiate
// them with double, the adjoint kernels with dual numbers (pg_dual.cuh).
#pragma once

#include "pg_common.cuh"

namespace pg {

template <class T>
constexpr bool is_double = false;
template <>
inline constexpr bool is_double<double> = true;

template <class T>
struct ParT {
    T sL, a, sR;
};
using Par = ParT<double>;

// The smaller / larger of two values by one comparison (no NaN rules; a NaN in
// the first operand stays).
template <class T>
__device__ __forceinline__ T lesser(T a, T b) { return (b < a) ? b : a; }
template <class T>
__device__ __forceinline__ T larger(T a, T b) { return (b > a) ? b : a; }

// a b + c in one rounding; of a derivative type, as it stands.  Which product of a sum the
// compiler contracts may depend on the code around it: where two instances of a kernel have
// to give the same bits, every product that is added is added by this.
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
template <class A, class B, class C>
__device__ __forceinline__ auto mad(const A& a, const B& b, const C& c) {
    return a * b + c;
}

// Reciprocal (of either sign) and reciprocal square root of a normal double within two
// ulp (NaN at zero and infinity): the hardware's approximation (rcp/rsqrt.approx.ftz.f64, which reads and
// returns the upper 32 bits of a double, so |e| < 2^-19) and one third-order step
// of Newton's iteration (Householder, "The Numerical Treatment of a Single
// Nonlinear Equation", 1970): with e = 1 - x y, y (1 + e + e^2) is off by e^3, and
// with e = 1 - x y^2, y (1 + e/2 + 3 e^2/8) by 5 e^3 / 16.  Three and five
// FP64 instructions and no branch, where the IEEE quotient and root take about
// ten each and a slow path: the sweeps are bound by this arithmetic's latency.
__device__ __forceinline__ double inv(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsq(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
template <class T>
__device__ __forceinline__ T inv(const T& x) { return 1.0 / x; }
template <class T>
__device__ __forceinline__ T rsq(const T& x) { return 1.0 / sqrt(x); }

// src/solver/recon/recon.cu:216-378 (slopes) + src/solver/recon/PPM.cu:64-91 (flattening,
// monotonicity).  w: {wL0,wL1,wL2, wR0,wR1,wR2} with sL = wL . (a[i-1]-a[i-2], a[i]-a[i-1],
// a[i+1]-a[i]) and sR = wR . (a[i]-a[i-1], a[i+1]-a[i], a[i+2]-a[i+1]).  Each slope takes
// the size min(|s|, |d|) and the sign of its neighbour difference d; both vanish at an
// extremum.  The reference's monotonicity test (sR + sL)^2 < 3 (sR + sL) (sL - sR) is, for
// slopes of one sign, 2 |sR| < |sL|, where it sets sL = 2 sR: the sizes are limited to
// twice each other.
template <class T>
__device__ __forceinline__ ParT<T> recon(const double* __restrict__ w, T am2, T am1, T a0, T ap1, T ap2, T flat) {
    const T d0 = am1 - am2, d1 = a0 - am1, d2 = ap1 - a0, d3 = ap2 - ap1;
    const T sL = w[0] * d0 + w[1] * d1 + w[2] * d2;
    const T sR = w[3] * d1 + w[4] * d2 + w[5] * d3;
    T l = lesser(fabs(sL), fabs(d1));
    T r = lesser(fabs(sR), fabs(d2));
    // a zero size makes both vanish below; for a derivative it has to be an exact zero here
    bool zero = signbit(d1) != signbit(d2);
    if constexpr (!is_double<T>) zero = zero || !(l > 0.0) || !(r > 0.0);
    if (zero) {
        l = 0.0;
        r = 0.0;
    }
    const T k = 1.0 - flat;
    return {copysign(lesser(l, 2.0 * r) * k, d1), a0, copysign(lesser(r, 2.0 * l) * k, d2)};
}

// Averages of the parabola over the fraction x of the cell touching its left /
// right edge (src/solver/recon/PPM.cu:95-113).  The x-only factors h = x/2 and
// g = 1 - x/1.5 are shared by every field averaged at the same x.
template <class T>
struct FracT {
    T h, g;
};
using Frac = FracT<double>;
// of the swept fraction y of the cell at the edge (1 - x / 1.5 in one FMA: within
// an ulp of 1 of the rounded quotient's)
template <class T>
__device__ __forceinline__ FracT<T> frac(T y) { return {0.5 * y, 1.0 - y * (2.0 / 3.0)}; }
template <class T>
__device__ __forceinline__ T aveL(const FracT<T>& f, const ParT<T>& p) {
    const T a6 = 3.0 * (p.sL - p.sR);
    const T aL = p.a - p.sL;
    const T S = p.sR + p.sL;
    return aL + f.h * (S + f.g * a6);
}
template <class T>
__device__ __forceinline__ T aveR(const FracT<T>& f, const ParT<T>& p) {
    const T a6 = 3.0 * (p.sL - p.sR);
    const T aR = p.a + p.sR;
    const T S = p.sR + p.sL;
    return aR - f.h * (S - f.g * a6);
}

template <class T>
__device__ __forceinline__ T exp_lim(T x) { return larger(1.0 + x, T(1.0e-6)); }  // solve.cu:29

// sqrt(gam p / r) with one reciprocal root and no division
template <class T>
__device__ __forceinline__ T sound_speed(double gam, T r, T p) {
    const T g = gam * p;
    return g * rsq(g * r);
}
// the product is rounded on its own, so that every pass that forms the CFL rate
// gets the same bits whatever it is added to
__device__ __forceinline__ double sound_speed(double gam, double r, double p) {
    const double g = gam * p;
    return __dmul_rn(g, rsq(g * r));
}

// Shock flattening coefficient of the middle cell (src/solver/recon/PPM.cu:7-62).
// The reference forms the Mach numbers (u0 - up1) / cs and (um1 - u0) / cs only
// to test their signs, which are those of the differences.  Its steepness
// |dp1 / dp2 - 1/2| - 1/4 of either side is (|dp1 - dp2 / 2| - |dp2| / 4) / |dp2|:
// the numerators decide whether there is a shock and which side is steeper, so
// one reciprocal is left, on cells that are flattened at all.
template <class T>
__device__ __forceinline__ T flatten(T p0, T pm2, T pm1, T pp1, T pp2, T um1, T u0, T up1) {
    const T dp1f = pp1 - p0, dp2f = pp2 - pm1;
    const T dp1b = p0 - pm1, dp2b = pp1 - pm2;
    const T wf = fabs(dp2f), wb = fabs(dp2b);
    const T nf = fabs(dp1f - 0.5 * dp2f) - 0.25 * wf;
    const T nb = fabs(dp1b - 0.5 * dp2b) - 0.25 * wb;
    T f = 0.0;
    if ((u0 > up1 || um1 > u0) && wf > 0.0 && wb > 0.0 && (nf > 0.0 || nb > 0.0)) {
        const bool back = nb * wf > nf * wb;
        const T big = larger(fabs(dp1f), fabs(dp1b));
        f = 10.0 * (back ? nb : nf) * big * inv((back ? wb : wf) * p0);
        f = lesser(T(0.5), f);
    }
    return f;
}

template <class T>
struct HalfT {
    T r, p, u, v, w;
};
using Half = HalfT<double>;

// Interface state on the LEFT edge of a cell = the right state of the face
// below it (src/solver/riemann/states.cu:151-206).  sx = dt / (rad (xr - xl)): the
// swept fraction per unit speed; cs0 = sqrt(gam p/r) of the cell averages r0c, p0c,
// u0c.  The reference forms the traced positions xl + speed dt and takes xl off
// again; the swept fraction comes directly from the speed, which only drops
// that cancellation.  With s = (gam p r)^-1/2 every quotient of the trace is a
// product: cs = gam p s, 1 / cs = r s, 1 / (r cs) = s.
template <class T>
__device__ __forceinline__ HalfT<T> state_at_left_edge(double gam, T sx, T cs0, T r0c, T p0c, T u0c, const ParT<T>& R,
                                                       const ParT<T>& Pp, const ParT<T>& U, const ParT<T>& V,
                                                       const ParT<T>& W) {
    const T one = 1.0, zero = 0.0;
    FracT<T> q = frac(lesser((cs0 - lesser(u0c, zero)) * sx, one));
    const T m = lesser(aveL(q, U), zero);
    q = frac(lesser(-m * sx, one));
    const T r0 = larger(aveL(q, R), r0c * 1.0e-10), p0 = larger(aveL(q, Pp), p0c * 1.0e-10);
    const T u0 = aveL(q, U);
    const T g = gam * p0;
    const T s = rsq(g * r0);
    q = frac(lesser((g * s - m) * sx, one));
    const T du = (u0 - aveL(q, U)) * (r0 * s), dp = aveL(q, Pp) - p0;
    return {r0 * exp_lim(du), p0 * exp_lim(gam * du), u0 - dp * s, aveL(q, V), aveL(q, W)};
}

// Interface state on the RIGHT edge of a cell = the left state of the face
// above it (src/solver/riemann/states.cu:210-264).
template <class T>
__device__ __forceinline__ HalfT<T> state_at_right_edge(double gam, T sx, T cs0, T r0c, T p0c, T u0c,
                                                        const ParT<T>& R, const ParT<T>& Pp, const ParT<T>& U,
                                                        const ParT<T>& V, const ParT<T>& W) {
    const T one = 1.0, zero = 0.0;
    FracT<T> q = frac(lesser((cs0 + larger(u0c, zero)) * sx, one));
    const T m = larger(aveR(q, U), zero);
    q = frac(lesser(m * sx, one));
    const T r0 = larger(aveR(q, R), r0c * 1.0e-10), p0 = larger(aveR(q, Pp), p0c * 1.0e-10);
    const T u0 = aveR(q, U);
    const T g = gam * p0;
    const T s = rsq(g * r0);
    q = frac(lesser((g * s + m) * sx, one));
    const T du = (aveR(q, U) - u0) * (r0 * s), dp = p0 - aveR(q, Pp);
    return {r0 * exp_lim(du), p0 * exp_lim(gam * du), u0 - dp * s, aveR(q, V), aveR(q, W)};
}

// src/EOS/EOS.cu:4-18 (EOS 0: isothermal, 2: ideal gas; ie: internal_e_flag)
template <class T>
__device__ __forceinline__ T energy(int eos, int ie, double gam, T r, T p, T u, T v, T w) {
    if (eos == 2) {
        T e = p / ((gam - 1.0) * r);
        if (ie == 0) e += u * u / 2.0 + v * v / 2.0 + w * w / 2.0;
        return e;
    }
    return p / r;
}

template <class T>
struct FluxT {
    T r, p, u, v, w, pres, uprs;
};
using Flux = FluxT<double>;

// Wave speeds (src/solver/riemann/wave_speeds.cu:24-35, 288-333) and the HLLC
// fluxes (src/solver/riemann/HLLC.cu:10-77) at one face, us = 0.  The reference
// forms all four candidate fluxes and picks one by the signs of sl, sr, sm
// (HLLC.cu:2-8); here the signs are tested first and only the selected
// candidate is formed.
template <class T>
__device__ __forceinline__ FluxT<T> hllc(int eos, int ie, double gam, const HalfT<T>& L, const HalfT<T>& R) {
    const T cl = sound_speed(gam, L.r, L.p), cr = sound_speed(gam, R.r, R.p);
    const T ic = inv(cl + cr);
    const T pm = 0.5 * (R.p + L.p) * exp_lim(gam * (L.u - R.u) * ic);
    // Roe's averages weighted with the roots of the densities, through their ratio
    const T q = R.r * rsq(L.r * R.r), iq = inv(1.0 + q);
    const T u_ = (L.u + q * R.u) * iq, du = R.u - L.u;
    const T c2 = (cl * cl + cr * cr * q) * iq + 0.5 * q * (iq * iq) * (du * du);
    const T cc = c2 * rsq(c2);
    const T sl = u_ - cc, sr = u_ + cc;
    const T ml = L.r * cl, mr = R.r * cr;
    const T sm = (ml * L.u + mr * R.u) * inv(ml + mr) + 2.0 * (L.p - R.p) * (inv(L.r + R.r) * ic);

    // side of every upwinded quantity: left iff sl >= 0, or sr >= 0 and sm >= 0
    const bool left = (signbit(sl) == 0) || (signbit(sr) == 0 && signbit(sm) == 0);
    const HalfT<T>& S = left ? L : R;
    FluxT<T> F;
    if (signbit(sl) == 0 || signbit(sr) != 0) {  // supersonic: the upwind state's own fluxes
        F.r = S.u * S.r;
        F.pres = S.p;
        F.uprs = (ie == 0) ? S.u * S.p : S.u;
    } else {  // star region on the side of the contact
        const T s_ = left ? sl : sr;
        const T is = inv(s_ - sm);
        F.r = sm * S.r * (s_ - S.u) * is;
        F.pres = (s_ * pm - sm * S.p) * is;
        if (ie == 0) F.uprs = sm * (s_ * pm - S.u * S.p) * is;
        else F.uprs = sm * (s_ * pm - S.u * S.p) / (s_ * pm - sm * S.p);
    }
    F.u = S.u * F.r;
    F.v = S.v * F.r;
    F.w = S.w * F.r;
    F.p = (eos > 0) ? energy<T>(eos, ie, gam, S.r, S.p, S.u, T(0.0), T(0.0)) * F.r : T(0.0);
    if (eos != 2) F.uprs = 0.0;
    return F;
}

// Viscous force density of the middle cell of a 3x3 stencil
// (src/viscosity/viscosity.cu:9-22, 84-194, ndim 2).  Stencil order: n<3 row j,
// 3..5 row j-1, 6..8 row j+1, columns i-1..i+1.  The grid spacings enter as
// per-index reciprocals: X = {1/(r2-r0), 1/(r2-r1), 1/(r1-r0), 1/(0.5(r2-r0)), 1/r1},
// Y = {1/(t2-t0), 1/(t2-t1), 1/(t1-t0), 1/(0.5(t2-t0))}.  Sums of products by mad: the
// kicks' instances give the same bits.
template <class T>
__device__ __forceinline__ void viscous(const double* __restrict__ X, const double* __restrict__ Y, const T* u,
                                        const T* v, const T* nr, T& fx_out, T& fy_out) {
    const double i_r20 = X[0], i_r21 = X[1], i_r10 = X[2], i_hr20 = X[3], i_r1 = X[4];
    const double i_t20 = Y[0], i_t21 = Y[1], i_t10 = Y[2], i_ht20 = Y[3];
    const T dudx = (u[2] - u[0]) * i_r20;
    const T d2udx2 = mad(u[2] - u[1], i_r21, (u[0] - u[1]) * i_r10) * i_hr20;
    const T dndx = (nr[2] - nr[0]) * i_r20;
    const T dvdx = (v[2] - v[0]) * i_r20;
    const T d2vdx2 = mad(v[2] - v[1], i_r21, (v[0] - v[1]) * i_r10) * i_hr20;
    const T dvdy = (v[7] - v[4]) * i_t20 * i_r1;
    const T d2vdy2 = mad(v[7] - v[1], i_t21, (v[4] - v[1]) * i_t10) * i_ht20 * i_r1 * i_r1;
    const T d2vdxy = (v[8] - v[6] - v[5] + v[3]) * i_r20 * i_t20 * i_r1;
    const T dudy = (u[7] - u[4]) * i_t20 * i_r1;
    const T d2udxy = (u[8] - u[6] - u[5] + u[3]) * i_r20 * i_t20;  // times i_r1
    const T d2udy2 = mad(u[7] - u[1], i_t21, (u[4] - u[1]) * i_t10) * i_ht20 * i_r1;  // times i_r1
    const T dndy = (nr[7] - nr[4]) * i_t20 * i_r1;
    const T shear = mad(v[2] - v[0], i_r20, dudy);  // dudy + dvdx

    const T sxx = 2.0 * nr[1] * dudx;
    const T syy = 2.0 * nr[1] * mad(u[1], i_r1, dvdy);
    const T sxy = nr[1] * mad(-v[1], i_r1, shear);
    // two chains each, whose latencies overlap: with one, and the planet's pull as it was, the
    // kicks took 2 % of a 1024x3072 step more
    const T fx = mad(sxx, i_r1, mad(2.0 * dndx, dudx, 2.0 * nr[1] * d2udx2));
    const T fy = mad(2.0 * dndy * u[1], i_r1, mad(2.0 * nr[1] * dudy, i_r1, mad(2.0 * dndy, dvdy, 2.0 * nr[1] * d2vdy2)));
    T gx = mad(dndy, shear, nr[1] * mad(d2udy2, i_r1, d2vdxy));
    gx = mad(-(dndy * v[1]), i_r1, gx);
    gx = mad(-(nr[1] * dvdy), i_r1, gx);
    fx_out = fx + mad(-syy, i_r1, gx);
    T gy = mad(dndx, shear, nr[1] * mad(d2udxy, i_r1, d2vdx2));
    gy = mad(-(dndx * v[1]), i_r1, gy);
    gy = mad(-(nr[1] * dvdx), i_r1, gy);
    gy = mad(nr[1] * v[1] * i_r1, i_r1, gy);
    fy_out = fy + mad(2.0 * sxy, i_r1, gy);
}

// Conservative update with floors (src/solver/sweeps.cu:218-261).  cs2: get_cs2
// at the cell.  For the isothermal EOS the energy slot is dead (it is
// overwritten by cs2 r), so it is not formed.  ISO: 2D isothermal, whose zero
// z-velocity stays as it is.
template <bool ISO = false>
__device__ __forceinline__ Cell update_cell(int eos, int ie, double gam, double cs2, Cell Q, const Cell& D,
                                            int* floor_hits) {
    const double r_min = fmax(Q.r * 1.0e-10, SMALLR);
    const double p_min = fmax(Q.p * 1.0e-10, SMALLP);
    const double u_old = Q.u, v_old = Q.v, w_old = Q.w;
    if (eos == 2) {
        Q.p = energy(eos, ie, gam, Q.r, Q.p, Q.u, Q.v, Q.w);
        Q.p *= Q.r;
    }
    Q.u *= Q.r;
    Q.v *= Q.r;
    if (!ISO) {
        Q.w *= Q.r;
        Q.w += D.w;
        Q.p += D.p;
    }
    Q.r += D.r;
    Q.u += D.u;
    Q.v += D.v;
    const double ir = inv(Q.r);
    Q.u *= ir;
    Q.v *= ir;
    if (!ISO) Q.w *= ir;
    if (Q.r < r_min) {
        Q.r = r_min;
        Q.p = p_min;
        Q.u = u_old;
        Q.v = v_old;
        Q.w = w_old;
        if (floor_hits) atomicAdd(floor_hits, 1);
    } else if (eos == 2) {
        const double gamm = gam - 1.0;
        if (ie == 0) Q.p = fmax(Q.p * gamm - gamm * Q.r * (Q.u * Q.u + Q.v * Q.v + Q.w * Q.w) / 2.0, p_min);
        else Q.p = fmax(Q.p * gamm, p_min);
    } else {
        Q.p = cs2 * Q.r;
    }
    return Q;
}

}  // namespace pg
