// FP32-mixed Godunov step for ensembles of 2D polar planet-disks (sm_100a).
//
// The same five fused passes as the FP64 kernels (kick1 C->T, radial sweep T->C,
// azimuthal sweep + orbital shift C->T, residual advection T->C, kick2 +
// damping + CFL rate C->T), on FP32 residual planes.  Every pass is ONE
// persistent launch over the concatenated runs of all disks in the ensemble (a run: some
// rows of 32 neighbouring radii of one disk), so disks of uneven size share the
// GPU without one launch per disk.
//
// A disk whose clock reached end_time has its runs copied through unchanged, so
// the two state buffers of all disks stay in step.
#include <cstdio>
#include <vector>

#include "pg_common.cuh"
#include "pg_f32.cuh"
#include "pg_internal.h"
#include "pg_planet.cuh"

namespace pg {
namespace f32 {

// A pass's work is cut into runs: a warp takes the rows j0 .. j1-1 of its 32
// neighbouring radii one after the other (int4 {disk, first lane's radius, j0, j1}, a
// table built with the ensemble).  Lanes along the radius make every access to a plane
// a coalesced row segment and every per-radius factor a register for the whole run;
// what a cell needs of its neighbours comes by shuffle or stays from the row before.
// No shared memory and no barrier: tiles whose phases met at __syncthreads spent half
// their instructions on table loads, tile addresses and the exchange, and waited on
// barriers and L1 for most of the rest (55 % of issue slots at 1024x3072).  There, us a
// pass, tiles -> runs: kick1 75 -> 53, sweep_x 148 -> 82, sweep_y 135 -> 72, advection
// 81 -> 39, kick2 140 -> 84; what bounds them is instruction issue.  All are compiled for 5
// CTAs of 4 warps per SM; at 3 / 4 / 6 / 7 kick1 takes 78 / 78 / 66 / 73, sweep_x
// 99 / 100 / 90 / 93, sweep_y 78 / 78 / 82 / 87, kick2 99 / 107 / 122 / 133, and the
// advection 39 / 39 / 43 / 45.
constexpr int MW = 4, MT = 32 * MW;  // warps of a CTA, independent of one another

__device__ __forceinline__ float up1(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float down1(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Planar multi-value tables: value m of slot group `slot` at index i.
template <int N>
__device__ __forceinline__ void xload(const View32& w, int slot, int i, float* out) {
#pragma unroll
    for (int m = 0; m < N; ++m) out[m] = w.tx[(size_t)(slot + m) * w.xn + i];
}
template <int N>
__device__ __forceinline__ void yload(const View32& w, int slot, int j, float* out) {
#pragma unroll
    for (int m = 0; m < N; ++m) out[m] = w.ty[(size_t)(slot + m) * w.yn + j];
}

// Interior cell (i, j) and its periodic azimuthal image (boundary.cu:141-209).
__device__ __forceinline__ void emit32(const View32& w, float* out, int i, int j, float a, float b, float c) {
    const size_t pl = w.plane();
    size_t m = (size_t)j * w.pitch + i;
    out[m] = a;
    out[pl + m] = b;
    out[2 * pl + m] = c;
    int jimg = -1;
    if (j < 2 * NPAD) jimg = j + w.yres;
    else if (j >= w.yres) jimg = j - w.yres;
    if (jimg >= 0) {
        m = (size_t)jimg * w.pitch + i;
        out[m] = a;
        out[pl + m] = b;
        out[2 * pl + m] = c;
    }
}

// What the marching passes read of the disk's descriptor in every row, in registers: the
// descriptor lies in global memory, and the rows' stores would make each use of it a load.
struct Disk32 {
    int pitch, yres, yn;
    size_t pl;
    const float* ty;
    float* out;
    __device__ __forceinline__ Disk32(const View32& w, int in)
        : pitch(w.pitch), yres(w.yres), yn(w.yn), pl(w.plane()), ty(w.ty), out(w.buf[in ^ 1]) {}
    __device__ __forceinline__ float y(int slot, int j) const { return ty[slot * yn + j]; }
    template <int N>
    __device__ __forceinline__ void ys(int slot, int j, float* o) const {
#pragma unroll
        for (int m = 0; m < N; ++m) o[m] = ty[(slot + m) * yn + j];
    }
    // the new residuals of interior cell (i, j) and their periodic image (emit32)
    __device__ __forceinline__ void emit(int i, int j, float a, float b, float c) const {
        float* o = out + ((size_t)j * pitch + i);
        o[0] = a;
        o[pl] = b;
        o[2 * pl] = c;
        if (j < 2 * NPAD || j >= yres) {
            o += (long long)(j < 2 * NPAD ? yres : -yres) * pitch;
            o[0] = a;
            o[pl] = b;
            o[2 * pl] = c;
        }
    }
};

// What the half-kicks need of a lane's radius.
struct Kick32 {
    float sbg, abg, v2r, ir, rad, dr;  // dr: r - x_p
    float nu, nul, nur, vb[7], X[5];   // viscosity here and at the neighbours, stencil factors
    float m, xp, rs2, ip2;             // the planet
    const float* trig;                 // per-row table of its angles, null without a planet
};
__device__ __forceinline__ Kick32 kick_tables(const View32& w, int i, int which) {
    Kick32 c;
    c.sbg = w.x(X_SBG)[i];
    c.abg = w.x(X_ABG)[i];
    c.v2r = w.x(X_V2R)[i];
    c.ir = w.x(X_IRAD)[i];
    c.rad = w.x(X_RAD)[i];
    c.dr = w.tcol()[2 * i + which];
    const float* s = w.tscal() + 4 * which;
    c.m = s[0];
    c.xp = s[1];
    c.rs2 = s[2];
    c.ip2 = s[3];
    c.trig = w.nplanet ? w.trig + 3 * which : nullptr;
    c.nu = c.nul = c.nur = 0.0f;
    if (w.visc) {
        const float* nu = w.x(X_NU);
        c.nu = nu[i];
        c.nul = nu[max(i - 1, 0)];
        c.nur = nu[min(i + 1, w.xarr - 1)];
        xload<7>(w, X_VBG, i, c.vb);
        xload<5>(w, X_VISX, i, c.X);
    }
    return c;
}

// Star + planet gravity (forces.cu:182-327) without the star term, which is in
// X_ABG.  |r - r_p|^2 = (r - x_p)^2 + 2 r x_p (1 - cos) + rs^2 has no cancellation.
__device__ __forceinline__ void gravity32(const Kick32& c, int j, float& gx, float& gy) {
    gx = 0.0f;
    gy = 0.0f;
    if (!c.trig) return;
    const float* tr = c.trig + TRIG_ROW * j;
    const float R2 = c.dr * c.dr + 2.0f * c.rad * c.xp * tr[2] + c.rs2;
    const float ir = rsq32(R2);
    const float rf = ir * ir * ir;
    gx = -c.m * (c.dr + c.xp * tr[2]) * rf - c.m * tr[1] * c.ip2;
    gy = -c.m * c.xp * tr[0] * rf + c.m * tr[0] * c.ip2;
}

// Half-kick of the residual velocities (sweeps.cu:597-711 with geomx 1):
// v^2/r - 1/r^2 = X_ABG + (2 v0/r + dv/r) dv.  mdt != 0 re-evaluates the
// curvature term at the mdt-predicted velocity (sweeps.cu:663-687).
__device__ __forceinline__ void kick32(const Kick32& c, float dS, float& du, float& dv, float vx, float vy, float gx,
                                       float gy, float mdt, float dt, bool visc) {
    const float iS = visc ? rcp32(c.sbg + dS) : 0.0f;
    float fx = c.abg + (c.v2r + dv * c.ir) * dv + vx * iS;
    const float fy = vy * iS;
    if (mdt != 0.0f) {
        const float dvT = dv + fy * mdt + gy * mdt;
        fx = c.abg + (c.v2r + dvT * c.ir) * dvT + vx * iS;
    }
    du = du + fx * dt + gx * dt;
    dv = dv + fy * dt + gy * dt;
}

// One row's residuals at the lane's radius, the velocities at its neighbours' too.
struct Row32 {
    float S, u[3], v[3];
};
__device__ __forceinline__ Row32 row32(float S, float u, float v) {
    return Row32{S, {up1(u), u, down1(u)}, {up1(v), v, down1(v)}};
}
// Viscous force density of the middle of three rows: residual part plus background
// part (viscosity.cu:84-194).
__device__ __forceinline__ void stress32(const Disk32& D, const Kick32& c, int j, const Row32& lo, const Row32& mid,
                                         const Row32& hi, float& vx, float& vy) {
    float Y[4];
    D.ys<4>(Y_VISY, j, Y);
    const float nr1 = (c.sbg + mid.S) * c.nu;
    const float dndx = (c.vb[6] + down1(mid.S) * c.nur - up1(mid.S) * c.nul) * c.X[0];
    const float dndy = (hi.S - lo.S) * c.nu * Y[0] * c.X[4];
    const float u[9] = {mid.u[0], mid.u[1], mid.u[2], lo.u[0], lo.u[1], lo.u[2], hi.u[0], hi.u[1], hi.u[2]};
    const float v[9] = {mid.v[0], mid.v[1], mid.v[2], lo.v[0], lo.v[1], lo.v[2], hi.v[0], hi.v[1], hi.v[2]};
    float fx, fy;
    viscous32(c.X, Y, u, v, nr1, dndx, dndy, fx, fy);
    vx = fx + c.vb[0] * nr1 + c.vb[1] * dndx + c.vb[2] * dndy;
    vy = fy + c.vb[3] * nr1 + c.vb[4] * dndx + c.vb[5] * dndy;
}

// CFL signal rate (timestep.cu:46-77) in FP64 from the residuals.
__device__ __forceinline__ double rate64(const View32& w, int i, int j, float du, float dv) {
    const DiskView& d = w.d64;
    const double cs = w.cs64[i];
    const double u = d.initx[5 * i + 2] + (double)du;
    const double vn = (d.initx[5 * i + 3] - d.radx[i] * d.frame_omega - d.rot[i]) + (double)dv;
    const double a = (fabs(u) + cs) * d.idx_x[i];
    const double b = (fabs(vn) + cs) * (d.idx_y[j] * d.irad[i]);
    return fmax(a, b);
}

// the dust's CFL rate (timestep.cu:64-74): its speeds without a sound speed
__device__ __forceinline__ double drate64(const View32& w, int i, int j, float du, float dv) {
    const DiskView& d = w.d64;
    const double u = d.initd[4 * i + 1] + (double)du;
    const double vn = (d.initd[4 * i + 2] - d.radx[i] * d.frame_omega - d.rot[i]) + (double)dv;
    return fmax(fabs(u) * d.idx_x[i], fabs(vn) * (d.idx_y[j] * d.irad[i]));
}

// ================================================================ dust
// One pressureless dust fluid (dust_flag) in the FP32-mixed form: residual
// planes {dSigma_d, dv_r,d, dv_phi,d} against init_CD, transported by the
// reference's upwind PPM fluxes with the compression factor and the flux
// limiter (src/solver/dust/dust.cu:6-147) and updated by update_Dust
// (dust.cu:149-176) in residual form, e.g. v_new - v = (D(Sigma v) - v D Sigma) /
// Sigma_new with the transported field taken relative to a neighbouring cell.
// Each sweep is one launch over the dusty disks' runs, laid out like the gas's: edge states,
// limited face fluxes and the update of a cell stay in registers, neighbours by shuffle or
// from the row before.  (As one launch per face and one per cell through a scratch array of
// fluxes, every face formed both its cells' states again: 65 us a sweep at 682x2046, three
// times the gas's.)  The dust planes carry no ghost images: rows wrap, and the
// radial ghosts of boundary 0 hold init_CD, i.e. zero residuals.
struct DR {
    float S, u, v;  // residuals
};
__device__ __forceinline__ int wrap32(const View32& w, int j) {
    if (j < NPAD) return j + w.yres;
    if (j >= NPAD + w.yres) return j - w.yres;
    return j;
}
__device__ __forceinline__ DR dload(const View32& w, const float* b, int i, int j) {
    if (i < NPAD || i >= NPAD + w.xres) return {0.0f, 0.0f, 0.0f};
    const size_t pl = w.plane(), m = (size_t)wrap32(w, j) * w.pitch + i;
    return {b[m], b[pl + m], b[2 * pl + m]};
}
__device__ __forceinline__ void dstore(const View32& w, float* b, int i, int j, const DR& c) {
    const size_t pl = w.plane(), m = (size_t)j * w.pitch + i;
    b[m] = c.S;
    b[pl + m] = c.u;
    b[2 * pl + m] = c.v;
}
__device__ __forceinline__ float exp_limf(float x) { return fmaxf(1.0f + x, 1.0e-6f); }

struct DEdge {
    float S, u, t;  // density and normal velocity (absolute), transported field relative to the cell
};
// One edge state of a dust cell (dust.cu:6-103; SIDE 0 left, 1 right) from its parabolas;
// sx = sdt / dx, uc the cell's normal velocity, Sc its density.
template <int SIDE>
__device__ __forceinline__ DEdge dust_edge(float sx, float Sc, float uc, const Par32& R, const Par32& U,
                                           const Par32& T) {
    auto away = [](float u) { return SIDE == 0 ? fmaxf(-u, 0.0f) : fmaxf(u, 0.0f); };
    auto ave = [](const Frac32& q, const Par32& p) { return SIDE == 0 ? aveL32(q, p) : aveR32(q, p); };
    const float d = away(SIDE == 0 ? uc - U.sL : uc + U.sR) * sx;  // swept fraction
    const float ud = ave(frac32(fminf(d, 1.0f)), U);
    const Frac32 q = frac32(fminf(away(uc + ud) * sx, 1.0f));
    const float c = sx * (SIDE == 0 ? ud : -ud) / (1.0f - d);  // the cell's compression
    return DEdge{(Sc + ave(q, R)) * exp_limf(c), uc + ave(q, U), ave(q, T)};
}
struct DFlux {
    float r, u, t;  // mass, normal momentum, transported field relative to the face's lower cell
};
// dust_flow's limited upwind flux (dust.cu:120-147) between lower cell a and upper cell b:
// no more than the cells hold (Sa sxa, Sb sxb); jump: the transported field from a to b
__device__ __forceinline__ DFlux dust_flux(float Sa, float sxa, const DEdge& a, float Sb, float sxb, const DEdge& b,
                                           float jump) {
    const float Fl = fminf(Sa * sxa, fmaxf(a.u * a.S, 0.0f));
    const float Fr = fmaxf(-Sb * sxb, fminf(b.u * b.S, 0.0f));
    return DFlux{Fl + Fr, Fl * a.u + Fr * b.u, Fl * a.t + Fr * (jump + b.t)};
}
// update_Dust (dust.cu:149-176) in residual form: DS and the increments Dn = D(Sigma u_n) -
// u_n D Sigma and Dt of the residuals n and t; true where the density fell to its floor
__device__ __forceinline__ void update_dust32(const View32& w, Scalars* sc, float sbg, float DS, float Dn, float Dt,
                                              float& S, float& n, float& t) {
    const float Sc = sbg + S, Sn = Sc + DS;
    const float rmin = fmaxf(Sc * 1.0e-10f, w.dust_rmin);
    if (Sn < rmin) {
        S = rmin - sbg;
    } else {
        const float iS = rcp32(Sn);
        S += DS;
        n += Dn * iS;
        t += Dt * iS;
    }
    if (!(Sn > 0.0f)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
}

// radial dust sweep: normal v_r, transported r v_phi
__global__ void __launch_bounds__(MT, 5) k32d_sweep_x(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                     int nruns, int in) {
    pdl_enter();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        if (!w.dust) continue;
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0;
        const float dtf = (float)sc->dt;
        const size_t pl = w.plane(), pitch = w.pitch;
        const int i = run.y + lane, c = min(i, w.xarr - 3);
        const bool output = lane >= 1 && lane <= 30 && i < NPAD + w.xres;
        const float* src = w.dbuf[in] + (size_t)run.z * pitch + c;
        float* dst = w.dbuf[in ^ 1] + (size_t)run.z * pitch + c;
        if (done) {
            for (int j = run.z; j < run.w; ++j, src += pitch, dst += pitch)
                if (output) {
                    dst[0] = src[0];
                    dst[pl] = src[pl];
                    dst[2 * pl] = src[2 * pl];
                }
            continue;
        }
        float db[12], wt[6], rad[5];
        xload<12>(w, X_DDBG, c, db);
        xload<6>(w, X_WX, c, wt);
#pragma unroll
        for (int m = 0; m < 5; ++m) rad[m] = w.x(X_RAD)[c - 2 + m];
        const float sbg = w.x(X_DSBG)[c], ubg = w.x(X_DUBG)[c], sx = dtf * w.x(X_IDX)[c];
        const float g0 = w.x(X_XA)[c], g1 = w.x(X_XA)[c + 1], f = dtf * w.x(X_IXV)[c], irad = w.x(X_IRAD)[c];
#pragma unroll 1
        for (int j = run.z; j < run.w; ++j, src += pitch, dst += pitch) {
            float aS[5], aU[5], aT[5];
            const float S0 = src[0], u0 = src[pl], v0 = src[2 * pl];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                if (m == 2) {
                    aS[m] = aU[m] = aT[m] = 0.0f;
                    continue;
                }
                const int kk = m < 2 ? m : m - 1;
                aS[m] = db[kk] + (src[m - 2] - S0);
                aU[m] = db[4 + kk] + (src[pl + m - 2] - u0);
                aT[m] = db[8 + kk] + (rad[m] * src[2 * pl + m - 2] - rad[2] * v0);
            }
            const Par32 R = recon32(wt, aS[0], aS[1], aS[3], aS[4], 0.0f);
            const Par32 U = recon32(wt, aU[0], aU[1], aU[3], aU[4], 0.0f);
            const Par32 T = recon32(wt, aT[0], aT[1], aT[3], aT[4], 0.0f);
            const float Sc = sbg + S0, uc = ubg + u0;
            const DEdge b = dust_edge<0>(sx, Sc, uc, R, U, T), e = dust_edge<1>(sx, Sc, uc, R, U, T);
            const float jump = up1(aT[3]);  // from the lower cell
            const DEdge a{up1(e.S), up1(e.u), up1(e.t)};
            const DFlux F = dust_flux(up1(Sc), up1(sx), a, Sc, sx, b, jump);
            const DFlux G{down1(F.r), down1(F.u), down1(F.t)};
            const float DS = (F.r * g0 - G.r * g1) * f;
            const float Dn = (g0 * (F.u - F.r * uc) - g1 * (G.u - G.r * uc)) * f;
            const float Dt = (g0 * (F.t - F.r * jump) - g1 * G.t) * f * irad;
            if (output) {
                float S = S0, u = u0, v = v0;
                update_dust32(w, sc, sbg, DS, Dn, Dt, S, u, v);
                dst[0] = S;
                dst[pl] = u;
                dst[2 * pl] = v;
            }
        }
    }
}

// Five rows of a dust column in registers and the next in flight; rows wrap.
struct DColumn {
    float S[5], u[5], v[5], nS, nu, nv;
    const float* p;  // row `row` of the column
    int row, end;
    size_t pl, pitch, wrap;
    __device__ __forceinline__ DColumn(const View32& w, int in, int c, int first) {
        pl = w.plane();
        pitch = w.pitch;
        wrap = pitch * w.yres;
        end = NPAD + w.yres;
        row = first < NPAD ? first + w.yres : first;
        p = w.dbuf[in] + (size_t)row * pitch + c;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            S[m] = p[0];
            u[m] = p[pl];
            v[m] = p[2 * pl];
            next();
        }
        fetch();
    }
    __device__ __forceinline__ void next() {
        p += pitch;
        if (++row == end) {
            row = NPAD;
            p -= wrap;
        }
    }
    __device__ __forceinline__ void fetch() {
        nS = p[0];
        nu = p[pl];
        nv = p[2 * pl];
        next();
    }
    __device__ __forceinline__ void shift() {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            S[m] = S[m + 1];
            u[m] = u[m + 1];
            v[m] = v[m + 1];
        }
        S[4] = nS;
        u[4] = nu;
        v[4] = nv;
    }
};

// azimuthal dust sweep (normal v_phi - orb_rot - r Omega, transported v_r) writing each cell
// at the gas's shifted row of its radius (orbit.cu:30-46)
__global__ void __launch_bounds__(MT, 5) k32d_sweep_y(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                     int nruns, int in) {
    pdl_enter();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        if (!w.dust) continue;
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0;
        const float dtf = (float)sc->dt;
        const Disk32 D(w, in);
        const int i = run.y + lane, c = min(i, NPAD + w.xres - 1);
        const bool active = i < NPAD + w.xres;
        float* dst = w.dbuf[in ^ 1];
        if (done) {
            for (int j = run.z; j < run.w; ++j)
                if (active) dstore(w, dst, i, j, dload(w, w.dbuf[in], i, j));
            continue;
        }
        int js = run.z - NPAD;
        if (w.orbadv) {
            js = (js + w.d64.inc[c]) % D.yres;
            if (js < 0) js += D.yres;
        }
        const float sbg = w.x(X_DSBG)[c], ubg = w.x(X_DEPS)[c], sdt = dtf * w.x(X_IRAD)[c];
        DColumn q(w, in, c, run.z - NPAD);
        DEdge pe{};  // the right edge of the cell below, its density and swept fraction
        float pS = 0.0f, psx = 0.0f;
        DFlux pf{};
#pragma unroll 1
        for (int t = run.z - 1; t <= run.w; ++t) {
            const int tw = t < NPAD ? t + D.yres : (t >= NPAD + D.yres ? t - D.yres : t);
            float wt[6];
            D.ys<6>(Y_WY, tw, wt);
            const float sx = sdt * D.y(Y_IDY, tw);
            const Par32 R = recon32(wt, q.S[0] - q.S[2], q.S[1] - q.S[2], q.S[3] - q.S[2], q.S[4] - q.S[2], 0.0f);
            const Par32 U = recon32(wt, q.v[0] - q.v[2], q.v[1] - q.v[2], q.v[3] - q.v[2], q.v[4] - q.v[2], 0.0f);
            const Par32 T = recon32(wt, q.u[0] - q.u[2], q.u[1] - q.u[2], q.u[3] - q.u[2], q.u[4] - q.u[2], 0.0f);
            const float Sc = sbg + q.S[2], uc = ubg + q.v[2];
            const DEdge b = dust_edge<0>(sx, Sc, uc, R, U, T), e = dust_edge<1>(sx, Sc, uc, R, U, T);
            const DFlux F = dust_flux(pS, psx, pe, Sc, sx, b, q.u[2] - q.u[1]);
            if (t > run.z) {  // the cell below has both its fluxes
                float S = q.S[1], u = q.u[1], v = q.v[1];
                const float f = sdt * D.y(Y_IYV, t - 1), un = ubg + v;
                const float DS = (pf.r - F.r) * f;
                const float Dn = ((pf.u - pf.r * un) - (F.u - F.r * un)) * f;
                const float Dt = ((pf.t - pf.r * (q.u[1] - q.u[0])) - F.t) * f;
                if (active) {
                    update_dust32(w, sc, sbg, DS, Dn, Dt, S, v, u);
                    dstore(w, dst, i, js + NPAD, DR{S, u, v});
                }
                if (++js == D.yres) js = 0;
            }
            pe = e;
            pS = Sc;
            psx = sx;
            pf = F;
            q.shift();
            q.fetch();
        }
    }
}

// residual advection of the dust by orb_res (advection.cu:175-357)
__global__ void __launch_bounds__(MT, 6) k32d_advect(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                    int nruns, int in) {
    pdl_enter();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        if (!w.dust) continue;
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0;
        const float dtf = (float)sc->dt;
        const Disk32 D(w, in);
        const int i = run.y + lane, c = min(i, NPAD + w.xres - 1);
        const bool active = i < NPAD + w.xres;
        float* dst = w.dbuf[in ^ 1];
        if (done) {
            for (int j = run.z; j < run.w; ++j)
                if (active) dstore(w, dst, i, j, dload(w, w.dbuf[in], i, j));
            continue;
        }
        const float speed = (float)w.d64.res[c], sbg = w.x(X_DSBG)[c], sdt = dtf * w.x(X_IRAD)[c];
        const float swept = fabsf(speed) * sdt;
        const bool up = speed > 0.0f;
        DColumn q(w, in, c, run.z - NPAD);
        float pr = 0.0f, pv = 0.0f, pu = 0.0f;  // the row before: mass flux and the carried v and u
#pragma unroll 1
        for (int t = run.z - 1; t <= run.w; ++t) {
            const int tw = t < NPAD ? t + D.yres : (t >= NPAD + D.yres ? t - D.yres : t);
            float wt[6];
            D.ys<6>(Y_WY, tw, wt);
            const Par32 R = recon32(wt, q.S[0] - q.S[2], q.S[1] - q.S[2], q.S[3] - q.S[2], q.S[4] - q.S[2], 0.0f);
            const Par32 N = recon32(wt, q.v[0] - q.v[2], q.v[1] - q.v[2], q.v[3] - q.v[2], q.v[4] - q.v[2], 0.0f);
            const Par32 T = recon32(wt, q.u[0] - q.u[2], q.u[1] - q.u[2], q.u[3] - q.u[2], q.u[4] - q.u[2], 0.0f);
            const Frac32 x = frac32(fminf(swept * D.y(Y_IDY, tw), 1.0f));
            const float F = ((sbg + q.S[2]) + (up ? aveR32(x, R) : aveL32(x, R))) * speed;
            // carried v and u, relative to the cell's own
            const float fv = up ? aveR32(x, N) : aveL32(x, N), fu = up ? aveR32(x, T) : aveL32(x, T);
            const int j = up ? t : t - 1;
            if (active && j >= run.z && j < run.w) {
                float S = up ? q.S[2] : q.S[1], u = up ? q.u[2] : q.u[1], v = up ? q.v[2] : q.v[1];
                const float f = sdt * D.y(Y_IYV, j);
                const float jv = q.v[2] - q.v[1], ju = q.u[2] - q.u[1];  // from the row below to this one
                const float Dv = (up ? pr * (pv - jv) - F * fv : pr * pv - F * (fv + jv)) * f;
                const float Du = (up ? pr * (pu - ju) - F * fu : pr * pu - F * (fu + ju)) * f;
                update_dust32(w, sc, sbg, (pr - F) * f, Dv, Du, S, v, u);
                dstore(w, dst, i, j, DR{S, u, v});
            }
            pr = F;
            pv = fv;
            pu = fu;
            q.shift();
            q.fetch();
        }
    }
}

// Drag of the dust towards the gas in a half-kick (sweeps.cu:626-707, the
// exponential integrator with t_s = St h / (c_s Sigma), dust.cu:1-4) in
// residual form.  gu, gv: the gas residuals the drag relaxes to at the start;
// with mdt != 0 the forces are re-evaluated at the mdt-predicted dust velocity
// and towards the mdt-predicted gas velocity (tu, tv).  gx, gy: planet gravity.
__device__ __forceinline__ void dust_drag32(const View32& w, int i, float Sg, float gu, float gv, float tu, float tv,
                                            float gx, float gy, float mdt, float dt, DR& D) {
    const float ts = w.st_h / (w.x(X_CS0)[i] * Sg);
    const float ir = w.x(X_IRAD)[i], dabg = w.x(X_DABG)[i], dv2r = w.x(X_DV2R)[i];
    const float dgu = w.x(X_DGU)[i], dgv = w.x(X_DGV)[i];
    float vd = D.v;  // dust v_phi residual entering the curvature term
    float ru = gu, rv = gv;
    if (mdt != 0.0f) {
        const float dtm = -expm1f(-mdt / ts);
        vd = D.v + dtm * ((dgv + gv - D.v) + ts * gy);
        ru = tu;
        rv = tv;
    }
    const float dtau = -expm1f(-dt / ts);
    const float fx = (dgu + ru - D.u) + ts * (dabg + (dv2r + vd * ir) * vd + gx);
    const float fy = (dgv + rv - D.v) + ts * gy;
    D.u += dtau * fx;
    D.v += dtau * fy;
}

// ============================================================ radial sweep
// Lanes 1..30 of a run update; lane l's left face takes its left state from lane l - 1, its right flux
// from lane l + 1.
__global__ void __launch_bounds__(MT, 5) k32_sweep_x(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                  int nruns, int in) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_enter();
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0;
        const float dtf = (float)sc->dt, gam = w.gam;
        const int i = run.y + lane, c = min(i, w.xarr - 3);  // c: the stencil stays in the row
        const bool output = lane >= 1 && lane <= 30 && i < NPAD + w.xres;
        const float* src = w.buf[in] + (size_t)run.z * w.pitch + c;
        const Disk32 D(w, in);
        if (done) {
            for (int j = run.z; j < run.w; ++j, src += D.pitch)
                if (output) D.emit(i, j, src[0], src[D.pl], src[2 * D.pl]);
            continue;
        }
        float db[16], wt[6], cs2[5], rad[5];
        xload<16>(w, X_DBG, c, db);
        xload<6>(w, X_WX, c, wt);
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            cs2[m] = w.x(X_CS2)[c - 2 + m];
            rad[m] = w.x(X_RAD)[c - 2 + m];
        }
        const float sbg = w.x(X_SBG)[c], pbg = w.x(X_PBG)[c], ubg = w.x(X_UBG)[c], sx = dtf * w.x(X_IDX)[c];
        const float g0 = w.x(X_XA)[c], g1 = w.x(X_XA)[c + 1], f = dtf * w.x(X_IXV)[c], irad = w.x(X_IRAD)[c];
#pragma unroll 1
        for (int j = run.z; j < run.w; ++j, src += D.pitch) {
            float dS[5], du[5], dv[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                dS[m] = src[m - 2];
                du[m] = src[D.pl + m - 2];
                dv[m] = src[2 * D.pl + m - 2];
            }
            float aS[5], aP[5], aU[5], aL[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                if (m == 2) {
                    aS[m] = aP[m] = aU[m] = aL[m] = 0.0f;
                    continue;
                }
                const int kk = m < 2 ? m : m - 1;
                aS[m] = (dS[m] - dS[2]) + db[kk];
                aP[m] = (cs2[m] * dS[m] - cs2[2] * dS[2]) + db[4 + kk];
                aU[m] = (du[m] - du[2]) + db[8 + kk];
                aL[m] = (rad[m] * dv[m] - rad[2] * dv[2]) + db[12 + kk];
            }
            const float Sc = sbg + dS[2];
            const float pc = pbg + cs2[2] * dS[2];
            const float uc = ubg + du[2];
            const float cs0 = gam * pc * rsq32(gam * pc * Sc);
            const float flat = flatten32(pc, aP[0], aP[1], aP[3], aP[4], aU[1], aU[3]);
            const Par32 R = recon32(wt, aS[0], aS[1], aS[3], aS[4], flat);
            const Par32 P = recon32(wt, aP[0], aP[1], aP[3], aP[4], flat);
            const Par32 U = recon32(wt, aU[0], aU[1], aU[3], aU[4], flat);
            const Par32 A = recon32(wt, aL[0], aL[1], aL[3], aL[4], flat);
            const HS a = edge32<0>(gam, sx, cs0, Sc, pc, uc, R, P, U, A);
            const HS b = edge32<1>(gam, sx, cs0, Sc, pc, uc, R, P, U, A);
            // HLLC at the left face, referenced to its left cell (jumps from there to this cell)
            const float jS = up1(aS[3]), jP = up1(aP[3]), jL = up1(aL[3]);
            const HS L{up1(b.rd), up1(b.pd), up1(b.u), up1(b.v)};
            const HS Rr{a.rd + jS, a.pd + jP, a.u, a.v + jL};
            const FX F = hllc32(gam, up1(Sc), up1(pc), L, Rr);
            // residual update (sweeps.cu:218-261, 300-335)
            const float Fr1 = down1(F.r);
            const float Dr = (F.r * g0 - Fr1 * g1) * f;
            // pres0 - pres1 = (p[s-1] - p[s]) + (pd0 - pd1)
            const float dpres = (F.pd - down1(F.pd)) - jP;
            const float Du = ((F.u * g0 - down1(F.u) * g1) + 0.5f * (g0 + g1) * dpres) * f;
            // D(Sigma v) - v D(Sigma) with l = r v: faces referenced to cells s-1 and s
            const float Dv = (g0 * F.r * (F.v - jL) - g1 * Fr1 * down1(F.v)) * f * irad;
            if (output) {
                float dSn = dS[2], dun = du[2], dvn = dv[2];
                const float Sn = Sc + Dr;
                const float rmin = fmaxf(Sc * 1.0e-10f, 1.0e-10f);
                if (Sn < rmin) {
                    dSn = rmin - sbg;
                    atomicAdd(&sc->floor_hits, 1);
                } else {
                    const float iS = rcp32(Sn);
                    dSn += Dr;
                    dun += (Du - uc * Dr) * iS;
                    dvn += Dv * iS;
                }
                if (!(Sn > 0.0f)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                D.emit(i, j, dSn, dun, dvn);
            }
        }
    }
}

// ========================================= azimuthal sweep + orbital shift
// A lane marches along its column: five rows of it in registers, the next in flight.
__global__ void __launch_bounds__(MT, 5) k32_sweep_y(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                  int nruns, int in) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_enter();
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0;
        const double dt = sc->dt;
        const float dtf = (float)dt, gam = w.gam;
        const int i = run.y + lane, c = min(i, NPAD + w.xres - 1);
        const bool active = i < NPAD + w.xres;
        const Disk32 D(w, in);
        if (done) {
            const float* src = w.buf[in] + (size_t)run.z * w.pitch + c;
            for (int j = run.z; j < run.w; ++j, src += D.pitch)
                if (active) D.emit(i, j, src[0], src[D.pl], src[2 * D.pl]);
            continue;
        }
        int js = run.z - NPAD;  // row the first output goes to (orbit.cu:30-46)
        if (w.orbadv) {
            // set_orbital_advection (src/orbit/orbit.cu:74-99) in FP64 for this column
            const DiskView& d = w.d64;
            const double dy = d.dy0 * d.radx[c];
            const double rot = d.rot[c];
            const int shift = __double2int_rd(rot * dt / dy + 0.5);
            double speed = shift * dy / dt;
            speed = rot - speed;
            if (run.z == NPAD && active) {
                d.res[i] = speed;
                d.inc[i] = shift;
            }
            js = (js + shift) % w.yres;
            if (js < 0) js += w.yres;
        }
        const float cs2 = w.x(X_CS2)[c], cs0 = w.x(X_CS0)[c], eps = w.x(X_EPS)[c], sbg = w.x(X_SBG)[c];
        const float pbg = w.x(X_PBG)[c], irad = w.x(X_IRAD)[c], sdt = dtf * irad;
        const float* next = w.buf[in] + (size_t)(run.z - NPAD) * w.pitch + c;
        float dS[5], du[5], dv[5], nS = 0.0f, nu = 0.0f, nv = 0.0f;
#pragma unroll
        for (int m = 0; m < 5; ++m, next += D.pitch) {
            dS[m] = next[0];
            du[m] = next[D.pl];
            dv[m] = next[2 * D.pl];
        }
        HS pb{};   // the right edge of the cell below
        FX pf{};   // the flux at the face below it
#pragma unroll 1
        for (int t = run.z - 1; t <= run.w; ++t, next += D.pitch) {
            if (t < run.w) {
                nS = next[0];
                nu = next[D.pl];
                nv = next[2 * D.pl];
            }
            float aS[5], aN[5], aT[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                aS[m] = dS[m] - dS[2];
                aN[m] = dv[m] - dv[2];
                aT[m] = du[m] - du[2];
            }
            const float Sc = sbg + dS[2];
            const float pc = cs2 * Sc;
            const float un = dv[2] + eps;
            // p = cs2 Sigma along the column: pressure ratios are density ratios
            const float flat = flatten32(Sc, aS[0], aS[1], aS[3], aS[4], aN[1], aN[3]);
            float wt[6];
            D.ys<6>(Y_WY, t, wt);
            const Par32 R = recon32(wt, aS[0], aS[1], aS[3], aS[4], flat);
            const Par32 N = recon32(wt, aN[0], aN[1], aN[3], aN[4], flat);
            const Par32 Tt = recon32(wt, aT[0], aT[1], aT[3], aT[4], flat);
            const Par32 P{cs2 * R.sL, cs2 * R.sR};
            const float sx = sdt * D.y(Y_IDY, t);
            HS a = edge32<0>(gam, sx, cs0, Sc, pc, un, R, P, N, Tt);
            HS b = edge32<1>(gam, sx, cs0, Sc, pc, un, R, P, N, Tt);
            // relative to the background, which is constant along the column
            a.rd += dS[2];
            a.pd += cs2 * dS[2];
            a.v += du[2];
            b.rd += dS[2];
            b.pd += cs2 * dS[2];
            b.v += du[2];
            FX F{};
            if (t >= run.z) F = hllc32(gam, sbg, pbg, pb, a);
            if (t > run.z) {  // the cell below has both its fluxes
                const int j = t - 1;
                const float dS0 = dS[1], du0 = du[1], dv0 = dv[1];
                const float f = dtf * D.y(Y_IYV, j) * irad;
                const float Dr = (pf.r - F.r) * f;
                const float Dn = ((pf.u - F.u) + (pf.pd - F.pd)) * f;
                const float Dt = (pf.r * (pf.v - du0) - F.r * (F.v - du0)) * f;
                if (active) {
                    float dSn = dS0, dun = du0, dvn = dv0;
                    const float S0 = sbg + dS0;
                    const float Sn = S0 + Dr;
                    const float rmin = fmaxf(S0 * 1.0e-10f, 1.0e-10f);
                    if (Sn < rmin) {
                        dSn = rmin - sbg;
                        atomicAdd(&sc->floor_hits, 1);
                    } else {
                        const float iS = rcp32(Sn);
                        dSn = dS0 + Dr;
                        dvn = dv0 + (Dn - (dv0 + eps) * Dr) * iS;
                        dun = du0 + Dt * iS;
                    }
                    if (!(Sn > 0.0f)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    D.emit(i, js + NPAD, dSn, dun, dvn);
                }
                if (++js == D.yres) js = 0;
            }
            pb = b;
            pf = F;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                dS[m] = dS[m + 1];
                du[m] = du[m + 1];
                dv[m] = dv[m + 1];
            }
            dS[4] = nS;
            du[4] = nu;
            dv[4] = nv;
        }
    }
}

// ===================================================== residual advection
// advection.cu:20-170.  The residual speed of a column has one sign: every cell feeds
// the same one of its two faces, and with this row's flux and the last one's the update
// of this row (upwards) or the last (downwards) is complete.
__global__ void __launch_bounds__(MT, 5) k32_advect(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                 int nruns, int in) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_enter();
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0;
        const double dt = sc->dt;
        const float dtf = (float)dt;
        const int i = run.y + lane, c = min(i, NPAD + w.xres - 1);
        const bool active = i < NPAD + w.xres;
        const Disk32 D(w, in);
        if (done) {
            const float* src = w.buf[in] + (size_t)run.z * w.pitch + c;
            for (int j = run.z; j < run.w; ++j, src += D.pitch)
                if (active) D.emit(i, j, src[0], src[D.pl], src[2 * D.pl]);
            continue;
        }
        const DiskView& d = w.d64;
        const double speed = d.res[c];
        const double* idy = d.idx_y;
        const double sx = fabs(speed) * (dt * d.irad[c]);
        const bool up = speed > 0.0;
        const float spf = (float)speed, sbg = w.x(X_SBG)[c], irad = w.x(X_IRAD)[c];
        const float* next = w.buf[in] + (size_t)(run.z - NPAD) * w.pitch + c;
        float dS[5], du[5], dv[5], nS = 0.0f, nu = 0.0f, nv = 0.0f;
#pragma unroll
        for (int m = 0; m < 5; ++m, next += D.pitch) {
            dS[m] = next[0];
            du[m] = next[D.pl];
            dv[m] = next[2 * D.pl];
        }
        float pr = 0.0f, pn = 0.0f, pt = 0.0f;  // the row before: mass flux and the carried v and u
#pragma unroll 1
        for (int t = run.z - 1; t <= run.w; ++t, next += D.pitch) {
            if (t < run.w) {
                nS = next[0];
                nu = next[D.pl];
                nv = next[2 * D.pl];
            }
            // the swept fraction in FP64: |res| dt / (r dphi)
            const Frac32 qf = frac32((float)fmin(sx * idy[t], 1.0));
            float wt[6];
            D.ys<6>(Y_WY, t, wt);
            const Par32 R = recon32(wt, dS[0] - dS[2], dS[1] - dS[2], dS[3] - dS[2], dS[4] - dS[2], 0.0f);
            const Par32 N = recon32(wt, dv[0] - dv[2], dv[1] - dv[2], dv[3] - dv[2], dv[4] - dv[2], 0.0f);
            const Par32 Tt = recon32(wt, du[0] - du[2], du[1] - du[2], du[3] - du[2], du[4] - du[2], 0.0f);
            const float fr = ((sbg + dS[2]) + (up ? aveR32(qf, R) : aveL32(qf, R))) * spf;
            const float fn = dv[2] + (up ? aveR32(qf, N) : aveL32(qf, N));
            const float ft = du[2] + (up ? aveR32(qf, Tt) : aveL32(qf, Tt));
            const int j = up ? t : t - 1;
            if (active && j >= run.z && j < run.w) {
                const float dS0 = up ? dS[2] : dS[1], du0 = up ? du[2] : du[1], dv0 = up ? dv[2] : dv[1];
                const float f = dtf * D.y(Y_IYV, j) * irad;
                const float Dr = (pr - fr) * f;
                const float Sn = (sbg + dS0) + Dr;
                const float iS = rcp32(Sn);
                if (!(Sn > 0.0f)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                D.emit(i, j, dS0 + Dr, du0 + (pr * (pt - du0) - fr * (ft - du0)) * f * iS,
                       dv0 + (pr * (pn - dv0) - fr * (fn - dv0)) * f * iS);
            }
            pr = fr;
            pn = fn;
            pt = ft;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                dS[m] = dS[m + 1];
                du[m] = du[m + 1];
                dv[m] = dv[m + 1];
            }
            dS[4] = nS;
            du[4] = nu;
            dv[4] = nv;
        }
    }
}

// ====================================================== kick 1 (+ stress)
// Lanes 1..30 of a run have an output; the stress stencil's rows stay in registers.
__global__ void __launch_bounds__(MT, 5) k32_kick1(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                int nruns, int in) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_enter();
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0, visc = w.visc != 0;
        const float hdt = (float)(0.5 * sc->dt);
        const int i = run.y + lane, c = min(i, w.xarr - 1);
        const bool output = lane >= 1 && lane <= 30 && i < NPAD + w.xres;
        const Disk32 D(w, in);
        const float* next = w.buf[in] + (size_t)run.z * w.pitch + c;
        if (done) {
            for (int j = run.z; j < run.w; ++j, next += D.pitch)
                if (output) {
                    D.emit(i, j, next[0], next[D.pl], next[2 * D.pl]);
                    if (w.dust) dstore(w, w.dbuf[in ^ 1], i, j, dload(w, w.dbuf[in], i, j));
                }
            continue;
        }
        const Kick32 K = kick_tables(w, c, 0);
        const bool dusty = w.dust != 0;
        float* vis = w.vis + ((size_t)run.z * D.pitch + c);
        const float* const last = next + (size_t)(run.w - run.z) * D.pitch;
        next -= D.pitch;
        Row32 lo{}, mid = row32(next[0], next[D.pl], next[2 * D.pl]);
        next += D.pitch;
        Row32 hi = row32(next[0], next[D.pl], next[2 * D.pl]);
        next += D.pitch;
        float nS = next[0], nu = next[D.pl], nv = next[2 * D.pl];  // a row ahead of the stencil
#pragma unroll 1
        for (int j = run.z; j < run.w; ++j, vis += D.pitch) {
            lo = mid;
            mid = hi;
            hi = row32(nS, nu, nv);
            if (next < last) {
                next += D.pitch;
                nS = next[0];
                nu = next[D.pl];
                nv = next[2 * D.pl];
            }
            float vx = 0.0f, vy = 0.0f;
            if (visc) stress32(D, K, j, lo, mid, hi, vx, vy);
            if (!output) continue;
            if (visc) {  // kept for the predictor of kick2, with the periodic image
                vis[0] = vx;
                vis[D.pl] = vy;
                if (j < 2 * NPAD || j >= D.yres) {
                    float* s = vis + (long long)(j < 2 * NPAD ? D.yres : -D.yres) * D.pitch;
                    s[0] = vx;
                    s[D.pl] = vy;
                }
            }
            float gx, gy, du = mid.u[1], dv = mid.v[1];
            gravity32(K, j, gx, gy);
            kick32(K, mid.S, du, dv, vx, vy, gx, gy, 0.0f, hdt, visc);
            D.emit(i, j, mid.S, du, dv);
            if (dusty) {
                DR q = dload(w, w.dbuf[in], i, j);
                dust_drag32(w, i, K.sbg + mid.S, mid.u[1], mid.v[1], 0.0f, 0.0f, gx, gy, 0.0f, hdt, q);
                dstore(w, w.dbuf[in ^ 1], i, j, q);
            }
        }
    }
}

// ============================================ kick 2 + damping + CFL speed
// A row is predicted (sweeps.cu:713-729, mdt = dt = dt/2) with the stress of kick1 when
// it enters; outside the radial range the ghosts keep init_C (zero residuals) as boundx2
// does for boundary 0 (boundary.cu:722-820).
__global__ void __launch_bounds__(MT, 5) k32_kick2(const View32* __restrict__ V, const int4* __restrict__ runs,
                                                int nruns, int in) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_enter();
    for (int it = blockIdx.x * MW + warp; it < nruns; it += gridDim.x * MW) {
        const int4 run = runs[it];
        const View32& w = V[run.x];
        Scalars* sc = w.d64.sc;
        const bool done = sc->done != 0, visc = w.visc != 0;
        const double dt = sc->dt;
        const float dtf = (float)dt, hdt = (float)(0.5 * dt);
        const int i = run.y + lane, c = min(i, w.xarr - 1);
        const bool inside = i >= NPAD && i < NPAD + w.xres;
        const bool output = inside && lane >= 1 && lane <= 30;
        const Disk32 D(w, in);
        const float* next = w.buf[in] + (size_t)run.z * w.pitch + c;
        if (done) {
            for (int j = run.z; j < run.w; ++j, next += D.pitch)
                if (output) {
                    D.emit(i, j, next[0], next[D.pl], next[2 * D.pl]);
                    if (w.dust) dstore(w, w.dbuf[in ^ 1], i, j, dload(w, w.dbuf[in], i, j));
                }
            continue;
        }
        const Kick32 K = kick_tables(w, c, 1);
        const DiskView& d = w.d64;
        // the CFL rate (timestep.cu:46-77) in FP64 from the residuals
        const double ubg = d.initx[5 * c + 2], vbg = d.initx[5 * c + 3] - d.radx[c] * d.frame_omega - d.rot[c];
        const double cs = w.cs64[c], idx = d.idx_x[c], irad = d.irad[c];
        float kw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (w.kill) xload<4>(w, X_KILL, c, kw);
        const double* idy = d.idx_y;
        const bool dusty = w.dust != 0, damped = kw[1] > 0.0f || kw[3] > 0.0f;
        double vmax = 0.0;
        int jn = run.z - 1;  // the next row to enter the stencil
        next -= D.pitch;
        const float* const last = next + (size_t)(run.w - run.z + 1) * D.pitch;
        const float* nvis = w.vis + ((size_t)jn * D.pitch + c);
        float u = 0.0f, v = 0.0f, gx = 0.0f, gy = 0.0f;      // the middle row before the kick, its gravity
        float un = 0.0f, vn = 0.0f, gxn = 0.0f, gyn = 0.0f;  // ... of the row that entered last
        float nS, nu, nv, nx = 0.0f, ny = 0.0f;              // the row after it and its stress, in flight
        auto fetch = [&]() {
            nS = next[0];
            nu = next[D.pl];
            nv = next[2 * D.pl];
            if (visc) {
                nx = nvis[0];
                ny = nvis[D.pl];
            }
        };
        Row32 lo{}, mid{}, hi{};
        auto enter = [&]() {
            const float S = nS, fx = nx, fy = ny;
            un = nu;
            vn = nv;
            if (next < last) {
                next += D.pitch;
                nvis += D.pitch;
                fetch();
            }
            gravity32(K, jn, gxn, gyn);
            float pu = un, pv = vn;
            if (visc) {
                if (inside) kick32(K, S, pu, pv, fx, fy, gxn, gyn, hdt, hdt, true);
                hi = row32(S, pu, pv);
            } else {
                hi.S = S;
            }
            ++jn;
        };
        fetch();
#pragma unroll 1
        for (int j = run.z - 2; j < run.w; ++j) {  // two rows enter before the first output
            lo = mid;
            mid = hi;
            u = un;
            v = vn;
            gx = gxn;
            gy = gyn;
            enter();
            if (j < run.z) continue;
            float vx = 0.0f, vy = 0.0f;
            if (visc) stress32(D, K, j, lo, mid, hi, vx, vy);
            if (!output) continue;
            float dS = mid.S, du = u, dv = v;
            if (dusty) {
                // the gas velocity predicted over mdt (sweeps.cu:679-687), towards which
                // the dust's corrector relaxes
                DR q = dload(w, w.dbuf[in], i, j);
                const float iS = visc ? rcp32(K.sbg + dS) : 0.0f;
                const float fx0 = K.abg + (K.v2r + dv * K.ir) * dv + vx * iS;
                const float tu = du + fx0 * hdt + gx * hdt, tv = dv + vy * iS * hdt + gy * hdt;
                dust_drag32(w, i, K.sbg + dS, du, dv, tu, tv, gx, gy, hdt, hdt, q);
                vmax = fmax(vmax, drate64(w, i, j, q.u, q.v));
                dstore(w, w.dbuf[in ^ 1], i, j, q);
            }
            kick32(K, dS, du, dv, vx, vy, gx, gy, hdt, hdt, visc);
            if (damped) {
                // killwave (killwave.cu:48-100): relax towards init_C, i.e. residuals towards 0
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const float itau = kw[2 * side + 1];
                    if (itau > 0.0f) {
                        const float f = kw[2 * side] * (dtf * itau);
                        dS -= f * dS;
                        du -= f * du;
                        dv -= f * dv;
                    }
                }
            }
            if (!(K.sbg + dS > 0.0f)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
            const double a = (fabs(ubg + (double)du) + cs) * idx;
            const double b = (fabs(vbg + (double)dv) + cs) * (idy[j] * irad);
            vmax = fmax(vmax, fmax(a, b));
            D.emit(i, j, dS, du, dv);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        if (lane == 0) atomic_max_pos(&sc->vmax_bits, vmax);
    }
}

// ================================================================ misc
// One block per disk: its first thread sets dt, clock and planet of the step, then all fill
// its planet table (see TRIG_ROW).
__global__ void __launch_bounds__(1024) k32_time(const View32* __restrict__ V) {
    pdl_enter();
    const View32& w = V[blockIdx.x];
    if (threadIdx.x == 0) advance_clock(w.d64);
    __syncthreads();
    const Scalars* sc = w.d64.sc;
    const pg_body& a = sc->planet_cur;
    const pg_body& b = sc->planet_next;
    const double ya = a.y + 0.0 * a.vy, yb = b.y + 0.0 * b.vy;
    for (int k = threadIdx.x; k < w.yarr; k += blockDim.x) {
        float* t = w.trig + (size_t)TRIG_ROW * k;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            double s, c;
            sincos(0.5 * (w.d64.ycj[k] - (which ? yb : ya)), &s, &c);
            t[3 * which] = (float)(2.0 * s * c);
            t[3 * which + 1] = (float)(1.0 - 2.0 * s * s);
            t[3 * which + 2] = (float)(2.0 * s * s);
        }
    }
    for (int k = threadIdx.x; k < w.xarr; k += blockDim.x) {
        float* c = w.trig + (size_t)TRIG_ROW * w.yn + 2 * k;
        c[0] = (float)(w.d64.radx[k] - a.x);
        c[1] = (float)(w.d64.radx[k] - b.x);
    }
    if (threadIdx.x == 0) {
        float* s = w.trig + (size_t)TRIG_ROW * w.yn + 2 * (size_t)w.xn;
        s[0] = (float)a.m;
        s[1] = (float)a.x;
        s[2] = (float)(a.rs * a.rs);
        s[3] = (float)(1.0 / a.x / a.x);
        s[4] = (float)b.m;
        s[5] = (float)b.x;
        s[6] = (float)(b.rs * b.rs);
        s[7] = (float)(1.0 / b.x / b.x);
    }
}

// Signal rate of a state just written by set_state (one disk).
__global__ void k32_cfl(const View32* __restrict__ V, int b) {
    const View32& w = *V;
    const float* buf = w.buf[b];
    const size_t pl = w.plane();
    const long long n = (long long)w.xres * w.yres;
    double vmax = 0.0;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const size_t c = (size_t)j * w.pitch + i;
        vmax = fmax(vmax, rate64(w, i, j, buf[pl + c], buf[2 * pl + c]));
        if (w.dust) vmax = fmax(vmax, drate64(w, i, j, w.dbuf[b][pl + c], w.dbuf[b][2 * pl + c]));
    }
    block_max_to<256>(&w.d64.sc->vmax_bits, vmax);
}

// dust (absolute FP64 interior arrays) <-> residual planes against init_CD
__global__ void k32_dfill(const View32* __restrict__ V, int b, const double* r, const double* u, const double* v) {
    const View32& w = *V;
    const long long n = (long long)w.xres * w.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const double* I = w.d64.initd + 4 * i;
        dstore(w, w.dbuf[b], i, j, DR{(float)(r[m] - I[0]), (float)(u[m] - I[1]), (float)(v[m] - I[2])});
    }
}
__global__ void k32_dextract(const View32* __restrict__ V, int b, double* r, double* u, double* v) {
    const View32& w = *V;
    const long long n = (long long)w.xres * w.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const double* I = w.d64.initd + 4 * i;
        const DR c = dload(w, w.dbuf[b], i, j);
        r[m] = I[0] + (double)c.S;
        u[m] = I[1] + (double)c.u;
        v[m] = I[2] + (double)c.v;
    }
}

// Host state (FP64 interior arrays) -> residual planes with their azimuthal images.
__global__ void k32_fill(const View32* __restrict__ V, int b, const double* r, const double* u, const double* v) {
    const View32& w = *V;
    const long long n = (long long)w.xres * w.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const double* I = w.d64.initx + 5 * i;
        emit32(w, w.buf[b], i, j, (float)(r[m] - I[0]), (float)(u[m] - I[2]), v ? (float)(v[m] - I[3]) : 0.0f);
    }
}

__global__ void k32_extract(const View32* __restrict__ V, int b, double* r, double* p, double* u, double* v) {
    const View32& w = *V;
    const float* buf = w.buf[b];
    const size_t pl = w.plane();
    const long long n = (long long)w.xres * w.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const size_t c = (size_t)j * w.pitch + i;
        const double* I = w.d64.initx + 5 * i;
        const double rr = I[0] + (double)buf[c];
        r[m] = rr;
        p[m] = w.d64.cs2x[i] * rr;
        u[m] = I[2] + (double)buf[pl + c];
        v[m] = I[3] + (double)buf[2 * pl + c];
    }
}

// Mass and angular momentum, sum Sigma dV and sum Sigma r v dV with dV = xv yv,
// in FP64 with compensated (Kahan) accumulation per thread, then one partial
// pair per block, summed on the host in block order (deterministic).
__global__ void k32_totals(const View32* __restrict__ V, int b, double* part) {
    const View32& w = *V;
    const DiskView& d = w.d64;
    const float* buf = w.buf[b];
    const size_t pl = w.plane();
    const long long n = (long long)w.xres * w.yres;
    double sm = 0.0, cm = 0.0, sl = 0.0, cl = 0.0;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const size_t c = (size_t)j * w.pitch + i;
        const double dV = d.xv[i] * d.yv[j];
        const double S = d.initx[5 * i] + (double)buf[c];
        const double vv = d.initx[5 * i + 3] + (double)buf[2 * pl + c];
        double y = S * dV - cm;
        double t = sm + y;
        cm = (t - sm) - y;
        sm = t;
        y = S * d.radx[i] * vv * dV - cl;
        t = sl + y;
        cl = (t - sl) - y;
        sl = t;
    }
    __shared__ double rm[256], rl[256];
    rm[threadIdx.x] = sm;
    rl[threadIdx.x] = sl;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            rm[threadIdx.x] += rm[threadIdx.x + h];
            rl[threadIdx.x] += rl[threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = rm[0];
        part[2 * blockIdx.x + 1] = rl[0];
    }
}

// Torque of the planet on the disk, as k_torque of the FP64 kernels
// (src/output/output.cu:336-412), in FP64 from the residual state.
__global__ void k32_torque(const View32* __restrict__ V, int b, double* part) {
    const View32& w = *V;
    const DiskView& d = w.d64;
    const pg_body p = d.sc->planet_next;
    const float* buf = w.buf[b];
    const long long n = (long long)w.xres * w.yres;
    double sum = 0.0, comp = 0.0;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % w.xres), j = NPAD + (int)(m / w.xres);
        const double rad = d.radx[i];
        double sinfac, cosfac;
        sincos(d.ycraw[j] - p.y, &sinfac, &cosfac);
        const double Rp = sqrt(rad * rad + p.x * p.x - 2.0 * p.x * rad * cosfac + p.rs * p.rs);
        const double rs_fac = 1.0 / Rp / Rp / Rp;
        const double gy = -p.m * p.x * sinfac * rs_fac + p.m * sinfac / p.x / p.x;
        const double dv = 0.5 * (d.xa[i + 1] * d.xa[i + 1] - d.xa[i] * d.xa[i]) * (d.ya[j + 1] - d.ya[j]);
        const double S = d.initx[5 * i] + (double)buf[(size_t)j * w.pitch + i];
        const double y = rad * gy * (S * dv) - comp;
        const double t = sum + y;
        comp = (t - sum) - y;
        sum = t;
    }
    __shared__ double red[256];
    red[threadIdx.x] = sum;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// FP32 tables of one disk from its FP64 tables (slots in pg_f32.cuh).
__global__ void k32_init_tables(const View32 w, float* tx, float* ty, double* cs64) {
    const DiskView& d = w.d64;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    auto X = [&](int slot) { return tx + (size_t)slot * w.xn; };
    auto Y = [&](int slot) { return ty + (size_t)slot * w.yn; };
    if (k < w.xarr) {
        const int i = k;
        const double* I = d.initx + 5 * i;
        X(X_SBG)[i] = (float)I[0];
        X(X_PBG)[i] = (float)I[1];
        X(X_UBG)[i] = (float)I[2];
        X(X_CS2)[i] = (float)d.cs2x[i];
        X(X_RAD)[i] = (float)d.radx[i];
        X(X_IRAD)[i] = (float)d.irad[i];
        X(X_IDX)[i] = (float)d.idx_x[i];
        X(X_IXV)[i] = (float)d.ixv[i];
        X(X_XA)[i] = (float)d.xa[i];
        if (i == w.xarr - 1) X(X_XA)[i + 1] = (float)d.xa[i + 1];
        X(X_NU)[i] = (float)d.nux[i];
        X(X_ABG)[i] = (float)(I[3] * I[3] * d.irad[i] + d.gstar[i]);
        X(X_V2R)[i] = (float)(2.0 * I[3] * d.irad[i]);
        X(X_EPS)[i] = (float)(I[3] - d.radx[i] * d.frame_omega - d.rot[i]);
        const double cs = sqrt(d.gam * d.cs2x[i]);
        X(X_CS0)[i] = (float)cs;
        cs64[i] = cs;

        const int offs[4] = {-2, -1, 1, 2};
        for (int kk = 0; kk < 4; ++kk) {
            const int ik = min(max(i + offs[kk], 0), w.xarr - 1);
            const double* J = d.initx + 5 * ik;
            X(X_DBG + kk)[i] = (float)(J[0] - I[0]);
            X(X_DBG + 4 + kk)[i] = (float)(J[1] - I[1]);
            X(X_DBG + 8 + kk)[i] = (float)(J[2] - I[2]);
            X(X_DBG + 12 + kk)[i] = (float)(d.radx[ik] * J[3] - d.radx[i] * I[3]);
        }
        for (int m = 0; m < 6; ++m) X(X_WX + m)[i] = (float)d.wx[6 * i + m];
        for (int m = 0; m < 5; ++m) X(X_VISX + m)[i] = (float)d.visx[5 * i + m];
        float vb[7] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (i >= 1 && i + 1 < w.xarr) {
            // the background's viscous force density, linear in (nr1, dndx, dndy): the
            // reference's stencil with v_r0, v_phi0 axisymmetric (all d/dphi terms vanish)
            const double* Xr = d.visx + 5 * i;
            const double i_r20 = Xr[0], i_r21 = Xr[1], i_r10 = Xr[2], i_hr20 = Xr[3], i_r1 = Xr[4];
            const double u0 = d.initx[5 * (i - 1) + 2], u1 = I[2], u2 = d.initx[5 * (i + 1) + 2];
            const double v0 = d.initx[5 * (i - 1) + 3], v1 = I[3], v2 = d.initx[5 * (i + 1) + 3];
            const double dudx = (u2 - u0) * i_r20;
            const double d2udx2 = ((u2 - u1) * i_r21 - (u1 - u0) * i_r10) * i_hr20;
            const double dvdx = (v2 - v0) * i_r20;
            const double d2vdx2 = ((v2 - v1) * i_r21 - (v1 - v0) * i_r10) * i_hr20;
            vb[0] = (float)(2.0 * d2udx2 + 2.0 * dudx * i_r1 - 2.0 * u1 * i_r1 * i_r1);
            vb[1] = (float)(2.0 * dudx);
            vb[2] = (float)(dvdx - v1 * i_r1);
            vb[3] = (float)(d2vdx2 - dvdx * i_r1 + v1 * i_r1 * i_r1 + 2.0 * (dvdx - v1 * i_r1) * i_r1);
            vb[4] = (float)(dvdx - v1 * i_r1);
            vb[5] = (float)(2.0 * u1 * i_r1);
            vb[6] = (float)(d.initx[5 * (i + 1)] * d.nux[i + 1] - d.initx[5 * (i - 1)] * d.nux[i - 1]);
        }
        for (int m = 0; m < 7; ++m) X(X_VBG + m)[i] = vb[m];
        if (d.initd) {
            const double* D = d.initd + 4 * i;
            X(X_DSBG)[i] = (float)D[0];
            X(X_DUBG)[i] = (float)D[1];
            X(X_DVBG)[i] = (float)D[2];
            X(X_DEPS)[i] = (float)(D[2] - d.radx[i] * d.frame_omega - d.rot[i]);
            X(X_DABG)[i] = (float)(D[2] * D[2] * d.irad[i] + d.gstar[i]);
            X(X_DV2R)[i] = (float)(2.0 * D[2] * d.irad[i]);
            X(X_DGU)[i] = (float)(I[2] - D[1]);
            X(X_DGV)[i] = (float)(I[3] - D[2]);
            for (int kk = 0; kk < 4; ++kk) {
                const int ik = min(max(i + offs[kk], 0), w.xarr - 1);
                const double* E = d.initd + 4 * ik;
                X(X_DDBG + kk)[i] = (float)(E[0] - D[0]);
                X(X_DDBG + 4 + kk)[i] = (float)(E[1] - D[1]);
                X(X_DDBG + 8 + kk)[i] = (float)(d.radx[ik] * E[2] - d.radx[i] * D[2]);
            }
        }
        const double* kt = d.killx + 4 * i;
        X(X_KILL + 0)[i] = (float)kt[0];
        X(X_KILL + 1)[i] = kt[1] > 0.0 ? (float)(1.0 / kt[1]) : 0.0f;
        X(X_KILL + 2)[i] = (float)kt[2];
        X(X_KILL + 3)[i] = kt[3] > 0.0 ? (float)(1.0 / kt[3]) : 0.0f;
    }
    if (k < w.yarr) {
        Y(Y_IDY)[k] = (float)d.idx_y[k];
        Y(Y_IYV)[k] = (float)d.iyv[k];
        for (int m = 0; m < 6; ++m) Y(Y_WY + m)[k] = (float)d.wy[6 * k + m];
        for (int m = 0; m < 4; ++m) Y(Y_VISY + m)[k] = (float)d.visy[4 * k + m];
    }
}

// test support: the edge states' root of a product
__global__ void k32_test_root(const float* ab, long long n, float* out) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
        out[k] = rsq32_product(ab[2 * k], ab[2 * k + 1]);
}

// ============================================================== launchers
static inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

static int sm_count32() {
    static int nsm = 0;
    if (nsm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (nsm <= 0) nsm = 148;
    }
    return nsm;
}

static unsigned persistent_grid(const void* kernel, int threads, size_t smem, long long ntiles, int cap = 0) {
    const int nsm = sm_count32();
    static const void* keys[16] = {nullptr};
    static int vals[16] = {0};
    int per_sm = 0;
    for (int n = 0; n < 16 && keys[n]; ++n)
        if (keys[n] == kernel) per_sm = vals[n];
    if (per_sm == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        for (int n = 0; n < 16; ++n)
            if (!keys[n]) {
                keys[n] = kernel;
                vals[n] = per_sm;
                break;
            }
    }
    if (cap > 0 && cap < per_sm) per_sm = cap;
    long long g = (long long)per_sm * nsm;
    if (g > ntiles) g = ntiles;
    return (unsigned)(g < 1 ? 1 : g);
}

static const void* pass_kernel(int pass) {
    static const void* const k[5] = {(const void*)k32_kick1, (const void*)k32_sweep_x, (const void*)k32_sweep_y,
                                     (const void*)k32_advect, (const void*)k32_kick2};
    return k[pass];
}

int pass_occupancy32(int pass) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pass_kernel(pass), MT, 0) != cudaSuccess)
        return 1;
    return per_sm < 1 ? 1 : per_sm;
}

// The runs of the three kinds (radial sweep; azimuthal sweep and advection; kicks) over
// disks of these sizes, as int4 {disk, first lane's radius, first row, last row + 1}.
// Long runs waste little on the rows that only feed the stencils at their ends and on the
// tables they load, short ones give the warps that hide latency: per kind the length with
// the least run_cost (pg_internal.h) at 20 resident warps an SM.  1024x3072, us a pass at
// 4 / 8 / 16 / 24 / 48 / 96 rows: radial sweep 82 / 78 / 77 / 85 / 80 / 115, azimuthal
// 96 / 82 / 73 / 74 / 76 / 98, kick2 105 / 90 / 88 / 89 / 82 / 128; by the rule 82, 72, 84.
// Variant 1 is half as long, for the autotuner to try.
void build_runs32(const int* xres, const int* yres, int nd, std::vector<int4>* runs, Runs32* R) {
    runs->clear();
    const int resident = 20 * sm_count32();
    for (int kind = 0; kind < 3; ++kind) {
        const int out = kind == 1 ? 32 : 30, first = kind == 1 ? NPAD : NPAD - 1;
        int len = 2;
        double best = 1e300;
        for (int l = 2; l <= 64; l += (l < 16 ? 1 : 4)) {
            long long warps = 0;
            for (int k = 0; k < nd; ++k) warps += (long long)((xres[k] + out - 1) / out) * ((yres[k] + l - 1) / l);
            const double cost = run_cost(warps, resident, l + (kind == 0 ? 1.5 : 3.5));
            if (cost < best) {
                best = cost;
                len = l;
            }
        }
        for (int v = 0; v < 2; ++v) {
            const int l = len >> v;
            R->first[v][kind] = (int)runs->size();
            for (int k = 0; k < nd; ++k)
                for (int j = 0; j < yres[k]; j += l)
                    for (int i = 0; i < xres[k]; i += out)
                        runs->push_back(make_int4(k, first + i, NPAD + j, NPAD + (j + l < yres[k] ? j + l : yres[k])));
            R->count[v][kind] = (int)runs->size() - R->first[v][kind];
        }
    }
}

void launch_time32(const View32* V, int nd, cudaStream_t s) { launch_step(k32_time, nd, 1024, 0, s, V); }
void launch_pass32(int pass, const View32* V, const Runs32& R, int in, cudaStream_t s, const Tune32& t) {
    static constexpr int KIND[5] = {2, 0, 1, 1, 2};
    const int v = t.v[pass], kind = KIND[pass], n = R.count[v][kind];
    const int4* runs = R.d + R.first[v][kind];
    const unsigned g = persistent_grid(pass_kernel(pass), MT, 0, cdiv(n, MW), t.cps[pass]);
    switch (pass) {
        case 0: launch_step(k32_kick1, g, MT, 0, s, V, runs, n, in); break;
        case 1: launch_step(k32_sweep_x, g, MT, 0, s, V, runs, n, in); break;
        case 2: launch_step(k32_sweep_y, g, MT, 0, s, V, runs, n, in); break;
        case 3: launch_step(k32_advect, g, MT, 0, s, V, runs, n, in); break;
        default: launch_step(k32_kick2, g, MT, 0, s, V, runs, n, in); break;
    }
}
void launch_cfl32(const View32* Vk, int b, cudaStream_t s) { k32_cfl<<<592, 256, 0, s>>>(Vk, b); }
// the dust part of pass 1 (radial sweep), 2 (azimuthal sweep), 3 (advection), on the gas's runs
void launch_dust_pass32(int pass, const View32* V, const Runs32& R, int in, cudaStream_t s) {
    auto go = [&](auto kernel, int kind) {
        const int n = R.count[0][kind];
        launch_step(kernel, persistent_grid((const void*)kernel, MT, 0, cdiv(n, MW)), MT, 0, s, V,
                    R.d + R.first[0][kind], n, in);
    };
    if (pass == 1) go(k32d_sweep_x, 0);
    else if (pass == 2) go(k32d_sweep_y, 1);
    else if (pass == 3) go(k32d_advect, 1);
}
void launch_dfill32(const View32* Vk, int b, const double* r, const double* u, const double* v, cudaStream_t s) {
    k32_dfill<<<592, 256, 0, s>>>(Vk, b, r, u, v);
}
void launch_dextract32(const View32* Vk, int b, double* r, double* u, double* v, cudaStream_t s) {
    k32_dextract<<<592, 256, 0, s>>>(Vk, b, r, u, v);
}
void launch_fill32(const View32* Vk, int b, const double* r, const double* u, const double* v, cudaStream_t s) {
    k32_fill<<<1184, 256, 0, s>>>(Vk, b, r, u, v);
}
void launch_extract32(const View32* Vk, int b, double* r, double* p, double* u, double* v, cudaStream_t s) {
    k32_extract<<<1184, 256, 0, s>>>(Vk, b, r, p, u, v);
}
void launch_totals32(const View32* Vk, int b, double* part, int nblocks, cudaStream_t s) {
    k32_totals<<<nblocks, 256, 0, s>>>(Vk, b, part);
}
void launch_torque32(const View32* Vk, int b, double* part, int nblocks, cudaStream_t s) {
    k32_torque<<<nblocks, 256, 0, s>>>(Vk, b, part);
}
void launch_init_tables32(const View32& w, float* tx, float* ty, double* cs64, cudaStream_t s) {
    const int n = w.xarr > w.yarr ? w.xarr : w.yarr;
    k32_init_tables<<<cdiv(n, 128), 128, 0, s>>>(w, tx, ty, cs64);
}

}  // namespace f32
}  // namespace pg

extern "C" pg_status pg_test_root32(const float* ab, long long n, float* out) {
    if (!ab || !out || n <= 0) return PG_ERR_ARG;
    float* d = nullptr;
    if (cudaMalloc(&d, 3 * n * sizeof(float)) != cudaSuccess) return PG_ERR_CUDA;
    cudaError_t e = cudaMemcpy(d, ab, 2 * n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        pg::f32::k32_test_root<<<592, 256>>>(d, n, d + 2 * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}
