// penguin_b200 3D form (ndim 3) for sm_100a: the reference's DS() with the
// polar sweep (src/solver/solve.cu:212-292 with ndim 3) as five passes over the
// AoS state, on the spherical (r, phi, theta) grid of the reference's 3D preset
// (include/para_files/Adiabatic_CPD.h: geometries 2/4/5) or on a cartesian box:
//
//   kick1   C -> T : first half-kick (src/solver/sweeps.cu:597-711, mdt = 0) with
//                    the spherical gravity and fictitious forces
//                    (src/solver/force/forces.cu:14-39, 110-327); radial ghost images
//   sweep_x T -> C : radial sweep (sweeps.cu:263-335); azimuthal ghost images
//   sweep_y C -> T : azimuthal sweep (sweeps.cu:361-433); polar ghost images
//   sweep_z T -> C : polar sweep (sweeps.cu:458-554)
//   kick2   C -> T : predictor + corrector half-kick, wave damping
//                    (src/killwave/killwave.cu:17-103) and the CFL signal rate
//                    (src/timestep/timestep.cu:18-97, ndim 3)
//
// plus the 2D form's one-block kernel of the clock and the per-row planet angles.  Lanes of a warp lie along the radius in every pass.  The radial sweep stages
// rows with TMA and exchanges edge states and fluxes between lanes by shuffle; the
// azimuthal and polar sweeps march along their direction with five cells of a column in
// registers (the 2D form's work layout, pg_kernels.cu, and its building blocks,
// pg_hydro.cuh).  Each pass writes the ghost cells the next pass reads (the images the
// reference's boundx/boundy/boundz copy in place), so no boundary pass runs between
// stages.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <vector>

#include "pg_common.cuh"
#include "pg_hydro.cuh"
#include "pg_internal.h"
#include "pg_planet.cuh"

namespace pg {

// ------------------------------------------------------------ work layout
constexpr int S3_WARPS = 4;                          // warps per CTA, independent of one another
constexpr int S3_THREADS = 32 * S3_WARPS;
constexpr int S3_OUT = 30;                           // radial sweep: outputs of a warp's 32 cells
constexpr int S3_ROWS = RX_TILE_ROWS;                // rows per TMA copy
constexpr int S3_STAGE = RX_TILE_CELLS * S3_ROWS * 5;  // doubles
constexpr int K3_THREADS = 256;
constexpr size_t S3_SMEM = (size_t)S3_WARPS * 2 * S3_STAGE * 8 + S3_WARPS * 16 + 128;
static_assert(S3_STAGE * 8 % 128 == 0, "128-byte aligned stages");
static_assert(RX_TILE_CELLS == S3_OUT + 6, "32 lanes and two stencil cells a side");

// Everything a 3D kernel reads: the 2D view's scalars, grid and tables for x
// and y (and the clock), plus the polar grid and the (x, z) tables.
struct View3 {
    DiskView d;
    int zres, zarr, geomz, bound_bom, bound_top, init3;
    double zmin;
    const double* za;
    const double* zv;
    const double* wz;      // 6 slope weights per polar index
    const double* idx_z;   // 1 / (za[k+1] - za[k])
    const double* zc;      // 0.5 (za[k+1] + za[k])
    const double* sinz;    // sin(zc) (the sweeps' and the CFL's rad_cyl)
    const double* sinpol;  // sincos(zc) (the planet's pull, forces.cu:18-21)
    const double* cospol;
    const double* tanz;    // tan(zc) (get_fz)
    const double* gfx;     // eval_gfac(geomx, xa[i]) (riemann.cu:5-11)
    const double* gfz;     // eval_gfac(geomz, za[k])
    const double* cs2;     // get_cs2(xc(i), zc(k)), xarr * zarr
    const double* initc;   // init_C(xc(i), zc(k)), 5 per (i, k)
};

__device__ __forceinline__ size_t at3(const View3& v, int i, int j, int k) {
    return (size_t)i + (size_t)v.d.xarr * ((size_t)j + (size_t)v.d.yarr * (size_t)k);
}
__device__ __forceinline__ void put3(Cell* out, const View3& v, int i, int j, int k, const Cell& c) {
    double* q = reinterpret_cast<double*>(out + at3(v, i, j, k));
    q[0] = c.r;
    q[1] = c.p;
    q[2] = c.u;
    q[3] = c.v;
    q[4] = c.w;
}
__device__ __forceinline__ Cell get3(const Cell* in, const View3& v, int i, int j, int k) {
    const double* q = reinterpret_cast<const double*>(in + at3(v, i, j, k));
    return Cell{q[0], q[1], q[2], q[3], q[4]};
}

// Ghost images.  Radial (kick1 output, read by the radial sweep; boundary.cu:13-62):
// bound 1 copies the edge cell, 2 mirrors it with u negated; bound-0 ghosts hold
// init_C and are never rewritten.
__device__ __forceinline__ void emit_x(const View3& v, Cell* out, int i, int j, int k, const Cell& c) {
    const DiskView& d = v.d;
    put3(out, v, i, j, k, c);
    const int nx = d.xres + NPAD;
    if (d.bound_lft == 1 && i == NPAD) {
        for (int n = 0; n < NPAD; ++n) put3(out, v, n, j, k, c);
    } else if (d.bound_lft == 2 && i < 2 * NPAD) {
        Cell m = c;
        m.u = -m.u;
        put3(out, v, 2 * NPAD - 1 - i, j, k, m);
    }
    if (d.bound_rgh == 1 && i == nx - 1) {
        for (int n = 0; n < NPAD; ++n) put3(out, v, nx + n, j, k, c);
    } else if (d.bound_rgh == 2 && i >= nx - NPAD) {
        Cell m = c;
        m.u = -m.u;
        put3(out, v, 2 * nx - 1 - i, j, k, m);
    }
}
// Azimuthal (radial sweep output, read by the azimuthal sweep): periodic
// (boundary.cu:140-209 with bound_bak / bound_frn 3).
__device__ __forceinline__ void emit_y(const View3& v, Cell* out, int i, int j, int k, const Cell& c) {
    put3(out, v, i, j, k, c);
    if (j < 2 * NPAD) put3(out, v, i, j + v.d.yres, k, c);
    else if (j >= v.d.yres) put3(out, v, i, j - v.d.yres, k, c);
}
// Polar (azimuthal sweep output, read by the polar sweep; boundary.cu:270-320):
// 1 zero gradient, 2 reflecting (w negated), 3 periodic; 0 holds init_C.
__device__ __forceinline__ void emit_z(const View3& v, Cell* out, int i, int j, int k, const Cell& c) {
    put3(out, v, i, j, k, c);
    const int nz = v.zres + NPAD;
    if (v.bound_bom == 2 && k < 2 * NPAD) {
        Cell m = c;
        m.w = -m.w;
        put3(out, v, i, j, 2 * NPAD - 1 - k, m);
    } else if (v.bound_bom == 1 && k == NPAD) {
        for (int n = 0; n < NPAD; ++n) put3(out, v, i, j, n, c);
    } else if (v.bound_bom == 3 && k >= v.zres) {
        put3(out, v, i, j, k - v.zres, c);
    }
    if (v.bound_top == 2 && k >= nz - NPAD) {
        Cell m = c;
        m.w = -m.w;
        put3(out, v, i, j, 2 * nz - 1 - k, m);
    } else if (v.bound_top == 1 && k == nz - 1) {
        for (int n = 0; n < NPAD; ++n) put3(out, v, i, j, nz + n, c);
    } else if (v.bound_top == 3 && k < 2 * NPAD) {
        put3(out, v, i, j, k + v.zres, c);
    }
}

// ================================================================ sweeps
__device__ __forceinline__ double up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double down1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Net flux through a cell's two faces.  The reference stores each flux times its area in
// shared memory before differencing, so the products are rounded on their own
// (__dmul_rn: no FMA).
__device__ __forceinline__ double net3(double f0, double g0, double f1, double g1) {
    return __dmul_rn(f0, g0) - __dmul_rn(f1, g1);
}
// the slots' increments (before the geometric factor) from the fluxes of the two faces
// (src/solver/riemann/riemann.cu:40-87)
__device__ __forceinline__ Cell increments(const DiskView& d, const Flux& a, double g0, const Flux& b, double g1) {
    Cell D;
    D.r = net3(a.r, g0, b.r, g1);
    D.u = net3(a.u, g0, b.u, g1) + 0.5 * (g0 + g1) * (a.pres - b.pres);
    D.v = net3(a.v, g0, b.v, g1);
    D.w = net3(a.w, g0, b.w, g1);
    D.p = 0.0;
    if (d.eos == 2) {
        double de = net3(a.uprs, g0, b.uprs, g1);
        if (d.ie != 0) de *= 0.5 * (a.pres + b.pres);
        D.p = net3(a.p, g0, b.p, g1) + de;
    }
    return D;
}

// Radial sweep (sweeps.cu:263-335) of rows j of one plane k: 4 rows of 36 cells per TMA
// copy, two copies in flight per warp; lane l holds cell 2 + 30 seg + l.  Compiled for MB
// CTAs per SM, 3 (168 registers) or 4 (128, some spilled): create3 picks.
template <int MB>
__global__ void __launch_bounds__(S3_THREADS, MB)
    k3_sweep_x(const __grid_constant__ CUtensorMap tm, const View3 v, Cell* __restrict__ out, int nseg, int len,
               int nchunk, int nitems) {
    extern __shared__ __align__(128) double smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* buf = smem_base128(smem_raw) + (size_t)warp * 2 * S3_STAGE;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_base128(smem_raw) + (size_t)S3_WARPS * 2 * S3_STAGE) + 2 * warp;
    const DiskView& d = v.d;
    Scalars* sc = d.sc;
    if (lane == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncwarp();
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt, gam = d.gam;
    int n = 0;  // copies waited for by this warp
    for (int item = blockIdx.x * S3_WARPS + warp; item < nitems; item += gridDim.x * S3_WARPS) {
        const int seg = item % nseg, rest = item / nseg;
        const int k = NPAD + rest / nchunk;
        const int j0 = NPAD + len * (rest % nchunk), j1 = min(j0 + len, NPAD + d.yres);
        auto issue = [&](int j, int m) {
            issue_begin(&bar[m & 1], S3_STAGE * 8);
            tma_load_3d(buf + (m & 1) * S3_STAGE, &tm, 5 * S3_OUT * seg, j, k, &bar[m & 1]);
        };
        if (lane == 0) {
            issue(j0, n);
            if (j0 + S3_ROWS < j1) issue(j0 + S3_ROWS, n + 1);
        }
        const int i = NPAD - 1 + S3_OUT * seg + lane, ic = min(i, d.xarr - 1);
        const bool output = lane >= 1 && lane <= S3_OUT && i < NPAD + d.xres;
        double w[6], rad[5];
#pragma unroll
        for (int m = 0; m < 6; ++m) w[m] = d.wx[6 * ic + m];
        // angular momenta r sin(theta) v_phi and r v_theta (sweeps.cu:283-300)
        const double sz = d.geomx == 2 ? v.sinz[k] : 1.0;
#pragma unroll
        for (int m = 0; m < 5; ++m) rad[m] = d.geomx != 0 ? d.radx[min(max(i - 2 + m, 0), d.xarr - 1)] : 1.0;
        const bool third = d.geomx == 2;
        const double sx = dt * d.idx_x[ic], f = dt * inv(d.xv[ic]);
        const double g0 = v.gfx[ic], g1 = v.gfx[ic + 1];
        const double ir = d.geomx != 0 ? inv(rad[2]) : 1.0, irs = d.geomx != 0 ? inv(rad[2] * sz) : 1.0;
        const double cs2 = v.cs2[ic + d.xarr * k];
#pragma unroll 1
        for (int j = j0; j < j1; j += S3_ROWS, ++n) {
            if (!warp_wait(&bar[n & 1], (uint32_t)((n >> 1) & 1), sc)) {
                if (lane == 0 && j + S3_ROWS < j1) mbar_wait(&bar[(n + 1) & 1], (uint32_t)(((n + 1) >> 1) & 1), sc);
                return;
            }
            const double* row = buf + (n & 1) * S3_STAGE + 5 * (lane + 2);
#pragma unroll 1
            for (int jj = j; jj < min(j + S3_ROWS, j1); ++jj, row += 5 * RX_TILE_CELLS) {
                const Cell C0{row[0], row[1], row[2], row[3], row[4]};
                const double cs0 = sound_speed(gam, C0.r, C0.p);
                const double flat = flatten(C0.p, row[-9], row[-4], row[6], row[11], row[-3], C0.u, row[7]);
                auto field = [&](int m) { return recon(w, row[m - 10], row[m - 5], row[m], row[m + 5], row[m + 10], flat); };
                auto momentum = [&](int m, double g) {
                    return recon(w, row[m - 10] * (rad[0] * g), row[m - 5] * (rad[1] * g), row[m] * (rad[2] * g),
                                 row[m + 5] * (rad[3] * g), row[m + 10] * (rad[4] * g), flat);
                };
                const Par R = field(0), P = field(1), U = field(2), A = momentum(3, sz);
                const Par Z = third ? momentum(4, 1.0) : field(4);
                const Half eL = state_at_left_edge(gam, sx, cs0, C0.r, C0.p, C0.u, R, P, U, A, Z);
                const Half eR = state_at_right_edge(gam, sx, cs0, C0.r, C0.p, C0.u, R, P, U, A, Z);
                const Half L{up1(eR.r), up1(eR.p), up1(eR.u), up1(eR.v), up1(eR.w)};
                const Flux F = hllc(d.eos, d.ie, gam, L, eL);
                const Flux G{down1(F.r), down1(F.p), down1(F.u), down1(F.v), down1(F.w), down1(F.pres), down1(F.uprs)};
                Cell D = increments(d, F, g0, G, g1);
                D.r *= f; D.p *= f; D.u *= f; D.v *= f * irs; D.w *= f;
                if (third) D.w *= ir;
                if (output) {
                    const Cell Q = update_cell(d.eos, d.ie, gam, cs2, C0, D, &sc->floor_hits);
                    if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    emit_y(v, out, i, jj, k, Q);
                }
            }
            __syncwarp();  // the copy's reads are done
            if (lane == 0 && j + 2 * S3_ROWS < j1) issue(j + 2 * S3_ROWS, n + 2);
        }
    }
}

// Azimuthal (DIR 1, sweeps.cu:361-433) and polar (DIR 2, :458-554) sweeps: a lane marches
// along its column with five cells in registers and the next in flight, like the 2D
// azimuthal sweep.  Lines of a plane k (DIR 1) or of a row j (DIR 2).  128x256x72, us a
// sweep, tiles -> runs: radial 250 -> 143, azimuthal 249 -> 133, polar 363 -> 144; FP64 issue
// and latency bound all three.  At 2 / 3 / 4 CTAs per SM azimuthal 150 / 133 / 164, polar
// 165 / 144 / 167.
template <int DIR>
__global__ void __launch_bounds__(S3_THREADS, 3)
    k3_march(const Cell* __restrict__ in, const View3 v, Cell* __restrict__ out, int ncol, int len, int nchunk,
             int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const DiskView& d = v.d;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt, gam = d.gam;
    const int res = DIR == 1 ? d.yres : v.zres;
    const bool sph = DIR == 1 ? d.geomy == 4 : v.geomz == 5;
    const double* wtab = DIR == 1 ? d.wy : v.wz;
    const double* idx = DIR == 1 ? d.idx_y : v.idx_z;
    const double* vol = DIR == 1 ? d.yv : v.zv;
    const size_t pitch = 5 * (DIR == 1 ? (size_t)d.xarr : (size_t)d.xarr * d.yarr);
    for (int item = blockIdx.x * S3_WARPS + warp; item < nitems; item += gridDim.x * S3_WARPS) {
        const int i = NPAD + 32 * (item % ncol) + lane, rest = item / ncol;
        const int s0 = NPAD + len * (rest % nchunk), s1 = min(s0 + len, NPAD + res);
        const int line = NPAD + rest / nchunk;  // k (DIR 1) or j (DIR 2)
        const bool active = i < NPAD + d.xres;
        const int ic = min(i, NPAD + d.xres - 1);
        // DIR 1 rad_cyl (sweeps.cu:380-386), DIR 2 rad (:486-489)
        const double rad = sph ? (DIR == 1 ? d.radx[ic] * v.sinz[line] : d.radx[ic]) : 1.0;
        const double irad = sph ? inv(rad) : 1.0;
        const double v0 = DIR == 1 && sph ? rad * d.frame_omega : 0.0;  // the frame's rotation (:388-396)
        const double sdt = dt * irad;  // set_state receives dt/rad (riemann.cu:111)
        const double* next = reinterpret_cast<const double*>(
            in + (DIR == 1 ? at3(v, ic, s0 - NPAD, line) : at3(v, ic, line, s0 - NPAD)));
        double q[5][5], nx[5];
#pragma unroll
        for (int m = 0; m < 5; ++m, next += pitch)
#pragma unroll
            for (int c = 0; c < 5; ++c) q[m][c] = next[c];
        Half pr{};
        Flux pf{};
#pragma unroll 1
        for (int t = s0 - 1; t <= s1; ++t, next += pitch) {
            if (t < s1) {
#pragma unroll
                for (int c = 0; c < 5; ++c) nx[c] = next[c];
            }
            const double* w = wtab + 6 * t;
            // sweep order: DIR 1 v_phi, v_theta, v_r; DIR 2 v_theta, v_r, r sin(theta) v_phi
            constexpr int cu = DIR == 1 ? 3 : 4, ca = DIR == 1 ? 4 : 2, cz = DIR == 1 ? 2 : 3;
            double u[5], z[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                u[m] = DIR == 1 ? q[m][cu] - v0 : q[m][cu];
                z[m] = q[m][cz];
                if (DIR == 2 && sph) z[m] *= rad * v.sinz[t - 2 + m];
            }
            const double cs0 = sound_speed(gam, q[2][0], q[2][1]);
            const double flat = flatten(q[2][1], q[0][1], q[1][1], q[3][1], q[4][1], u[1], u[2], u[3]);
            const double sx = sdt * idx[t];
            auto field = [&](int m) { return recon(w, q[0][m], q[1][m], q[2][m], q[3][m], q[4][m], flat); };
            const Par R = field(0), P = field(1), A = field(ca);
            const Par U = recon(w, u[0], u[1], u[2], u[3], u[4], flat);
            const Par Z = recon(w, z[0], z[1], z[2], z[3], z[4], flat);
            const Half eL = state_at_left_edge(gam, sx, cs0, q[2][0], q[2][1], u[2], R, P, U, A, Z);
            const Half eR = state_at_right_edge(gam, sx, cs0, q[2][0], q[2][1], u[2], R, P, U, A, Z);
            Flux F{};
            if (t >= s0) F = hllc(d.eos, d.ie, gam, pr, eL);
            if (t > s0) {  // the cell below has both its fluxes
                const int s = t - 1;
                const double g0 = DIR == 1 ? 1.0 : v.gfz[s], g1 = DIR == 1 ? 1.0 : v.gfz[s + 1];
                Cell D = increments(d, pf, g0, F, g1);
                const double f = sdt * inv(vol[s]);
                D.r *= f; D.p *= f; D.u *= f; D.v *= f; D.w *= f;
                const Cell C0{q[1][0], q[1][1], q[1][2], q[1][3], q[1][4]};
                if (DIR == 1) {  // sweeps.cu:403-425 (orb_rot 0)
                    D = Cell{D.r, D.p, D.w, D.u + v0 * D.r, D.v};
                } else {  // sweeps.cu:507-532
                    double Dz = D.w;
                    if (sph) Dz *= inv(rad * v.sinz[s]);
                    D = Cell{D.r, D.p, D.v, Dz, D.u};
                }
                if (active) {
                    const int k = DIR == 1 ? line : s;
                    const Cell Q = update_cell(d.eos, d.ie, gam, v.cs2[i + d.xarr * k], C0, D, &sc->floor_hits);
                    if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    if (DIR == 1) emit_z(v, out, i, s, line, Q);
                    else put3(out, v, i, line, s, Q);
                }
            }
            pr = eR;
            pf = F;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                q[0][c] = q[1][c];
                q[1][c] = q[2][c];
                q[2][c] = q[3][c];
                q[3][c] = q[4][c];
                q[4][c] = nx[c];
            }
        }
    }
}

// ================================================================= kicks
// Gravity of the star and the planet and the fictitious forces in spherical
// coordinates (get_gx/gy/gz, star_planet_grav and get_fx/fy/fz of
// src/solver/force/forces.cu:14-39, 110-327, twobd_flag 0; cartesian: none).
struct Grav3 {
    double gx, gy, gz;
};
// the planet's factors of a pass
struct Planet3 {
    double m, x, ix2, irs, irs3;
};
__device__ __forceinline__ Planet3 planet3(const pg_body& p) {
    const double irs = 1.0 / p.rs;
    return Planet3{p.m, p.x, 1.0 / p.x / p.x, irs, irs * irs * irs};
}
__device__ __forceinline__ Grav3 gravity3(const View3& v, int j, int k, double rad, double irad, double pol,
                                          const Planet3& pl, int which) {
    const DiskView& d = v.d;
    Grav3 g{0.0, 0.0, 0.0};
    if (d.geomx != 2) return g;
    g.gx = -irad * irad;
    if (d.nplanet > 0) {
        const double sinfac = d.trig[4 * j + 2 * which], cosfac = d.trig[4 * j + 2 * which + 1];
        const double sinpol = v.sinpol[k], cospol = v.cospol[k];
        const double plm = pl.m, plx = pl.x;
        const double R2 = rad * rad + plx * plx - 2.0 * plx * rad * cosfac * sinpol;
        const double ir = rsq(R2);
        // max(4 - 3 Rp / rs, 1) / max(rs^3, Rp^3)
        const double rs_fac = fmax(4.0 - 3.0 * (R2 * ir) * pl.irs, 1.0) * fmin(pl.irs3, ir * ir * ir);
        g.gx += -plm * (rad - plx * cosfac * sinpol) * rs_fac - plm * sinpol * cosfac * pl.ix2;
        g.gy += -plm * plx * sinfac * rs_fac + plm * sinpol * sinfac * pl.ix2;
        g.gz += plm * plx * cosfac * cospol * rs_fac - plm * cospol * cosfac * inv(sinpol) * pl.ix2;
    }
    if (pol < v.zmin) g.gz *= -1.0;
    return g;
}
__device__ __forceinline__ void fict3(const View3& v, double irad, double itan, double pol, const Cell& T, double& fx,
                                      double& fy, double& fz) {
    fx = 0.0;
    fy = 0.0;
    fz = 0.0;
    if (v.d.geomx == 2) {
        const double c = T.v * T.v * irad;
        fx = c + T.w * T.w * irad;
        fz = c * itan;
        if (pol < v.zmin) fz *= -1.0;
    }
}

// CFL signal rate of one cell (src/timestep/timestep.cu:46-88, ndim 3, orb_rot 0).
__device__ __forceinline__ double rate3(const View3& v, const Cell& c, int i, int j, int k) {
    const DiskView& d = v.d;
    double rad = 1.0, rad_cyl = 1.0;
    if (d.geomy == 4) {
        rad = d.radx[i];
        rad_cyl = rad * v.sinz[k];
    }
    const double cs = sound_speed(d.gam, c.r, c.p);
    double spd = fabs(c.u) + cs;
    double tmp = fmax(spd * d.idx_x[i], 0.0);
    spd = fabs(c.v - rad_cyl * d.frame_omega - 0.0) + cs;
    tmp = fmax(spd * d.idx_y[j] * inv(rad_cyl), tmp);
    spd = fabs(c.w) + cs;
    tmp = fmax(spd * v.idx_z[k] * inv(rad), tmp);
    return tmp;
}

// PASS 1: first half-kick with the bodies of the previous step; PASS 2: the
// predictor / corrector half-kick with the bodies at t + dt, then wave damping
// and the signal rate of the result.  A warp takes rows (j, k) and its lanes the cells of
// a row: the row's factors are found once per row, not divided out of a cell's index.
template <int PASS>
__global__ void __launch_bounds__(K3_THREADS, 4) k3_kick(const View3 v, const Cell* __restrict__ in, Cell* __restrict__ out) {
    const DiskView& d = v.d;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt, hdt = 0.5 * dt;
    const Planet3 pl = planet3(PASS == 1 ? sc->planet_cur : sc->planet_next);
    const int rows = d.yres * v.zres, lane = threadIdx.x & 31;
    const bool sph = d.geomx == 2;
    double vmax = 0.0;
    for (int row = (blockIdx.x * K3_THREADS + threadIdx.x) >> 5; row < rows; row += gridDim.x * (K3_THREADS / 32)) {
        const int j = NPAD + row % d.yres, k = NPAD + row / d.yres;
        const double pol = v.zc[k], itan = sph ? inv(v.tanz[k]) : 0.0;
        for (int i = NPAD + lane; i < NPAD + d.xres; i += 32) {
            const Cell C = get3(in, v, i, j, k);
            const double rad = d.radx[i], irad = sph ? inv(rad) : 0.0;
            const Grav3 g = gravity3(v, j, k, rad, irad, pol, pl, PASS - 1);
            double fx, fy, fz;
            fict3(v, irad, itan, pol, C, fx, fy, fz);
            if (PASS == 2) {  // the predictor over mdt = dt/2 (sweeps.cu:658-675)
                Cell T = C;
                T.u = C.u + fx * hdt + g.gx * hdt;
                T.v = C.v + fy * hdt + g.gy * hdt;
                T.w = C.w + fz * hdt + g.gz * hdt;
                fict3(v, irad, itan, pol, T, fx, fy, fz);
            }
            Cell Q;
            Q.u = C.u + fx * hdt + g.gx * hdt;
            Q.v = C.v + fy * hdt + g.gy * hdt;
            Q.w = C.w + fz * hdt + g.gz * hdt;
            Q.r = C.r;
            Q.p = C.p;
            if (PASS == 1) {
                emit_x(v, out, i, j, k, Q);
                continue;
            }
            if (d.kill) {  // relax towards init_C (killwave.cu:48-100)
                const double* kt = d.killx + 4 * i;
                const double* I = v.initc + 5 * ((size_t)i + (size_t)d.xarr * k);
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const double tau = kt[2 * side + 1];
                    if (tau > 0.0) {
                        double f = kt[2 * side];
                        f *= dt / tau;
                        Q.r += f * (I[0] - Q.r);
                        Q.p += f * (I[1] - Q.p);
                        Q.u += f * (I[2] - Q.u);
                        Q.v += f * (I[3] - Q.v);
                        Q.w += f * (I[4] - Q.w);
                    }
                }
            }
            if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
            put3(out, v, i, j, k, Q);
            vmax = fmax(vmax, rate3(v, Q, i, j, k));
        }
    }
    if (PASS == 2) block_max_to<K3_THREADS>(&sc->vmax_bits, vmax);
}

__global__ void __launch_bounds__(K3_THREADS) k3_cfl(const View3 v, const Cell* __restrict__ in) {
    const DiskView& d = v.d;
    const long long n = (long long)d.xres * d.yres * v.zres;
    double vmax = 0.0;
    for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % d.xres);
        const long long rest = m / d.xres;
        const int j = NPAD + (int)(rest % d.yres);
        const int k = NPAD + (int)(rest / d.yres);
        vmax = fmax(vmax, rate3(v, get3(in, v, i, j, k), i, j, k));
    }
    block_max_to<K3_THREADS>(&d.sc->vmax_bits, vmax);
}

// ======================================================== state transfer
// Both buffers: interior from the planes (x fastest, then y, then z), every
// ghost cell init_C (fill_grid, src/init/init.cu:502-519, as the device
// evaluates it for the bound-0 ghosts of boundary.cu:30-33, 276-318).
__global__ void k3_fill(const View3 v, Cell* a, Cell* b, const double* r, const double* p, const double* u,
                        const double* vv, const double* w) {
    const DiskView& d = v.d;
    const long long n = (long long)d.xarr * d.yarr * v.zarr;
    for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(m % d.xarr);
        const long long rest = m / d.xarr;
        const int j = (int)(rest % d.yarr);
        const int k = (int)(rest / d.yarr);
        Cell c;
        if (i >= NPAD && i < NPAD + d.xres && j >= NPAD && j < NPAD + d.yres && k >= NPAD && k < NPAD + v.zres) {
            const size_t q = (size_t)(i - NPAD) + (size_t)d.xres * ((size_t)(j - NPAD) + (size_t)d.yres * (k - NPAD));
            c = Cell{r[q], p[q], u[q], vv[q], w[q]};
        } else {
            const double* I = v.initc + 5 * ((size_t)i + (size_t)d.xarr * k);
            c = Cell{I[0], I[1], I[2], I[3], I[4]};
        }
        put3(a, v, i, j, k, c);
        put3(b, v, i, j, k, c);
    }
}

__global__ void k3_extract(const View3 v, const Cell* in, double* r, double* p, double* u, double* vv, double* w) {
    const DiskView& d = v.d;
    const long long n = (long long)d.xres * d.yres * v.zres;
    for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % d.xres);
        const long long rest = m / d.xres;
        const int j = NPAD + (int)(rest % d.yres);
        const int k = NPAD + (int)(rest / d.yres);
        const Cell c = get3(in, v, i, j, k);
        r[m] = c.r;
        p[m] = c.p;
        u[m] = c.u;
        vv[m] = c.v;
        w[m] = c.w;
    }
}

// The bound-0 radial and polar ghosts of a caller's buffer: init_C as the device
// evaluates it (boundary.cu:30-33, 56-59, 293-294, 315-316); never rewritten.
__global__ void k3_analytic_ghosts(const View3 v, Cell* buf) {
    const DiskView& d = v.d;
    const long long n = (long long)d.xarr * d.yarr * v.zarr;
    for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(m % d.xarr);
        const long long rest = m / d.xarr;
        const int j = (int)(rest % d.yarr);
        const int k = (int)(rest / d.yarr);
        const bool gx = (i < NPAD && d.bound_lft == 0) || (i >= NPAD + d.xres && d.bound_rgh == 0);
        const bool gz = (k < NPAD && v.bound_bom == 0) || (k >= NPAD + v.zres && v.bound_top == 0);
        if (!gx && !gz) continue;
        const double* I = v.initc + 5 * ((size_t)i + (size_t)d.xarr * k);
        put3(buf, v, i, j, k, Cell{I[0], I[1], I[2], I[3], I[4]});
    }
}

// ================================================================ tables
// Evaluated on the device with its own sin / cos / tan / pow / exp / sqrt, as
// the reference evaluates them in its kernels.
struct Tab3Args {
    double sc_h, planet_radius, p_alpha, p_beta, xmin, xmax, kill_width, kill_width_out;
    int geomx, init_flag, kill;
};
__device__ inline double t3_cs2(const Tab3Args& a, double x, double z) {  // init.cu:7-17
    const double coeff = a.sc_h * a.sc_h * (1.0 / a.planet_radius);
    if (a.geomx == 0) return coeff;
    return coeff * pow(x * sin(z) / a.planet_radius, -a.p_beta);
}
__device__ inline double t3_h(const Tab3Args& a, double x, double z) {  // init.cu:20-29
    if (a.geomx == 0) return a.sc_h;
    return sqrt(t3_cs2(a, x, z) * pow(x * sin(z), 3));
}
__device__ inline double t3_rho(const Tab3Args& a, double x, double z) {  // init.cu:53-71, 90-91 (init_flag 3)
    const double cs2 = t3_cs2(a, x, z);
    const double r = x * sin(z);
    return pow(x * sin(z) / a.planet_radius, -a.p_alpha) * exp((1.0 / x - 1.0 / r) / cs2);
}
__device__ inline double t3_p(const Tab3Args& a, double x, double z) { return t3_cs2(a, x, z) * t3_rho(a, x, z); }

__global__ void k3_tables(const View3 v, Tab3Args a, double* zc, double* sinz, double* sinpol, double* cospol,
                          double* tanz, double* idx_z, double* gfx, double* gfz, double* radx, double* idx_x,
                          double* killx, double* ycj, double* idx_y, double* cs2, double* initc) {
    const DiskView& d = v.d;
    const long long nxz = (long long)d.xarr * v.zarr;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid <= v.zarr) gfz[tid] = (v.geomz == 5) ? sin(v.za[tid]) : 1.0;
    if (tid <= d.xarr) {
        const double x = d.xa[tid];
        gfx[tid] = (d.geomx == 2) ? x * x : (d.geomx == 1 ? x : 1.0);
    }
    if (tid < v.zarr) {
        const int k = (int)tid;
        const double z = 0.5 * (v.za[k + 1] + v.za[k]);
        zc[k] = z;
        sinz[k] = sin(z);
        sincos(z, &sinpol[k], &cospol[k]);
        tanz[k] = tan(z);
        idx_z[k] = 1.0 / (v.za[k + 1] - v.za[k]);
    }
    if (tid < d.yarr) {
        const int j = (int)tid;
        ycj[j] = 0.5 * (d.ya[j + 1] + d.ya[j]);
        idx_y[j] = 1.0 / (d.ya[j + 1] - d.ya[j]);
    }
    if (tid < d.xarr) {
        const int i = (int)tid;
        const double x = 0.5 * (d.xa[i + 1] + d.xa[i]);
        radx[i] = x;
        idx_x[i] = 1.0 / (d.xa[i + 1] - d.xa[i]);
        // killwave.cu:24-34 with the ndim-3 scale height at the midplane
        const double d_in = t3_h(a, a.xmin, HPI) * a.kill_width;
        const double d_out = t3_h(a, a.xmax, HPI) * a.kill_width_out;
        const double inner = a.xmin + d_in, outer = a.xmax - d_out;
        double* kt = killx + 4 * i;
        kt[0] = kt[1] = kt[2] = kt[3] = 0.0;
        if (a.kill && i >= NPAD && i < NPAD + d.xres) {
            if (x < inner) {
                kt[1] = (a.geomx == 0) ? 1.0 : pow(x, 1.5);
                double f = __sinf(HPI * ((inner - x) / d_in));  // get_ramping_fac (killwave.cu:8-14)
                kt[0] = f * f;
            }
            if (x > outer) {
                kt[3] = (a.geomx == 0) ? 1.0 : pow(x, 1.5);
                double f = __sinf(HPI * ((x - outer) / d_out));
                kt[2] = f * f;
            }
        }
    }
    if (tid < nxz) {
        const int i = (int)(tid % d.xarr), k = (int)(tid / d.xarr);
        const double x = 0.5 * (d.xa[i + 1] + d.xa[i]);
        const double z = 0.5 * (v.za[k + 1] + v.za[k]);
        cs2[tid] = t3_cs2(a, x, z);
        double* q = initc + 5 * tid;
        if (a.init_flag == 3) {  // init_C of init_flag 3 (init.cu:90-91, 157-158, 196-198, 269-274, 322-323)
            const double r = x * sin(z);
            q[0] = t3_rho(a, x, z);
            q[1] = t3_p(a, x, z);
            q[2] = -1.5 * 0.0 / r;
            const double rho = t3_rho(a, x, z);
            const double dr = 1.1514178e-7;
            const double dP_dr = (t3_p(a, x + dr, z) - t3_p(a, x - dr, z)) / (2.0 * dr);
            q[3] = sqrt(1.0 / x + (x / rho) * dP_dr);
            q[4] = 0.0;
        } else {
            q[0] = 1.0;
            q[1] = 1.0;
            q[2] = q[3] = q[4] = 0.0;
        }
    }
}

// ================================================================ engine
struct Engine3 {
    pg_params P{};
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    View3 v{};
    Cell* buf[2] = {nullptr, nullptr};
    bool own_buffers = true;  // false: the caller's Grid buffers (pg_grid_*)
    CUtensorMap maps[2];  // per buffer: the radial sweep's box
    const void* map_base[2] = {nullptr, nullptr};
    std::vector<const void*> ghosted;  // caller buffers whose bound-0 ghosts hold the device init_C
    std::vector<double> hxa, hya, hza; // host faces of each axis (ghosts included), for snapshots
    double* tables = nullptr;
    double* stage = nullptr;
    size_t stage_n = 0;
    HostCopy readback;  // staging of large reads of the state
    Scalars* sc = nullptr;
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    int cur = 0;
    int cur_base = 0;
    long long steps_base = 0;
    bool pending = false;
    bool fresh = true;
    // of each sweep: CTAs, warps across the radius, rows of a run, runs per line, runs
    bool dense = false;  // the radial sweep's instance: 4 CTAs per SM, else 3
    unsigned grid_sweep[3] = {0, 0, 0};
    int across[3], len[3], chunks[3], items[3];
    unsigned grid_kick = 0;
};

static pg_status fail3(pg_status s, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    set_last_error(buf);
    return s;
}

#define PG3_CUDA(call)                                                                                     \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess)                                                                             \
            return fail3(PG_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
    } while (0)

static pg_status check3(const pg_params* P) {
    if (!P) return fail3(PG_ERR_ARG, "null params");
    if (P->ndim != 3) return fail3(PG_ERR_CONFIG, "the 3D form needs ndim 3");
    const bool sph = P->geomx == 2 && P->geomy == 4 && P->geomz == 5;
    const bool cart = P->geomx == 0 && P->geomy == 0 && P->geomz == 0;
    if (!sph && !cart) return fail3(PG_ERR_CONFIG, "3D geometries: spherical (2, 4, 5) or cartesian (0, 0, 0)");
    if (P->xres < 2 * NPAD || P->yres < 2 * NPAD || P->zres < 2 * NPAD || P->xres % 2)
        return fail3(PG_ERR_CONFIG, "3D resolutions: at least 6 cells per axis, even xres");
    if (P->gridx < 0 || P->gridx > 4 || P->gridy < 0 || P->gridy > 4 || P->gridz < 0 || P->gridz > 4)
        return fail3(PG_ERR_CONFIG, "grids must be 0 to 4");
    if (P->eos_flag != 0 && P->eos_flag != 2) return fail3(PG_ERR_CONFIG, "EOS_flag must be 0 or 2");
    if (P->bound_lft < 0 || P->bound_lft > 2 || P->bound_rgh < 0 || P->bound_rgh > 2)
        return fail3(PG_ERR_CONFIG, "radial boundaries must be 0, 1 or 2");
    if (P->bound_bom < 0 || P->bound_bom > 3 || P->bound_top < 0 || P->bound_top > 3)
        return fail3(PG_ERR_CONFIG, "polar boundaries must be 0 to 3");
    if (P->visc_flag || P->orbadv_flag || P->dust_flag || P->cool_flag || P->twobd_flag)
        return fail3(PG_ERR_CONFIG, "3D runs without viscosity, orbital advection, dust, cooling and two-body frame");
    if (P->n_planet < 0 || P->n_planet > 1) return fail3(PG_ERR_CONFIG, "n_planet must be 0 or 1");
    const bool analytic = P->kill_flag || P->bound_lft == 0 || P->bound_rgh == 0 || P->bound_bom == 0 ||
                          P->bound_top == 0;
    if (analytic && (!sph || P->init_flag != 3))
        return fail3(PG_ERR_CONFIG, "analytic ghosts or wave damping need the spherical disk (init_flag 3)");
    return PG_OK;
}

static unsigned occupancy_grid(const void* kernel, int threads, size_t smem, long long work) {
    int dev = 0, nsm = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
    long long g = (long long)nsm * (per > 0 ? per : 1);
    if (g > work) g = work;
    return (unsigned)(g > 0 ? g : 1);
}

static pg_status make_maps(Engine3& E, int b) {
    const DiskView& d = E.v.d;
    const uint64_t d0 = 5ull * d.xarr, d1 = d.yarr, d2 = E.v.zarr;
    pg_status s;
    if ((s = make_map3_f64(&E.maps[b], E.buf[b], d0, d1, d2, 5 * RX_TILE_CELLS, S3_ROWS, 1)) != PG_OK) return s;
    E.map_base[b] = E.buf[b];
    return PG_OK;
}

// one sweep from buffer b to the other
static void enqueue_sweep(Engine3& E, int dir, int b) {
    Cell* out = E.buf[1 - b];
    const int a = E.across[dir], l = E.len[dir], c = E.chunks[dir], n = E.items[dir];
    if (dir == 0) launch_step(E.dense ? k3_sweep_x<4> : k3_sweep_x<3>, E.grid_sweep[0], S3_THREADS, S3_SMEM, E.stream, E.maps[b], E.v, out, a, l, c, n);
    else if (dir == 1) launch_step(k3_march<1>, E.grid_sweep[1], S3_THREADS, 0, E.stream, E.buf[b], E.v, out, a, l, c, n);
    else launch_step(k3_march<2>, E.grid_sweep[2], S3_THREADS, 0, E.stream, E.buf[b], E.v, out, a, l, c, n);
}

// the five passes of one step from buffer c (newest state ends in 1 - c)
static void enqueue_passes(Engine3& E, int c) {
    const View3& v = E.v;
    cudaStream_t s = E.stream;
    Cell* A = E.buf[c];
    Cell* B = E.buf[1 - c];
    launch_step(k3_kick<1>, E.grid_kick, K3_THREADS, 0, s, v, A, B);
    enqueue_sweep(E, 0, 1 - c);
    enqueue_sweep(E, 1, c);
    enqueue_sweep(E, 2, 1 - c);
    launch_step(k3_kick<2>, E.grid_kick, K3_THREADS, 0, s, v, A, B);
}

static pg_status resolve3(Engine3& E) {
    if (!E.pending) return PG_OK;
    long long steps = 0;
    PG3_CUDA(cudaMemcpyAsync(&steps, &E.sc->steps, sizeof(steps), cudaMemcpyDeviceToHost, E.stream));
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    E.cur = (int)((E.cur_base + (steps - E.steps_base)) & 1);
    E.pending = false;
    return PG_OK;
}

static pg_status stage_buffer(Engine3& E, size_t n, double** out) {
    if (E.stage_n < n) {
        if (E.stage) cudaFree(E.stage);
        E.stage = nullptr;
        E.stage_n = 0;
        PG3_CUDA(cudaMalloc(&E.stage, n * sizeof(double)));
        E.stage_n = n;
    }
    *out = E.stage;
    return PG_OK;
}

static void release3(Engine3* E) {
    if (!E) return;
    for (int b = 0; b < 2; ++b) {
        if (E->graph[b]) cudaGraphExecDestroy(E->graph[b]);
        if (E->buf[b] && E->own_buffers) cudaFree(E->buf[b]);
    }
    if (E->tables) cudaFree(E->tables);
    if (E->stage) cudaFree(E->stage);
    if (E->sc) cudaFree(E->sc);
    if (E->own_stream && E->stream) cudaStreamDestroy(E->stream);
    delete E;
}

static pg_status create3(const pg_params* P, int device, cudaStream_t stream, Engine3** out, bool own = true) {
    pg_status s = check3(P);
    if (s != PG_OK) return s;
    PG3_CUDA(cudaSetDevice(device));
    Engine3* E = new Engine3();
    E->P = *P;
    if (E->P.kill_width_out <= 0.0) E->P.kill_width_out = E->P.kill_width;
    E->device = device;
    auto bad = [&](pg_status st) {
        release3(E);
        return st;
    };
    if (stream) {
        E->stream = stream;
    } else {
        if (cudaStreamCreateWithFlags(&E->stream, cudaStreamNonBlocking) != cudaSuccess)
            return bad(fail3(PG_ERR_CUDA, "stream creation failed"));
        E->own_stream = true;
    }
    const pg_params& Q = E->P;
    const int xarr = Q.xres + 2 * NPAD, yarr = Q.yres + 2 * NPAD, zarr = Q.zres + 2 * NPAD;
    std::vector<double> xa(xarr + 1), xv(xarr), ya(yarr + 1), yv(yarr), za(zarr + 1), zv(zarr);
    make_grid(xa.data(), xv.data(), Q.xmin, Q.xmax, Q.xres, NPAD, Q.geomx, Q.gridx, &Q);
    make_grid(ya.data(), yv.data(), Q.ymin, Q.ymax, Q.yres, NPAD, Q.geomy, Q.gridy, &Q);
    make_grid(za.data(), zv.data(), Q.zmin, Q.zmax, Q.zres, NPAD, Q.geomz, Q.gridz, &Q);
    for (double a : xa) if (!std::isfinite(a)) return bad(fail3(PG_ERR_CONFIG, "the radial spacing needs more cells"));
    for (double a : ya) if (!std::isfinite(a)) return bad(fail3(PG_ERR_CONFIG, "the azimuthal spacing needs more cells"));
    for (double a : za) if (!std::isfinite(a)) return bad(fail3(PG_ERR_CONFIG, "the polar spacing needs more cells"));
    E->hxa = xa;
    E->hya = ya;
    E->hza = za;
    // table block: faces and volumes, weights, per-index and (x, z) tables, trig
    const size_t nxz = (size_t)xarr * zarr;
    const size_t ntab = (xarr + 1) + xarr + (yarr + 1) + yarr + (zarr + 1) + zarr   // grid
                        + 6 * (size_t)(xarr + yarr + zarr)                             // slope weights
                        + 6 * (size_t)zarr + (zarr + 1) + (xarr + 1)                   // zc sinz sinpol cospol tanz idx_z gfz gfx
                        + 2 * (size_t)xarr + 4 * (size_t)xarr                          // radx idx_x killx
                        + 2 * (size_t)yarr                                             // ycj idx_y
                        + nxz + 5 * nxz                                                // cs2 initc
                        + 4 * (size_t)yarr + 2;                                        // trig
    if (cudaMalloc(&E->tables, ntab * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&E->sc, sizeof(Scalars)) != cudaSuccess)
        return bad(fail3(PG_ERR_CUDA, "table allocation failed"));
    const size_t ncell = (size_t)xarr * yarr * zarr;
    E->own_buffers = own;
    for (int b = 0; own && b < 2; ++b)
        if (cudaMalloc(&E->buf[b], ncell * sizeof(Cell)) != cudaSuccess)
            return bad(fail3(PG_ERR_CUDA, "state allocation failed (%zu cells)", ncell));
    cudaMemsetAsync(E->sc, 0, sizeof(Scalars), E->stream);
    double* t = E->tables;
    auto take = [&](size_t n) {
        double* p = t;
        t += n;
        return p;
    };
    double* dxa = take(xarr + 1);
    double* dxv = take(xarr);
    double* dya = take(yarr + 1);
    double* dyv = take(yarr);
    double* dza = take(zarr + 1);
    double* dzv = take(zarr);
    double* wx = take(6 * (size_t)xarr);
    double* wy = take(6 * (size_t)yarr);
    double* wz = take(6 * (size_t)zarr);
    double* zc = take(zarr);
    double* sinz = take(zarr);
    double* sinpol = take(zarr);
    double* cospol = take(zarr);
    double* tanz = take(zarr);
    double* idx_z = take(zarr);
    double* gfz = take(zarr + 1);
    double* gfx = take(xarr + 1);
    double* radx = take(xarr);
    double* idx_x = take(xarr);
    double* killx = take(4 * (size_t)xarr);
    double* ycj = take(yarr);
    double* idx_y = take(yarr);
    double* cs2 = take(nxz);
    double* initc = take(5 * nxz);
    double* trig = take(4 * (size_t)yarr + 2);
    cudaMemcpyAsync(dxa, xa.data(), xa.size() * 8, cudaMemcpyHostToDevice, E->stream);
    cudaMemcpyAsync(dxv, xv.data(), xv.size() * 8, cudaMemcpyHostToDevice, E->stream);
    cudaMemcpyAsync(dya, ya.data(), ya.size() * 8, cudaMemcpyHostToDevice, E->stream);
    cudaMemcpyAsync(dyv, yv.data(), yv.size() * 8, cudaMemcpyHostToDevice, E->stream);
    cudaMemcpyAsync(dza, za.data(), za.size() * 8, cudaMemcpyHostToDevice, E->stream);
    cudaMemcpyAsync(dzv, zv.data(), zv.size() * 8, cudaMemcpyHostToDevice, E->stream);
    // 4th-order slope weights of each direction from the reference's own rounded
    // grid moments (evaluated on the device with its expressions)
    std::vector<double> w(6 * (size_t)std::max(xarr, std::max(yarr, zarr)));
    const int geoms[3] = {Q.geomx, Q.geomy, Q.geomz};
    const int ns[3] = {xarr, yarr, zarr};
    const double* faces[3] = {dxa, dya, dza};
    double* wdst[3] = {wx, wy, wz};
    for (int a = 0; a < 3; ++a) {
        s = recon_weights(geoms[a], faces[a], ns[a], w.data(), E->stream);
        if (s != PG_OK) return bad(s);
        cudaMemcpyAsync(wdst[a], w.data(), 6 * (size_t)ns[a] * 8, cudaMemcpyHostToDevice, E->stream);
        if (cudaStreamSynchronize(E->stream) != cudaSuccess) return bad(fail3(PG_ERR_CUDA, "weight upload failed"));
    }
    DiskView& d = E->v.d;
    d.xres = Q.xres;
    d.yres = Q.yres;
    d.xarr = xarr;
    d.yarr = yarr;
    d.ypad = NPAD;
    d.ndim = 3;
    d.geomx = Q.geomx;
    d.geomy = Q.geomy;
    d.eos = Q.eos_flag;
    d.ie = Q.internal_e_flag;
    d.bound_lft = Q.bound_lft;
    d.bound_rgh = Q.bound_rgh;
    d.kill = Q.kill_flag;
    d.nplanet = Q.n_planet;
    d.gam = Q.gam;
    d.cfl = Q.cfl;
    d.frame_omega = Q.frame_omega;
    d.planet_mass = Q.planet_mass;
    d.ramp_time = Q.ramp_time;
    d.xa = dxa;
    d.xv = dxv;
    d.wx = wx;
    d.wy = wy;
    d.ya = dya;
    d.yv = dyv;
    d.radx = radx;
    d.ycj = ycj;
    d.ycraw = ycj;
    d.killx = killx;
    d.idx_x = idx_x;
    d.idx_y = idx_y;
    d.trig = trig;
    d.sc = E->sc;
    View3& v = E->v;
    v.zres = Q.zres;
    v.zarr = zarr;
    v.geomz = Q.geomz;
    v.bound_bom = Q.bound_bom;
    v.bound_top = Q.bound_top;
    v.init3 = Q.init_flag == 3;
    v.zmin = Q.zmin;
    v.za = dza;
    v.zv = dzv;
    v.wz = wz;
    v.idx_z = idx_z;
    v.zc = zc;
    v.sinz = sinz;
    v.sinpol = sinpol;
    v.cospol = cospol;
    v.tanz = tanz;
    v.gfx = gfx;
    v.gfz = gfz;
    v.cs2 = cs2;
    v.initc = initc;
    Tab3Args ta{Q.sc_h, Q.planet_radius, Q.p_alpha, Q.p_beta, Q.xmin, Q.xmax, Q.kill_width, E->P.kill_width_out,
                Q.geomx, Q.init_flag, Q.kill_flag};
    const long long nt = std::max((long long)nxz, (long long)std::max(xarr, std::max(yarr, zarr)) + 1);
    k3_tables<<<(unsigned)((nt + 127) / 128), 128, 0, E->stream>>>(v, ta, zc, sinz, sinpol, cospol, tanz, idx_z, gfx,
                                                                      gfz, radx, idx_x, killx, ycj, idx_y, cs2, initc);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(E->stream) != cudaSuccess)
        return bad(fail3(PG_ERR_CUDA, "table kernel failed"));
    for (int b = 0; own && b < 2; ++b)
        if ((s = make_maps(*E, b)) != PG_OK) return bad(s);
    // The radial sweep at 3 CTAs per SM is 1 to 10 % faster than at 4 with its spills (us:
    // 48x40x36 13.2 / 14.6, 96x192x54 68 / 75, 192x384x108 409 / 429), unless its runs fill
    // their last wave so badly that the other count's finer waves win (128x256x72 166 / 143,
    // 96x96x96 69 / 64): by run_cost, with a wave's time proportional to its warps, those are
    // the grids where 4 looks better by 3.5 % or more (0.957 and 0.962; 120x112x112, 0.948, loses 2.5 %).
    double cost[2];
    for (int k = 0; k < 2; ++k) {
        const void* f = k == 0 ? (const void*)k3_sweep_x<3> : (const void*)k3_sweep_x<4>;
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S3_SMEM);
        cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        const long long fit = S3_WARPS * (long long)occupancy_grid(f, S3_THREADS, S3_SMEM, 1ll << 40);
        const long long lines = (long long)((Q.xres + S3_OUT - 1) / S3_OUT) * Q.zres;
        const int len = run_length(lines, Q.yres, fit, 1.5);
        cost[k] = (double)fit * run_cost(lines * ((Q.yres + len - 1) / len), fit, len + 1.5);
    }
    E->dense = cost[1] < 0.965 * cost[0];
    const void* sweep_x = E->dense ? (const void*)k3_sweep_x<4> : (const void*)k3_sweep_x<3>;
    const int along[3] = {Q.yres, Q.yres, Q.zres};  // rows a run is cut from
    const int lines[3] = {Q.zres, Q.zres, Q.yres};
    for (int a = 0; a < 3; ++a) {
        E->across[a] = (Q.xres + (a == 0 ? S3_OUT : 32) - 1) / (a == 0 ? S3_OUT : 32);
        const void* kernel = a == 0 ? sweep_x : (a == 1 ? (const void*)k3_march<1> : (const void*)k3_march<2>);
        const size_t smem = a == 0 ? S3_SMEM : 0;
        const long long resident = S3_WARPS * (long long)occupancy_grid(kernel, S3_THREADS, smem, 1ll << 40);
        E->len[a] = run_length((long long)E->across[a] * lines[a], along[a], resident, a == 0 ? 1.5 : 3.5);
        E->chunks[a] = (along[a] + E->len[a] - 1) / E->len[a];
        E->items[a] = E->across[a] * E->chunks[a] * lines[a];
        E->grid_sweep[a] = occupancy_grid(kernel, S3_THREADS, smem, (E->items[a] + S3_WARPS - 1) / S3_WARPS);
    }
    E->grid_kick = occupancy_grid((const void*)k3_kick<2>, K3_THREADS, 0,
                                  ((long long)Q.yres * Q.zres + K3_THREADS / 32 - 1) / (K3_THREADS / 32));
    *out = E;
    return PG_OK;
}

// ------------------------------------------------------- drop-in (Grid)
// pg_grid_* with ndim 3: the engine's tables for the caller's grid, keyed by
// its device xa; the state lives in the caller's C and T.
static std::map<const double*, Engine3*> g_grids3;

pg_status check_params3(const pg_params* P) { return check3(P); }

static pg_status grid3_engine(const pg_params& P, pg_grid* dev, Engine3** out) {
    if (!dev) return fail3(PG_ERR_ARG, "null grid");
    if (dev->xres != P.xres || dev->yres != P.yres || dev->zres != P.zres)
        return fail3(PG_ERR_CONFIG, "grid dimensions differ from the configured parameters");
    if (dev->xbgn != 0) return fail3(PG_ERR_CONFIG, "radial domain decomposition is not supported");
    auto it = g_grids3.find(dev->xa);
    if (it != g_grids3.end()) {
        *out = it->second;
        return PG_OK;
    }
    int device = 0;
    PG3_CUDA(cudaGetDevice(&device));
    Engine3* E = nullptr;
    pg_status s = create3(&P, device, (cudaStream_t)dev->stream, &E, false);
    if (s != PG_OK) return s;
    g_grids3[dev->xa] = E;
    *out = E;
    return PG_OK;
}

pg_status grid3_init_orbadv(const pg_params& P, pg_grid* dev) {
    Engine3* E = nullptr;
    pg_status s = grid3_engine(P, dev, &E);
    if (s != PG_OK) return s;
    // init_OrbAdv (src/orbit/orbit.cu:51-72) without OrbAdv_flag: orb_rot 0, orb_shf 0
    const size_t nxz = (size_t)dev->xarr * dev->zarr;
    if (dev->orb_rot) PG3_CUDA(cudaMemsetAsync(dev->orb_rot, 0, sizeof(double) * nxz, E->stream));
    if (dev->orb_shf) PG3_CUDA(cudaMemsetAsync(dev->orb_shf, 0, sizeof(int) * nxz, E->stream));
    PG3_CUDA(cudaStreamSynchronize(E->stream));
    return PG_OK;
}

pg_status grid3_global_dt(const pg_params& P, pg_grid* dev, double dt_prev, double* dt_out) {
    Engine3* E = nullptr;
    pg_status s = grid3_engine(P, dev, &E);
    if (s != PG_OK) return s;
    PG3_CUDA(cudaMemsetAsync(&E->sc->vmax_bits, 0, sizeof(unsigned long long), E->stream));
    k3_cfl<<<E->grid_kick, K3_THREADS, 0, E->stream>>>(E->v, reinterpret_cast<const Cell*>(dev->C));
    PG3_CUDA(cudaGetLastError());
    unsigned long long bits = 0;
    PG3_CUDA(cudaMemcpyAsync(&bits, &E->sc->vmax_bits, sizeof(bits), cudaMemcpyDeviceToHost, E->stream));
    PG3_CUDA(cudaStreamSynchronize(E->stream));
    double vmax;
    std::memcpy(&vmax, &bits, sizeof vmax);
    const double dt = E->P.cfl / vmax;  // get_dt_lv2 (timestep.cu:108)
    double tmp = dt_prev * 1.1;         // timestep.cu:133-139
    if (dt < tmp) tmp = dt;
    *dt_out = tmp;
    return PG_OK;
}

pg_status grid3_solve(const pg_params& P, pg_grid* dev, double time, double dt) {
    Engine3* E = nullptr;
    pg_status s = grid3_engine(P, dev, &E);
    if (s != PG_OK) return s;
    E->buf[0] = reinterpret_cast<Cell*>(dev->C);
    E->buf[1] = reinterpret_cast<Cell*>(dev->T);
    for (int b = 0; b < 2; ++b) {
        if (E->map_base[b] != E->buf[b] && (s = make_maps(*E, b)) != PG_OK) return s;
        if (std::find(E->ghosted.begin(), E->ghosted.end(), E->buf[b]) == E->ghosted.end()) {
            k3_analytic_ghosts<<<1184, 256, 0, E->stream>>>(E->v, E->buf[b]);
            E->ghosted.push_back(E->buf[b]);
        }
    }
    if (E->v.d.nplanet > 0 && dev->planets) k_grid_planet_in<<<1, 1, 0, E->stream>>>(E->sc, dev->planets, 0);
    launch_set_time(E->v.d, time, dt, E->stream);
    enqueue_passes(*E, 0);
    if (E->v.d.nplanet > 0 && dev->planets) k_grid_planet_out<<<1, 1, 0, E->stream>>>(E->sc, dev->planets, 0);
    PG3_CUDA(cudaGetLastError());
    // the newest state is in T: swap like the reference (src/solver/sweeps.cu:353-355, 550-552)
    pg_cell* t = dev->C;
    dev->C = dev->T;
    dev->T = t;
    return PG_OK;
}

void grid3_release() {
    for (auto& kv : g_grids3) release3(kv.second);
    g_grids3.clear();
}

// Device-clocked steps from here on run towards end_time (main.cu:322-339).
static pg_status begin_run(Engine3& E, double end_time) {
    PG3_CUDA(cudaSetDevice(E.device));
    pg_status s = resolve3(E);
    if (s != PG_OK) return s;
    Scalars h{};
    PG3_CUDA(cudaMemcpyAsync(&h, E.sc, sizeof(Scalars), cudaMemcpyDeviceToHost, E.stream));
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    // main.cu:144 + 322: the first cap on dt is end_time - t after a (re)start;
    // a run that stopped on a clip at its end_time continues like main.cu after a
    // dump (main.cu:333-338, 425)
    if (E.fresh) h.dt_prev = end_time - h.t;
    else if (h.dt_hold > 0.0) h.dt_prev = h.dt_hold;
    h.dt_hold = 0.0;
    h.end_time = end_time;
    h.done = 0;
    h.pad_ = 0;
    PG3_CUDA(cudaMemcpyAsync(E.sc, &h, sizeof(Scalars), cudaMemcpyHostToDevice, E.stream));
    E.fresh = false;
    E.cur_base = E.cur;
    E.steps_base = h.steps;
    E.pending = true;
    return PG_OK;
}

}  // namespace pg

using namespace pg;

struct pg_disk3 {
    Engine3* E;
};

extern "C" {

pg_status pg_make_axis(const pg_params* P, int axis, double* a, double* v) {
    if (!P || !a || !v || axis < 0 || axis > 2) return fail3(PG_ERR_ARG, "bad argument");
    const int pad = (axis == 0 || (axis == 1 && P->ndim > 1) || (axis == 2 && P->ndim > 2)) ? NPAD : 0;
    if (axis == 0) make_grid(a, v, P->xmin, P->xmax, P->xres, pad, P->geomx, P->gridx, P);
    else if (axis == 1) make_grid(a, v, P->ymin, P->ymax, P->yres, pad, P->geomy, P->gridy, P);
    else make_grid(a, v, P->zmin, P->zmax, P->zres, pad, P->geomz, P->gridz, P);
    return PG_OK;
}

pg_status pg_disk3_create(const pg_params* P, int device, void* stream, pg_disk3** out) {
    if (!out) return fail3(PG_ERR_ARG, "null argument");
    Engine3* E = nullptr;
    pg_status s = create3(P, device, (cudaStream_t)stream, &E);
    if (s != PG_OK) return s;
    *out = new pg_disk3{E};
    return PG_OK;
}

pg_status pg_disk3_destroy(pg_disk3* dk) {
    if (!dk) return PG_OK;
    cudaSetDevice(dk->E->device);
    cudaStreamSynchronize(dk->E->stream);
    release3(dk->E);
    delete dk;
    return PG_OK;
}

pg_status pg_disk3_set_state(pg_disk3* dk, double t, const double* r, const double* p, const double* u,
                             const double* v, const double* w) {
    if (!dk || !r || !p || !u || !v || !w) return fail3(PG_ERR_ARG, "null argument");
    Engine3& E = *dk->E;
    PG3_CUDA(cudaSetDevice(E.device));
    const size_t n = (size_t)E.P.xres * E.P.yres * E.P.zres;
    double* st = nullptr;
    pg_status s = stage_buffer(E, 5 * n, &st);
    if (s != PG_OK) return s;
    const double* src[5] = {r, p, u, v, w};
    for (int f = 0; f < 5; ++f)
        PG3_CUDA(cudaMemcpyAsync(st + f * n, src[f], n * sizeof(double), cudaMemcpyHostToDevice, E.stream));
    k3_fill<<<1184, 256, 0, E.stream>>>(E.v, E.buf[0], E.buf[1], st, st + n, st + 2 * n, st + 3 * n, st + 4 * n);
    PG3_CUDA(cudaGetLastError());
    E.cur = 0;
    E.pending = false;
    E.fresh = true;
    launch_init_planet(E.v.d, E.P, t, E.stream);
    Scalars h{};
    PG3_CUDA(cudaMemcpyAsync(&h, E.sc, sizeof(Scalars), cudaMemcpyDeviceToHost, E.stream));
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    h.t = t;
    h.dt = 0.0;
    h.dt_prev = 0.0;
    h.end_time = 1.0e30;
    h.vmax_bits = 0ull;
    h.steps = 0;
    h.done = 0;
    h.pad_ = 0;
    h.err = 0;
    h.floor_hits = 0;
    h.dt_hold = 0.0;
    PG3_CUDA(cudaMemcpyAsync(E.sc, &h, sizeof(Scalars), cudaMemcpyHostToDevice, E.stream));
    k3_cfl<<<E.grid_kick, K3_THREADS, 0, E.stream>>>(E.v, E.buf[0]);
    PG3_CUDA(cudaGetLastError());
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    return PG_OK;
}

pg_status pg_disk3_get_state(pg_disk3* dk, double* r, double* p, double* u, double* v, double* w, double* t_out) {
    if (!dk || !r || !p || !u || !v || !w) return fail3(PG_ERR_ARG, "null argument");
    Engine3& E = *dk->E;
    PG3_CUDA(cudaSetDevice(E.device));
    pg_status s = resolve3(E);
    if (s != PG_OK) return s;
    const size_t n = (size_t)E.P.xres * E.P.yres * E.P.zres;
    double* st = nullptr;
    if ((s = stage_buffer(E, 5 * n, &st)) != PG_OK) return s;
    k3_extract<<<1184, 256, 0, E.stream>>>(E.v, E.buf[E.cur], st, st + n, st + 2 * n, st + 3 * n, st + 4 * n);
    PG3_CUDA(cudaGetLastError());
    double* dst[5] = {r, p, u, v, w};
    PG3_CUDA(copy_planes_out(E.readback, E.device, st, dst, 5, n, E.stream));
    if (t_out) PG3_CUDA(cudaMemcpyAsync(t_out, &E.sc->t, sizeof(double), cudaMemcpyDeviceToHost, E.stream));
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    return PG_OK;
}

pg_status pg_disk3_global_dt(pg_disk3* dk, double dt_prev, double* dt_out) {
    if (!dk || !dt_out) return fail3(PG_ERR_ARG, "null argument");
    Engine3& E = *dk->E;
    PG3_CUDA(cudaSetDevice(E.device));
    unsigned long long bits = 0;
    PG3_CUDA(cudaMemcpyAsync(&bits, &E.sc->vmax_bits, sizeof(bits), cudaMemcpyDeviceToHost, E.stream));
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    double vmax;
    std::memcpy(&vmax, &bits, sizeof vmax);
    const double dt = E.P.cfl / vmax;  // get_dt_lv2 (timestep.cu:108)
    double tmp = dt_prev * 1.1;        // timestep.cu:133-139
    if (dt < tmp) tmp = dt;
    *dt_out = tmp;
    return PG_OK;
}

pg_status pg_disk3_solve(pg_disk3* dk, double t, double dt) {
    if (!dk) return fail3(PG_ERR_ARG, "null disk");
    Engine3& E = *dk->E;
    PG3_CUDA(cudaSetDevice(E.device));
    pg_status s = resolve3(E);
    if (s != PG_OK) return s;
    launch_set_time(E.v.d, t, dt, E.stream);
    enqueue_passes(E, E.cur);
    PG3_CUDA(cudaGetLastError());
    E.cur = 1 - E.cur;
    E.fresh = false;
    return PG_OK;
}

pg_status pg_disk3_run(pg_disk3* dk, int nsteps, double end_time) {
    if (!dk) return fail3(PG_ERR_ARG, "null disk");
    if (nsteps <= 0) return PG_OK;
    Engine3& E = *dk->E;
    pg_status s = begin_run(E, end_time);
    if (s != PG_OK) return s;
    const bool may_finish = end_time < 1.0e29;
    for (int step = 0; step < nsteps; ++step) {
        if (may_finish && step > 0 && step % 256 == 0) {
            int done = 0;
            PG3_CUDA(cudaMemcpyAsync(&done, &E.sc->done, sizeof(int), cudaMemcpyDeviceToHost, E.stream));
            PG3_CUDA(cudaStreamSynchronize(E.stream));
            if (done) break;
        }
        const int c0 = E.cur;
        if (!E.graph[c0]) {  // one step (clock + five passes) from buffer c0, captured once
            cudaGraph_t g;
            PG3_CUDA(cudaStreamBeginCapture(E.stream, cudaStreamCaptureModeThreadLocal));
            launch_time_step(E.v.d, E.stream);
            enqueue_passes(E, c0);
            cudaError_t ce = cudaStreamEndCapture(E.stream, &g);
            PG3_CUDA(ce);
            PG3_CUDA(cudaGraphInstantiate(&E.graph[c0], g, 0));
            cudaGraphDestroy(g);
        }
        PG3_CUDA(cudaGraphLaunch(E.graph[c0], E.stream));
        E.cur = 1 - c0;
    }
    if (!may_finish) E.pending = false;
    else E.cur = E.cur_base;  // resolved from the device step count on next use
    return PG_OK;
}

pg_status pg_disk3_clock(pg_disk3* dk, double* t, double* dt, long long* steps) {
    if (!dk) return fail3(PG_ERR_ARG, "null disk");
    Scalars h{};
    PG3_CUDA(cudaMemcpyAsync(&h, dk->E->sc, sizeof(Scalars), cudaMemcpyDeviceToHost, dk->E->stream));
    PG3_CUDA(cudaStreamSynchronize(dk->E->stream));
    if (t) *t = h.t;
    if (dt) *dt = h.dt;
    if (steps) *steps = h.steps;
    return PG_OK;
}

pg_status pg_disk3_check(pg_disk3* dk) {
    if (!dk) return fail3(PG_ERR_ARG, "null disk");
    Engine3& E = *dk->E;
    int err = 0;
    PG3_CUDA(cudaMemcpyAsync(&err, &E.sc->err, sizeof(int), cudaMemcpyDeviceToHost, E.stream));
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    const int zero = 0;
    PG3_CUDA(cudaMemcpy(&E.sc->err, &zero, sizeof(int), cudaMemcpyHostToDevice));
    if (err & (1 << PG_ERR_TIMEOUT)) return fail3(PG_ERR_TIMEOUT, "a device wait timed out");
    if (err & (1 << PG_ERR_NAN)) return fail3(PG_ERR_NAN, "non-positive or NaN density produced");
    return PG_OK;
}

// Average device time of each pass over nsteps device-clocked steps (CUDA
// events on the disk's stream): clock, kick1, sweep_x, sweep_y, sweep_z, kick2.
pg_status pg_disk3_pass_times(pg_disk3* dk, int nsteps, double* ms6) {
    if (!dk || !ms6 || nsteps <= 0) return fail3(PG_ERR_ARG, "bad argument");
    Engine3& E = *dk->E;
    pg_status s = begin_run(E, 1.0e30);
    if (s != PG_OK) return s;
    E.pending = false;  // no end_time: every step runs
    cudaEvent_t ev[7];
    for (auto& e : ev) PG3_CUDA(cudaEventCreate(&e));
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const View3& v = E.v;
    for (int step = 0; step < nsteps; ++step) {
        const int c = E.cur;
        Cell* A = E.buf[c];
        Cell* B = E.buf[1 - c];
        cudaEventRecord(ev[0], E.stream);
        launch_time_step(v.d, E.stream);
        cudaEventRecord(ev[1], E.stream);
        k3_kick<1><<<E.grid_kick, K3_THREADS, 0, E.stream>>>(v, A, B);
        cudaEventRecord(ev[2], E.stream);
        enqueue_sweep(E, 0, 1 - c);
        cudaEventRecord(ev[3], E.stream);
        enqueue_sweep(E, 1, c);
        cudaEventRecord(ev[4], E.stream);
        enqueue_sweep(E, 2, 1 - c);
        cudaEventRecord(ev[5], E.stream);
        k3_kick<2><<<E.grid_kick, K3_THREADS, 0, E.stream>>>(v, A, B);
        cudaEventRecord(ev[6], E.stream);
        PG3_CUDA(cudaGetLastError());
        PG3_CUDA(cudaEventSynchronize(ev[6]));
        for (int k = 0; k < 6; ++k) {
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
            acc[k] += ms;
        }
        E.cur = 1 - c;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    for (int k = 0; k < 6; ++k) ms6[k] = acc[k] / nsteps;
    return PG_OK;
}

// write_check_point (src/output/output.cu:125-180, ndim 3): t, the interior
// faces of x, y and z, then the r, p, u, v, w planes (x fastest, then y, then z)
pg_status pg_disk3_write_snapshot(pg_disk3* dk, const char* path) {
    if (!dk || !path) return fail3(PG_ERR_ARG, "null argument");
    Engine3& E = *dk->E;
    const size_t n = (size_t)E.P.xres * E.P.yres * E.P.zres;
    std::vector<double> h(5 * n);
    double t = 0.0;
    pg_status s = pg_disk3_get_state(dk, h.data(), h.data() + n, h.data() + 2 * n, h.data() + 3 * n, h.data() + 4 * n, &t);
    if (s != PG_OK) return s;
    FILE* f = std::fopen(path, "wb");
    if (!f) return fail3(PG_ERR_ARG, "cannot open %s", path);
    bool ok = std::fwrite(&t, sizeof(double), 1, f) == 1;
    ok = ok && std::fwrite(&E.hxa[NPAD], sizeof(double), E.P.xres + 1, f) == (size_t)E.P.xres + 1;
    ok = ok && std::fwrite(&E.hya[NPAD], sizeof(double), E.P.yres + 1, f) == (size_t)E.P.yres + 1;
    ok = ok && std::fwrite(&E.hza[NPAD], sizeof(double), E.P.zres + 1, f) == (size_t)E.P.zres + 1;
    ok = ok && std::fwrite(h.data(), sizeof(double), 5 * n, f) == 5 * n;
    ok = (std::fclose(f) == 0) && ok;
    return ok ? PG_OK : fail3(PG_ERR_ARG, "short write to %s", path);
}

// load_grid (src/output/output.cu:182-248, ndim 3): t and the five planes of a
// checkpoint file (the faces are skipped), then a restart at t like set_state
pg_status pg_disk3_read_snapshot(pg_disk3* dk, const char* path, double* t_out) {
    if (!dk || !path) return fail3(PG_ERR_ARG, "null argument");
    Engine3& E = *dk->E;
    const size_t n = (size_t)E.P.xres * E.P.yres * E.P.zres;
    std::vector<double> h(5 * n);
    double t = 0.0;
    FILE* f = std::fopen(path, "rb");
    if (!f) return fail3(PG_ERR_ARG, "cannot open %s", path);
    bool ok = std::fread(&t, sizeof(double), 1, f) == 1;
    ok = ok && std::fseek(f, (long)sizeof(double) * (1 + E.P.xres + 1 + E.P.yres + 1 + E.P.zres + 1), SEEK_SET) == 0;
    ok = ok && std::fread(h.data(), sizeof(double), 5 * n, f) == 5 * n;
    std::fclose(f);
    if (!ok) return fail3(PG_ERR_ARG, "%s is not a checkpoint of this grid", path);
    if (t_out) *t_out = t;
    return pg_disk3_set_state(dk, t, h.data(), h.data() + n, h.data() + 2 * n, h.data() + 3 * n, h.data() + 4 * n);
}

// test support: one step with host t and dt (as pg_disk3_solve), copying the
// whole buffer (ghosts included, xarr*yarr*zarr cells) after each of the five
// passes into out (5 x that many cells): kick1, sweep_x, sweep_y, sweep_z,
// kick2 (with the damping).  Blocking.
pg_status pg_disk3_stages(pg_disk3* dk, double t, double dt, pg_cell* out) {
    if (!dk || !out) return fail3(PG_ERR_ARG, "null argument");
    Engine3& E = *dk->E;
    PG3_CUDA(cudaSetDevice(E.device));
    pg_status s = resolve3(E);
    if (s != PG_OK) return s;
    const View3& v = E.v;
    const size_t n = (size_t)v.d.xarr * v.d.yarr * v.zarr;
    const int c = E.cur;
    Cell* A = E.buf[c];
    Cell* B = E.buf[1 - c];
    launch_set_time(v.d, t, dt, E.stream);
    auto grab = [&](const Cell* src, int k) {
        return cudaMemcpyAsync(out + k * n, src, n * sizeof(Cell), cudaMemcpyDeviceToHost, E.stream);
    };
    k3_kick<1><<<E.grid_kick, K3_THREADS, 0, E.stream>>>(v, A, B);
    PG3_CUDA(grab(B, 0));
    enqueue_sweep(E, 0, 1 - c);
    PG3_CUDA(grab(A, 1));
    enqueue_sweep(E, 1, c);
    PG3_CUDA(grab(B, 2));
    enqueue_sweep(E, 2, 1 - c);
    PG3_CUDA(grab(A, 3));
    k3_kick<2><<<E.grid_kick, K3_THREADS, 0, E.stream>>>(v, A, B);
    PG3_CUDA(grab(B, 4));
    PG3_CUDA(cudaGetLastError());
    PG3_CUDA(cudaStreamSynchronize(E.stream));
    E.cur = 1 - c;
    E.fresh = false;
    return PG_OK;
}

}  // extern "C"
