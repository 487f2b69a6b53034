// penguin_b200 kernels for sm_100a: one Godunov timestep of PEnGUIn
// (src/solver/solve.cu:212-292) as five fused passes over the AoS state:
//
//   kick1   C -> T : viscous stress (src/viscosity/viscosity.cu:34-197) + first half-kick
//                    (src/solver/sweeps.cu:597-711, mdt = 0); stores the stress for kick2
//   sweep_x T -> C : radial Godunov sweep (src/solver/sweeps.cu:263-335)
//   sweep_y C -> T : azimuthal sweep (sweeps.cu:361-433) writing each cell at its
//                    orbital-advection shifted row (src/orbit/orbit.cu:17-99)
//   advect  T -> C : residual orbital advection (src/solver/advection/advection.cu:1-173)
//   kick2   C -> T : predictor kick, viscous stress of the predicted state and
//                    corrector kick (solve.cu:266-269), wave damping
//                    (src/killwave/killwave.cu:17-103) and the CFL signal speed
//                    for the next step (src/timestep/timestep.cu:18-97)
//
// plus a one-block clock kernel (dt, planet and its table).  Every pass writes each cell
// together with its ghost images, so no separate boundary pass is needed between stages.
#include <cstdio>

#include "pg_common.cuh"
#include "pg_hydro.cuh"
#include "pg_internal.h"
#include "pg_planet.cuh"
#include "pg_dust.cuh"

namespace pg {

// ------------------------------------------------- the sweeps' work layout
// Lanes of a warp lie along the radius, which is contiguous in memory, in every
// pass, and a warp takes `len` rows of its 30 or 32 radii one after the other.  No
// barrier separates the phases of a cell: what a cell needs of its neighbours comes
// by shuffle (radial sweep) or stays in registers from the row before (azimuthal
// passes).  Tiles of 32 x 8 cells whose phases met at __syncthreads and exchanged
// states and fluxes through shared memory spent 900-1000 instructions a cell, 350 of
// them FP64, and a quarter of their time at the barriers; the sweeps spend 720-770 now.
// What is left to bound them is FP64 issue and latency: the FP64 pipe is 57-60 % busy in
// the sweeps, at a third of the copy rate.  1024x3072, us a pass, tiles -> runs: kick1
// 108 -> 87, sweep_x 298 -> 124, sweep_y 328 -> 123, advection 154 -> 71, kick2 177 -> 140.
// Each kernel is compiled for the CTAs per SM that were fastest there, at 2 / 3 / 4 / 5:
// sweep_x 134 / 124 / 128 / 149, sweep_y 148 / 123 / 138 / 246, advection 76 / 76 / 71 / 72
// (adiabatic 512x1536: 26.5 / 26.2 / 25.7 / 31.6), kick1 138 / 106 / 87 / 96.
constexpr int SW_WARPS = 4;                       // warps per CTA, independent of one another
constexpr int RX_OUT = 30;                        // radial sweep: outputs of a warp's 32 cells
constexpr int RX_ROWS = RX_TILE_ROWS;             // rows per TMA copy
constexpr int RX_STAGE = RX_TILE_CELLS * RX_ROWS * 5;  // doubles
static_assert(RX_TILE_CELLS == RX_OUT + 6, "32 lanes and two stencil cells a side");
static_assert(RX_STAGE * 8 % 128 == 0, "128-byte aligned stages");
constexpr size_t RX_SMEM = (size_t)SW_WARPS * 2 * RX_STAGE * 8 + SW_WARPS * 16 + 128;

constexpr int KK_OUT = 30;                        // half-kicks: outputs of a warp's 32 cells

// --------------------------------------------------------- source terms
struct Grav {
    double gx, gy, gz;
};
// Star + planet gravity in the 2D cylindrical frame (src/solver/force/forces.cu:41-58,
// 182-327 with twobd_flag 0, pol = 0).  The star term is a per-radius table; the
// planet's angle enters through the per-row sin/cos table of this step
// (planet_rows) and 1/x_p^2 through the table's tail.
__device__ __forceinline__ Grav gravity_at(const DiskView& d, double gstar, double rad, double sinfac,
                                           double cosfac, double iplx2, const pg_body& p) {
    Grav g{0.0, 0.0, 0.0};
    if (d.geomx == 1) {
        g.gx = gstar;
        g.gz = -0.0;
        if (d.nplanet > 0) {
            const double plm = p.m, plx = p.x;
            const double ir = rsq(mad(-2.0 * plx * rad, cosfac, mad(rad, rad, mad(plx, plx, p.rs * p.rs))));
            const double rs_fac = ir * ir * ir;
            g.gx = mad(-plm, mad(cosfac, iplx2, mad(-plx, cosfac, rad) * rs_fac), g.gx);
            g.gy = plm * (sinfac * mad(-plx, rs_fac, iplx2));
        }
    }
    return g;
}
__device__ __forceinline__ Grav gravity(const DiskView& d, int i, double rad, double sinfac, double cosfac,
                                        double iplx2, const pg_body& p) {
    return gravity_at(d, d.geomx == 1 ? d.gstar[i] : 0.0, rad, sinfac, cosfac, iplx2, p);
}

// One body of the two-body frame as an inertial point mass
// (star_planet_grav_cyl_inertial, src/solver/force/forces.cu:89-106, z = 0).
__device__ __forceinline__ void inertial_pull(double rad, double sinfac, double cosfac, const pg_body& p, Grav& g) {
    const double plm = p.m, plx = p.x;
    const double Rp = sqrt(rad * rad + plx * plx - 2.0 * plx * rad * cosfac + 0.0 * 0.0 + p.rs * p.rs);
    const double rs_fac = 1.0 / Rp / Rp / Rp;
    g.gx += -plm * (rad - plx * cosfac) * rs_fac;
    g.gy += -plm * plx * sinfac * rs_fac;
    g.gz += -plm * 0.0 * rs_fac;
}

// Gravity at cell (i, j) with the bodies of the first half-kick (which 0) or at
// t + dt (which 1).  In the two-body frame (twobd_flag 1, forces.cu:182-327)
// the star (planets[0]) and the planet (planets[1]) pull as inertial point
// masses and the fixed-star term and the indirect term drop out.
__device__ __forceinline__ Grav body_gravity(const DiskView& d, int i, int j, int which, const pg_body& pl,
                                             const pg_body& st) {
    const double* tr = d.trig + 4 * j + 2 * which;
    if (!d.twobd) return gravity(d, i, d.radx[i], tr[0], tr[1], d.trig[4 * d.yarr + which], pl);
    Grav g{0.0, 0.0, 0.0};
    if (d.geomx == 1) {
        const double* ts = d.strig + 4 * j + 2 * which;
        inertial_pull(d.radx[i], ts[0], ts[1], st, g);
        inertial_pull(d.radx[i], tr[0], tr[1], pl, g);
    }
    return g;
}

// One cell of apply_source_terms (src/solver/sweeps.cu:597-711): curvature,
// gravity and viscous acceleration; with mdt != 0 the forces are re-evaluated
// at the mdt-predicted velocities (sweeps.cu:663-687).

// Newtonian cooling of the pressure over dt (src/solver/cool/cool.cu:1-33): the
// specific energy p/r relaxes towards cs^2(xc) with t_c = beta r_cyl^1.5
// (cool 1, tabulated) or beta / r sqrt(p/r) / h (cool 2, r the density).
__device__ __forceinline__ double p_cool(const DiskView& d, int i, double p, double r, double dt) {
    const double tc = (d.cool == 1) ? d.coolx[i] : d.beta_cool * (1.0 / r) * (sqrt(p / r) / d.sc_h);
    const double e = p / r;
    const double e0 = d.cs2x[i];
    return r * (e0 + (e - e0) * exp(-dt / tc));
}

template <bool VISC>
__device__ __forceinline__ Cell kick(const DiskView& d, const Cell& C, double ix, const Grav& g, double vx,
                                     double vy, double mdt, double dt, double* Tu = nullptr, double* Tv = nullptr) {
    Cell T = C;
    const double ir = VISC ? inv(C.r) : 0.0;  // T.r == C.r throughout
    double fx = (d.geomx == 1) ? T.v * T.v * ix : 0.0;
    const double fy = VISC ? vy * ir : 0.0, fz = 0.0;  // stress in 2D only
    if (VISC) fx = mad(vx, ir, fx);
    if (mdt != 0.0) {
        T.u = mad(g.gx, mdt, mad(fx, mdt, C.u));
        T.v = mad(g.gy, mdt, mad(fy, mdt, C.v));
        if (Tu) *Tu = T.u;  // the gas velocity the dust drag relaxes towards (sweeps.cu:679-687)
        if (Tv) *Tv = T.v;
        fx = (d.geomx == 1) ? T.v * T.v * ix : 0.0;
        if (VISC) fx = mad(vx, ir, fx);
    }
    Cell o;
    o.u = mad(g.gx, dt, mad(fx, dt, C.u));
    o.v = mad(g.gy, dt, mad(fy, dt, C.v));
    o.w = mad(g.gz, dt, mad(fz, dt, C.w));
    o.r = C.r;
    o.p = C.p;
    return o;
}

// add_grid (src/output/output.cu:250-275): A += C (0.5 dt) / T on the interior
__device__ __forceinline__ void accumulate_average(const DiskView& d, int i, int j, const Cell& C, double hdt) {
    const double fac = hdt / d.ave_T;
    Cell* a = d.ave + (size_t)i + (size_t)d.xarr * j;
    a->r += C.r * fac;
    a->p += C.p * fac;
    a->u += C.u * fac;
    a->v += C.v * fac;
    a->w += C.w * fac;
}

__device__ __forceinline__ double signal_rate(const DiskView& d, const Cell& c, int i, int j,
                                              const DCell* dc = nullptr) {
    // src/timestep/timestep.cu:46-77 (cell widths as reciprocals); with dust the
    // dust speeds also bound dt (:64-74)
    const double rad_cyl = (d.geomy == 3) ? d.radx[i] : 1.0;
    const double cs = sound_speed(d.gam, c.r, c.p);
    double spd = fabs(c.u) + cs;
    if (dc) spd = fmax(fabs(dc->u), spd);
    double tmp = fmax(spd * d.idx_x[i], 0.0);
    if (d.ndim > 1) {
        spd = fabs(mad(-rad_cyl, d.frame_omega, c.v) - d.rot[i]) + cs;
        if (dc) spd = fmax(fabs(mad(-rad_cyl, d.frame_omega, dc->v) - d.rot[i]), spd);
        tmp = fmax(spd * (d.idx_y[j] * ((d.geomy == 3) ? d.irad[i] : 1.0)), tmp);
    }
    return tmp;
}

// What a marching pass writes: cell (i, j) at `o` and its periodic azimuthal image; a cell
// with radial images (bound 1 and 2, a lane at the edge) takes emit's general way.
struct Emitter {
    int lo, hi;        // rows below lo have an image yres rows up, rows from hi on yres rows down
    long long image;   // doubles between a row and its image
    bool edge;
    __device__ __forceinline__ Emitter(const DiskView& d, int i) {
        lo = d.ndim > 1 ? 2 * NPAD : 0;
        hi = d.ndim > 1 ? d.yres : 0x7fffffff;
        image = 5ll * d.xarr * d.yres;
        const int nx = d.xres + NPAD;
        edge = (d.bound_lft != 0 && i < 2 * NPAD) || (d.bound_rgh != 0 && i >= nx - NPAD);
    }
    __device__ __forceinline__ void put(double* o, const Cell& c) const {
        o[0] = c.r;
        o[1] = c.p;
        o[2] = c.u;
        o[3] = c.v;
        o[4] = c.w;
    }
    __device__ __forceinline__ void operator()(const DiskView& d, Cell* out, double* o, int i, int j, const Cell& c) const {
        put(o, c);
        if (j < lo || j >= hi) put(o + (j < lo ? image : -image), c);
        if (edge) emit(d, out, i, j, c);
    }
};
__device__ __forceinline__ double* cell_at(const DiskView& d, Cell* out, int i, int j) {
    return reinterpret_cast<double*>(out + ((size_t)i + (size_t)d.xarr * j));
}

// ================================================================ sweeps
// ISO: a 2D isothermal gas, which needs neither the energy flux nor the z-velocity
// (identically zero in 2D): nothing is computed that the equation of state does not use.
// The passes are bound by the latency and issue of their FP64 arithmetic (0.3 of the
// copy rate), so what counts is instructions: reciprocals and roots without their
// IEEE tails (pg_hydro.cuh).

__device__ __forceinline__ double up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double down1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Radial sweep (src/solver/sweeps.cu:263-335).  A warp stages 4 rows of 36 cells per
// TMA copy, two copies in flight; lane l holds cell 2 + 30 seg + l: it reconstructs it,
// takes its left face's left state from the lane below and its right face's flux from
// the lane above, and lanes 1..30 update.
template <bool ISO>
__global__ void __launch_bounds__(32 * SW_WARPS, 3)
    k_sweep_x(const __grid_constant__ CUtensorMap tm, const DiskView d, Cell* __restrict__ out, int nseg, int len,
              int nitems) {
    extern __shared__ __align__(128) double smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* buf = smem_base128(smem_raw) + (size_t)warp * 2 * RX_STAGE;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_base128(smem_raw) + (size_t)SW_WARPS * 2 * RX_STAGE) + 2 * warp;
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
    const int eos = ISO ? 0 : d.eos;
    const int jend = d.ypad + d.yres;
    int k = 0;  // copies waited for by this warp
    for (int item = blockIdx.x * SW_WARPS + warp; item < nitems; item += gridDim.x * SW_WARPS) {
        const int seg = item % nseg, j0 = d.ypad + len * (item / nseg), j1 = min(j0 + len, jend);
        auto issue = [&](int j, int n) {  // rows j .. j + 3 into copy n
            issue_begin(&bar[n & 1], RX_STAGE * 8);
            issue_box(buf + (n & 1) * RX_STAGE, &tm, 5 * RX_OUT * seg, j, &bar[n & 1]);
        };
        if (lane == 0) {
            issue(j0, k);
            if (j0 + RX_ROWS < j1) issue(j0 + RX_ROWS, k + 1);
        }
        const int i = NPAD - 1 + RX_OUT * seg + lane, ic = min(i, d.xarr - 1);
        const bool output = lane >= 1 && lane <= RX_OUT && i < NPAD + d.xres;
        const Emitter emit_to(d, i);
        double* o = cell_at(d, out, ic, j0);
        double w[6], rad[5];
#pragma unroll
        for (int m = 0; m < 6; ++m) w[m] = d.wx[6 * ic + m];
#pragma unroll
        for (int m = 0; m < 5; ++m) rad[m] = d.geomx == 1 ? d.radx[min(max(i - 2 + m, 0), d.xarr - 1)] : 1.0;
        const double sx = dt * d.idx_x[ic];
        const double f = dt * d.ixv[ic];
        const double irad = d.geomx == 1 ? d.irad[ic] : 1.0;
        const double cs2 = d.cs2x[ic];
        const double g0 = d.geomx == 1 ? d.xa[ic] : 1.0, g1 = d.geomx == 1 ? d.xa[ic + 1] : 1.0;  // riemann.cu:5-11
        for (int j = j0; j < j1; j += RX_ROWS, ++k) {
            if (!warp_wait(&bar[k & 1], (uint32_t)((k >> 1) & 1), sc)) {
                if (lane == 0 && j + RX_ROWS < j1) mbar_wait(&bar[(k + 1) & 1], (uint32_t)(((k + 1) >> 1) & 1), sc);
                return;
            }
            const double* row = buf + (k & 1) * RX_STAGE + 5 * (lane + 2);
#pragma unroll 1
            for (int jj = j; jj < min(j + RX_ROWS, j1); ++jj, row += 5 * RX_TILE_CELLS) {
                auto field = [&](int m, double flat) {
                    return recon(w, row[m - 10], row[m - 5], row[m], row[m + 5], row[m + 10], flat);
                };
                const Cell C0{row[0], row[1], row[2], row[3], row[4]};
                const double cs0 = sound_speed(gam, C0.r, C0.p);
                const double flat = flatten(C0.p, row[-9], row[-4], row[6], row[11], row[-3], C0.u, row[7]);
                const Par R = field(0, flat), P = field(1, flat), U = field(2, flat);
                // angular momentum (geomx 1)
                const Par A = recon(w, row[-7] * rad[0], row[-2] * rad[1], C0.v * rad[2], row[8] * rad[3],
                                    row[13] * rad[4], flat);
                Par Z{0.0, 0.0, 0.0};
                if (!ISO && d.ndim != 2) Z = field(4, flat);  // in 2D the z-velocity is identically zero
                const Half eL = state_at_left_edge(gam, sx, cs0, C0.r, C0.p, C0.u, R, P, U, A, Z);
                const Half eR = state_at_right_edge(gam, sx, cs0, C0.r, C0.p, C0.u, R, P, U, A, Z);
                const Half L{up1(eR.r), up1(eR.p), up1(eR.u), up1(eR.v), ISO ? 0.0 : up1(eR.w)};
                const Flux F = hllc(eos, d.ie, gam, L, eL);
                // net_source (src/solver/riemann/riemann.cu:40-87) and the flux differences
                auto net = [&](double x) { return x * g0 - down1(x) * g1; };
                const double pres1 = down1(F.pres);
                Cell D;
                D.r = net(F.r) * f;
                D.u = (net(F.u) + 0.5 * (g0 + g1) * (F.pres - pres1)) * f;
                D.v = net(F.v) * f * irad;
                D.w = D.p = 0.0;
                if (!ISO) {
                    D.w = net(F.w) * f;
                    double de = net(F.uprs);
                    if (d.ie != 0) de *= 0.5 * (F.pres + pres1);
                    D.p = (net(F.p) + (eos == 2 ? de : 0.0)) * f;
                }
                if (output) {
                    const Cell Q = update_cell<ISO>(eos, d.ie, gam, cs2, C0, D, &sc->floor_hits);
                    if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    emit_to(d, out, o, i, jj, Q);
                }
                o += 5 * (size_t)d.xarr;
            }
            __syncwarp();  // the copy's reads are done
            if (lane == 0 && j + 2 * RX_ROWS < j1) issue(j + 2 * RX_ROWS, k + 2);
        }
    }
}

// r, p, u, v of one cell of a column
__device__ __forceinline__ void load4(const double* c, double* q) {
#pragma unroll
    for (int m = 0; m < 4; ++m) q[m] = c[m];
}

// Azimuthal sweep (sweeps.cu:361-433) with the orbital shift (orbit.cu:17-99): a lane
// marches along its own column.  Five rows of it are in registers, the next one in
// flight; each row costs one reconstruction, one trace of both edges, the flux at the
// face below it and the update of the cell below that, written len rows long at its
// shifted place.  The per-radius factors are loop constants and the per-row tables
// the same for the whole warp.
template <bool ISO>
__global__ void __launch_bounds__(32 * SW_WARPS, 3)
    k_sweep_y(const Cell* __restrict__ in, const DiskView d, Cell* __restrict__ out, int ncol, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt, gam = d.gam;
    const int eos = ISO ? 0 : d.eos;
    for (int item = blockIdx.x * SW_WARPS + warp; item < nitems; item += gridDim.x * SW_WARPS) {
        const int i = NPAD + 32 * (item % ncol) + lane;
        const bool active = i < NPAD + d.xres;
        const int ic = min(i, NPAD + d.xres - 1);
        const int s0 = NPAD + len * (item / ncol), s1 = min(s0 + len, NPAD + d.yres);
        const double rad = (d.geomy == 3) ? d.radx[ic] : 1.0, irad = (d.geomy == 3) ? d.irad[ic] : 1.0;
        const double rot = d.rot[ic], cs2 = d.cs2x[ic];
        const double v0 = (d.geomy == 3) ? rot + rad * d.frame_omega : rot;
        // set_orbital_advection (src/orbit/orbit.cu:74-99) for this column
        int shift = 0;
        if (d.orbadv) {
            const double dy = d.dy0 * d.radx[ic];
            shift = __double2int_rd(rot * dt / dy + 0.5);
            double speed = shift * dy / dt;
            speed = rot - speed;
            if (s0 == NPAD && active) {
                d.res[i] = speed;
                d.inc[i] = shift;
            }
        }
        const double sdt = dt * irad;
        // row the first output goes to: T[(j+inc) mod N] = C[j] (orbit.cu:30-46)
        int js = (s0 - d.ypad + shift) % d.yres;
        if (js < 0) js += d.yres;
        const double* col = reinterpret_cast<const double*>(in + ic);
        const size_t pitch = 5 * (size_t)d.xarr;
        const Emitter emit_to(d, i);
        double* o = cell_at(d, out, ic, js + d.ypad);
        const double* next = col + pitch * (s0 - NPAD);
        double q[5][4], nx[4];  // rows t-2 .. t+2 and t+3: r, p, v_r, v_phi
#pragma unroll
        for (int m = 0; m < 5; ++m, next += pitch) load4(next, q[m]);
        Half pr{};   // the state at the right edge of the cell below
        Flux pf{};   // the flux at the face below it
#pragma unroll 1
        for (int t = s0 - 1; t <= s1; ++t) {
            if (t < s1) load4(next, nx);
            next += pitch;
            double u[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) u[m] = q[m][3] - v0;
            const double* w = d.wy + 6 * t;
            auto field = [&](int m, double flat) { return recon(w, q[0][m], q[1][m], q[2][m], q[3][m], q[4][m], flat); };
            const double cs0 = sound_speed(gam, q[2][0], q[2][1]);
            const double flat = flatten(q[2][1], q[0][1], q[1][1], q[3][1], q[4][1], u[1], u[2], u[3]);
            const double sx = sdt * d.idx_y[t];
            const Par R = field(0, flat), P = field(1, flat), A = field(2, flat);
            const Par U = recon(w, u[0], u[1], u[2], u[3], u[4], flat);
            const Par Z{0.0, 0.0, 0.0};
            const Half eL = state_at_left_edge(gam, sx, cs0, q[2][0], q[2][1], u[2], R, P, U, A, Z);
            const Half eR = state_at_right_edge(gam, sx, cs0, q[2][0], q[2][1], u[2], R, P, U, A, Z);
            Flux F{};
            if (t >= s0) F = hllc(eos, d.ie, gam, pr, eL);
            if (t > s0) {  // the cell below has both its fluxes
                const double f = sdt * d.iyv[t - 1];
                Cell D;
                D.r = (pf.r - F.r) * f;
                D.v = ((pf.u - F.u) + (pf.pres - F.pres)) * f + v0 * D.r;
                D.u = (pf.v - F.v) * f;
                D.w = D.p = 0.0;
                if (!ISO) {
                    double de = pf.uprs - F.uprs;
                    if (d.ie != 0) de *= 0.5 * (pf.pres + F.pres);
                    D.p = ((pf.p - F.p) + (eos == 2 ? de : 0.0)) * f;
                }
                if (active) {
                    const Cell C0{q[1][0], q[1][1], q[1][2], q[1][3], 0.0};
                    const Cell Q = update_cell<ISO>(eos, d.ie, gam, cs2, C0, D, &sc->floor_hits);
                    if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    emit_to(d, out, o, i, js + d.ypad, Q);
                }
                o += pitch;
                if (++js == d.yres) {
                    js = 0;
                    o -= pitch * d.yres;
                }
            }
            pr = eR;
            pf = F;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                q[0][m] = q[1][m];
                q[1][m] = q[2][m];
                q[2][m] = q[3][m];
                q[3][m] = q[4][m];
                q[4][m] = nx[m];
            }
        }
    }
}

// ===================================================== residual advection
// advection.cu:1-173, marching like the azimuthal sweep.  The residual speed of a column
// has one sign, so every cell feeds one face, the same of its two for the whole column:
// with this row's flux and the last one's the update of this row (upwards) or of the
// last (downwards) is complete.
template <bool ISO>
__global__ void __launch_bounds__(32 * SW_WARPS, 4)
    k_advect(const Cell* __restrict__ in, const DiskView d, Cell* __restrict__ out, int ncol, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt;
    for (int item = blockIdx.x * SW_WARPS + warp; item < nitems; item += gridDim.x * SW_WARPS) {
        const int i = NPAD + 32 * (item % ncol) + lane;
        const bool active = i < NPAD + d.xres;
        const int ic = min(i, NPAD + d.xres - 1);
        const int s0 = NPAD + len * (item / ncol), s1 = min(s0 + len, NPAD + d.yres);
        const double speed = d.res[ic], cs2 = d.cs2x[ic];
        const double sdt = dt * ((d.geomy == 3) ? d.irad[ic] : 1.0);
        const double sx = fabs(speed) * sdt;
        const bool up = speed > 0.0;
        const size_t pitch = 5 * (size_t)d.xarr;
        const double* next = reinterpret_cast<const double*>(in + ic) + pitch * (s0 - NPAD);
        const Emitter emit_to(d, i);
        double* o = cell_at(d, out, ic, up ? s0 - 1 : s0 - 2);  // the row updated at t = s0 - 1
        double q[5][4], nx[4];
#pragma unroll
        for (int m = 0; m < 5; ++m, next += pitch) load4(next, q[m]);
        double pm = 0.0, pu = 0.0, pv = 0.0, pp = 0.0;  // what the row before carries through its face
#pragma unroll 1
        for (int t = s0 - 1; t <= s1; ++t) {
            if (t < s1) load4(next, nx);
            next += pitch;
            const double* w = d.wy + 6 * t;
            const Frac x = frac(lesser(sx * d.idx_y[t], 1.0));
            auto ave = [&](int m) {
                const Par a = recon(w, q[0][m], q[1][m], q[2][m], q[3][m], q[4][m], 0.0);
                return up ? aveR(x, a) : aveL(x, a);
            };
            const double fm = ave(0) * speed, fu = ave(2) * fm, fv = ave(3) * fm;
            const double fp = (!ISO && d.eos != 0) ? ave(1) * speed : 0.0;
            const int row = up ? t : t - 1;
            if (active && row >= s0 && row < s1) {
                const double f = sdt * d.iyv[row];
                Cell Q{up ? q[2][0] : q[1][0], up ? q[2][1] : q[1][1], up ? q[2][2] : q[1][2], up ? q[2][3] : q[1][3],
                       0.0};
                const double r = Q.r + (pm - fm) * f;
                const double ir = inv(r);
                Q.u = (Q.u * Q.r + (pu - fu) * f) * ir;
                Q.v = (Q.v * Q.r + (pv - fv) * f) * ir;
                if (!ISO) Q.p += (pp - fp) * f;
                Q.r = r;
                if (ISO || d.eos == 0) Q.p = cs2 * r;
                if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                emit_to(d, out, o, i, row, Q);
            }
            o += pitch;
            pm = fm;
            pu = fu;
            pv = fv;
            pp = fp;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                q[0][m] = q[1][m];
                q[1][m] = q[2][m];
                q[2][m] = q[3][m];
                q[3][m] = q[4][m];
                q[4][m] = nx[m];
            }
        }
    }
}

// ================================================================== kicks
// Both half-kicks march along the rows like the azimuthal passes, lanes along the
// radius with one halo cell a side (30 outputs of 32): a row is loaded, predicted
// (kick 2) and exchanged with the neighbouring lanes once and stays in registers while
// it is the upper, the middle and the lower row of the 3 x 3 stress stencil.  The
// 32 x 8 tiles they replace predicted 340 cells for 256 outputs in two rounds and
// spent 460 (kick 1) and 880 (kick 2) instructions a cell, mostly on table loads and
// shared-memory addresses.
struct Column {  // the per-radius factors of a lane
    int i, ic;   // cell index, and clamped to the array for loads
    double rad, irad, gstar, nu;
    bool inside, output;
};
__device__ __forceinline__ Column column(const DiskView& d, int seg, int lane) {
    Column c;
    c.i = NPAD - 1 + KK_OUT * seg + lane;
    c.ic = min(c.i, d.xarr - 1);
    c.inside = c.i >= NPAD && c.i < NPAD + d.xres;
    c.output = c.inside && lane >= 1 && lane <= KK_OUT;
    c.rad = d.radx[c.ic];
    c.irad = d.irad[c.ic];
    c.gstar = d.geomx == 1 ? d.gstar[c.ic] : 0.0;
    c.nu = d.nux[c.ic];
    return c;
}
template <bool PLAIN = false>
__device__ __forceinline__ Grav row_gravity(const DiskView& d, const Column& c, int j, int which, const pg_body& pl,
                                            const pg_body& st) {
    if (!PLAIN && d.twobd) return body_gravity(d, c.ic, j, which, pl, st);
    const double* tr = d.trig + 4 * j + 2 * which;
    return gravity_at(d, c.gstar, c.rad, tr[0], tr[1], d.trig[4 * d.yarr + which], pl);
}
// u and v of one row at the lane's column and its two neighbours'
struct Row3 {
    double u[3], v[3], nr;  // left, own, right; own density times viscosity
};
__device__ __forceinline__ Row3 row3(double u, double v, double nr) {
    return Row3{{up1(u), u, down1(u)}, {up1(v), v, down1(v)}, nr};
}
// viscous force of the middle of three rows (viscous' stencil order: middle, lower, upper)
__device__ __forceinline__ void row_stress(const DiskView& d, const Column& c, int j, const Row3& lo, const Row3& mid,
                                           const Row3& hi, double& vx, double& vy) {
    const double u[9] = {mid.u[0], mid.u[1], mid.u[2], lo.u[0], lo.u[1], lo.u[2], hi.u[0], hi.u[1], hi.u[2]};
    const double v[9] = {mid.v[0], mid.v[1], mid.v[2], lo.v[0], lo.v[1], lo.v[2], hi.v[0], hi.v[1], hi.v[2]};
    const double nr[9] = {up1(mid.nr), mid.nr, down1(mid.nr), 0.0, lo.nr, 0.0, 0.0, hi.nr, 0.0};
    viscous(d.visx + 5 * c.ic, d.visy + 4 * j, u, v, nr, vx, vy);
}

template <bool VISC>
__global__ void __launch_bounds__(32 * SW_WARPS, 4)
    k_kick1(const Cell* __restrict__ in, const DiskView d, Cell* __restrict__ out, double* __restrict__ vis,
            const pg_dust* __restrict__ din, pg_dust* __restrict__ dout, int nseg, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double hdt = 0.5 * sc->dt;
    const pg_body pl = sc->planet_cur, star = sc->star_cur;
    const size_t pitch = 5 * (size_t)d.xarr;
    for (int item = blockIdx.x * SW_WARPS + warp; item < nitems; item += gridDim.x * SW_WARPS) {
        const Column c = column(d, item % nseg, lane);
        const int j0 = d.ypad + len * (item / nseg), j1 = min(j0 + len, d.ypad + d.yres);
        const double* next = reinterpret_cast<const double*>(in + c.ic) + pitch * (VISC ? j0 - 1 : j0);
        const Emitter emit_to(d, c.i);
        double* o = cell_at(d, out, c.ic, j0);
        double q[4], up[4], nx[4];  // the middle row, the one above and the next in flight: r, p, v_r, v_phi
        double w = 0.0, uw = 0.0, nw = 0.0;  // ... and in 1D v_z, zero in 2D
        Row3 lo{}, mid{}, hi{};
        int jl = VISC ? j0 - 1 : j0;             // the next row to load, and the last one
        const int jlast = VISC ? j1 : j1 - 1;
        auto fetch = [&]() {
            if (jl <= jlast) {
                load4(next, nx);
                if (!VISC && d.ndim == 1) nw = next[4];
            }
            next += pitch;
            ++jl;
        };
        auto enter = [&]() {
#pragma unroll
            for (int m = 0; m < 4; ++m) up[m] = nx[m];
            uw = nw;
            fetch();
            if (VISC) hi = row3(up[2], up[3], __dmul_rn(up[0], c.nu));
        };
        fetch();
        if (VISC) {
            enter();
            mid = hi;
        }
        enter();
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
#pragma unroll
            for (int m = 0; m < 4; ++m) q[m] = up[m];
            w = uw;
            const Grav g = row_gravity(d, c, j, 0, pl, star);
            double vx = 0.0, vy = 0.0;
            if (VISC) {
                lo = mid;
                mid = hi;
            }
            enter();
            if (VISC) {
                row_stress(d, c, j, lo, mid, hi, vx, vy);
            }
            double* const oj = o;
            o += pitch;
            if (!c.output) continue;
            if (VISC) {
                // the stress is kept for the predictor of kick2, with its periodic images
                double2* s = reinterpret_cast<double2*>(vis) + (size_t)c.i + (size_t)d.xarr * j;
                *s = double2{vx, vy};
                if (j < 2 * NPAD) s[(size_t)d.xarr * d.yres] = double2{vx, vy};
                else if (j >= d.yres) *(s - (size_t)d.xarr * d.yres) = double2{vx, vy};
            }
            const Cell C{q[0], q[1], q[2], q[3], w};
            Cell Q = kick<VISC>(d, C, c.irad, g, vx, vy, 0.0, hdt);
            if (d.cool) Q.p = p_cool(d, c.i, C.p, C.r, hdt);  // sweeps.cu:695-699
            emit_to(d, out, oj, c.i, j, Q);
            if (d.ave) accumulate_average(d, c.i, j, C, hdt);  // averaging(dev, 0.5 dt, T) before solve
            if (din) {  // dust half-kick: drag towards the gas cell C (sweeps.cu:626-707, mdt = 0)
                const DCell D = dust_kick(d, C, C.u, C.v, C.p, load_dust(din, d.xarr, c.i, j), g.gx, g.gy, g.gz,
                                          c.irad, 0.0, hdt);
                emit_dust(d, dout, c.i, j, D);
            }
        }
    }
}

// Kick 2 with damping and the CFL rate.  A row is predicted (sweeps.cu:713-729 with
// mdt = dt = dt/2) when it enters, with kick 1's stress and the bodies at t + dt; the
// corrector re-uses its gravity.
// PLAIN: no cooling, averages, dust or second body, whose code holds registers also where it
// does not run: 1024x3072 158 us with that code in, without it 190 / 150 / 140 / 175 at 2 / 3 /
// 4 / 5 CTAs per SM (at 4 92 bytes are spilled); the general instance, averaging, 260 / 209 / 244
// at 2 / 3 / 4.  Kick 1 has no such instance (87 us with and without that code).  The
// gas's sums of products are added by mad: both instances give the same bits, so a disk that
// averages or carries dust moves like one that does not.
template <bool VISC, bool PLAIN>
__global__ void __launch_bounds__(32 * SW_WARPS, PLAIN ? 4 : 3)
    k_kick2(const Cell* __restrict__ in, const double* __restrict__ vis, const DiskView d, Cell* __restrict__ out,
            const pg_dust* __restrict__ din, pg_dust* __restrict__ dout, int nseg, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt, hdt = 0.5 * dt;
    const pg_body pl = sc->planet_next, star = sc->star_next;
    const size_t pitch = 5 * (size_t)d.xarr;
    double vmax = 0.0;
    for (int item = blockIdx.x * SW_WARPS + warp; item < nitems; item += gridDim.x * SW_WARPS) {
        const Column c = column(d, item % nseg, lane);
        const int j0 = d.ypad + len * (item / nseg), j1 = min(j0 + len, d.ypad + d.yres);
        int jn = VISC ? j0 - 1 : j0;  // the next row to enter
        const double* next = reinterpret_cast<const double*>(in + c.ic) + pitch * jn;
        const double2* nvis = reinterpret_cast<const double2*>(vis) + (size_t)c.ic + (size_t)d.xarr * jn;
        const Emitter emit_to(d, c.i);
        double* o = cell_at(d, out, c.ic, j0);
        const int jlast = VISC ? j1 : j1 - 1;
        double q[4], up[4], nx[4];  // the middle row, the one above, the next in flight (with its stress)
        double2 nf{0.0, 0.0};
        double w = 0.0, uw = 0.0, nw = 0.0;  // v_z in 1D, zero in 2D
        auto fetch = [&](int j) {
            if (j <= jlast) {
                load4(next, nx);
                if (VISC) nf = *nvis;
                else if (d.ndim == 1) nw = next[4];
            }
            next += pitch;
            nvis += d.xarr;
        };
        Grav g{}, gup{};
        Row3 lo{}, mid{}, hi{};
        auto enter = [&]() {  // row jn into `up`, its prediction into `hi`
#pragma unroll
            for (int m = 0; m < 4; ++m) up[m] = nx[m];
            uw = nw;
            const double2 f = nf;
            fetch(jn + 1);
            // without stress the last call finds no row; in 1D the planet's table has none to read either
            if (VISC || jn <= jlast) gup = row_gravity<PLAIN>(d, c, jn, 1, pl, star);
            ++jn;
            if (!VISC) return;
            double u = up[2], v = up[3];
            if (c.inside) {
                const Cell P = kick<true>(d, Cell{up[0], up[1], u, v, 0.0}, c.irad, gup, f.x, f.y, hdt, hdt);
                u = P.u;
                v = P.v;
            }
            // radial ghosts of the predicted state (boundx2, src/boundary/boundary.cu:722-820): bound 0
            // keeps the analytic state; a copy or a reflection of the edge cell otherwise
            if (d.bound_lft != 0) {
                const double a = down1(u), b = down1(v);
                if (c.i == NPAD - 1) {
                    u = d.bound_lft == 2 ? -a : a;
                    v = b;
                }
            }
            if (d.bound_rgh != 0) {
                const double a = up1(u), b = up1(v);
                if (c.i == NPAD + d.xres) {
                    u = d.bound_rgh == 2 ? -a : a;
                    v = b;
                }
            }
            hi = row3(u, v, __dmul_rn(up[0], c.nu));
        };
        fetch(jn);
        enter();
        if (VISC) {
            mid = hi;
            enter();
        }
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
#pragma unroll
            for (int m = 0; m < 4; ++m) q[m] = up[m];
            w = uw;
            g = gup;
            double vx = 0.0, vy = 0.0;
            if (VISC) {
                lo = mid;
                mid = hi;
                enter();
                row_stress(d, c, j, lo, mid, hi, vx, vy);
            } else {
                enter();
            }
            double* const oj = o;
            o += pitch;
            if (!c.output) continue;
            const int i = c.i;
            const Cell C{q[0], q[1], q[2], q[3], w};
            double Tu = C.u, Tv = C.v;
            Cell Q = kick<VISC>(d, C, c.irad, g, vx, vy, hdt, hdt, &Tu, &Tv);
            // cooling over dt/2; the predictor cools over mdt = dt/2 as well, so Q.p is also
            // the predicted pressure the dust's second stopping time reads (sweeps.cu:668-699)
            if (!PLAIN && d.cool) Q.p = p_cool(d, i, C.p, C.r, hdt);
            const double Tp = Q.p;
            if (d.kill) {
                // killwave (src/killwave/killwave.cu:48-100): relax towards init_C
                const double* I = d.initx + 5 * i;
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const double tau = d.killx[4 * i + 2 * side + 1];
                    if (tau > 0.0) {
                        const double f = d.killx[4 * i + 2 * side] * (dt / tau);
                        Q.r = mad(f, I[0] - Q.r, Q.r);
                        Q.p = mad(f, I[1] - Q.p, Q.p);
                        Q.u = mad(f, I[2] - Q.u, Q.u);
                        Q.v = mad(f, I[3] - Q.v, Q.v);
                        if (!VISC) Q.w = mad(f, I[4] - Q.w, Q.w);
                    }
                }
            }
            if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
            if (!PLAIN && din) {  // dust corrector half-kick towards the predicted gas velocity (sweeps.cu:663-707)
                const DCell D = dust_kick(d, C, Tu, Tv, Tp, load_dust(din, d.xarr, i, j), g.gx, g.gy, g.gz, c.irad,
                                          hdt, hdt);
                emit_dust(d, dout, i, j, D);
                vmax = fmax(vmax, signal_rate(d, Q, i, j, &D));
            } else {
                vmax = fmax(vmax, signal_rate(d, Q, i, j));
            }
            emit_to(d, out, oj, i, j, Q);
            if (!PLAIN && d.ave) accumulate_average(d, i, j, Q, hdt);  // ... and after it
        }
    }
    block_max_to<32 * SW_WARPS>(&sc->vmax_bits, vmax);
}

// ================================================================ misc
__global__ void k_cfl(const DiskView d, const Cell* __restrict__ in, const pg_dust* __restrict__ din) {
    const long long n = (long long)d.xres * d.yres;
    double vmax = 0.0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(k % d.xres);
        const int j = d.ypad + (int)(k / d.xres);
        if (din) {
            const DCell D = load_dust(din, d.xarr, i, j);
            vmax = fmax(vmax, signal_rate(d, load_cell(in, d.xarr, i, j), i, j, &D));
        } else {
            vmax = fmax(vmax, signal_rate(d, load_cell(in, d.xarr, i, j), i, j));
        }
    }
    block_max_to<256>(&d.sc->vmax_bits, vmax);
}

__global__ void k_reset_vmax(Scalars* sc) { sc->vmax_bits = 0ull; }

// Opens a device-resident run without a host round trip.  main.cu:144 + 322:
// the first step after a (re)start is capped by end_time - t; after a clip at
// end_time the step the clip replaced caps the next one (main.cu:333-338, 425).
__global__ void k_run_begin(Scalars* sc, double end_time, int fresh) {
    if (fresh) sc->dt_prev = end_time - sc->t;
    else if (sc->dt_hold > 0.0) sc->dt_prev = sc->dt_hold;
    sc->dt_hold = 0.0;
    sc->end_time = end_time;
    sc->done = 0;
    sc->pad_ = 0;
}

// Per row, sin and cos of (azimuth - planet angle) for the planet of the first
// half-kick and for the planet at t+dt, and 1/x_p^2 of both (forces.cu:41-58).  By the
// one block whose first thread has just set the clock: as a launch of its own the table
// cost a step of the 126x389 disk 2 us.
__device__ __forceinline__ void planet_rows(const DiskView& d) {
    __syncthreads();
    const Scalars* sc = d.sc;
    const pg_body& a = sc->planet_cur;
    const pg_body& b = sc->planet_next;
    const double ya = a.y + 0.0 * a.vy, yb = b.y + 0.0 * b.vy;
    for (int j = threadIdx.x; j < d.yarr; j += blockDim.x) {
        double* t = d.trig + 4 * j;
        sincos(d.ycj[j] - ya, &t[0], &t[1]);
        sincos(d.ycj[j] - yb, &t[2], &t[3]);
        if (d.twobd) {
            double* u = d.strig + 4 * j;
            sincos(d.ycj[j] - (sc->star_cur.y + 0.0 * sc->star_cur.vy), &u[0], &u[1]);
            sincos(d.ycj[j] - (sc->star_next.y + 0.0 * sc->star_next.vy), &u[2], &u[3]);
        }
    }
    if (threadIdx.x == 0) {
        d.trig[4 * d.yarr] = 1.0 / a.x / a.x;
        d.trig[4 * d.yarr + 1] = 1.0 / b.x / b.x;
    }
}

// Host-supplied t, dt (pg_*_solve): planet for this step, reset of the signal-speed max.
__global__ void __launch_bounds__(1024) k_set_time(const DiskView d, double t, double dt, pg_body* planets) {
    pdl_enter();
    if (threadIdx.x == 0) {
        Scalars* sc = d.sc;
        sc->done = 0;
        sc->dt = dt;
        sc->planet_cur = sc->planet_next;
        sc->star_cur = sc->star_next;
        evolve_bodies(d, sc, t + dt);  // evolve_planet (solve.cu:264)
        sc->t = t + dt;
        sc->dt_prev = dt;
        sc->vmax_bits = 0ull;
        sc->steps += 1;
        if (planets) {  // recorded for the adjoint
            planets[0] = sc->planet_cur;
            planets[1] = sc->planet_next;
        }
    }
    planet_rows(d);
}

// Device-resident loop step of one disk (advance_clock).
__global__ void __launch_bounds__(1024) k_time_step(const DiskView d) {
    pdl_enter();
    if (threadIdx.x == 0) advance_clock(d);
    planet_rows(d);
}

__global__ void k_init_planet(const DiskView d, double a, double e, double rs, double t) {
    // init_planet (src/planet/planet.cu:319-402): one planet, or the star-planet
    // pair of the two-body frame (the star unsmoothed)
    pg_body b{}, s{};
    b.a = s.a = a;
    b.e = s.e = e;
    b.rs = 0.0;
    if (d.twobd) two_body_solution(d, s, b, t);
    else orbit_solution(d, b, t);
    b.rs = rs;
    d.sc->planet_next = b;
    d.sc->planet_cur = b;
    d.sc->star_next = s;
    d.sc->star_cur = s;
}

// Per-index tables evaluated with the device's own pow/sqrt/__sinf so they carry
// the same bits as the reference's device-side evaluations.
struct TabArgs {
    double sc_h, planet_radius, p_alpha, p_beta, ss_alpha, frame_omega;
    double xmin, xmax, kill_width, kill_width_out;
    int visc, orbadv, kill, init_flag, geomx;
};
__device__ inline double d_cs2(const TabArgs& a, double x) {  // init.cu:7-17
    double coeff = a.sc_h * a.sc_h * (1.0 / a.planet_radius);
    if (a.geomx == 0) return coeff;
    return coeff * pow(x / a.planet_radius, -a.p_beta);
}
__device__ inline double d_h(const TabArgs& a, double x) {  // init.cu:20-29
    if (a.geomx == 0) return a.sc_h;
    return sqrt(d_cs2(a, x) * pow(x, 3));
}
__device__ inline double d_nu(const TabArgs& a, double x) {  // init.cu:31-50
    if (!a.visc) return 0.0;
    double coeff = a.ss_alpha * sqrt(d_cs2(a, a.planet_radius)) * d_h(a, a.planet_radius);
    if (a.geomx == 0) return coeff;
    return coeff * pow(x / a.planet_radius, a.p_alpha);
}
__device__ inline double d_r(const TabArgs& a, double x) { return pow(x / a.planet_radius, -a.p_alpha) * 1.0; }
__device__ inline double d_p(const TabArgs& a, double x) { return d_cs2(a, x) * d_r(a, x); }
__device__ inline void d_initC(const TabArgs& a, double x, double* q) {  // init.cu:431-442 (init_flag 2)
    if (a.init_flag == 2) {
        q[0] = d_r(a, x);
        q[1] = d_p(a, x);
        q[2] = -1.5 * d_nu(a, x) / x;
        const double rho = d_r(a, x);
        const double dr = 1.1514178e-7;
        const double dP_dr = (d_p(a, x + dr) - d_p(a, x - dr)) / (2.0 * dr);
        q[3] = sqrt(1.0 / x + (x / rho) * dP_dr);
        q[4] = 0.0;
    } else {
        q[0] = 1.0; q[1] = 1.0; q[2] = 0.0; q[3] = 0.0; q[4] = 0.0;
    }
}
__device__ inline double ramping_fac(double x) {  // killwave.cu:8-14
    double f = __sinf(HPI * x);
    f *= f;
    return f;
}

__global__ void k_init_tables(const DiskView d, TabArgs a, double* radx, double* cs2x, double* nux, double* initx,
                              double* killx, double* rot, double* ycraw, double* ycj, double* xrec, double* yrec) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < d.xarr) {
        const double x = 0.5 * (d.xa[k + 1] + d.xa[k]);
        radx[k] = x;
        cs2x[k] = d_cs2(a, x);
        nux[k] = d_nu(a, x);
        d_initC(a, x, initx + 5 * k);
        // orb_rot (src/orbit/orbit.cu:57-69)
        if (rot) rot[k] = a.orbadv ? initx[5 * k + 3] - x * a.frame_omega : 0.0;
        // cooling time of cool_flag 1 (src/solver/cool/cool.cu:1-12, 15-27)
        if (d.coolx) const_cast<double*>(d.coolx)[k] = pow((a.geomx == 1) ? x : 1.0, 1.5) * d.beta_cool;
        const double d_in = d_h(a, a.xmin) * a.kill_width;
        const double d_out = d_h(a, a.xmax) * a.kill_width_out;
        const double inner = a.xmin + d_in;
        const double outer = a.xmax - d_out;
        double* kt = killx + 4 * k;
        kt[0] = kt[1] = kt[2] = kt[3] = 0.0;
        if (a.kill && k >= NPAD && k < NPAD + d.xres) {
            if (x < inner) {
                double f = (inner - x) / d_in;
                kt[1] = (a.geomx == 0) ? 1.0 : pow(x, 1.5);
                kt[0] = ramping_fac(f);
            }
            if (x > outer) {
                double f = (x - outer) / d_out;
                kt[3] = (a.geomx == 0) ? 1.0 : pow(x, 1.5);
                kt[2] = ramping_fac(f);
            }
        }
        // reciprocals and star gravity; xrec layout: idx_x, ixv, irad, gstar [xarr each], visx [5 xarr]
        xrec[k] = 1.0 / (d.xa[k + 1] - d.xa[k]);
        xrec[d.xarr + k] = 1.0 / d.xv[k];
        xrec[2 * d.xarr + k] = 1.0 / x;
        if (a.geomx == 1) {
            const double dis = sqrt(x * x + 0.0 * 0.0);
            xrec[3 * d.xarr + k] = -x / dis / dis / dis;  // forces.cu:203-204
        } else {
            xrec[3 * d.xarr + k] = 0.0;
        }
        double* vx = xrec + 4 * d.xarr + 5 * k;
        vx[0] = vx[1] = vx[2] = vx[3] = vx[4] = 0.0;
        if (k >= 1 && k + 1 < d.xarr) {
            const double r0 = 0.5 * (d.xa[k] + d.xa[k - 1]), r2 = 0.5 * (d.xa[k + 2] + d.xa[k + 1]);
            vx[0] = 1.0 / (r2 - r0);
            vx[1] = 1.0 / (r2 - x);
            vx[2] = 1.0 / (x - r0);
            vx[3] = 1.0 / (0.5 * (r2 - r0));
            vx[4] = 1.0 / x;
        }
    }
    if (k < d.yarr) {
        ycraw[k] = 0.5 * (d.ya[k + 1] + d.ya[k]);
        int jm = k;
        if (d.ndim > 1) {
            if (k < d.ypad) jm = k + d.yres;
            else if (k >= d.ypad + d.yres) jm = k - d.yres;
        }
        ycj[k] = 0.5 * (d.ya[jm + 1] + d.ya[jm]);
        // yrec layout: idx_y, iyv [yarr each], visy [4 yarr]
        yrec[k] = 1.0 / (d.ya[k + 1] - d.ya[k]);
        yrec[d.yarr + k] = 1.0 / d.yv[k];
        double* vy = yrec + 2 * d.yarr + 4 * k;
        vy[0] = vy[1] = vy[2] = vy[3] = 0.0;
        if (k >= 1 && k + 1 < d.yarr) {
            const double t0 = 0.5 * (d.ya[k] + d.ya[k - 1]), t1 = 0.5 * (d.ya[k + 1] + d.ya[k]);
            const double t2 = 0.5 * (d.ya[k + 2] + d.ya[k + 1]);
            vy[0] = 1.0 / (t2 - t0);
            vy[1] = 1.0 / (t2 - t1);
            vy[2] = 1.0 / (t1 - t0);
            vy[3] = 1.0 / (0.5 * (t2 - t0));
        }
    }
}

// Bound-0 radial ghosts hold init_C (src/boundary/boundary.cu:30-33, 56-59) in every
// row, of blockIdx.y consecutive buffers.
__global__ void k_init_xghosts(const DiskView d, Cell* buf) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 2 * NPAD * d.yarr) return;
    const int j = k / (2 * NPAD);
    const int n = k % (2 * NPAD);
    const int i = n < NPAD ? n : d.xres + n;
    const int bnd = n < NPAD ? d.bound_lft : d.bound_rgh;
    if (bnd != 0) return;
    const double* I = d.initx + 5 * i;
    store_cell(buf + (size_t)blockIdx.y * d.xarr * d.yarr, d.xarr, i, j, Cell{I[0], I[1], I[2], I[3], I[4]});
}

// boundy then boundx (src/boundary/boundary.cu:141-209, 13-62) on one buffer.
__global__ void k_bound_y(const DiskView d, Cell* buf) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (d.ndim < 2 || k >= d.xarr * NPAD) return;
    const int i = k % d.xarr, n = k / d.xarr;
    store_cell(buf, d.xarr, i, n, load_cell(buf, d.xarr, i, d.yres + n));
    store_cell(buf, d.xarr, i, d.yres + NPAD + n, load_cell(buf, d.xarr, i, NPAD + n));
}
__global__ void k_bound_x(const DiskView d, Cell* buf) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= d.yarr) return;
    const int nx = d.xres + NPAD;
    for (int n = 0; n < NPAD; ++n) {
        if (d.bound_lft == 2) {
            Cell c = load_cell(buf, d.xarr, 2 * NPAD - 1 - n, j);
            c.u *= -1.0;
            store_cell(buf, d.xarr, n, j, c);
        } else if (d.bound_lft == 1) {
            store_cell(buf, d.xarr, n, j, load_cell(buf, d.xarr, NPAD, j));
        }
        if (d.bound_rgh == 2) {
            Cell c = load_cell(buf, d.xarr, nx - 1 - n, j);
            c.u *= -1.0;
            store_cell(buf, d.xarr, nx + n, j, c);
        } else if (d.bound_rgh == 1) {
            store_cell(buf, d.xarr, nx + n, j, load_cell(buf, d.xarr, nx - 1, j));
        }
    }
}

// Torque of the planet on the disk (src/output/output.cu:336-412 with g_phi of
// src/output/forces.cu:39-57 at z = 0, 2D polar): one compensated partial sum of
// r g_phi Sigma dV per thread, summed per block, dV = (xa[i+1]^2 - xa[i]^2)/2 (ya[j+1] - ya[j]).
__global__ void k_torque(const DiskView d, const Cell* __restrict__ buf, double* part) {
    const pg_body p = d.sc->planet_next;
    const long long n = (long long)d.xres * d.yres;
    double sum = 0.0, comp = 0.0;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % d.xres), j = d.ypad + (int)(m / d.xres);
        const double rad = d.radx[i];
        double sinfac, cosfac;
        sincos(d.ycraw[j] - p.y, &sinfac, &cosfac);
        const double Rp = sqrt(rad * rad + p.x * p.x - 2.0 * p.x * rad * cosfac + p.rs * p.rs);
        const double rs_fac = 1.0 / Rp / Rp / Rp;
        // the planet's pull (output_gy, src/output/forces.cu:103-127): with the indirect
        // term, or as an inertial point mass in the two-body frame (global_sum(.., 1))
        const double gy = d.twobd ? -p.m * p.x * sinfac * rs_fac
                                  : -p.m * p.x * sinfac * rs_fac + p.m * sinfac / p.x / p.x;
        const double dv = 0.5 * (d.xa[i + 1] * d.xa[i + 1] - d.xa[i] * d.xa[i]) * (d.ya[j + 1] - d.ya[j]);
        const double y = rad * gy * (load_cell(buf, d.xarr, i, j).r * dv) - comp;
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

// ============================================================== launchers
static inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

cudaError_t set_kernel_attributes() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* f, size_t bytes) {
        cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (r != cudaSuccess) e = r;
        r = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (r != cudaSuccess) e = r;
    };
    set((const void*)k_sweep_x<true>, RX_SMEM);
    set((const void*)k_sweep_x<false>, RX_SMEM);
    return e;
}

void launch_init_tables(const DiskView& d, const pg_params& P, double* tab, cudaStream_t s) {
    TabArgs a{P.sc_h, P.planet_radius, P.p_alpha, P.p_beta, P.ss_alpha, P.frame_omega, P.xmin, P.xmax,
              P.kill_width, P.kill_width_out > 0.0 ? P.kill_width_out : P.kill_width,
              P.visc_flag, P.orbadv_flag, P.kill_flag, P.init_flag, P.geomx};
    // tab layout (doubles), see table_layout() in pg_engine.cu
    double* radx = tab;
    double* cs2x = radx + d.xarr;
    double* nux = cs2x + d.xarr;
    double* initx = nux + d.xarr;
    double* killx = initx + 5 * d.xarr;
    double* xrec = killx + 4 * d.xarr;    // 9 xarr
    double* ycraw = xrec + 9 * d.xarr;
    double* ycj = ycraw + d.yarr;
    double* yrec = ycj + d.yarr;          // 6 yarr
    const int n = d.xarr > d.yarr ? d.xarr : d.yarr;
    k_init_tables<<<cdiv(n, 128), 128, 0, s>>>(d, a, radx, cs2x, nux, initx, killx, const_cast<double*>(d.rot),
                                                ycraw, ycj, xrec, yrec);
}

void launch_torque(const DiskView& d, const Cell* buf, double* part, int nblocks, cudaStream_t s) {
    k_torque<<<nblocks, 256, 0, s>>>(d, buf, part);
}

void launch_init_xghosts(const DiskView& d, Cell* buf, cudaStream_t s, int nbuf) {
    k_init_xghosts<<<dim3(cdiv(2 * NPAD * d.yarr, 256), nbuf), 256, 0, s>>>(d, buf);
}

void launch_bound(const DiskView& d, Cell* buf, cudaStream_t s) {
    if (d.ndim > 1) k_bound_y<<<cdiv(d.xarr * NPAD, 256), 256, 0, s>>>(d, buf);
    if (d.bound_lft != 0 || d.bound_rgh != 0) k_bound_x<<<cdiv(d.yarr, 256), 256, 0, s>>>(d, buf);
}

void launch_cfl(const DiskView& d, const Cell* buf, cudaStream_t s, const pg_dust* dbuf) {
    k_reset_vmax<<<1, 1, 0, s>>>(d.sc);
    const long long n = (long long)d.xres * d.yres;
    unsigned blocks = cdiv(n, 256);
    if (blocks > 148u * 8u) blocks = 148u * 8u;
    k_cfl<<<blocks, 256, 0, s>>>(d, buf, dbuf);
}

// threads of the clock's block: up to 1024, the rows of the planet table
static unsigned clock_threads(const DiskView& d) { return d.yarr < 1024 ? (unsigned)(d.yarr + 31) / 32 * 32 : 1024; }
void launch_set_time(const DiskView& d, double t, double dt, cudaStream_t s, pg_body* planets) {
    launch_step(k_set_time, 1, clock_threads(d), 0, s, d, t, dt, planets);
}
void launch_run_begin(Scalars* sc, double end_time, bool fresh, cudaStream_t s) {
    k_run_begin<<<1, 1, 0, s>>>(sc, end_time, fresh ? 1 : 0);
}

void launch_time_step(const DiskView& d, cudaStream_t s) {
    launch_step(k_time_step, 1, clock_threads(d), 0, s, d);
}

void launch_init_planet(const DiskView& d, const pg_params& P, double t, cudaStream_t s) {
    const double a = P.planet_radius;
    const double rs = (P.ndim == 2) ? P.rs_fac * P.sc_h * a : P.rs_fac * pow(P.planet_mass / 3.0, 1.0 / 3.0) * a;
    k_init_planet<<<1, 1, 0, s>>>(d, a, P.planet_ecc, rs, t);
}

static int kernel_occupancy(const void* kernel, int threads, size_t smem);

static int sm_count() {
    static int nsm = 0;
    if (nsm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (nsm <= 0) nsm = 148;
    }
    return nsm;
}

// Persistent grid: as many CTAs as fit on the GPU at once (at most cps per SM
// when cps > 0), each looping over its work.
static unsigned persistent_grid(const void* kernel, int threads, size_t smem, long long ntiles, int cps = 0) {
    int per_sm = kernel_occupancy(kernel, threads, smem);
    if (cps > 0 && cps < per_sm) per_sm = cps;
    long long g = (long long)per_sm * sm_count();
    if (g > ntiles) g = ntiles;
    return (unsigned)(g < 1 ? 1 : g);
}

static int kernel_occupancy(const void* kernel, int threads, size_t smem) {
    // occupancy of each kernel, queried once (launches repeat every step)
    static const void* keys[128] = {nullptr};
    static int vals[128] = {0};
    int per_sm = 0;
    for (int n = 0; n < 128 && keys[n]; ++n)
        if (keys[n] == kernel) per_sm = vals[n];
    if (per_sm == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        for (int n = 0; n < 128; ++n)
            if (!keys[n]) {
                keys[n] = kernel;
                vals[n] = per_sm;
                break;
            }
    }
    return per_sm;
}

// the 2D isothermal instances of the sweeps and the advection apply
static bool iso_2d(const DiskView& d) { return d.eos == 0 && d.ndim == 2; }

// the instance of kick 2 without cooling, averages, dust and a second body applies
static bool plain_kick(const DiskView& d) { return !d.cool && !d.ave && !d.dust && !d.twobd; }

// Rows a warp of a pass takes one after the other: the tuned length, or the one of least
// run_cost (pg_internal.h).  1024x3072, us a pass at 4 / 8 / 16 / 24 / 48 / 64 / 96 rows:
// radial sweep 124 / 124 / 123 / 120 / 150 / 124 / 139, azimuthal 173 / 146 / 137 / 143 / 168 /
// 137 / 171 (1776 warps fit: 48 rows are 2048 runs, a full wave and a sixth), advection 84 /
// 82 / 78 / 77 / 74 / 90 / 124; with the rule's 64, 56 and 44 rows 124, 123 and 71.
static int pass_length(const Tune* t, int k, const void* kernel, size_t smem, int lines, int rows, double extra) {
    const int len = (t && k >= 0) ? SWEEP_LENGTHS[t->v[k]] : 0;
    if (len > 0) return len;
    const long long resident = (long long)SW_WARPS * sm_count() * kernel_occupancy(kernel, 32 * SW_WARPS, smem);
    return run_length(lines, rows, resident, extra);
}
// CTAs for `items` warps of work, at most what fits at once (cps > 0: at most cps per SM)
static unsigned sweep_grid(const void* kernel, size_t smem, long long items, int cps) {
    return persistent_grid(kernel, 32 * SW_WARPS, smem, (items + SW_WARPS - 1) / SW_WARPS, cps);
}

// one marching pass: runs of `lines` warps across the radius
template <class K, class... A>
static void march(const Tune* t, int k, int cps, K kernel, size_t smem, const DiskView& d, int lines, double extra,
                  cudaStream_t s, A... a) {
    const int len = pass_length(t, k, (const void*)kernel, smem, lines, d.yres, extra);
    const int items = lines * (int)cdiv(d.yres, len);
    launch_step(kernel, sweep_grid((const void*)kernel, smem, items, t ? t->cps[cps] : 0), 32 * SW_WARPS, smem, s, a...,
                lines, len, items);
}

void launch_sweep_x(const DiskView& d, const CellMaps& in, Cell* out, cudaStream_t s, const Tune* t) {
    const int n = (int)cdiv(d.xres, RX_OUT);
    if (iso_2d(d)) march(t, 0, 1, k_sweep_x<true>, RX_SMEM, d, n, 1.5, s, in.sx, d, out);
    else march(t, 0, 1, k_sweep_x<false>, RX_SMEM, d, n, 1.5, s, in.sx, d, out);
}
void launch_sweep_y(const DiskView& d, const Cell* in, Cell* out, cudaStream_t s, const Tune* t) {
    const int n = (int)cdiv(d.xres, 32);
    if (iso_2d(d)) march(t, 1, 2, k_sweep_y<true>, 0, d, n, 3.5, s, in, d, out);
    else march(t, 1, 2, k_sweep_y<false>, 0, d, n, 3.5, s, in, d, out);
}
void launch_advect(const DiskView& d, const Cell* in, Cell* out, cudaStream_t s, const Tune* t) {
    const int n = (int)cdiv(d.xres, 32);
    if (iso_2d(d)) march(t, 2, 3, k_advect<true>, 0, d, n, 3.5, s, in, d, out);
    else march(t, 2, 3, k_advect<false>, 0, d, n, 3.5, s, in, d, out);
}
void launch_kick1(const DiskView& d, const Cell* in, Cell* out, double* vis, cudaStream_t s, const pg_dust* din,
                  pg_dust* dout, const Tune* t) {
    const int n = (int)cdiv(d.xres, KK_OUT);
    if (d.visc && d.ndim == 2) march(t, -1, 0, k_kick1<true>, 0, d, n, 2.0, s, in, d, out, vis, din, dout);
    else march(t, -1, 0, k_kick1<false>, 0, d, n, 1.0, s, in, d, out, vis, din, dout);
}
void launch_kick2(const DiskView& d, const Cell* in, const double* vis, Cell* out, cudaStream_t s, const pg_dust* din,
                  pg_dust* dout, const Tune* t) {
    const int n = (int)cdiv(d.xres, KK_OUT);
    if (!(d.visc && d.ndim == 2)) march(t, -1, 4, k_kick2<false, false>, 0, d, n, 1.0, s, in, vis, d, out, din, dout);
    else if (plain_kick(d)) march(t, -1, 4, k_kick2<true, true>, 0, d, n, 2.5, s, in, vis, d, out, din, dout);
    else march(t, -1, 4, k_kick2<true, false>, 0, d, n, 2.5, s, in, vis, d, out, din, dout);
}

// CTAs per SM that fit for a pass (0 kick1, 1 sweep_x, 2 sweep_y, 3 advect, 4 kick2)
int pass_occupancy(const DiskView& d, int pass) {
    const bool vis = d.visc && d.ndim == 2, iso = iso_2d(d);
    constexpr int nt = 32 * SW_WARPS;
    switch (pass) {
        case 0: return kernel_occupancy(vis ? (const void*)k_kick1<true> : (const void*)k_kick1<false>, nt, 0);
        case 1: return kernel_occupancy(iso ? (const void*)k_sweep_x<true> : (const void*)k_sweep_x<false>, nt, RX_SMEM);
        case 2: return kernel_occupancy(iso ? (const void*)k_sweep_y<true> : (const void*)k_sweep_y<false>, nt, 0);
        case 3: return kernel_occupancy(iso ? (const void*)k_advect<true> : (const void*)k_advect<false>, nt, 0);
        default:
            if (!vis) return kernel_occupancy((const void*)k_kick2<false, false>, nt, 0);
            return kernel_occupancy(plain_kick(d) ? (const void*)k_kick2<true, true> : (const void*)k_kick2<true, false>, nt, 0);
    }
}

// threads per CTA of the sweeps and the CTAs per SM their registers were compiled for
void sweep_launch_shape(int* threads, int* minb) {
    *threads = 32 * SW_WARPS;
    *minb = 3;
}

int kernels_per_step(const DiskView& d) {
    if (tube_applies(d)) return 1;  // at most: the device loop's launch takes many steps
    int n = 1 /*clock and planet table*/ + 1 /*kick1*/ + 1 /*sweep x*/ + 1 /*kick2*/;
    if (d.ndim > 1) n += 1;
    if (d.ndim > 1 && d.orbadv) n += 1;
    if (d.dust) n += 1 + (d.ndim > 1 ? 1 : 0) + (d.ndim > 1 && d.orbadv ? 1 : 0);  // dust sweeps, advection
    return n;
}

}  // namespace pg

namespace pg {
// test support: the radial sweeps' bounded wait on tiles whose copies are never issued: the
// barriers of a warp's two stages expect `bytes` that nothing delivers, so the warp gives up
// after the wait's limit, PG_ERR_TIMEOUT is recorded and it leaves as the sweeps' warps do,
// after a wait for the other stage; nothing is in flight when it does.
__global__ void k_test_bounded_wait(Scalars* sc, uint32_t bytes, int* left) {
    __shared__ __align__(8) uint64_t bars[2][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* bar = bars[warp];
    if (lane == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncwarp();
    if (lane == 0) {
        issue_begin(&bar[0], bytes);
        issue_begin(&bar[1], bytes);
    }
    if (!warp_wait(&bar[0], 0, sc)) {
        if (lane == 0) mbar_wait(&bar[1], 0, sc);
        if (threadIdx.x == 0) *left = 1;
        return;
    }
    if (threadIdx.x == 0) *left = 2;  // the copy "landed": not expected
}

// test support: frac (pg_hydro.cuh)
__global__ void k_test_frac(const double* x, long long n, double* out) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const Frac f = frac(x[k]);
        out[2 * k] = f.h;
        out[2 * k + 1] = f.g;
    }
}
// test support: inv and rsq (pg_hydro.cuh)
__global__ void k_test_inv_rsq(const double* x, long long n, double* out) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        out[2 * k] = inv(x[k]);
        out[2 * k + 1] = rsq(x[k]);
    }
}
}  // namespace pg

extern "C" pg_status pg_test_bounded_wait(int* err_bits, int* left, float* ms) {
    if (!err_bits || !left || !ms) return PG_ERR_ARG;
    pg::Scalars* sc = nullptr;
    int* dleft = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t e = cudaMalloc(&sc, sizeof(pg::Scalars));
    if (e == cudaSuccess) e = cudaMalloc(&dleft, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(sc, 0, sizeof(pg::Scalars));
    if (e == cudaSuccess) e = cudaMemset(dleft, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e == cudaSuccess) {
        cudaEventRecord(e0);
        pg::k_test_bounded_wait<<<1, 64>>>(sc, 4096, dleft);
        e = cudaGetLastError();
        cudaEventRecord(e1);
    }
    if (e == cudaSuccess) e = cudaEventSynchronize(e1);
    if (e == cudaSuccess) e = cudaEventElapsedTime(ms, e0, e1);
    pg::Scalars h{};
    if (e == cudaSuccess) e = cudaMemcpy(&h, sc, sizeof(h), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(left, dleft, sizeof(int), cudaMemcpyDeviceToHost);
    *err_bits = h.err;
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(sc);
    cudaFree(dleft);
    return e == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}

// out2[2n] on the host from a kernel (x, n, out) over x[n]
static pg_status test_pairs(void (*kernel)(const double*, long long, double*), const double* x, long long n,
                            double* out2) {
    if (!x || !out2 || n <= 0) return PG_ERR_ARG;
    double *dx = nullptr, *dout = nullptr;
    if (cudaMalloc(&dx, n * sizeof(double)) != cudaSuccess) return PG_ERR_CUDA;
    if (cudaMalloc(&dout, 2 * n * sizeof(double)) != cudaSuccess) {
        cudaFree(dx);
        return PG_ERR_CUDA;
    }
    cudaError_t e = cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        kernel<<<592, 256>>>(dx, n, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out2, dout, 2 * n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dout);
    return e == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}
extern "C" pg_status pg_test_frac(const double* x, long long n, double* out2) {
    return test_pairs(pg::k_test_frac, x, n, out2);
}
extern "C" pg_status pg_test_inv_rsq(const double* x, long long n, double* out2) {
    return test_pairs(pg::k_test_inv_rsq, x, n, out2);
}
