// Dust passes of the FP64 step (dust_flag): the radial and azimuthal dust
// sweeps (src/solver/dust/dust.cu:6-326; the azimuthal one writes each cell at
// its orbital-advection shifted row like the gas, src/orbit/orbit.cu:17-49) and
// the dust residual advection (src/solver/advection/advection.cu:175-357).
// The dust half-kicks are fused into the gas kick passes (pg_kernels.cu).
//
// The reference's dust reconstruction reads the recon_flag 6 flattening
// coefficient from shared memory that dust_flow / advection never write
// (src/solver/recon/PPM.cu:68-77); it is 0 here, which is what the reference
// computes when that memory holds zeros.
#include "pg_common.cuh"
#include "pg_dust.cuh"
#include "pg_hydro.cuh"
#include "pg_internal.h"

namespace pg {

// Lanes of a warp lie along the radius and the warp takes a run of rows one after the
// other, as in the gas's passes (pg_kernels.cu): neighbours come by shuffle (radial sweep)
// or stay in registers from the row before (azimuthal passes), no barrier and no shared
// memory.  Bound by FP64 issue and latency; with tiles of 32 x 4 cells whose phases met at
// barriers the sweeps and the advection of gas and dust took 133 us at 384x1024, with these
// 103.  Compiled for 4 CTAs per SM: at 5 the azimuthal sweep spills (38 -> 41 us with the
// gas's, the advection 28 -> 30).  The w velocity is identically zero (dust runs in 2D) and
// stays as it is.
constexpr int DS_WARPS = 4;  // warps per CTA, independent of one another
constexpr int DS_THREADS = 32 * DS_WARPS;
constexpr int DS_OUT = 30;   // radial sweep: outputs of a warp's 32 cells

// src/solver/riemann/riemann.cu:5-11
__device__ __forceinline__ double gfac(int geom, double x) {
    if (geom == 1) return x;
    if (geom == 2) return x * x;
    return 1.0;
}

// A cell's states at one of its faces (dust_flux, dust.cu:6-103): mass density times the
// compression factor, normal and transported velocity.  SIDE 0: its left face, 1: its right.
struct DEdge {
    double r, u, a;
};
template <int SIDE>
__device__ __forceinline__ DEdge dust_edge(double sx, double uc, const Par& R, const Par& U, const Par& A) {
    auto ave = [](const Frac& f, const Par& p) { return SIDE == 0 ? aveL(f, p) : aveR(f, p); };
    // sx: swept fraction per unit speed; the traced positions of the reference enter only
    // as fractions of the cell
    const double m = (SIDE == 0 ? lesser(U.a - U.sL, 0.0) : larger(U.a + U.sR, 0.0)) * sx;
    const double un = ave(frac(lesser(SIDE == 0 ? -m : m, 1.0)), U);
    const Frac x = frac(lesser((SIDE == 0 ? -lesser(un, 0.0) : larger(un, 0.0)) * sx, 1.0));
    const double e = (SIDE == 0) ? exp_lim(sx * (un - uc) * inv(1.0 + m)) : exp_lim(sx * (uc - un) * inv(1.0 - m));
    return DEdge{ave(x, R) * e, ave(x, U), ave(x, A)};
}
struct DFlux {
    double r, u, a;
};
// limited mass flux and the upwind transport at a face between the cells of densities rL, rR
__device__ __forceinline__ DFlux dust_flux(double rL, double sxL, const DEdge& L, double rR, double sxR, const DEdge& R) {
    const double ml = lesser(rL * sxL, larger(L.u * L.r, 0.0));
    const double mr = larger(-rR * sxR, lesser(R.u * R.r, 0.0));
    return DFlux{ml + mr, ml * L.u + mr * R.u, ml * L.a + mr * R.a};
}
__device__ __forceinline__ double up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double down1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }
// r, v_r, v_phi of a cell
__device__ __forceinline__ void load3(const pg_dust* c, double& r, double& u, double& v) {
    const double2* q = reinterpret_cast<const double2*>(c);
    const double2 ru = q[0];
    r = ru.x;
    u = ru.y;
    v = q[1].x;
}

// ============================================================ dust sweeps
// Radial (fields r, u, r v): lane l holds cell 2 + 30 seg + l, lanes 1..30 update.
__global__ void __launch_bounds__(DS_THREADS, 4)
    k_dsweep_x(const pg_dust* __restrict__ in, const DiskView d, pg_dust* __restrict__ out, int nseg, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt;
    for (int item = blockIdx.x * DS_WARPS + warp; item < nitems; item += gridDim.x * DS_WARPS) {
        const int i = NPAD - 1 + DS_OUT * (item % nseg) + lane;
        const int c = min(i, d.xarr - 3);  // the stencil stays in the row
        const bool output = lane >= 1 && lane <= DS_OUT && i < NPAD + d.xres;
        const int j0 = d.ypad + len * (item / nseg), j1 = min(j0 + len, d.ypad + d.yres);
        double w[6], rad[5];
#pragma unroll
        for (int m = 0; m < 6; ++m) w[m] = d.wx[6 * c + m];
#pragma unroll
        for (int m = 0; m < 5; ++m) rad[m] = (d.geomx == 1) ? d.radx[c - 2 + m] : 1.0;
        const double sx = dt * d.idx_x[c], f = dt * d.ixv[c], irad = (d.geomx == 1) ? d.irad[c] : 1.0;
        const double g0 = gfac(d.geomx, d.xa[c]), g1 = gfac(d.geomx, d.xa[c + 1]), sxl = up1(sx);
        const pg_dust* src = in + c + (size_t)d.xarr * j0;
#pragma unroll 1
        for (int j = j0; j < j1; ++j, src += d.xarr) {
            double r[5], u[5], a[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) load3(src + m - 2, r[m], u[m], a[m]);
            const double v = a[2];
#pragma unroll
            for (int m = 0; m < 5; ++m) a[m] *= rad[m];
            const Par R = recon(w, r[0], r[1], r[2], r[3], r[4], 0.0);
            const Par U = recon(w, u[0], u[1], u[2], u[3], u[4], 0.0);
            const Par A = recon(w, a[0], a[1], a[2], a[3], a[4], 0.0);
            const DEdge b = dust_edge<0>(sx, u[2], R, U, A), e = dust_edge<1>(sx, u[2], R, U, A);
            const DFlux F = dust_flux(up1(r[2]), sxl, DEdge{up1(e.r), up1(e.u), up1(e.a)}, r[2], sx, b);
            const double Dr = (F.r * g0 - down1(F.r) * g1) * f;
            const double Du = (F.u * g0 - down1(F.u) * g1) * f;
            const double Da = (F.a * g0 - down1(F.a) * g1) * f * irad;
            if (output) {
                const DCell N = update_dust(d, DCell{r[2], u[2], v, 0.0}, DCell{Dr, Du, Da, 0.0});
                if (!(N.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                emit_dust(d, out, i, j, N);
            }
        }
    }
}

// the five rows of a lane's column that a marching pass holds, and the next one in flight
struct DColumn {
    double r[5], u[5], v[5], nr = 0.0, nu = 0.0, nv = 0.0;
    const pg_dust* next;
    int pitch;
    __device__ __forceinline__ DColumn(const pg_dust* first, int pitch_) : next(first), pitch(pitch_) {
#pragma unroll
        for (int m = 0; m < 5; ++m, next += pitch) load3(next, r[m], u[m], v[m]);
    }
    __device__ __forceinline__ void fetch() {
        load3(next, nr, nu, nv);
        next += pitch;
    }
    __device__ __forceinline__ void shift() {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            r[m] = r[m + 1];
            u[m] = u[m + 1];
            v[m] = v[m + 1];
        }
        r[4] = nr;
        u[4] = nu;
        v[4] = nv;
    }
};

// Azimuthal (fields r, v - orb_rot - r Omega, u) and the orbital shift.
__global__ void __launch_bounds__(DS_THREADS, 4)
    k_dsweep_y(const pg_dust* __restrict__ in, const DiskView d, pg_dust* __restrict__ out, int ncol, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt;
    for (int item = blockIdx.x * DS_WARPS + warp; item < nitems; item += gridDim.x * DS_WARPS) {
        const int i = NPAD + 32 * (item % ncol) + lane;
        const bool active = i < NPAD + d.xres;
        const int c = min(i, NPAD + d.xres - 1);
        const int s0 = NPAD + len * (item / ncol), s1 = min(s0 + len, NPAD + d.yres);
        double v0 = d.rot[c];
        if (d.geomy == 3) v0 += d.radx[c] * d.frame_omega;
        const double sdt = dt * ((d.geomy == 3) ? d.irad[c] : 1.0);
        int shift = 0;
        if (d.orbadv) {  // the gas's set_orbital_advection (orbit.cu:74-99): the same shift for the dust
            const double dy = d.dy0 * d.radx[c];
            shift = __double2int_rd(d.rot[c] * dt / dy + 0.5);
        }
        int js = (s0 - d.ypad + shift) % d.yres;  // TD[(j+inc) mod N] = CD[j] (orbit.cu:30-46)
        if (js < 0) js += d.yres;
        DColumn q(in + c + (size_t)d.xarr * (s0 - NPAD), d.xarr);
        DEdge pe{};  // the right edge of the cell below, its swept fraction per unit speed
        double psx = 0.0;
        DFlux pf{};  // the flux at the face below it
#pragma unroll 1
        for (int t = s0 - 1; t <= s1; ++t) {
            if (t < s1) q.fetch();
            double u[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) u[m] = q.v[m] - v0;
            const double* w = d.wy + 6 * t;
            const double sx = sdt * d.idx_y[t];
            const Par R = recon(w, q.r[0], q.r[1], q.r[2], q.r[3], q.r[4], 0.0);
            const Par U = recon(w, u[0], u[1], u[2], u[3], u[4], 0.0);
            const Par A = recon(w, q.u[0], q.u[1], q.u[2], q.u[3], q.u[4], 0.0);
            const DEdge b = dust_edge<0>(sx, u[2], R, U, A), e = dust_edge<1>(sx, u[2], R, U, A);
            const DFlux F = dust_flux(q.r[1], psx, pe, q.r[2], sx, b);
            if (t > s0) {  // the cell below has both its fluxes
                const double f = sdt * d.iyv[t - 1], Dr = (pf.r - F.r) * f;
                if (active) {
                    const DCell N = update_dust(d, DCell{q.r[1], q.u[1], q.v[1], 0.0},
                                                DCell{Dr, (pf.a - F.a) * f, (pf.u - F.u) * f + v0 * Dr, 0.0});
                    if (!(N.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    emit_dust(d, out, i, js + d.ypad, N);
                }
                if (++js == d.yres) js = 0;
            }
            pe = e;
            psx = sx;
            pf = F;
            q.shift();
        }
    }
}

// ===================================================== dust residual advection
// advection() on Dust (advection.cu:175-233) + advecty (:235-290): the gas's residual speed
// orb_res, fields (r, v, u), update_Dust.  The speed of a column has one sign: every row
// feeds the same one of its two faces.
__global__ void __launch_bounds__(DS_THREADS, 4)
    k_dadvect(const pg_dust* __restrict__ in, const DiskView d, pg_dust* __restrict__ out, int ncol, int len, int nitems) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Scalars* sc = d.sc;
    pdl_enter();
    if (sc->done) return;
    const double dt = sc->dt;
    for (int item = blockIdx.x * DS_WARPS + warp; item < nitems; item += gridDim.x * DS_WARPS) {
        const int i = NPAD + 32 * (item % ncol) + lane;
        const bool active = i < NPAD + d.xres;
        const int c = min(i, NPAD + d.xres - 1);
        const int s0 = NPAD + len * (item / ncol), s1 = min(s0 + len, NPAD + d.yres);
        const double speed = d.res[c], sdt = dt * ((d.geomy == 3) ? d.irad[c] : 1.0), sx = fabs(speed) * sdt;
        const bool up = speed > 0.0;  // a row is upwind of its upper face, else of its lower one
        DColumn q(in + c + (size_t)d.xarr * (s0 - NPAD), d.xarr);
        DFlux pf{};  // the flux that the row below fed
#pragma unroll 1
        for (int t = s0 - 1; t <= s1; ++t) {
            if (t < s1) q.fetch();
            const double* w = d.wy + 6 * t;
            const Frac x = frac(lesser(sx * d.idx_y[t], 1.0));
            auto ave = [&](const double* a) {
                const Par A = recon(w, a[0], a[1], a[2], a[3], a[4], 0.0);
                return up ? aveR(x, A) : aveL(x, A);
            };
            const double m = ave(q.r) * speed;
            const DFlux F{m, ave(q.u) * m, ave(q.v) * m};
            const int j = up ? t : t - 1;  // the row that has both its fluxes now
            if (active && j >= s0 && j < s1) {
                const double f = sdt * d.iyv[j];
                const DCell Q{up ? q.r[2] : q.r[1], up ? q.u[2] : q.u[1], up ? q.v[2] : q.v[1], 0.0};
                const DCell N = update_dust(d, Q, DCell{(pf.r - F.r) * f, (pf.u - F.u) * f, (pf.a - F.a) * f, 0.0});
                if (!(N.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                emit_dust(d, out, i, j, N);
            }
            pf = F;
            q.shift();
        }
    }
}

// ================================================================ misc
// init_CD everywhere (fill_grid, src/init/init.cu:502-519): the dust of a restart
// (the reference's load_grid reads the gas only, src/output/output.cu:182-248).
__global__ void k_dust_init(const DiskView d, pg_dust* buf) {
    const long long n = (long long)d.xarr * d.yarr;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(k % d.xarr), j = (int)(k / d.xarr);
        const double* I = d.initd + 4 * i;
        store_dust(buf, d.xarr, i, j, DCell{I[0], I[1], I[2], I[3]});
    }
}

// Bound-0 radial ghosts of a dust buffer: init_CD (boundx_dust,
// src/boundary/boundary.cu:64-113), every row.
__global__ void k_dust_xghosts(const DiskView d, pg_dust* buf) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 2 * NPAD * d.yarr) return;
    const int j = k / (2 * NPAD), n = k % (2 * NPAD);
    const int i = n < NPAD ? n : d.xres + n;  // 0..NPAD-1 and NPAD+xres..xarr-1
    const bool bound0 = (n < NPAD) ? d.bound_lft == 0 : d.bound_rgh == 0;
    if (!bound0) return;
    const double* I = d.initd + 4 * i;
    store_dust(buf, d.xarr, i, j, DCell{I[0], I[1], I[2], I[3]});
}

// The ghost images of every interior dust cell (boundy_dust and the bound 1/2
// radial ghosts), for a dust state written by the caller.
__global__ void k_dust_images(const DiskView d, pg_dust* buf) {
    const long long n = (long long)d.xres * d.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % d.xres), j = d.ypad + (int)(m / d.xres);
        emit_dust(d, buf, i, j, load_dust(buf, d.xarr, i, j));
    }
}

// Interior dust from host arrays (r, u, v) with its ghost images.
__global__ void k_dust_fill(const DiskView d, pg_dust* buf, const double* r, const double* u, const double* v) {
    const long long n = (long long)d.xres * d.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % d.xres), j = d.ypad + (int)(m / d.xres);
        emit_dust(d, buf, i, j, DCell{r[m], u[m], v[m], 0.0});
    }
}

__global__ void k_dust_extract(const DiskView d, const pg_dust* buf, double* r, double* u, double* v) {
    const long long n = (long long)d.xres * d.yres;
    for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
        const int i = NPAD + (int)(m % d.xres), j = d.ypad + (int)(m / d.xres);
        const DCell c = load_dust(buf, d.xarr, i, j);
        r[m] = c.r;
        u[m] = c.u;
        v[m] = c.v;
    }
}

// ============================================================== launchers
static inline unsigned dcdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// CTAs of a kernel that fit on the device
template <auto K>
static int dust_resident() {
    static const int n = [] {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 148;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K, DS_THREADS, 0) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        return sms * per_sm;
    }();
    return n;
}
// one marching pass: runs of `lines` warps across the radius, of the length of least run_cost
template <auto K>
static void march_dust(const DiskView& d, int lines, double extra, const pg_dust* in, pg_dust* out, cudaStream_t s) {
    const int fit = dust_resident<K>();
    const int len = run_length(lines, d.yres, (long long)DS_WARPS * fit, extra);
    const int items = lines * (int)dcdiv(d.yres, len), all = (int)dcdiv(items, DS_WARPS);
    launch_step(K, (unsigned)(all < fit ? all : fit), DS_THREADS, 0, s, in, d, out, lines, len, items);
}
void launch_dsweep_x(const DiskView& d, const pg_dust* in, pg_dust* out, cudaStream_t s) {
    march_dust<k_dsweep_x>(d, (int)dcdiv(d.xres, DS_OUT), 1.5, in, out, s);
}
void launch_dsweep_y(const DiskView& d, const pg_dust* in, pg_dust* out, cudaStream_t s) {
    march_dust<k_dsweep_y>(d, (int)dcdiv(d.xres, 32), 3.5, in, out, s);
}
void launch_dadvect(const DiskView& d, const pg_dust* in, pg_dust* out, cudaStream_t s) {
    march_dust<k_dadvect>(d, (int)dcdiv(d.xres, 32), 3.5, in, out, s);
}
void launch_dust_init(const DiskView& d, pg_dust* buf, cudaStream_t s) { k_dust_init<<<592, 256, 0, s>>>(d, buf); }
void launch_dust_xghosts(const DiskView& d, pg_dust* buf, cudaStream_t s) {
    k_dust_xghosts<<<(2 * NPAD * d.yarr + 255) / 256, 256, 0, s>>>(d, buf);
}
void launch_dust_images(const DiskView& d, pg_dust* buf, cudaStream_t s) { k_dust_images<<<592, 256, 0, s>>>(d, buf); }
void launch_dust_fill(const DiskView& d, pg_dust* buf, const double* r, const double* u, const double* v,
                      cudaStream_t s) {
    k_dust_fill<<<592, 256, 0, s>>>(d, buf, r, u, v);
}
void launch_dust_extract(const DiskView& d, const pg_dust* buf, double* r, double* u, double* v, cudaStream_t s) {
    k_dust_extract<<<592, 256, 0, s>>>(d, buf, r, u, v);
}

}  // namespace pg
