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

// Tiles of 32 outputs x 4 pencils: 160 threads and 25 KB of shared memory, so that 6
// CTAs per SM hide the FP64 latency the passes are bound by.  The w velocity is
// identically zero (dust runs in 2D) and stays as it is: three fields go through the
// phases.
constexpr int DS_LEN = 32, DS_W = DUST_W;
constexpr int DS_TL = DS_LEN + 2 * NPAD;               // 38
constexpr int DS_P1 = DS_LEN + 2, DS_P2 = DS_LEN + 1;  // cells with edge states, faces per pencil
constexpr int DS_THREADS = 160;
constexpr int DS_MINB = 5;
constexpr int DS_NST = DS_P1 * DS_W, DS_NFX = DS_P2 * DS_W;
static_assert(DS_NST <= DS_THREADS, "one cell per thread in each phase");
constexpr int DS_TILE = 4 * DS_TL * DS_W;              // doubles; a cell is 32 bytes, so any column starts a TMA box
constexpr int DS_STAGE = (DS_TILE + 15) / 16 * 16;     // 128-B aligned stages
constexpr size_t DS_SMEM = (size_t)(2 * DS_STAGE + 6 * DS_NST + 3 * DS_NFX) * 8 + 16 + 128;
constexpr int DA_NF = DS_TL * DS_W;                    // advection faces per tile
constexpr size_t DA_SMEM = (size_t)(2 * DS_STAGE + 3 * DA_NF) * 8 + 16 + 128;

// src/solver/riemann/riemann.cu:5-11
__device__ __forceinline__ double gfac(int geom, double x) {
    if (geom == 1) return x;
    if (geom == 2) return x * x;
    return 1.0;
}

// ============================================================ dust sweeps
// DIR 0: radial pencils of rows (fields r, u, r v); DIR 1: azimuthal pencils of
// columns (r, v - orb_rot - r Omega, u).
template <int DIR>
__global__ void __launch_bounds__(DS_THREADS, DS_MINB)
    k_dsweep(const __grid_constant__ CUtensorMap tm, const DiskView d, pg_dust* __restrict__ out, int ntx, int ntiles) {
    extern __shared__ __align__(128) double smem_raw[];
    double* smem = smem_base128(smem_raw);
    auto stage = [&](int n) { return smem + (n & 1) * DS_STAGE; };
    double* st = smem + 2 * DS_STAGE;  // [6][DS_NST]: right state of the left face, left state of the right face
    double* fl = st + 6 * DS_NST;      // [3][DS_NFX]
    uint64_t* bar = reinterpret_cast<uint64_t*>(fl + 3 * DS_NFX);
    __shared__ int s_inc[DS_W];
    Scalars* sc = d.sc;
    if (sc->done) return;
    const int tid = threadIdx.x;
    const double dt = sc->dt;
    const double* idx = (DIR == 0) ? d.idx_x : d.idx_y;  // one over a cell's width
    auto origin = [&](int tile, int& s0, int& q0) {
        s0 = NPAD + DS_LEN * (tile % ntx);
        q0 = (DIR == 0 ? d.ypad : NPAD) + DS_W * (tile / ntx);
    };
    auto issue = [&](int tile, int k) {
        int s0, q0;
        origin(tile, s0, q0);
        issue_begin(&bar[k & 1], DS_TILE * 8);
        if (DIR == 0) tma_load_2d(stage(k), &tm, 4 * (s0 - NPAD), q0, &bar[k & 1]);
        else tma_load_2d(stage(k), &tm, 4 * q0, s0 - NPAD, &bar[k & 1]);
    };
    // tile cell (position along the pencil t, pencil q) -> its 4 doubles
    auto cellp = [&](const double* T, int t, int q) { return T + ((DIR == 0) ? q * DS_TL + t : t * DS_W + q) * 4; };
    // dt over the pencil's radius (azimuthal sweeps: dust_flow, dust.cu:120-121)
    auto pencil_dt = [&](int q) { return dt * ((DIR == 1 && d.geomy == 3) ? d.irad[min(q, d.xarr - 1)] : 1.0); };
    pipe_init(bar);
    if ((int)blockIdx.x >= ntiles) return;
    if (tid == 0) issue(blockIdx.x, 0);
    int kt = 0;
    for (int tile_id = blockIdx.x; tile_id < ntiles; tile_id += gridDim.x, ++kt) {
        if (tid == 0 && tile_id + (int)gridDim.x < ntiles) issue(tile_id + gridDim.x, kt + 1);
        int s0, q0;
        origin(tile_id, s0, q0);
        const double* T = stage(kt);
        if (DIR == 1 && tid < DS_W) {
            // the gas's set_orbital_advection (orbit.cu:74-99): the same shift for the dust
            const int i = q0 + tid;
            int shift = 0;
            if (d.orbadv && i < NPAD + d.xres) {
                const double dy = d.dy0 * d.radx[i];
                shift = __double2int_rd(d.rot[i] * dt / dy + 0.5);
            }
            s_inc[tid] = shift;
        }
        if (!pipe_wait(bar, kt, sc)) {
            pipe_drain(bar, kt, tile_id + (int)gridDim.x < ntiles, sc);
            return;
        }

        // ---- P1: per cell, the state at its left face (seen from the right) and at
        // its right face (seen from the left), dust_flux (dust.cu:6-103)
        if (tid < DS_NST) {
            const int q = (DIR == 0) ? tid / DS_P1 : tid % DS_W;
            const int t = 2 + ((DIR == 0) ? tid % DS_P1 : tid / DS_W);
            const int s = s0 - NPAD + t;
            const int sc_ = (DIR == 0) ? min(s, d.xarr - 1) : min(s, d.yarr - 1);
            double v0 = 0.0;
            if (DIR == 1) {
                const int i = min(q0 + q, d.xarr - 1);
                v0 = d.rot[i];
                if (d.geomy == 3) v0 += d.radx[i] * d.frame_omega;
            }
            double r[5], u[5], a[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                // 16-byte loads: 8-byte ones at this 32-byte stride conflict 4 ways
                const double2* c = reinterpret_cast<const double2*>(cellp(T, t - 2 + m, q));
                const double2 ru = c[0], vw = c[1];
                r[m] = ru.x;
                u[m] = (DIR == 0) ? ru.y : vw.x - v0;
                a[m] = (DIR == 0) ? vw.x : ru.y;
                if (DIR == 0 && d.geomx == 1) a[m] *= d.radx[min(max(s - 2 + m, 0), d.xarr - 1)];
            }
            const double* wt = ((DIR == 0) ? d.wx : d.wy) + 6 * sc_;
            const Par R = recon(wt, r[0], r[1], r[2], r[3], r[4], 0.0);
            const Par U = recon(wt, u[0], u[1], u[2], u[3], u[4], 0.0);
            const Par A = recon(wt, a[0], a[1], a[2], a[3], a[4], 0.0);
            // swept fraction per unit speed: the traced positions of the reference enter
            // only as fractions of the cell
            const double sx = pencil_dt(q0 + q) * idx[sc_];
            // left face, from this cell
            double m = lesser(U.a - U.sL, 0.0) * sx;
            const double ur = aveL(frac(lesser(-m, 1.0)), U);
            Frac x = frac(lesser(-lesser(ur, 0.0) * sx, 1.0));
            double* o = st + tid;
            o[0] = aveL(x, R) * exp_lim(sx * (ur - u[2]) * inv(1.0 + m));
            o[DS_NST] = aveL(x, U);
            o[2 * DS_NST] = aveL(x, A);
            // right face, from this cell
            m = larger(U.a + U.sR, 0.0) * sx;
            const double ul = aveR(frac(lesser(m, 1.0)), U);
            x = frac(lesser(larger(ul, 0.0) * sx, 1.0));
            o[3 * DS_NST] = aveR(x, R) * exp_lim(sx * (u[2] - ul) * inv(1.0 - m));
            o[4 * DS_NST] = aveR(x, U);
            o[5 * DS_NST] = aveR(x, A);
        }
        __syncthreads();

        // ---- P2: limited mass flux and the upwind transport at every face
        if (tid < DS_NFX) {
            const int q = (DIR == 0) ? tid / DS_P2 : tid % DS_W;
            const int f = (DIR == 0) ? tid % DS_P2 : tid / DS_W;  // between tile cells 2+f and 3+f
            const double* R = st + ((DIR == 0) ? q * DS_P1 + f + 1 : (f + 1) * DS_W + q);
            const double* L = st + 3 * DS_NST + ((DIR == 0) ? q * DS_P1 + f : f * DS_W + q);
            const int sfc = min(s0 + f, (DIR == 0 ? d.xarr : d.yarr) - 1);  // face index = index of the right cell
            const double sdt = pencil_dt(q0 + q);
            const double rL = cellp(T, 2 + f, q)[0], rR = cellp(T, 3 + f, q)[0];
            const double ml = lesser(rL * sdt * idx[sfc - 1], larger(L[DS_NST] * L[0], 0.0));
            const double mr = larger(-rR * sdt * idx[sfc], lesser(R[DS_NST] * R[0], 0.0));
            fl[tid] = ml + mr;
            fl[DS_NFX + tid] = ml * L[DS_NST] + mr * R[DS_NST];
            fl[2 * DS_NFX + tid] = ml * L[2 * DS_NST] + mr * R[2 * DS_NST];
        }
        __syncthreads();

        // ---- P3: flux differences and update_Dust (dust.cu:149-235, 256-326)
        if (tid < DS_LEN * DS_W) {
            const int q = (DIR == 0) ? tid / DS_LEN : tid % DS_W;
            const int o = (DIR == 0) ? tid % DS_LEN : tid / DS_W;
            const int s = s0 + o, qq = q0 + q;
            const bool valid = (DIR == 0) ? (s < NPAD + d.xres && qq < d.ypad + d.yres)
                                          : (s < NPAD + d.yres && qq < NPAD + d.xres);
            if (valid) {
                const double* f0 = fl + ((DIR == 0) ? q * DS_P2 + o : o * DS_W + q);
                const double* f1 = f0 + ((DIR == 0) ? 1 : DS_W);
                const double g0 = (DIR == 0) ? gfac(d.geomx, d.xa[s]) : 1.0;
                const double g1 = (DIR == 0) ? gfac(d.geomx, d.xa[s + 1]) : 1.0;
                const double f = (DIR == 0) ? dt * d.ixv[s] : pencil_dt(qq) * d.iyv[s];
                auto net = [&](int k) { return (f0[k * DS_NFX] * g0 - f1[k * DS_NFX] * g1) * f; };
                const double* c = cellp(T, NPAD + o, q);
                const DCell Q{c[0], c[1], c[2], c[3]};
                const double Dr = net(0);
                if (DIR == 0) {
                    const double Da = net(2) * (d.geomx == 1 ? d.irad[s] : 1.0);
                    const DCell N = update_dust(d, Q, DCell{Dr, net(1), Da, 0.0});
                    if (!(N.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    emit_dust(d, out, s, qq, N);
                } else {
                    double v0 = d.rot[qq];
                    if (d.geomy == 3) v0 += d.radx[qq] * d.frame_omega;
                    const DCell N = update_dust(d, Q, DCell{Dr, net(2), net(1) + v0 * Dr, 0.0});
                    if (!(N.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                    int j = s;
                    if (d.orbadv) {  // TD[(j+inc) mod N] = CD[j] (orbit.cu:30-46)
                        int js = (s - d.ypad + s_inc[q]) % d.yres;
                        if (js < 0) js += d.yres;
                        j = js + d.ypad;
                    }
                    emit_dust(d, out, qq, j, N);
                }
            }
        }
        __syncthreads();
    }
}

// ===================================================== dust residual advection
// advection() on Dust (advection.cu:175-233) + advecty (:235-290): the gas's
// residual speed orb_res, fields (r, v, u), update_Dust.
__global__ void __launch_bounds__(DS_THREADS, DS_MINB)
    k_dadvect(const __grid_constant__ CUtensorMap tm, const DiskView d, pg_dust* __restrict__ out, int ntx, int ntiles) {
    extern __shared__ __align__(128) double smem_raw[];
    double* smem = smem_base128(smem_raw);
    auto stage = [&](int n) { return smem + (n & 1) * DS_STAGE; };
    double* fl = smem + 2 * DS_STAGE;  // [3][DA_NF] upwind fluxes, indexed by face t
    uint64_t* bar = reinterpret_cast<uint64_t*>(fl + 3 * DA_NF);
    Scalars* sc = d.sc;
    if (sc->done) return;
    const int tid = threadIdx.x;
    const double dt = sc->dt;
    auto origin = [&](int tile, int& s0, int& q0) {
        s0 = NPAD + DS_LEN * (tile % ntx);
        q0 = NPAD + DS_W * (tile / ntx);
    };
    auto issue = [&](int tile, int k) {
        int s0, q0;
        origin(tile, s0, q0);
        issue_begin(&bar[k & 1], DS_TILE * 8);
        tma_load_2d(stage(k), &tm, 4 * q0, s0 - NPAD, &bar[k & 1]);
    };
    pipe_init(bar);
    if ((int)blockIdx.x >= ntiles) return;
    if (tid == 0) issue(blockIdx.x, 0);
    int kt = 0;
    for (int tile_id = blockIdx.x; tile_id < ntiles; tile_id += gridDim.x, ++kt) {
        if (tid == 0 && tile_id + (int)gridDim.x < ntiles) issue(tile_id + gridDim.x, kt + 1);
        int s0, q0;
        origin(tile_id, s0, q0);
        const double* T = stage(kt);
        if (!pipe_wait(bar, kt, sc)) {
            pipe_drain(bar, kt, tile_id + (int)gridDim.x < ntiles, sc);
            return;
        }
        if (tid < DS_NST) {
            const int q = tid % DS_W, t = 2 + tid / DS_W;
            const int s = min(s0 - NPAD + t, d.yarr - 1);
            const int i = min(q0 + q, d.xarr - 1);
            const double speed = d.res[i];
            const double sdt = dt * ((d.geomy == 3) ? d.irad[i] : 1.0);
            const double* wt = d.wy + 6 * s;
            const Frac x = frac(lesser(fabs(speed) * (sdt * d.idx_y[s]), 1.0));
            const bool up = speed > 0.0;  // this cell is upwind of its upper face, else of its lower one
            double r[5], u[5], v[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                const double2* c = reinterpret_cast<const double2*>(T + ((t - 2 + m) * DS_W + q) * 4);
                const double2 ru = c[0];
                r[m] = ru.x;
                u[m] = ru.y;
                v[m] = c[1].x;
            }
            auto ave = [&](const double* a) {
                const Par A = recon(wt, a[0], a[1], a[2], a[3], a[4], 0.0);
                return up ? aveR(x, A) : aveL(x, A);
            };
            const double m = ave(r) * speed;
            double* o = fl + (t + (up ? 1 : 0)) * DS_W + q;
            o[0] = m;
            o[DA_NF] = ave(u) * m;
            o[2 * DA_NF] = ave(v) * m;
        }
        __syncthreads();
        if (tid < DS_LEN * DS_W) {
            const int q = tid % DS_W, o = tid / DS_W;
            const int s = s0 + o, i = q0 + q;
            if (s < NPAD + d.yres && i < NPAD + d.xres) {
                const int t = NPAD + o;
                const double* f0 = fl + t * DS_W + q;
                const double f = dt * d.iyv[s] * ((d.geomy == 3) ? d.irad[i] : 1.0);
                auto net = [&](int k) { return (f0[k * DA_NF] - f0[k * DA_NF + DS_W]) * f; };
                const double* c = T + (t * DS_W + q) * 4;
                const DCell N = update_dust(d, DCell{c[0], c[1], c[2], c[3]}, DCell{net(0), net(1), net(2), 0.0});
                if (!(N.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
                emit_dust(d, out, i, s, N);
            }
        }
        __syncthreads();
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

static unsigned dust_grid(const void* kernel, size_t smem, long long ntiles) {
    static int nsm = 0;
    if (nsm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (nsm <= 0) nsm = 148;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, DS_THREADS, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    long long g = (long long)per_sm * nsm;
    if (g > ntiles) g = ntiles;
    return (unsigned)(g < 1 ? 1 : g);
}

cudaError_t set_dust_attributes() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* f, size_t bytes) {
        cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (r != cudaSuccess) e = r;
    };
    set((const void*)k_dsweep<0>, DS_SMEM);
    set((const void*)k_dsweep<1>, DS_SMEM);
    set((const void*)k_dadvect, DA_SMEM);
    return e;
}

void launch_dsweep_x(const DiskView& d, const DustMaps& in, pg_dust* out, cudaStream_t s) {
    const int ntx = (int)dcdiv(d.xres, DS_LEN), nt = ntx * (int)dcdiv(d.yres, DS_W);
    k_dsweep<0><<<dust_grid((const void*)k_dsweep<0>, DS_SMEM, nt), DS_THREADS, DS_SMEM, s>>>(in.sweep_x, d, out, ntx, nt);
}
void launch_dsweep_y(const DiskView& d, const DustMaps& in, pg_dust* out, cudaStream_t s) {
    const int ntx = (int)dcdiv(d.yres, DS_LEN), nt = ntx * (int)dcdiv(d.xres, DS_W);
    k_dsweep<1><<<dust_grid((const void*)k_dsweep<1>, DS_SMEM, nt), DS_THREADS, DS_SMEM, s>>>(in.sweep_y, d, out, ntx, nt);
}
void launch_dadvect(const DiskView& d, const DustMaps& in, pg_dust* out, cudaStream_t s) {
    const int ntx = (int)dcdiv(d.yres, DS_LEN), nt = ntx * (int)dcdiv(d.xres, DS_W);
    k_dadvect<<<dust_grid((const void*)k_dadvect, DA_SMEM, nt), DS_THREADS, DA_SMEM, s>>>(in.sweep_y, d, out, ntx, nt);
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
