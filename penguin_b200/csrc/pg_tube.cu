// The device-resident loop of a 1D cartesian tube (ndim 1, geomx 0, no damping or
// cooling): many steps per launch, on one thread-block cluster.
//
// A tube's step is one sweep: without curvature, gravity and stress the half-kicks
// add zeros.  As one launch per pass it takes 16 us up to 7682 cells, launch gaps
// and the kernels' ramps, for work of under a microsecond.  Here every cell stays in
// shared memory from step to step; a step costs the latency of one cell's
// reconstruction, trace, HLLC flux and update plus one cluster barrier, which
// publishes the edge cells and the signal rate: 3.7 us at 1024 cells, 3300 us for the
// 897 steps of the Sod tube to t = 0.2.
//
// Layout: CTA k owns cells k m .. k m + m - 1 (m = 30 per warp) and holds three
// more on either side, copies of its neighbours' cells or the tube's ghosts.  Lane l
// of a warp computes the edge states of cell base + l - 1; the left face's flux
// takes the left neighbour's state by shuffle and the update the right face's flux,
// so 30 of 32 lanes have an output and no barrier is needed inside a step.  The
// states are double-buffered: a step reads one copy, writes the other, its own
// cells here and the copies of edge cells through distributed shared memory.
#include <cooperative_groups.h>

#include "pg_common.cuh"
#include "pg_hydro.cuh"
#include "pg_internal.h"
#include "pg_planet.cuh"

namespace cg = cooperative_groups;

namespace pg {

constexpr int TB_OUT = 30;                    // outputs per warp
constexpr int TB_MAXWARPS = 16;               // 512 threads: 128 registers
constexpr int TB_MAXCTAS = 16;
constexpr int TB_CELLS = TB_OUT * TB_MAXWARPS + 2 * NPAD;

struct TubeShared {
    double f[2][5][TB_CELLS];      // r, p, u, v, w of the CTA's cells and their halo, two copies
    double rate[2][TB_MAXCTAS];    // every CTA's largest signal rate
    double wmax[2][TB_MAXWARPS];
    int moving;                    // some transverse velocity is not zero
};

__device__ __forceinline__ double shfl_up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double shfl_down1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

__global__ void __launch_bounds__(32 * TB_MAXWARPS, 1)
    k_tube(const DiskView d, Cell* __restrict__ b0, Cell* __restrict__ b1, const Cell* __restrict__ in, int nsteps,
           double host_t, double host_dt) {
    __shared__ TubeShared S;
    cg::cluster_group cl = cg::this_cluster();
    Scalars* sc = d.sc;
    const bool host = host_dt != 0.0;  // one step of the caller's t and dt (k_set_time)
    if (sc->done && !host) return;  // the same for every CTA
    const int rank = (int)cl.block_rank(), nc = (int)cl.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int m = TB_OUT * nw, n = d.xres;
    const int lo = rank * m;              // first cell owned (interior index, 0 .. n-1)
    const int g = lo + TB_OUT * warp + lane - 1;  // this lane's cell
    const bool output = lane >= 1 && lane <= TB_OUT && g < n;

    // both copies of this CTA's window (cells beyond the far ghosts: the last ghost)
    if (tid == 0) S.moving = 0;
    __syncthreads();
    bool moving = false;
    for (int q = tid; q < m + 2 * NPAD; q += blockDim.x) {
        const Cell c = load_cell(in, d.xarr, min(lo + q, d.xarr - 1), d.ypad);
        for (int k = 0; k < 2; ++k) {
            S.f[k][0][q] = c.r;
            S.f[k][1][q] = c.p;
            S.f[k][2][q] = c.u;
            S.f[k][3][q] = c.v;
            S.f[k][4][q] = c.w;
        }
        moving = moving || c.v != 0.0 || c.w != 0.0;
    }
    cl.sync();  // S.moving of every CTA is cleared
    if (moving)
        for (int k = 0; k < nc; ++k) *cl.map_shared_rank(&S.moving, k) = 1;

    // cell q (interior index, ghosts beyond 0 .. n-1) into every window that holds it
    auto put = [&](int copy, int q, const Cell& c) {
        const int own = min(max(q, 0) / m, nc - 1);
        for (int k = max(own - 1, 0); k <= min(own + 1, nc - 1); ++k) {
            const int s = q - (k * m - NPAD);
            if (s < 0 || s >= m + 2 * NPAD) continue;
            double* f = (k == rank) ? &S.f[copy][0][s] : cl.map_shared_rank(&S.f[copy][0][s], k);
            f[0] = c.r;
            f[TB_CELLS] = c.p;
            f[2 * TB_CELLS] = c.u;
            f[3 * TB_CELLS] = c.v;
            f[4 * TB_CELLS] = c.w;
        }
    };

    const int gi = min(max(g + NPAD, 0), d.xarr - 1);  // array index of the lane's cell
    const int ws = TB_OUT * warp + lane - 1 + NPAD;    // its place in the window
    const double* wt = d.wx + 6 * gi;
    const double w0 = wt[0], w1 = wt[1], w2 = wt[2], w3 = wt[3], w4 = wt[4], w5 = wt[5];
    const double idx = d.idx_x[gi], ixv = d.ixv[gi], cs2 = d.cs2x[gi], gam = d.gam;
    double t = sc->t, dt_prev = sc->dt_prev, dt = sc->dt, dt_hold = sc->dt_hold, t_prev = t;
    const double end_time = sc->end_time;
    double vmax = __longlong_as_double((long long)sc->vmax_bits);
    int clipped = host ? 0 : sc->pad_, done = 0, taken = 0;
    Cell Q{};
    cl.sync();
    const bool trans = S.moving != 0;

    for (; taken < nsteps; ++taken) {
        const int c0 = taken & 1, c1 = c0 ^ 1;
        if (taken > 0) {
            vmax = 0.0;
            for (int k = 0; k < nc; ++k) vmax = fmax(vmax, S.rate[c0][k]);
        }
        // advance_clock (pg_planet.cuh): every thread holds the same clock
        if (host) {
            t = host_t;
            dt = host_dt;
        } else {
            if (clipped || t >= end_time) {
                done = 1;
                break;
            }
            const double dtc = d.cfl / vmax, lim = dt_prev * 1.1;
            dt = (dtc < lim) ? dtc : lim;
            if (t + dt > end_time) {
                dt_hold = dt;
                dt = end_time - t;
                clipped = 1;
            }
        }
        t_prev = t;
        t = t + dt;
        dt_prev = dt;

        const double* f = &S.f[c0][0][0] + min(max(ws, 2), m + 2 * NPAD - 3);
        const double w[6] = {w0, w1, w2, w3, w4, w5};
        auto rec = [&](int k, double flat) {
            const double* a = f + k * TB_CELLS;
            return recon(w, a[-2], a[-1], a[0], a[1], a[2], flat);
        };
        const double* p = f + TB_CELLS;
        const double* u = f + 2 * TB_CELLS;
        const Cell C0{f[0], p[0], u[0], f[3 * TB_CELLS], f[4 * TB_CELLS]};
        const double cs0 = sound_speed(gam, C0.r, C0.p);
        const double flat = flatten(p[0], p[-2], p[-1], p[1], p[2], u[-1], u[0], u[1]);
        const double sx = dt * 1.0 * idx;
        const Par R = rec(0, flat), P = rec(1, flat), U = rec(2, flat);
        Par A{0.0, 0.0, 0.0}, Z{0.0, 0.0, 0.0};
        if (trans) {
            A = rec(3, flat);
            Z = rec(4, flat);
        }
        const Half eL = state_at_left_edge(gam, sx, cs0, C0.r, C0.p, C0.u, R, P, U, A, Z);
        const Half eR = state_at_right_edge(gam, sx, cs0, C0.r, C0.p, C0.u, R, P, U, A, Z);
        Half L{shfl_up1(eR.r), shfl_up1(eR.p), shfl_up1(eR.u), 0.0, 0.0};
        if (trans) {
            L.v = shfl_up1(eR.v);
            L.w = shfl_up1(eR.w);
        }
        const Flux F = hllc(d.eos, d.ie, gam, L, eL);
        const double ff = dt * ixv;
        const double pres1 = shfl_down1(F.pres);
        Cell D;
        D.r = (F.r - shfl_down1(F.r)) * ff;
        D.u = ((F.u - shfl_down1(F.u)) + 0.5 * (1.0 + 1.0) * (F.pres - pres1)) * ff;
        double de = 0.0;
        if (d.eos == 2) {
            const double du = F.uprs - shfl_down1(F.uprs);
            de = (d.ie == 0) ? du : 0.5 * (F.pres + pres1) * du;
        }
        D.p = ((F.p - shfl_down1(F.p)) + de) * ff;
        D.v = D.w = 0.0;
        if (trans) {
            D.v = (F.v - shfl_down1(F.v)) * ff;
            D.w = (F.w - shfl_down1(F.w)) * ff;
        }
        double rate = 0.0;
        if (output) {
            Q = update_cell(d.eos, d.ie, gam, cs2, C0, D, &sc->floor_hits);
            if (!(Q.r > 0.0)) atomicOr(&sc->err, 1 << PG_ERR_NAN);
            rate = fmax((fabs(Q.u) + sound_speed(gam, Q.r, Q.p)) * idx, 0.0);
            S.f[c1][0][ws] = Q.r;
            S.f[c1][1][ws] = Q.p;
            S.f[c1][2][ws] = Q.u;
            S.f[c1][3][ws] = Q.v;
            S.f[c1][4][ws] = Q.w;
            // the copies that other CTAs hold, and the tube's ghosts (emit, pg_common.cuh)
            if (g - lo < NPAD || lo + m - 1 - g < NPAD || g >= n - NPAD) {
                put(c1, g, Q);
                Cell M = Q;
                M.u = -M.u;
                if (d.bound_lft == 1 && g == 0) {
                    for (int k = 1; k <= NPAD; ++k) put(c1, -k, Q);
                } else if (d.bound_lft == 2 && g < NPAD) {
                    put(c1, -1 - g, M);
                }
                if (d.bound_rgh == 1 && g == n - 1) {
                    for (int k = 0; k < NPAD; ++k) put(c1, n + k, Q);
                } else if (d.bound_rgh == 2 && g >= n - NPAD) {
                    put(c1, 2 * n - 1 - g, M);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rate = fmax(rate, __shfl_xor_sync(0xffffffffu, rate, o));
        if (lane == 0) S.wmax[c1][warp] = rate;
        __syncthreads();
        if (tid < nc) {  // this CTA's largest rate to every CTA
            double r = 0.0;
            for (int k = 0; k < nw; ++k) r = fmax(r, S.wmax[c1][k]);
            *cl.map_shared_rank(&S.rate[c1][rank], tid) = r;
        }
        cl.sync();
    }

    // the newest state into both buffers (either may be the one read next), ghosts included
    if (taken > 0 && output) {
        emit(d, b0, g + NPAD, d.ypad, Q);
        emit(d, b1, g + NPAD, d.ypad, Q);
    }
    if (rank == 0 && tid == 0) {
        if (taken > 0) {
            vmax = 0.0;
            for (int k = 0; k < nc; ++k) vmax = fmax(vmax, S.rate[taken & 1][k]);
            sc->vmax_bits = (unsigned long long)__double_as_longlong(vmax);
            sc->t = t;
            sc->dt = dt;
            sc->dt_prev = dt_prev;
            sc->dt_hold = dt_hold;
            sc->steps += taken;
            // the bodies are functions of time alone: those of the last two steps' ends
            if (taken > 1) evolve_bodies(d, sc, t_prev);
            sc->planet_cur = sc->planet_next;
            sc->star_cur = sc->star_next;
            evolve_bodies(d, sc, t);
        }
        if (!host) sc->pad_ = clipped;
        sc->done = done;
    }
}

// The launch of a tube of n cells: enough CTAs that each scheduler has one warp
// (120 cells a CTA), at most a cluster of 16, then more warps.
static bool tube_shape(int n, int maxc, int* nc, int* warps) {
    *nc = 1;
    while (*nc < maxc && *nc * 4 * TB_OUT < n) *nc *= 2;
    *warps = (n + *nc * TB_OUT - 1) / (*nc * TB_OUT);
    return *warps <= TB_MAXWARPS;
}

static cudaError_t tube_launch(const DiskView& d, int nc, int warps, Cell* b0, Cell* b1, const Cell* in, int nsteps,
                               double t, double dt, cudaStream_t s, int* clusters) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(32 * warps);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (clusters) return cudaOccupancyMaxActiveClusters(clusters, k_tube, &cfg);
    return cudaLaunchKernelEx(&cfg, k_tube, d, b0, b1, in, nsteps, t, dt);
}

// CTAs of the largest cluster of full CTAs that the current device runs: 16 where it grants
// the non-portable size, else 8, or 0 (no tube loop).  Asked when a tube is made, for its own
// device: the attribute that allows 16 belongs to the device's context.
int tube_max_cluster() {
    const bool big = cudaFuncSetAttribute(k_tube, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    for (int nc = big ? TB_MAXCTAS : 8; nc >= 8; nc /= 2) {
        int got = 0;
        if (tube_launch(DiskView{}, nc, TB_MAXWARPS, nullptr, nullptr, nullptr, 0, 0.0, 0.0, nullptr, &got) == cudaSuccess &&
            got > 0)
            return nc;
    }
    cudaGetLastError();
    return 0;
}

// A tube whose half-kicks are identities, of a size that one cluster holds: 7680 cells with
// 16 CTAs take 4.9 us a step, 1024 cells 3.7; 7682 as separate launches 16.4.
bool tube_applies(const DiskView& d) {
    int nc, warps;
    return d.ndim == 1 && d.geomx == 0 && !d.kill && !d.cool && !d.ave && !d.dust && !d.twobd && d.tube > 0 &&
           tube_shape(d.xres, d.tube, &nc, &warps);
}

// nsteps of the device's clock, or with dt != 0 one step of the caller's t and dt
cudaError_t launch_tube(const DiskView& d, Cell* b0, Cell* b1, const Cell* in, int nsteps, double t, double dt,
                        cudaStream_t s) {
    int nc, warps;
    if (!tube_shape(d.xres, d.tube, &nc, &warps)) return cudaErrorInvalidConfiguration;
    return tube_launch(d, nc, warps, b0, b1, in, nsteps, t, dt, s, nullptr);
}

}  // namespace pg
