// Host-side declarations shared by the engine and the kernel launchers.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

#include "pg_common.cuh"

namespace pg {

// Rows a warp of the FP64 sweeps and the residual advection takes one after the other
// (pg_kernels.cu): the autotuner's variants.  0: run_length picks by the grid's size.
constexpr int NSWEEP_VARIANTS = 10;
constexpr int SWEEP_LENGTHS[NSWEEP_VARIANTS] = {0, 4, 6, 8, 12, 16, 24, 48, 64, 96};
// Time of `warps` runs of `rows` rows each (the extra rows at a run's ends included) in units
// of a row's time on a full GPU, where `resident` warps fit at once: whole waves of runs when
// there are more, and with fewer a row that is quicker for the idle issue slots, down to its
// latency.  The weights are those of the azimuthal sweeps measured from 126x389 to 1024x3072.
inline double run_cost(long long warps, long long resident, double rows) {
    if (warps <= resident) return rows * (0.55 + 0.45 * (double)warps / (double)resident);
    return rows * (double)((warps + resident - 1) / resident);
}
// The run length of least run_cost for `lines` warps across and `rows` rows of each line
inline int run_length(long long lines, int rows, long long resident, double extra) {
    int best = 2;
    double least = 1e300;
    for (int len = 2; len <= 64; len += (len < 16 ? 1 : 4)) {
        const double cost = run_cost(lines * ((rows + len - 1) / len), resident, len + extra);
        if (cost < least) {
            least = cost;
            best = len;
        }
    }
    return best;
}
constexpr int RX_TILE_CELLS = 36, RX_TILE_ROWS = 4;  // the radial sweep's TMA box

// Tensor map of one AoS cell buffer.
struct CellMaps {
    const void* base = nullptr;
    CUtensorMap sx;                        // box {5*36, 4}: the radial sweep
};
// Launch configuration of the FP64 passes (pg_disk_autotune).
struct Tune {
    int v[3] = {0, 0, 0};          // variant of sweep_x, sweep_y, advect (SWEEP_LENGTHS)
    int cps[5] = {0, 0, 0, 0, 0};  // CTAs per SM: kick1, sweep_x, sweep_y, advect, kick2 (0: all that fit)
};

// Pass inputs of one FP64 step, saved for its adjoint (pg_adjoint.cu).
struct StepRecord {
    Cell* stage[5];     // inputs of kick1, sweep_x, sweep_y, advect, kick2 (xarr*yarr AoS each; bound-0
                        // radial ghosts already in place)
    Cell* next;         // where kick2 leaves the new state: the next step's stage[0], or null (the disk's buffer)
    bool entered;       // stage[0] holds the step's input already
    double* vis;        // kick1's viscous force density (2 per cell, xarr*yarr)
    pg_body* planets;   // planet of the first half-kick, planet at t + dt
    double* res;        // orbital-advection residual speed per radius (xarr)
    int* inc;           // orbital-advection shift per radius (xarr)
};

// grid, slope weights and tensor maps (pg_engine.cu)
void make_grid(double* a, double* v, double amin, double amax, int res, int pad, int geom, int grid,
               const pg_params* P);
pg_status recon_weights(int geom, const double* dev_x, int ncell, double* w, cudaStream_t s);
pg_status make_map3_f64(CUtensorMap* m, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t b0,
                        uint32_t b1, uint32_t b2);

// the caller's planets array in and out of the device scalars (pg_engine.cu)
__global__ void k_grid_planet_in(Scalars* sc, const pg_body* planets, int twobd);
__global__ void k_grid_planet_out(const Scalars* sc, pg_body* planets, int twobd);
// the drop-in entry points with ndim 3 (pg_3d.cu)
pg_status check_params3(const pg_params* P);
pg_status grid3_init_orbadv(const pg_params& P, pg_grid* dev);
pg_status grid3_global_dt(const pg_params& P, pg_grid* dev, double dt_prev, double* dt_out);
pg_status grid3_solve(const pg_params& P, pg_grid* dev, double time, double dt);
void grid3_release();

// launch helpers (pg_kernels.cu)
void launch_init_tables(const DiskView& d, const pg_params& P, double* tab_base, cudaStream_t s);
void launch_init_xghosts(const DiskView& d, Cell* buf, cudaStream_t s, int nbuf = 1);
void launch_bound(const DiskView& d, Cell* buf, cudaStream_t s);
void launch_cfl(const DiskView& d, const Cell* buf, cudaStream_t s, const pg_dust* dbuf = nullptr);
void launch_set_time(const DiskView& d, double t, double dt, cudaStream_t s, pg_body* planets = nullptr);
void launch_time_step(const DiskView& d, cudaStream_t s);
void launch_run_begin(Scalars* sc, double end_time, bool fresh, cudaStream_t s);
void launch_kick1(const DiskView& d, const Cell* in, Cell* out, double* vis, cudaStream_t s,
                  const pg_dust* din = nullptr, pg_dust* dout = nullptr, const Tune* t = nullptr);
void launch_sweep_x(const DiskView& d, const CellMaps& in, Cell* out, cudaStream_t s, const Tune* t = nullptr);
void launch_sweep_y(const DiskView& d, const Cell* in, Cell* out, cudaStream_t s, const Tune* t = nullptr);
void launch_advect(const DiskView& d, const Cell* in, Cell* out, cudaStream_t s, const Tune* t = nullptr);
void launch_kick2(const DiskView& d, const Cell* in, const double* vis, Cell* out, cudaStream_t s,
                  const pg_dust* din = nullptr, pg_dust* dout = nullptr, const Tune* t = nullptr);
int pass_occupancy(const DiskView& d, int pass);
void sweep_launch_shape(int* threads, int* minb);
// the ghost rows of the periodic azimuth take the weights of the rows they image
void periodic_seam_weights(double* wy, int ypad, int yres);
void launch_init_planet(const DiskView& d, const pg_params& P, double t, cudaStream_t s);
void launch_torque(const DiskView& d, const Cell* buf, double* part, int nblocks, cudaStream_t s);
// compensated sum of n doubles in index order
double compensated_sum(const double* a, int n);
int kernels_per_step(const DiskView& d);
// many steps of a 1D cartesian tube in one launch (pg_tube.cu)
int tube_max_cluster();
bool tube_applies(const DiskView& d);
cudaError_t launch_tube(const DiskView& d, Cell* b0, Cell* b1, const Cell* in, int nsteps, double t, double dt,
                        cudaStream_t s);
void set_last_error(const char* msg);

// `planes` planes of `count` doubles, back to back in device memory, to host arrays
// (pg_hostcopy.cu), ordered after s's work; the caller synchronizes s.  The pinned staging
// (2 MB) is kept with the disk from its first large read on.
constexpr int COPY_THREADS = 4;
struct HostCopy {
    static constexpr size_t SLOT = (size_t)1 << 15;  // doubles
    double* pinned = nullptr;
    cudaEvent_t ev[COPY_THREADS][2] = {};
    HostCopy() = default;
    HostCopy(const HostCopy&) = delete;
    HostCopy& operator=(const HostCopy&) = delete;
    ~HostCopy();
    double* slot(int w, int k) const { return pinned + (2 * w + k) * SLOT; }
};
cudaError_t copy_planes_out(HostCopy& h, int device, const double* src, double* const* dst, int planes, size_t count,
                            cudaStream_t s);

// tables-only disks and FP32 tensor maps for the FP32 form (pg_engine.cu)
struct Engine;
// FP64 disks driven by the adjoint (pg_engine.cu)
Engine* disk_engine(pg_disk* d);
pg_status engine_set_state_device(Engine* E, double t, const double* r, const double* p, const double* u,
                                  const double* v);
pg_status engine_step(Engine* E, double t, double dt, const StepRecord* rec);
pg_status engine_save(Engine* E, Cell* cells, Scalars* sc);
pg_status engine_restore(Engine* E, const Cell* cells, const Scalars* sc, Cell* into = nullptr);
// the stream the engine launches on; returns the previous one
cudaStream_t engine_set_stream(Engine* E, cudaStream_t s);
pg_status engine_extract_device(Engine* E, double* r, double* p, double* u, double* v);
pg_status engine_run_pass(Engine* E, int pass, const Cell* in, Cell* out, const double* vis_in, double* vis_out);
pg_status table_engine_create(const pg_params* P, int device, cudaStream_t s, Engine** out);
void engine_destroy(Engine* E);
const DiskView& engine_view(const Engine* E);
void engine_init_planet(Engine* E, double t);
cudaError_t set_kernel_attributes();

// dust passes (pg_dust.cu)
void launch_dsweep_x(const DiskView& d, const pg_dust* in, pg_dust* out, cudaStream_t s);
void launch_dsweep_y(const DiskView& d, const pg_dust* in, pg_dust* out, cudaStream_t s);
void launch_dadvect(const DiskView& d, const pg_dust* in, pg_dust* out, cudaStream_t s);
void launch_dust_init(const DiskView& d, pg_dust* buf, cudaStream_t s);
void launch_dust_xghosts(const DiskView& d, pg_dust* buf, cudaStream_t s);
void launch_dust_images(const DiskView& d, pg_dust* buf, cudaStream_t s);
void launch_dust_fill(const DiskView& d, pg_dust* buf, const double* r, const double* u, const double* v,
                      cudaStream_t s);
void launch_dust_extract(const DiskView& d, const pg_dust* buf, double* r, double* u, double* v, cudaStream_t s);


namespace f32 {
struct View32;
// FP32-form launchers (pg_f32.cu); pass 0 kick1, 1 radial sweep, 2 azimuthal sweep,
// 3 advection, 4 kick2, reading buffer `in` and writing the other one
void launch_time32(const View32* V, int nd, cudaStream_t s);
// Launch configuration of the five FP32 passes (kick1, sweep x, sweep y, advect,
// kick2): which of the two lists of runs (0 or 1) and a CTAs-per-SM cap (0 = none).
struct Tune32 {
    int v[5];
    int cps[5];
};
// The runs of an ensemble's passes in device memory: per list (0 or 1) and kind (radial
// sweep; azimuthal sweep and advection; kicks) the first and how many.
struct Runs32 {
    int4* d;
    int first[2][3], count[2][3];
};
void launch_pass32(int pass, const View32* V, const Runs32& R, int in, cudaStream_t s, const Tune32& t);
void build_runs32(const int* xres, const int* yres, int nd, std::vector<int4>* runs, Runs32* R);
int pass_occupancy32(int pass);
void launch_cfl32(const View32* Vk, int b, cudaStream_t s);
void launch_dust_pass32(int pass, const View32* V, const Runs32& R, int in, cudaStream_t s);
void launch_dfill32(const View32* Vk, int b, const double* r, const double* u, const double* v, cudaStream_t s);
void launch_dextract32(const View32* Vk, int b, double* r, double* u, double* v, cudaStream_t s);
void launch_fill32(const View32* Vk, int b, const double* r, const double* u, const double* v, cudaStream_t s);
void launch_extract32(const View32* Vk, int b, double* r, double* p, double* u, double* v, cudaStream_t s);
void launch_totals32(const View32* Vk, int b, double* part, int nblocks, cudaStream_t s);
void launch_torque32(const View32* Vk, int b, double* part, int nblocks, cudaStream_t s);
void launch_init_tables32(const View32& w, float* tx, float* ty, double* cs64, cudaStream_t s);
}  // namespace f32

}  // namespace pg
