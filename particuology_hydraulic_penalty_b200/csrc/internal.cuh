// Internal declarations shared by the .cu translation units of libpscb200.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>

#include <string>

#include "../../include/psc_b200.h"

namespace psc {

// Thread-local last-error slot behind psc_last_error(), and the number of
// errors set on this thread (a handle copies the message when it changes).
void set_error(const std::string& msg);
uint64_t error_seq();
const std::string& last_error_string();
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t err, const char* what);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per device).
int sm_count();

constexpr int STEP_THREADS = 256;

// launchers (return cudaError_t of the launch)
cudaError_t launch_step_exact(const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags, bool moving,
                              int grid_ctas, cudaStream_t stream);
cudaError_t launch_step_fast(int store, const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags,
                             bool moving, int cpt, int grid_ctas, cudaStream_t stream);
cudaError_t launch_step_tma(int store, const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags,
                            bool moving, int grid_ctas, int stages, uint32_t stage_bytes, cudaStream_t stream);
cudaError_t launch_step_pair(int store, const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags,
                             bool moving, int grid_ctas, cudaStream_t stream);
cudaError_t read_device_status(int* out, bool clear);
cudaError_t read_pair_status(int* out, bool clear);
cudaError_t read_loads_status(int* out, bool clear);
// Window sums of the step partials into out[nwin][PSC_NRED] and, where given, out2 (device or
// page-locked host memory).
cudaError_t launch_reduce_windows(const psc_window* d_windows, int nwin, double* out, cudaStream_t stream,
                                  double* out2 = nullptr);
// One check of the lbm_converge criterion (couple_psc_liggghts.py:284-296) on a window's mean u_z
// after step `step`, made with the sums of the state after it.
struct ConvergeCheck {
    const double* pre;   // the sums taken by step `step` (the state before it and its IMB momentum)
    double* state;       // [0] mean u_z of the last check, [1] its step, [2] converged, [3] stopping step,
                         // [4] residual; [kConvState ..) the two rows of sums of the stopping step
    psc_window* tab[2];  // the window's descriptors: marked inactive on convergence
    int step, min_steps, last;  // last: keep the rows whether or not the step converges
    double tol, cells;
};
constexpr int kConvState = 8;
// The sums of one window into out, then the check.
cudaError_t launch_reduce_converge(const psc_window* d_window, double* out, const ConvergeCheck& cc,
                                   cudaStream_t stream);
cudaError_t launch_init_equilibrium(int store, double scale, void* f, int64_t ncells, cudaStream_t stream);
// inlet = {rho, ux, uy, uz} when open_x (PSC_WIN_OPEN_X faces), else unused
cudaError_t launch_stream_push(int store, double scale, const void* src, double* dst, int nx, int ny, int nz,
                               cudaStream_t stream, bool open_x = false, const double* inlet = nullptr);
// A launch that may start before the kernel ahead of it on its stream has ended (chained): its CTAs take the
// SMs as they fall free and set up what that kernel does not write; then every CTA waits (chain_wait) before
// it touches anything else, and lets its own successor in only then, so at most two kernels
// of a stream overlap.  What the kernel ahead writes is read after the wait by ordinary loads only: the
// read-only path (ld.global.nc, const __restrict__) is for data that nothing in the chain writes.  A step in a row of steps: 64^3 FP32 8.9 -> 7.7 us,
// 75^3 FP32 12.0 -> 10.5, 24^3 exact 4.65 -> 3.86, 96^3 exact 55.8 -> 54.1 us.
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                                  bool chained, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
    return cudaGetLastError();
}
// Waits until the kernels ahead on the stream have ended and their results are visible; then the next one may
// take the SMs that this one leaves.
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

cudaError_t launch_stream_pull_store(int store, double scale, const double* src, void* dst, int nx, int ny, int nz,
                                     cudaStream_t stream, bool open_x = false, const double* inlet = nullptr);

// One window of a rebuild: its geometry, room for its load-chunk descriptors (launch_chunk_desc; written by the
// build) or null, page-locked room for its entry and chunk totals (written by the plan) or null, and
// the solid velocity [3][N] (us_type 0 = float64, 1 = float32).
struct GeoJob {
    psc_geometry g;
    double* desc;
    int64_t* host_totals;
    void* us;
    int32_t us_type;
};
constexpr int kGeoJobs = 12;  // kernel parameters of 4 KB
static_assert(kGeoJobs * sizeof(GeoJob) <= 4000, "kernel parameters");
cudaError_t launch_geometry_plan(const GeoJob* jobs, int count, cudaStream_t stream);
cudaError_t launch_geometry_build(const GeoJob* jobs, int count, cudaStream_t stream);
cudaError_t launch_solid_velocity(const GeoJob* jobs, int count, cudaStream_t stream);
// desc: the chunk descriptors of this geometry (launch_chunk_desc), or null: made on every call in the
// chunks' partial rows.  host_diag: page-locked copy of diag, or null.
cudaError_t launch_particle_loads(const psc_geometry& g, int imb_type, const void* imb, double* chunk_partials,
                                  const double* imb_sums, double* forces, double* torques, double* diag,
                                  cudaStream_t stream, const double* desc = nullptr, double* host_diag = nullptr);
// The load-chunk descriptors of one geometry, 6 doubles per chunk.
cudaError_t launch_chunk_desc(const psc_geometry& g, double* desc, cudaStream_t stream);

// Arrays of doubles to consecutive places of one array (page-locked host memory), in one launch per
// kRowCopies of them.
struct RowCopy {
    const double* src;
    int64_t at, n;
};
constexpr int kRowCopies = 128;
cudaError_t launch_copy_rows(const RowCopy* rows, int count, double* dst, cudaStream_t stream);

// One window of a many-window particle-loads launch (a device table).
struct LoadsJob {
    psc_geometry g;
    const void* imb;          // IMB field [3][N] of the window (one imb_type for all jobs)
    const double* imb_sums;   // sum of the IMB field (3)
    double* forces;           // [P][3]
    double* torques;          // [P][3]
    double* diag;             // [PSC_NDIAG]
    double* host_diag;        // page-locked copy of diag, or null
};
// Particle loads and load diagnostics of njobs windows, one launch per stage for all of them.
// d_chunk_base / d_particle_base: [njobs + 1] exclusive prefix sums of the
// jobs' chunk and particle counts (the totals are their last entries, also
// passed by value); part: total_chunks rows of 6 doubles.  all_lists: every
// job gives loads-list arrays (the list path: the lists of the jobs whose list
// is not current are built first); list_ready: every job's list is current.
// Without all_lists the loads are reduced over the whole boxes.  desc: room for the chunk descriptors
// (6 doubles per chunk), which hold what an earlier call with the same jobs wrote when desc_ready.
// max_particles: the largest particle count of a job.
cudaError_t launch_particle_loads_multi(const LoadsJob* d_jobs, const int64_t* d_chunk_base,
                                        const int64_t* d_particle_base, int njobs, int64_t total_chunks,
                                        int64_t total_particles, int imb_type, int max_subsamples,
                                        bool all_lists, bool list_ready, double* part, double* desc, bool desc_ready,
                                        int max_particles, cudaStream_t stream);

cudaError_t launch_adjoint_seed(const psc_adjoint_args& a, cudaStream_t stream);
cudaError_t launch_adjoint_step(const psc_adjoint_args& a, cudaStream_t stream);
cudaError_t launch_adjoint_geometry_grad(const psc_geometry& g, const psc_adjoint_args& a, double* part,
                                         double* grad, cudaStream_t stream);

cudaError_t launch_vox_spheres(const double* pts, int M, const double* lo, const double* dx, double radius, int nx,
                               int ny, int nz, uint8_t* solid, cudaStream_t s);
cudaError_t launch_bb_step(const double* src, double* dst, const uint8_t* solid, int nx, int ny, int nz, double tau,
                           double fx, double fy, double fz, unsigned flags, double* mom, cudaStream_t s);

cudaError_t launch_equilibrium(const double* rho, const double* ux, const double* uy, const double* uz, double* out,
                               int64_t n, cudaStream_t s);
cudaError_t launch_guo(double fx, double fy, double fz, const double* ux, const double* uy, const double* uz,
                       double tau, double* out, int64_t n, cudaStream_t s);

// exclusive scan of int32 counts -> int32 offsets, out has n + 1 entries
size_t scan_tmp_bytes(int64_t n);

}  // namespace psc
