// Internal plan layout and kernel launchers shared by the translation units.
#pragma once

#include <string>
#include <vector>

#include "vg_advect_fx.cuh"
#include "vg_common.cuh"
#include "vg_f32_plan.cuh"
#include "vg_fft.cuh"
#include "vg_moments_fx.cuh"
#include "vg_poisson_fx.cuh"
#include "vlagpu.h"

struct vg_plan {
  void* arena;  // the plan's device memory (all arrays below but the spline's)
  // scalars of the run
  int nx, nv, precision, collision, integrator, n_pulses;
  double dt, nu, dx, dv, dv_sq, nudt, root_most;
  int nx_pow2, nv_pow2;
  // device constants
  double* x;
  double* v;
  double* kx;
  double* kv;
  double* inv_kx;
  double* v_pow;     // [5][nv]
  double* f_bg;      // [nv] (delta-f background) or null
  vg_pulse* pulses;  // [n_pulses]
  vg::cx<double>* tw64;  // [FFT_NMAX]
  vg::cx<float>* tw32;   // [FFT_NMAX]
  // fixed-point advection: its table (null: none), the grids' steps, and whether
  // each wavenumber grid is uniform (else the transforms in doubles)
  vg::FxTables* fx_tables;
  vg::fxw* tw_fx;
  vg::FxStep kv1, kx1;
  int kv_uniform, kx_uniform;
  // what the wavenumbers are off their grid's step by
  float* rest_v;
  float* rest_x;
  // lengths that are not powers of two: their angle tables and the bins' scratch
  vg::fxw* dft_v;
  vg::fxw* dft_x;
  void* dft_work;
  // fixed-point storage moments: the velocity powers and the logarithm's table
  vg::FxPowers fx_pw;
  vg::FxLogEntry* fx_log;
  // Green's function of the Poisson solve (null: by transforms)
  int2* green;
  int* green_e;
  int* pw_v;   // NumPy pairwise tree over nv-1 trapz terms
  int* pw_x;   // NumPy pairwise tree over nx values (x-means)
  int pw_v_leaves, pw_x_leaves, pw_v_words, pw_x_words;
  int pw_v_levels;  // pw_v ends with the additions by height (pairwise_table)
  // scratch
  double* dens;   // [nx]
  double* mom;    // [nx][MOM_STRIDE]
  double* bb;     // Thomas elimination scratch, thomas_scratch doubles (null: none is needed; FP64 mode)
  double* rho;    // [nx]
  double* etmp;   // [nx]
  int* flags;     // status bits raised on the device (VG_FLAG_*; null: none kept)
  // semi-Lagrangian steps (allocated by their first call): spline second
  // derivatives [(nx + 2) * (nv + 2)] and the Thomas pivot table [max(nx, nv)]
  double* sl_m;
  double* sl_w;
  // graph cache and per-kernel profiling state
  void* graph_cache;
  void* prof;
  // FP32 delta-f state (null in FP64 mode)
  vg::F32Plan* f32;
};

namespace vg {

constexpr int MOM_STRIDE = 8;

// moment kinds for the pairwise-trapz row kernel
enum MomKind : int { MOM_ONE = 0, MOM_W = 1, MOM_SQ = 2, MOM_FLOGF = 3, MOM_DG2 = 4, MOM_V = 5 };
struct MomSpec {
  int nm;
  int kind[MOM_STRIDE];
  int arg[MOM_STRIDE];  // MOM_W: row of v_pow; MOM_DG2: index of the vbar moment
};

// Per-kernel event timing shared by plans and sweeps: while enabled, each
// launcher call is bracketed by two events on its stream.
struct ProfState {
  bool enabled = false;
  std::vector<cudaEvent_t> pool;
  size_t used = 0;
  struct Rec {
    int kind;
    cudaEvent_t b, e;
  };
  std::vector<Rec> recs;
  ~ProfState() {
    for (cudaEvent_t ev : pool) cudaEventDestroy(ev);
  }
  cudaEvent_t next() {
    if (used == pool.size()) {
      cudaEvent_t ev;
      if (cudaEventCreate(&ev) != cudaSuccess) return nullptr;
      pool.push_back(ev);
    }
    return pool[used++];
  }
};

template <typename Fn>
cudaError_t prof_call(ProfState* ps, int kind, cudaStream_t s, Fn fn) {
  if (!ps || !ps->enabled) return fn();
  cudaEvent_t b = ps->next(), e = ps->next();
  if (!b || !e) return cudaErrorMemoryAllocation;
  cudaError_t err = cudaEventRecord(b, s);
  if (err != cudaSuccess) return err;
  err = fn();
  if (err != cudaSuccess) return err;
  err = cudaEventRecord(e, s);
  ps->recs.push_back({kind, b, e});
  return err;
}

// Sum the recorded launches per kind into vg_prof_entry lines (clears the record).
int prof_collect(ProfState* ps, int n_kinds, const char* const* names, const double* bytes_per_launch,
                 vg_prof_entry* out, int max, int* n_out);

void set_error(const std::string& msg);
// NumPy's pairwise summation tree over n terms as [n_leaves, n_prog,
// (start, len) per leaf, post-order program] (leaf index, -1 = combine)
std::vector<int> pairwise_table(int n);
int cuda_status(cudaError_t err, const char* what);
// raise a kernel's dynamic shared-memory limit once (not a stream operation,
// so it is legal while a stream is being captured)
cudaError_t ensure_smem(const void* kernel, size_t bytes);

// longest line the direct-DFT advection takes (lengths that are not powers of
// two; its shared memory holds 5 N doubles)
constexpr int DFT_ADVECT_NMAX = 4096;

// launchers (return cudaError_t of the launch)
cudaError_t launch_edfdv_f64(const vg_plan& p, double* f, const double* e, double dt, cudaStream_t s);
cudaError_t launch_vdfdx_f64(const vg_plan& p, double* f, double dt, cudaStream_t s);
// alternative FP64 operators (vg_advect_alt_f64.cu); out of place
cudaError_t ensure_sl_scratch(vg_plan& p);
cudaError_t launch_vdfdx_sl_f64(const vg_plan& p, const double* fin, double* fout, double dt, cudaStream_t s);
cudaError_t launch_edfdv_sl_f64(const vg_plan& p, const double* fin, const double* e, double* fout, double dt,
                                cudaStream_t s);
cudaError_t launch_edfdv_cd2_f64(const vg_plan& p, const double* fin, const double* e, double* fout, double dt,
                                 cudaStream_t s);
// the storage moments of all rows (layout of launch_moments_fx), in fixed point
// where the plan has its tables, else in doubles
cudaError_t launch_storage_moments_f64(const vg_plan& p, const double* f, double* out, int stride, bool full,
                                       cudaStream_t s);
// the density, or the collision operators' moments (columns 0: vbar, 1: v0t^2;
// column 0 is not written for LB), as NumPy sums them
enum TrapzOp { TRAPZ_DENSITY = 0, TRAPZ_DG = 1, TRAPZ_LB = 2 };
cudaError_t launch_trapz_f64(const vg_plan& p, int op, const double* f, double* out, int stride, cudaStream_t s);
cudaError_t launch_row_moments_f64(const vg_plan& p, const double* f, const MomSpec& spec,
                                   double* out, int out_stride, cudaStream_t s);
// e = [driver or pulses(t)] + Re IFFT(i/kx FFT(rho)), rho = 1 - dens (dens_is_density) or dens
struct FieldTime {
  const double* t_ptr;  // device time value (time_batch + i) or null -> t_host
  double t_host;
  int nadd;
  double add[6];        // sub-step offsets added left to right
  int use_pulses;
};
cudaError_t launch_poisson_f64(const vg_plan& p, const double* dens, int dens_is_density,
                               const double* driver, const FieldTime& ft, double* e, cudaStream_t s);
// tridiagonal solve of rows with scratch of thomas_scratch doubles (it grows with nrows);
// nudt_row (per row, 0: leave the row as it is) or nudt for all; root_most: an upper
// estimate of the rows' mean of sqrt(nudt vth) (speed only)
cudaError_t launch_thomas_f64(double* f, int nrows, int nv, const double* v, const double* mom, int mstride,
                              int vbar_col, int vth_col, int dougherty, double nudt, const double* nudt_row,
                              double root_most, double dv, double dv_sq, double* scratch, cudaStream_t s);
// root_most of rows with a mean square root of nudt of `root`: 2 max|v| of it (vth <= n v^2, n <= 4)
double thomas_root_most(double root, const double* v, int nv);
// longest row whose chunked solve keeps all its arrays in shared memory, and
// longest row it takes at all
constexpr int THOMAS_SMEM_NV = 4096;
constexpr int THOMAS_CHUNK_NV = 8192;
// rows from which the one-thread-per-row solve fills the FP64 pipes itself (it
// spends fewer FP64 instructions, the chunked one needs fewer rows): 8192 x 1024
// 1.63 ms serial against 0.72 (nu 1e-4) to 1.01 ms (3e-3) in chunks, 16384 x
// 1024 1.72 against 1.45 to 2.01, 65536 x 1024 4.59 against 5.7 to 7.9; the same
// rows cross at nv = 256 (0.43 against 0.37 to 0.41 at 16384) and 2048
constexpr int THOMAS_SERIAL_ROWS = 12288;
// doubles per scratch array of a row: whole chunks of 32 for a whole number of warps
__host__ __device__ constexpr size_t thomas_pad(int nv) { return ((size_t)nv + 1023) / 1024 * 1024; }
// rows that may go either way, by their collisionality (see launch_thomas_f64)
constexpr bool thomas_either(int nrows, int nv) { return (long long)nrows * nv >= (1 << 20) || nv >= 4096; }
constexpr size_t thomas_scratch(int nrows, int nv) {
  return nv > THOMAS_SMEM_NV ? 2 * (size_t)nrows * thomas_pad(nv)
         : nv < 16 || nrows >= THOMAS_SERIAL_ROWS || thomas_either(nrows, nv) ? 2 * (size_t)nrows * nv
                                                                              : 0;
}
cudaError_t launch_storage_f64(const vg_plan& p, const double* f, const double* e, const double* de,
                               const vg_history& h, int i, cudaStream_t s);
cudaError_t launch_driver(const vg_plan& p, const FieldTime& ft, double* out, cudaStream_t s);
cudaError_t launch_twiddles(vg_plan& p, cudaStream_t s);

// FP32 delta-f path (vg_step_f32.cu)
cudaError_t launch_col_f32(const vg_plan& p, float* g, double dt, cudaStream_t s);
cudaError_t launch_field_f32(const vg_plan& p, const double* driver, const FieldTime& ft, double* e,
                             cudaStream_t s);
cudaError_t launch_dens_rows_f32(const vg_plan& p, const float* g, double* rho_out, int as_density,
                                 cudaStream_t s);
cudaError_t launch_poisson_only_f32(const vg_plan& p, const double* rho, const double* driver,
                                    const FieldTime& ft, double* e, cudaStream_t s);
cudaError_t launch_row_f32(const vg_plan& p, float* g, const double* e, double dt1, double dt2, int fp, int mom,
                           int n_modes, cudaStream_t s);
// FP32 copy of a caller-provided field for the kicks
cudaError_t launch_e_to_f32(const vg_plan& p, const double* e, cudaStream_t s);
cudaError_t launch_store_f32(const vg_plan& p, const float* g, const double* e, const double* de,
                             const vg_history& h, int i, int n_modes, cudaStream_t s);

}  // namespace vg
