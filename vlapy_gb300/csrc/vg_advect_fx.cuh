// Launch interface of the fixed-point FP64 advection (vg_edfdv_fx.cu,
// vg_vdfdx_fx.cu; the arithmetic is in vg_fx.cuh).
#pragma once

#include <vector>

#include "vg_fx.cuh"
#include "vg_moments_fx.cuh"

namespace vg {

// The constant tables of the fixed-point kernels on the current device: the
// twiddles (FX_TABLE entries) and the logarithm's entries.  Plans and batches
// hold them together: the first to ask uploads them, the last to let go frees
// them (both under one lock).
struct FxTables {
  int device, refs;
  fxw* tw;
  FxLogEntry* log;
};
cudaError_t fx_tables_acquire(FxTables** out);
void fx_tables_release(FxTables* t);
// the step k1 of a wavenumber grid k[m] = m k1, h + l
struct FxStep {
  double h, l;
  float own;  // the largest modulus of fx_step_rest's
};
// turns per index and unit field or velocity of the phase ((-k) dt) c with k =
// m k1: A = -k1 dt / (2 pi) to 62 bits; false when it is not finite
bool fx_make_turn(FxStep k1, double dt, FxTurn* out);
// true when k[m] is m k[1] to a few roundings for m <= n / 2 (fftfreq's grid): the
// fixed-point phases step from index to index, by the grid's least-squares step
// (k[1]'s own rounding, taken m times, would be an error of up to 2^-53 of every phase
// beside those that the k[m] have)
bool fx_uniform(const double* k, int n, FxStep* k1);
// what is left of the wavenumbers k[0 .. n / 2] past the step, (k[m] - m k1) 2^64 / (2 pi)
std::vector<float> fx_step_rest(const double* k, int n, FxStep* k1);

// v-advection of nrows rows of nv (a power of two <= 8192); rest: fx_step_rest's
// of kv; tw64 for the row pairs that go through doubles
cudaError_t launch_edfdv_fx(double* f, int nrows, int nv, const double* e, FxTurn turn, const float* rest,
                            const fxw* tw, const cx<double>* tw64, cudaStream_t s);

// One run of the x-advection: f[nx][nv] at f + f_off
struct FxColRun {
  long long f_off;
  int nv;
  const double* v;
  const float* rest;  // fx_step_rest's of kx
  FxTurn turn;
};
// column pairs per CTA for nx (a power of two <= 8192) when `pairs` pairs are advanced together
int fx_col_pairs(int nx, long long pairs);
// x-advection: items null: run `one`, all its tiles; else (run, tile) items of
// one nx over runs, tiles of S pairs
cudaError_t launch_vdfdx_fx(double* f, int nx, const FxColRun* runs, const int2* items, int n_items, FxColRun one, int S,
                            const fxw* tw, const cx<double>* tw64, cudaStream_t s);

// Lines whose length N is not a power of two (vg_dft_fx.cu): n_lines lines of N
// elements es apart, line l at l ls with the phase ((-k) dt) c of its double c[l];
// angles: the N angles' table; rest: fx_step_rest's; scratch: dft_fx_scratch bytes for the larger of the directions
// a plan uses
size_t dft_fx_scratch(int nx, int nv, bool x, bool v);
cudaError_t build_dft_table(int N, const fxw* tw, fxw* out, cudaStream_t s);
cudaError_t launch_dft_fx(double* f, int N, int n_lines, long long es, long long ls, const double* c, FxTurn turn,
                          const float* rest, double dt, const fxw* tw, const fxw* angles, void* scratch, cudaStream_t s);

}  // namespace vg
