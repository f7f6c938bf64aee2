// The spectral Poisson solve as an exact circular sum (vg_poisson_fx.cu).
#pragma once

#include "vg_fx.cuh"

namespace vg {

// longest nx that is solved this way (a plan's table grows with nx, its set-up with nx^2)
constexpr int POISSON_FX_NX = 4096;

// One run's Green's function: g[nx] in Q62 of 2^*e, split as fxw's components
struct PoissonFx {
  const int2* g;
  const int* e;
};
// Builds n_runs tables of one nx: inv_kx[r] are DEVICE arrays of nx, g and e the
// runs' tables, work DEVICE scratch of nx doubles per run and nx more
cudaError_t build_poisson_fx(const double* inv_kx, int nx, int n_runs, int2* g, int* e, double* work, cudaStream_t s);

}  // namespace vg
