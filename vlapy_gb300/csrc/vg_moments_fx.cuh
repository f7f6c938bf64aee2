// Launch interface of the fixed-point storage moments (vg_moments_fx.cu).
#pragma once

#include <vector>

#include "vg_fx.cuh"

namespace vg {

// -log(c / 2^15) in Q56 and the 16-bit reciprocal c of a mantissa interval
struct FxLogEntry {
  long long l;
  int c, pad;
};
constexpr int FX_LOG_ENTRIES = 1024;
const FxLogEntry* fx_log_host();

// v, v^2 .. v^5 as Q62 fractions of 2^e, split as fxw's components, [5][nv]
struct FxPowers {
  int e[5];
};
// longest row the tables are made for (40 bytes a point)
constexpr int FX_MOMENTS_NV = 65536;
// false when a power is not finite or its scale is out of range
bool fx_powers_host(const double* v, const double* v_pow, int nv, std::vector<int2>* out, FxPowers* pw);

// the moments of nrows rows into out[row * stride ..]: n, j, the second to fifth
// powers, f^2, f log f (full), or n, j, the second power, f^2, f log f
cudaError_t launch_moments_fx(const double* f, int nrows, int nv, const int2* vp, const FxPowers& pw,
                              const FxLogEntry* table, double dv, double* out, int stride, bool full, cudaStream_t s);

}  // namespace vg
