// Launch interface of the fixed-point storage moments (vg_moments_fx.cu).
#pragma once

#include "vg_fx.cuh"

namespace vg {

// -log(c / 2^15) in Q56 and the 16-bit reciprocal c of a mantissa interval
struct FxLogEntry {
  long long l;
  int c, pad;
};
constexpr int FX_LOG_ENTRIES = 1024;
const FxLogEntry* fx_log_host();

// v, v^2 .. v^5: mantissas of 2^61 .. 2^62 split as fxw's components ([5][nv]), and by
// how much each exponent is below the largest of its power, e (16 bits each)
struct FxPowers {
  int e[5];
  const int4* drop;  // null: no tables, the moments in doubles
  const int2* mant;
};
// longest row the tables are made for (56 bytes a point)
constexpr int FX_MOMENTS_NV = 65536;
// the powers' scales, or false when a power is not finite or its scale is out of range
bool fx_powers_scale(const double* v, const double* v_pow, int nv, FxPowers* pw);
// the tables in mem (fx_powers_bytes), from the powers on the device
size_t fx_powers_bytes(int nv);
cudaError_t build_fx_powers(const double* v, const double* v_pow, int nv, void* mem, FxPowers* pw, cudaStream_t s);

// the moments of nrows rows into out[row * stride ..]: n, j, the second to fifth
// powers, f^2, f log f (full), or n, j, the second power, f^2, f log f
cudaError_t launch_moments_fx(const double* f, int nrows, int nv, const double* v, const double* v_pow, const FxPowers& pw,
                              const FxLogEntry* table, double dv, double* out, int stride, bool full, cudaStream_t s);

}  // namespace vg
