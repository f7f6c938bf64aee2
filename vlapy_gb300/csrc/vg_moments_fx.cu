// Storage moments of the FP64 mode in fixed point: per row trapz(f v^p), p = 0 ..
// 5, trapz(f^2) and trapz(f log f) (vlapy/core/step.py:164-223).
//
// In doubles these eight moments are some 60 FP64 instructions per cell (a log is
// 30 of them), 64 cycles each and scheduler: 1.32 ms at 2048 x 4096 with the
// memory system idle.  Here a row is scaled to 64-bit integers by its own power of
// two (vg_fx.cuh), the velocity powers are Q62 fractions of their largest value,
// every product is three wide multiplies and every sum is exact (96 bits), so that
// only the products round, at 2^-60 of the row's maximum times the power's
// (NumPy's pairwise sums round at 2^-53 of the partial sums).  The density that the Poisson solve takes and the
// moments of the collision operator stay NumPy's own sums, bit for bit
// (k_row_moments_f64).
//
// log f: f = m 2^e with 1 <= m < 2; c = one of 1024 16-bit reciprocals of m, so
// that r = m c - 1 (exact in 64 bits) is below 2^-10.9, and log m = -log c + r -
// r^2 (1/2 - r/3 + r^2/4), the rest below 2^-57 (a table-driven logarithm in the
// manner of P. T. P. Tang, ACM Trans. Math. Softw. 16, 1990).
#include <algorithm>
#include <cmath>
#include <vector>

#include "vg_internal.cuh"
#include "vg_moments_fx.cuh"

namespace vg {

namespace {

struct Sum96 {
  long long hi, lo;  // hi 2^48 + lo
};
// the warp's sum, through its 32-bit adders in four parts of 24 bits
__device__ __forceinline__ Sum96 warp_sum(Acc96 s) {
  const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)(s.lo & 0xffffffu));
  const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)((s.lo >> 24) & 0xffffffu));
  const unsigned up = __reduce_add_sync(0xffffffffu, (unsigned)(s.lo >> 48) | (((unsigned)s.hi & 0xffu) << 16));
  const int hi = __reduce_add_sync(0xffffffffu, s.hi >> 8);
  return {((long long)hi << 24) + (long long)up, ((long long)mid << 24) + (long long)lo};
}
__device__ __forceinline__ double sum_to_double(Sum96 s) {
  return fma((double)s.hi, 281474976710656.0, (double)s.lo);  // 2^48
}

// log f - (E - 1023) log 2 in Q56 for f > 0 of a row of scale E, f >= 2^-60 of the largest
__device__ __forceinline__ long long log_q56(double f, int E, const FxLogEntry* __restrict__ table) {
  unsigned long long u = (unsigned long long)__double_as_longlong(f);
  int e = (int)(u >> 52);
  unsigned long long m = u & 0xfffffffffffffull;
  if (e == 0) {  // subnormal: bring the leading one to the implicit place
    const int z = __clzll((long long)m) - 11;
    m = (m << z) & 0xfffffffffffffull;
    e = 1 - z;
  }
  const FxLogEntry t = table[(unsigned)(m >> 42)];
  m |= 1ull << 52;
  const long long r = (long long)(m * (unsigned long long)t.c);  // (m c - 1) 2^67 modulo 2^64
  const long long r6 = r << 6;                                   // Q73
  const int rh = fx_hi(r6), rl = fx_lo(r6);
  const long long r2 = fx_rmul<0>(r6, rh, rl);                   // r^2, Q82
  const long long third = fx_rmul<0>(r6, fx_hi(1537228672809129301ll), fx_lo(1537228672809129301ll));  // r / 3, Q71
  const long long p = (1ll << 61) - (third >> 9) + (r2 >> 22);   // 1/2 - r/3 + r^2/4, Q62
  const long long q = fx_rmul<0>(r2, fx_hi(p), fx_lo(p));        // r^2 p, Q80
  return t.l + (r >> 11) - (q >> 24) + (long long)(e - E) * 49946518145322874ll;  // log 2 in Q56
}

// One CTA per row.  FULL: slots n, j, v^2 .. v^5, f^2, f log f; else n, j, v^2, f^2, f log f.
template <bool FULL>
__global__ void __launch_bounds__(256) k_moments_fx(const double* __restrict__ f, int nv, const int2* __restrict__ vp,
                                                    FxPowers pw, const FxLogEntry* __restrict__ table, double dv,
                                                    double* __restrict__ out, int stride) {
  constexpr int NP = FULL ? 6 : 3;       // velocity powers
  constexpr int NQ = NP + 2;
  __shared__ unsigned smax[8], sbad[8];
  __shared__ Sum96 part[NQ][8];
  const double* fr = f + (size_t)blockIdx.x * nv;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // scale of the row; a value that is not above zero makes the entropy NaN, as log f does
  unsigned mx = 0;
  bool low = false;
  for (int j = threadIdx.x; j < nv; j += blockDim.x) {
    const double x = fr[j];
    mx = max(mx, fx_exp_bits(x));
    low = low || !(__double_as_longlong(x) > 0);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  const unsigned anylow = __any_sync(0xffffffffu, low);
  if (lane == 0) {
    smax[w] = mx;
    sbad[w] = anylow;
  }
  __syncthreads();
  unsigned bad = 0;
  for (int q = 0; q < nw; ++q) {
    mx = max(mx, smax[q]);
    bad |= sbad[q];
  }
  const int E = fx_exp(mx);
  double* o = out + (size_t)blockIdx.x * stride;
  if (E == FX_NONFINITE) {
    // plain sums, for the infinities' and NaNs' sake: a thread per moment
    if (threadIdx.x < NQ) {
      const int q = threadIdx.x;
      double acc = 0.0;
      for (int j = 0; j < nv; ++j) {
        const double x = fr[j];
        double t = x;
        if (q >= 1 && q < NP) t = x * ldexp((double)(((long long)vp[(size_t)(q - 1) * nv + j].x << 32) + vp[(size_t)(q - 1) * nv + j].y), pw.e[q - 1] - 62);
        else if (q == NP) t = x * x;
        else if (q == NP + 1) t = x * log(x);
        acc += (j == 0 || j == nv - 1) ? 0.5 * t : t;
      }
      o[q] = dv * acc;
    }
    return;
  }
  Acc96 s[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q] = {0, 0};
  for (int j = threadIdx.x; j < nv; j += blockDim.x) {
    const double x = fr[j];
    const long long F = fx_from_double(x, E);
    const long long lg = (bad || F == 0) ? 0 : log_q56(x, E, table);
    const int half = (j == 0 || j == nv - 1) ? 1 : 0;  // the trapz weight of the ends
    acc_add(s[0], (F << 3) >> half);
#pragma unroll
    for (int p = 1; p < NP; ++p) {
      const int2 c = vp[(size_t)(p - 1) * nv + j];
      acc_add(s[p], fx_rmul<3>(F, c.x, c.y) >> half);
    }
    acc_add(s[NP], fx_rmul<3>(F, fx_hi(F), fx_lo(F)) >> half);
    acc_add(s[NP + 1], fx_rmul<3>(F, fx_hi(lg), fx_lo(lg)) >> half);
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const Sum96 t = warp_sum(s[q]);
    if (lane == 0) part[q][w] = t;
  }
  __syncthreads();
  if (threadIdx.x >= NQ) return;
  const int q = threadIdx.x;
  Sum96 t = part[q][0];
  for (int k = 1; k < nw; ++k) {
    t.hi += part[q][k].hi;
    t.lo += part[q][k].lo;
  }
  const double sum = nv < 2 ? 0.0 : dv * sum_to_double(t);
  // sums of 8 F, and of F V, F^2, F L over 2^61 (V in Q62 of 2^e, L in Q56)
  double r;
  if (q == 0) r = ldexp(sum, E - FX_SCALE - 3);
  else if (q < NP) r = ldexp(sum, E - FX_SCALE - 1 + pw.e[q - 1]);
  else if (q == NP) r = ldexp(ldexp(sum, E - FX_SCALE + 30), E - FX_SCALE + 31);
  else {
    Sum96 n = part[0][0];
    for (int k = 1; k < nw; ++k) {
      n.hi += part[0][k].hi;
      n.lo += part[0][k].lo;
    }
    const double nsum = dv * sum_to_double(n) * 0.125;
    r = ldexp(fma(nsum, (double)(E - 1023) * 0.69314718055994530942, sum * 32.0), E - FX_SCALE);
    if (nv < 2) r = 0.0;
    else if (bad) r = __longlong_as_double(0x7ff8000000000000ll);
  }
  o[q] = r;
}

// log(c / 2^15) by the series of 2 atanh((c - 2^15) / (c + 2^15)) in double-double
struct dd {
  double h, l;
};
dd dd_norm(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
dd dd_mul(dd a, dd b) {
  const double p = a.h * b.h;
  return dd_norm(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
dd dd_div(double a, double b) {
  const double q = a / b;
  return dd_norm(q, std::fma(-q, b, a) / b);
}
long long log_of(int c) {
  const dd z = dd_div((double)(c - 32768), (double)(c + 32768)), z2 = dd_mul(z, z);
  dd term = z, sum = z;
  for (int n = 3; n < 60; n += 2) {
    term = dd_mul(term, z2);
    const dd t = dd_mul(term, dd_div(1.0, (double)n));
    const dd s = dd_norm(sum.h, t.h);
    sum = dd_norm(s.h, s.l + (sum.l + t.l));
  }
  return 2 * ((long long)std::llrint(std::ldexp(sum.h, 56)) + (long long)std::llrint(std::ldexp(sum.l, 56)));
}

std::vector<FxLogEntry> build_log() {
  std::vector<FxLogEntry> t(FX_LOG_ENTRIES);
  for (int i = 0; i < FX_LOG_ENTRIES; ++i) {
    // the 16-bit reciprocal of the interval's middle, 2^15 / m
    const int c = (int)std::lround(32768.0 * 1024.0 / (1024.0 + i + 0.5));
    t[i] = {(long long)-log_of(c), c, 0};
  }
  return t;
}

}  // namespace

const FxLogEntry* fx_log_host() {
  static const std::vector<FxLogEntry> table = build_log();
  return table.data();
}

bool fx_powers_host(const double* v, const double* v_pow, int nv, std::vector<int2>* out, FxPowers* pw) {
  out->assign(5 * (size_t)nv, make_int2(0, 0));
  // v, then v^2, v^3, v^4, v^5 as v_pow's rows 1 .. 4 hold them
  for (int p = 0; p < 5; ++p) {
    const double* a = p == 0 ? v : v_pow + (size_t)p * nv;
    double mx = 0.0;
    for (int j = 0; j < nv; ++j) {
      if (!std::isfinite(a[j])) return false;
      mx = std::max(mx, std::fabs(a[j]));
    }
    int e = 0;
    std::frexp(mx, &e);
    if (mx == 0.0) e = 0;
    if (e > 900 || e < -900) return false;
    pw->e[p] = e;
    const double up = std::ldexp(1.0, 62 - e);
    for (int j = 0; j < nv; ++j) {
      const long long q = (long long)std::llrint(a[j] * up);
      (*out)[(size_t)p * nv + j] = make_int2(fx_hi(q), fx_lo(q));
    }
  }
  return true;
}

cudaError_t launch_moments_fx(const double* f, int nrows, int nv, const int2* vp, const FxPowers& pw,
                              const FxLogEntry* table, double dv, double* out, int stride, bool full, cudaStream_t s) {
  // four to eight elements a thread, whole warps
  const int block = nv >= 1024 ? 256 : nv >= 512 ? 128 : 64;
  if (full) k_moments_fx<true><<<nrows, block, 0, s>>>(f, nv, vp, pw, table, dv, out, stride);
  else k_moments_fx<false><<<nrows, block, 0, s>>>(f, nv, vp, pw, table, dv, out, stride);
  return cudaGetLastError();
}

}  // namespace vg
