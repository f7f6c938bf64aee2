// Storage moments of the FP64 mode in fixed point: per row trapz(f v^p), p = 0 ..
// 5, trapz(f^2) and trapz(f log f) (vlapy/core/step.py:164-223).
//
// In doubles these eight moments are some 60 FP64 instructions per cell (a log is
// 30 of them), 64 cycles each and scheduler: 1.32 ms at 2048 x 4096 with the
// memory system idle, here 0.16 (0.127 with one scale for a row and a power, see below;
// a row close to one: 0.58).
//
// Precision.  A factor is its mantissa, brought to [2^61, 2^62), and its exponent, so
// that a product (three wide multiplies) rounds at 2^-58 of itself; it is then shifted
// to the scale of the largest product of its row and power, which a first pass over the
// exponents finds, and added exactly (96 bits).  An error of a sum is therefore a few
// times 2^-59 of its own largest term, whatever the shape of the row, where a product
// of doubles rounds at 2^-53 of itself and NumPy's pairwise sums at 2^-53 of the
// partial sums.  (With one scale for a row and one for a power, max f max|v|^p, the
// fifth moment of a row of vth 0.3 on |v| < 6.4 was known to 1e-13 only.)  The values
// are not NumPy's bit for bit; the density that the Poisson solve takes and the moments
// of the collision operator are (k_trapz_f64).
//
// log f: f = m 2^e with 1 <= m < 2; c = one of 1024 16-bit reciprocals of m, so
// that r = m c - 1 (exact in 64 bits) is below 2^-10.9, and log m = -log c + r -
// r^2 (1/2 - r/3 + r^2/4), the rest below 2^-57 (a table-driven logarithm in the
// manner of P. T. P. Tang, ACM Trans. Math. Softw. 16, 1990).  It is good to some
// 2^-56, so a row whose f is close to one (sum f |log f| below a quarter of sum f)
// takes its entropy in doubles.
#include <algorithm>
#include <cmath>
#include <vector>

#include "vg_dd.cuh"
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
// rounded once, the same for every split of the rows over warps (the warps' lows add up
// to more than a double's 53 bits: carry first)
__device__ __forceinline__ double sum_to_double(Sum96 s) {
  return fma((double)(s.hi + (s.lo >> 48)), 281474976710656.0, (double)(s.lo & 0xffffffffffffll));  // 2^48
}

// A double as n 2^(e - 1084), |n| in [2^61, 2^62), or n = 0 with an exponent below all others
struct FxNum {
  long long n;
  int e;
};
constexpr int FX_ZERO_E = -16384;
__device__ __forceinline__ FxNum fx_num(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  int e = (int)((u >> 52) & 0x7ff);
  unsigned long long m = u & 0xfffffffffffffull;
  if (e) {
    m |= 1ull << 52;
  } else {
    if (m == 0) return {0, FX_ZERO_E};
    const int z = __clzll((long long)m) - 11;  // subnormal
    m <<= z;
    e = 1 - z;
  }
  const long long n = (long long)(m << 9);
  return {(long long)u < 0 ? -n : n, e};
}
// the exponent alone
__device__ __forceinline__ int fx_num_e(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  return e ? e : fx_num(x).e;
}
// a / 2^k rounded, k >= 0
__device__ __forceinline__ long long fx_shr(long long a, int k) {
  k = min(k, 62);
  return (a + ((1ll << k) >> 1)) >> k;
}

// log f - (e0 - 1023) log 2 in Q56 of f = num > 0
__device__ __forceinline__ long long log_q56(FxNum num, int e0, const FxLogEntry* __restrict__ table) {
  const unsigned long long m = (unsigned long long)num.n >> 9;  // 53 bits
  const FxLogEntry t = table[(unsigned)(m >> 42) & 1023u];
  const long long r = (long long)(m * (unsigned long long)t.c);  // (m c - 1) 2^67 modulo 2^64
  const long long r6 = r << 6;                                   // Q73
  const int rh = fx_hi(r6), rl = fx_lo(r6);
  const long long r2 = fx_rmul<0>(r6, rh, rl);                   // r^2, Q82
  const long long third = fx_rmul<0>(r6, fx_hi(1537228672809129301ll), fx_lo(1537228672809129301ll));  // r / 3, Q71
  const long long p = (1ll << 61) - (third >> 9) + (r2 >> 22);   // 1/2 - r/3 + r^2/4, Q62
  const long long q = fx_rmul<0>(r2, fx_hi(p), fx_lo(p));        // r^2 p, Q80
  return t.l + (r >> 11) - (q >> 24) + (long long)(num.e - e0) * 49946518145322874ll;  // log 2 in Q56
}

constexpr double LN2 = 0.69314718055994530942;

// One CTA per row.  FULL: slots n, j, v^2 .. v^5, f^2, f log f; else n, j, v^2, f^2, f log f.
// v, v_pow: the powers as doubles, for rows that are not finite.
template <bool FULL, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_moments_fx(const double* __restrict__ f, int nv, FxPowers pw,
                                                    const FxLogEntry* __restrict__ table, double dv,
                                                    const double* __restrict__ v, const double* __restrict__ v_pow,
                                                    double* __restrict__ out, int stride) {
  constexpr int NP = FULL ? 6 : 3;       // velocity powers
  constexpr int NQ = NP + 2;
  __shared__ int smax[NP][WARPS];
  __shared__ unsigned sbad[WARPS];
  __shared__ float ssize[WARPS];
  __shared__ Sum96 part[NQ][WARPS];
  __shared__ double red[WARPS];
  __shared__ int redo, top[NP];
  const double* fr = f + (size_t)blockIdx.x * nv;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // the largest exponent of f and of its products with the powers; a value that is not
  // above zero makes the entropy NaN, as log f does
  int mx[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) mx[p] = 2 * FX_ZERO_E;
  bool low = false;
  for (int j = threadIdx.x; j < nv; j += blockDim.x) {
    const double x = fr[j];
    const int e = fx_num_e(x);
    low = low || !(__double_as_longlong(x) > 0);
    mx[0] = max(mx[0], e);
    const int4 d = pw.drop[j];
    const int dd[3] = {d.x, d.y, d.z};
#pragma unroll
    for (int p = 1; p < NP; ++p) mx[p] = max(mx[p], e - ((dd[(p - 1) / 2] >> (16 * ((p - 1) & 1))) & 0xffff));
  }
  const unsigned anylow = __any_sync(0xffffffffu, low);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    mx[p] = __reduce_max_sync(0xffffffffu, mx[p]);
    if (lane == 0) smax[p][w] = mx[p];
  }
  if (lane == 0) sbad[w] = anylow;
  if (threadIdx.x == 0) redo = 0;
  __syncthreads();
  unsigned bad = 0;
  for (int q = 0; q < nw; ++q) {
#pragma unroll
    for (int p = 0; p < NP; ++p) mx[p] = max(mx[p], smax[p][q]);
    bad |= sbad[q];
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int p = 0; p < NP; ++p) top[p] = mx[p];
  }
  const int E = mx[0];
  double* o = out + (size_t)blockIdx.x * stride;
  if (E == FX_NONFINITE) {
    // plain sums, for the infinities' and NaNs' sake: a thread per moment
    if (threadIdx.x < NQ) {
      const int q = threadIdx.x;
      double acc = 0.0;
      for (int j = 0; j < nv; ++j) {
        const double x = fr[j];
        double t = x;
        if (q >= 1 && q < NP) t = x * (q == 1 ? v[j] : v_pow[(size_t)(q - 1) * nv + j]);
        else if (q == NP) t = x * x;
        else if (q == NP + 1) t = x * log(x);
        acc += (j == 0 || j == nv - 1) ? 0.5 * t : t;
      }
      o[q] = dv * acc;
    }
    return;
  }
  // logarithms against 2^(e0 - 1023): log f itself unless f is far from one.  All
  // f |log| <= 2^(E + 1 - 1023) (0.7 |E - e0| + 1.07) <= 2^(E - 1022 + up)
  const int far = abs(E - 1023) <= 40 ? abs(E - 1023) : 0, e0 = abs(E - 1023) <= 40 ? 1023 : E;
  const int up = far == 0 ? 1 : far <= 1 ? 1 : far <= 4 ? 2 : far <= 9 ? 3 : far <= 21 ? 4 : 5;
  Acc96 s[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q] = {0, 0};
  double xn = threadIdx.x < nv ? fr[threadIdx.x] : 0.0;  // (the next element, on its way)
  float size = 0.f;  // sum of f |log|, in units of 2^32 of its sum
  for (int j = threadIdx.x; j < nv; j += blockDim.x) {
    const FxNum F = fx_num(xn);
    xn = fr[min(j + (int)blockDim.x, nv - 1)];
    const int half = (j == 0 || j == nv - 1) ? 1 : 0;  // the trapz weight of the ends
    const int down = E - F.e;
    acc_add(s[0], fx_shr(F.n, down + half));
    const int4 d = pw.drop[j];
    const int dd[3] = {d.x, d.y, d.z};
#pragma unroll
    for (int p = 1; p < NP; ++p) {
      const int2 c = pw.mant[(size_t)(p - 1) * nv + j];
      const int drop = (dd[(p - 1) / 2] >> (16 * ((p - 1) & 1))) & 0xffff;
      acc_add(s[p], fx_shr(fx_rmul<0>(F.n, c.x, c.y), mx[p] - (F.e - drop) + half));
    }
    acc_add(s[NP], fx_shr(fx_rmul<0>(F.n, fx_hi(F.n), fx_lo(F.n)), 2 * down + half));
    if (!bad && down <= 70) {
      const long long lg = log_q56(F, e0, table);
      const int z = __clzll(lg < 0 ? -lg : lg) - 2;  // (62: lg is zero)
      const long long ln = z >= 0 ? lg << z : lg >> 1;
      const long long t = fx_rmul<0>(F.n, fx_hi(ln), fx_lo(ln));  // at least 2^58
      const int k = down + z - (8 - up) + half;                   // (-4 or more)
      const long long u = fx_shr(t << max(-k, 0), max(k, 0));     // at most 2^62
      acc_add(s[NP + 1], u);
      size += fabsf((float)(int)(u >> 32));
    }
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const Sum96 t = warp_sum(s[q]);
    if (lane == 0) part[q][w] = t;
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) size += __shfl_xor_sync(0xffffffffu, size, m);
  if (lane == 0) ssize[w] = size;
  __syncthreads();
  if (threadIdx.x < NQ) {
    const int q = threadIdx.x;
    Sum96 t = part[q][0];
    for (int k = 1; k < nw; ++k) {
      t.hi += part[q][k].hi;
      t.lo += part[q][k].lo;
    }
    const double sum = nv < 2 ? 0.0 : dv * sum_to_double(t);
    // f = F 2^(e - 1084), a product of two such numbers was divided by 2^64
    double r;
    if (q == 0) r = ldexp(sum, E - 1084);
    else if (q < NP) r = ldexp(sum, top[q] + pw.e[q - 1] - 2104);
    else if (q == NP) r = ldexp(sum, 2 * E - 2104);
    else {
      // F times a logarithm in Q56, divided by 2^64, times 2^(8 - up)
      r = ldexp(sum, E - 1084 + 64 - 56 - (8 - up));
      Sum96 n = part[0][0];
      for (int k = 1; k < nw; ++k) {
        n.hi += part[0][k].hi;
        n.lo += part[0][k].lo;
      }
      const double nsum = ldexp(dv * sum_to_double(n), E - 1084);
      if (e0 != 1023) r = fma(nsum, (double)(e0 - 1023) * LN2, r);
      if (nv < 2) r = 0.0;
      else if (bad) r = __longlong_as_double(0x7ff8000000000000ll);
      else if (e0 == 1023) {
        // the sum of f |log f| against a quarter of f's
        float a = 0.f;
        for (int k = 0; k < nw; ++k) a += ssize[k];
        redo = ldexp((double)a, 32 + 8 - (8 - up)) < 0.25 * fabs(sum_to_double(n));
      }
    }
    o[q] = r;
  }
  __syncthreads();
  if (!redo) return;
  // (logarithms near zero: the entropy in doubles)
  double acc = 0.0;
  for (int j = threadIdx.x; j < nv; j += blockDim.x) {
    const double x = fr[j], t = x * log(x);
    acc += (j == 0 || j == nv - 1) ? 0.5 * t : t;
  }
  for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if (lane == 0) red[w] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < nw; ++k) acc += red[k];
    o[NP + 1] = dv * acc;
  }
}

// the powers' mantissas and by how much their exponents are below the largest
__global__ void k_powers(const double* __restrict__ v, const double* __restrict__ v_pow, int nv, FxPowers pw, int4* drop,
                         int2* mant) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nv) return;
  int d[6] = {};
  for (int p = 0; p < 5; ++p) {
    const FxNum a = fx_num(p == 0 ? v[j] : v_pow[(size_t)p * nv + j]);
    mant[(size_t)p * nv + j] = make_int2(fx_hi(a.n), fx_lo(a.n));
    d[p] = min(pw.e[p] - a.e, 0xffff);
  }
  drop[j] = make_int4(d[0] | d[1] << 16, d[2] | d[3] << 16, d[4], 0);
}

// log(c / 2^15) by the series of 2 atanh((c - 2^15) / (c + 2^15)) in double-double
long long log_of(int c) {
  const dd z = dd_div({(double)(c - 32768), 0.0}, (double)(c + 32768)), z2 = dd_mul(z, z);
  dd term = z, sum = z;
  for (int n = 3; n < 60; n += 2) {
    term = dd_mul(term, z2);
    sum = dd_add(sum, dd_mul(term, dd_div({1.0, 0.0}, (double)n)));
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

bool fx_powers_scale(const double* v, const double* v_pow, int nv, FxPowers* pw) {
  // v, then v^2, v^3, v^4, v^5 as v_pow's rows 1 .. 4 hold them
  for (int p = 0; p < 5; ++p) {
    const double* a = p == 0 ? v : v_pow + (size_t)p * nv;
    double mx = 0.0;
    bool finite = true;
    for (int j = 0; j < nv; ++j) {
      finite = finite && std::isfinite(a[j]);
      mx = std::max(mx, std::fabs(a[j]));
    }
    if (!finite) return false;
    int e = 0;
    std::frexp(mx, &e);
    if (mx == 0.0) e = 0;
    if (e > 900 || e < -900) return false;
    pw->e[p] = e + 1022;  // the largest exponent field
  }
  return true;
}

size_t fx_powers_bytes(int nv) { return (size_t)nv * (sizeof(int4) + 5 * sizeof(int2)); }

cudaError_t build_fx_powers(const double* v, const double* v_pow, int nv, void* mem, FxPowers* pw, cudaStream_t s) {
  int4* drop = static_cast<int4*>(mem);
  int2* mant = reinterpret_cast<int2*>(drop + nv);
  pw->drop = drop;
  pw->mant = mant;
  k_powers<<<div_up(nv, 128), 128, 0, s>>>(v, v_pow, nv, *pw, drop, mant);
  return cudaGetLastError();
}

cudaError_t launch_moments_fx(const double* f, int nrows, int nv, const double* v, const double* v_pow, const FxPowers& pw,
                              const FxLogEntry* table, double dv, double* out, int stride, bool full, cudaStream_t s) {
  // four to eight elements a thread, whole warps; two where the rows do not fill the chip
  // (64 x 1024: 15.4 -> 14.4 us)
  int block = nv >= 1024 ? 256 : nv >= 512 ? 128 : 64;
  if (nrows <= GB300_SMS) block *= 2;
  auto run = [&](auto kernel) { kernel<<<nrows, block, 0, s>>>(f, nv, pw, table, dv, v, v_pow, out, stride); };
  if (block > 256) run(full ? k_moments_fx<true, 16> : k_moments_fx<false, 16>);
  else run(full ? k_moments_fx<true, 8> : k_moments_fx<false, 8>);
  return cudaGetLastError();
}

}  // namespace vg
