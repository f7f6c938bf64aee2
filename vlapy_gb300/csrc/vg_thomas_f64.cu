// The FP64 tridiagonal solve of the implicit Fokker-Planck step
// (vlapy/core/collisions.py:26-160 builds the diagonals, :222-265 eliminates),
// bit for bit the reference's serial Thomas order, by two kernels: one thread
// per row (k_thomas_serial, thomas_row_f64), and the lanes of a row together
// (k_thomas_chunks).
//
// What bounds it.  GB300 issues one FP64 warp instruction per 64 cycles and
// scheduler whatever the number of active lanes, and does not overlap two of
// one warp (measured: a chain of FMAs and four independent chains cost the
// same per FMA), so a row per thread is 50 instructions x 64 cycles per
// element on a handful of warps: 1.59 ms for 64 x 1024, 6.4 ms for 2048 x
// 4096, with most schedulers idle.
//
// k_thomas_chunks.  Each of the three recurrences (pivots p_j, forward values
// d_j, solution x_j) is a map value -> next value that contracts.  Lane t owns
// the chunk j in [t L, t L + L) and starts it from a guess of the value that
// enters it; after each sweep it takes the value its neighbour really ended
// with, and sweeps again if that differs in any bit from the one it used.  A
// repeated sweep stops at the first element that comes out as it was (what
// follows is unchanged).  When no lane's incoming value changes, every element
// is the reference's own operation on the reference's own operands: by
// induction over the lanes from the first, whose start is exact, the result is
// the serial one bit for bit.  The k-th sweep leaves at least k lanes exact,
// so there are never more sweeps than lanes; contraction makes it two
// (the pivots forget their start by a factor a c / p^2 per element, below 0.6
// for c = nu dt vth / dv^2 up to 13; strongly collisional rows of a full chip are left
// to one thread each, see launch_thomas_f64).  Measured: 64 x 1024 from 1.59 to 0.03 ms,
// 2048 x 4096 from 6.4 to 1.07 ms, against one thread per row.
//
// Divisions that share a divisor (by 2 dv, by a pivot) go through its
// correctly rounded reciprocal y and remainder term yl: q = n y + n yl is
// within an ulp of n / d, r = n - q d is exact, and q + r y rounds to the IEEE
// quotient (P. Markstein, Computation of elementary functions on the IBM RISC
// System/6000 processor, IBM J. Res. Dev. 34, 1990): four FP64 instructions
// instead of about eight.  Operands near the ends of the exponent range take
// the IEEE division itself.
//
// The guesses.  What a guess is off by costs sweeps: the values forget it by a factor
// m = a / p an element, 0.58 at c = 3, so from three digits a double takes 55 elements
// to come out the same, seven chunks of eight.  So each lane first runs the recurrence
// over the elements before its chunk (K of them, WARM_BITS / -log2 m) in double-float:
// that is some 90 cycles an element on the FP32 and integer pipes, where the FP64
// sweep takes 130 to 600, and leaves about nine elements to sweep again: two sweeps
// instead of two to eight, 2048 x 4096 from 1.31 to 1.07 ms, 64 x 1024 from 45 to 33 us.
#include <algorithm>
#include <cmath>

#include "vg_internal.cuh"
#include "vg_f32.cuh"
#include "vg_f64_body.cuh"

namespace vg {

namespace {

// true when a quotient of n by a divisor of ordinary size meets no underflow
// or overflow on the way: n's exponent in [2^-900, 2^900]
__device__ __forceinline__ bool ordinary(double n) {
  const unsigned e = ((unsigned)__double2hiint(n) >> 20) & 0x7ffu;
  return e - 123u < 1800u;
}

struct Recip {
  double d, y, yl;
  bool ok;  // the divisor itself is ordinary: [2^-60, 2^60]
};
__device__ __forceinline__ Recip recip_of(double d) {
  Recip r;
  r.d = d;
  r.y = __drcp_rn(d);
  r.yl = __dmul_rn(__fma_rn(-d, r.y, 1.0), r.y);
  const unsigned e = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
  r.ok = e - 963u < 121u;
  return r;
}
// the IEEE quotient n / r.d
__device__ __forceinline__ double div_recip(double n, const Recip& r) {
  if (!(r.ok && ordinary(n))) return __ddiv_rn(n, r.d);
  const double q = __fma_rn(n, r.y, __dmul_rn(n, r.yl));
  return __fma_rn(__fma_rn(-q, r.d, n), r.y, q);
}

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// The double v 2^k as double-float, by integer arithmetic (conversions between the
// two run on the FP64 pipe); 0 outside FP32's range, and for infinities and NaN.
__device__ __forceinline__ df32 df_of(double v, int k) {
  const int h = __double2hiint(v);
  const unsigned l = (unsigned)__double2loint(v);
  const int e = ((h >> 20) & 0x7ff) + k - 896;
  const bool ok = (unsigned)(e - 53) < 202u;  // (lo's exponent is 52 below)
  const unsigned sign = (unsigned)h & 0x80000000u;
  const float hi = __uint_as_float(sign | (unsigned)e << 23 | (__funnelshift_l(l, (unsigned)h, 3) & 0x7fffffu));
  const float lo = __uint2float_rn(l & 0x1fffffffu) * __uint_as_float(sign | (unsigned)(e - 52) << 23);
  return {ok ? hi : 0.f, ok ? lo : 0.f};
}
// and back: a 2^-k, or `other` where that is not an ordinary number
__device__ __forceinline__ double df_back(df32 a, int k, double other) {
  const double d = __dadd_rn((double)a.hi, (double)a.lo);
  const int e = (__double2hiint(d) >> 20) & 0x7ff;
  if (!(fabsf(a.hi) > 0.f && fabsf(a.hi) <= 3e38f) || e - k < 1 || e - k > 2046) return other;
  return __hiloint2double(__double2hiint(d) - (k << 20), __double2loint(d));
}
__device__ __forceinline__ df32 df_neg(df32 a) { return {-a.hi, -a.lo}; }
// a / b, |error| some 2^-45
__device__ __forceinline__ df32 df_div(df32 a, df32 b) {
  const float r = __frcp_rn(b.hi);
  const float q = a.hi * r;
  const float rem = fmaf(-q, b.hi, a.hi) + fmaf(-q, b.lo, a.lo);
  const float q1 = rem * r;
  const float hi = q + q1;
  return {hi, q1 - (hi - q)};
}
constexpr float WARM_BITS = 36.f;  // a 2^-44 or so from a guess good to two digits (28, 34, 40: within 1 %)
constexpr int WARM_MAX = 96;

}  // namespace

struct ThomasArgs {
  double* f;
  int nrows, nv;
  const double* v;
  const double* mom;
  int mstride, vbar_col, vth_col, dougherty;
  double nudt;
  const double* nudt_row;  // per row (0: leave the row as it is), or null: nudt
  double dv, dv_sq;
  double* scratch;
  // either: both kernels run, and the rows' collisionality says which of them solves
  // (all_stiff); stiff: 32 times the limit of the mean of sqrt(nudt vth)
  bool either;
  float stiff;
};
// Whether the launch is k_thomas_serial's: the same answer in every warp of both
// kernels, from 32 rows spread over all (whole warps call it)
__device__ __forceinline__ bool all_stiff(const ThomasArgs& a) {
  const size_t row = (size_t)((threadIdx.x & 31) * (unsigned)a.nrows / 32);
  const double nudt = a.nudt_row ? a.nudt_row[row] : a.nudt;
  float q = __fsqrt_rn(__double2float_rn(__dmul_rn(nudt, a.mom[row * a.mstride + a.vth_col])));
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, m));
  return q > a.stiff;  // (NaN: no)
}

__global__ void k_thomas_serial(ThomasArgs a) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (a.either && !all_stiff(a)) return;
  if (row >= a.nrows) return;
  const double nudt = a.nudt_row ? a.nudt_row[row] : a.nudt;
  if (a.nudt_row && nudt == 0.0) return;
  const double vbar = a.dougherty ? a.mom[(size_t)row * a.mstride + a.vbar_col] : 0.0;
  const double vth = a.mom[(size_t)row * a.mstride + a.vth_col];
  thomas_row_f64(a.f + (size_t)row * a.nv, a.scratch + (size_t)row * 2 * a.nv, a.nv, a.v, vbar, vth, a.dougherty,
                 nudt, a.dv, a.dv_sq);
}

// T lanes per row: WIDE, a CTA of T threads (a multiple of 32) per row; else a
// warp of 32 / T rows (T a power of two <= 32).  Five values per element live in
// arrays indexed [i][lane] (element i of the lane's chunk: consecutive lanes,
// consecutive words; the row stride S is odd, so the copy out, which walks i
// first, is free of bank conflicts too): a (then the solution x), c, the
// pivots p, m (then the pivots' reciprocals), d (at
// first f).  GLOBAL_AC: a and c in the
// scratch instead of shared memory (rows of more than 4096).
template <int L, bool WIDE, bool GLOBAL_AC>
__global__ void __launch_bounds__(WIDE ? 512 : 32) k_thomas_chunks(ThomasArgs g, int T) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double edge[WIDE ? 512 : 1];
  const int lane = threadIdx.x;
  const int N = g.nv;
  const int rows_per = WIDE ? 1 : 32 / T;
  const int t = WIDE ? lane : lane & (T - 1);
  const int row = blockIdx.x * rows_per + (WIDE ? 0 : lane / T);
  const int S = (WIDE ? T : 32) | 1;
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* sa = GLOBAL_AC ? g.scratch + (size_t)blockIdx.x * 2 * thomas_pad(N) : sm + 3 * L * S;
  double* sc = sa + (GLOBAL_AC ? (size_t)thomas_pad(N) : (size_t)L * S);
  const int SG = GLOBAL_AC ? T : S;  // row stride of a and c
  double* sp = sm;
  double* smm = sm + L * S;
  double* sd = sm + 2 * L * S;
  const bool valid = row < g.nrows;
  const double nudt = !valid ? 0.0 : (g.nudt_row ? g.nudt_row[row] : g.nudt);
  // rows of collisionless runs are left as they are (the lanes stay for the exchanges)
  const bool live_row = valid && !(g.nudt_row && nudt == 0.0);
  if (WIDE && !live_row) return;
  if (g.either && all_stiff(g)) return;
  const int j0 = t * L, j1 = live_row ? min(j0 + L, N) : 0;
  const int n = max(j1 - j0, 0);  // this lane's elements
  double* fr = g.f + (size_t)(live_row ? row : 0) * N;

  auto sync = [&]() {
    if constexpr (WIDE) __syncthreads();
    else __syncwarp();
  };
  auto any = [&](bool p) -> bool {
    if constexpr (WIDE) return __syncthreads_or(p) != 0;
    else return __any_sync(0xffffffffu, p);
  };
  // the value of the lane to the left (dir = -1) or right (+1) in the row
  auto neighbour = [&](double x, int dir) -> double {
    if constexpr (WIDE) {
      __syncthreads();
      edge[lane] = x;
      __syncthreads();
      const int q = lane + dir;
      return (q >= 0 && q < T) ? edge[q] : x;
    } else {
      return dir < 0 ? __shfl_up_sync(0xffffffffu, x, 1, T) : __shfl_down_sync(0xffffffffu, x, 1, T);
    }
  };

  const double vbar = (live_row && g.dougherty) ? g.mom[(size_t)row * g.mstride + g.vbar_col] : 0.0;
  const double vth = live_row ? g.mom[(size_t)row * g.mstride + g.vth_col] : 1.0;
  const double A = __ddiv_rn(-vth, g.dv_sq);
  const double b = add_rn(1.0, mul_rn(nudt, __ddiv_rn(mul_rn(2.0, vth), g.dv_sq)));
  // drift(j) = ((v_j - vbar) 0.5) / dv = (v_j - vbar) / (2 dv): the factor 2 is exact
  const Recip two_dv = recip_of(2.0 * g.dv);
  // element j's place in an array of row stride st
  auto at = [&](int j, int st) { return (int)((unsigned)j % L) * st + (lane - t) + (int)((unsigned)j / L); };
  // v waits in the pivots' place and f in the forward values' (a lane's walk along its
  // chunk in global memory touches 32 lines a load)
  if constexpr (WIDE) {
    for (int j = lane; j < N; j += T) {
      sp[at(j, S)] = g.v[j];
      sd[at(j, S)] = fr[j];
    }
  } else {
    for (int r = 0; r < rows_per; ++r) {
      const int rr = min(blockIdx.x * rows_per + r, g.nrows - 1);
      for (int j = lane; j < N; j += 32) {
        const int q = (int)((unsigned)j % L) * S + r * T + (int)((unsigned)j / L);
        sp[q] = g.v[j];
        sd[q] = g.f[(size_t)rr * N + j];
      }
    }
  }
  sync();
  auto drift = [&](int j) {
    const double vj = sp[at(j, S)];
    return div_recip(g.dougherty ? sub_rn(vj, vbar) : vj, two_dv);
  };

  // the diagonals: a[j] of row j + 1, c[j] of row j (a is stored at j + 1's place)
  double c_in = 0.0;  // c[j0 - 1]
  if (n > 0) {
    double dm = j0 > 0 ? drift(j0 - 1) : 0.0, d0 = drift(j0);
    if (j0 > 0) c_in = mul_rn(nudt, sub_rn(A, d0));
    for (int i = 0; i < n; ++i) {
      const int j = j0 + i;
      sa[i * SG + lane] = mul_rn(nudt, add_rn(A, dm));  // a[j - 1]; unused for j = 0
      const double dp = j + 1 < N ? drift(j + 1) : 0.0;
      sc[i * SG + lane] = mul_rn(nudt, sub_rn(A, dp));  // c[j]; unused for j = N - 1
      dm = d0;
      d0 = dp;
    }
  }
  sync();

  // elements of the warm-ups
  int K;
  {
    const float c = (float)nudt * (float)vth / (float)g.dv_sq, bf = 1.f + 2.f * c;
    const float m = 2.f * c / (bf + sqrtf(fmaxf(bf * bf - 4.f * c * c, 0.f)));
    K = (int)fminf(WARM_BITS / fmaxf(-__log2f(m), 0.1f), (float)WARM_MAX) + 2;
  }

  // ---- pivots: p_0 = b, m_j = a[j-1] / p_{j-1}, p_j = b - m_j c[j-1] ----------
  double in = b;
  if (n > 0 && t > 0) {
    // the map's fixed point with the coefficients there, in FP32; then the map (the
    // pivots forget twice as fast as the values)
    const int js = max(j0 - 1 - (K + 1) / 2, 0);
    const df32 bd = df_of(b, 0);
    df32 P = bd;
    if (js > 0) {
      const float ac = df_of(sa[at(js, SG)], 0).hi * df_of(sc[at(js - 1, SG)], 0).hi;
      P = {0.5f * (bd.hi + sqrtf(fmaxf(bd.hi * bd.hi - 4.f * ac, 0.f))), 0.f};
    }
    // (in batches: the conversions of four elements, which do not wait for one
    // another, then the chain)
    for (int j = js + 1; j < j0; j += 4) {
      df32 ac[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = min(j + u, j0 - 1);
        ac[u] = df_mul(df_of(sa[at(q, SG)], 0), df_of(sc[at(q - 1, SG)], 0));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j + u < j0) P = df_add(bd, df_neg(df_div(ac[u], P)));
    }
    in = df_back(P, 0, b);
  }
  sync();  // (the pivots go where v waits)
  double out = in;
  bool act = n > 0, first = true;
  for (int sweep = 0; sweep <= T; ++sweep) {
    if (act) {
      double pp = in, cp = c_in;
      int i = 0;
      if (t == 0) {
        sp[lane] = b;
        smm[lane] = 0.0;
        pp = b;
        cp = sc[lane];
        i = 1;
      }
      bool merged = false;
      for (; i < n; ++i) {
        const double m = __ddiv_rn(sa[i * SG + lane], pp);
        pp = sub_rn(b, mul_rn(m, cp));
        smm[i * S + lane] = m;
        if (!first && same_bits(pp, sp[i * S + lane])) {
          merged = true;
          break;
        }
        sp[i * S + lane] = pp;
        cp = sc[i * SG + lane];
      }
      if (!merged) out = pp;
    }
    first = false;
    const double nb = neighbour(out, -1);
    act = n > 0 && t > 0 && !same_bits(nb, in);
    in = nb;
    if (!any(act)) break;
  }

  // ---- forward values: d_0 = f_0, d_j = f_j - m_j d_{j-1} ----------------------
  sync();
  in = 0.0;
  int sh = 0;  // the warm-ups' scale: f is about 1 there
  if (n > 0) sh = 1023 - ((__double2hiint(sd[at(j0, S)]) >> 20) & 0x7ff);
  if (n > 0 && t > 0) {
    const int js = max(j0 - 1 - K, 0);
    df32 D = df_of(sd[at(js, S)], sh);
    if (js > 0) D = {__fdividef(D.hi, 1.f + df_of(smm[at(js, S)], 0).hi), 0.f};
    for (int j = js + 1; j < j0; j += 4) {
      df32 f4[4], m4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = min(j + u, j0 - 1);
        f4[u] = df_of(sd[at(q, S)], sh);
        m4[u] = df_neg(df_of(smm[at(q, S)], 0));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j + u < j0) D = df_add(f4[u], df_mul(m4[u], D));
    }
    in = df_back(D, sh, sd[at(j0 - 1, S)]);
  }
  sync();  // (the forward values go where f waits)
  out = in;
  act = n > 0;
  first = true;
  for (int sweep = 0; sweep <= T; ++sweep) {
    if (act) {
      double dp = in;
      int i = 0;
      if (t == 0) {
        dp = fr[0];
        sd[lane] = dp;
        i = 1;  // (sd holds f_j the first time, the last sweep's d_j afterwards)
      }
      bool merged = false;
      for (; i < n; ++i) {
        dp = sub_rn(first ? sd[i * S + lane] : fr[j0 + i], mul_rn(smm[i * S + lane], dp));
        if (!first && same_bits(dp, sd[i * S + lane])) {
          merged = true;
          break;
        }
        sd[i * S + lane] = dp;
      }
      if (!merged) out = dp;
    }
    first = false;
    const double nb = neighbour(out, -1);
    act = n > 0 && t > 0 && !same_bits(nb, in);
    in = nb;
    if (!any(act)) break;
  }

  // ---- back substitution: x_{N-1} = d / p, x_j = (d_j - c_j x_{j+1}) / p_j -----
  for (int i = 0; i < n; ++i) smm[i * S + lane] = __drcp_rn(sp[i * S + lane]);
  sync();
  in = 0.0;
  if (n > 0 && j1 < N) {
    // from the old value there: the step moves f little
    const int js = min(j1 + K, N - 1);
    df32 X = js == N - 1 ? df_mul(df_of(sd[at(js, S)], sh), df_of(smm[at(js, S)], 0)) : df_of(fr[js], sh);
    for (int j = js - 1; j >= j1; j -= 4) {
      df32 d4[4], c4[4], y4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = max(j - u, j1);
        d4[u] = df_of(sd[at(q, S)], sh);
        c4[u] = df_neg(df_of(sc[at(q, SG)], 0));
        y4[u] = df_of(smm[at(q, S)], 0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j - u >= j1) X = df_mul(df_add(d4[u], df_mul(c4[u], X)), y4[u]);
    }
    in = df_back(X, sh, fr[j1]);
  }
  out = in;
  act = n > 0;
  first = true;
  for (int sweep = 0; sweep <= T; ++sweep) {
    if (act) {
      double x = in;
      bool merged = false;
      for (int i = n - 1; i >= 0; --i) {
        Recip r;
        r.d = sp[i * S + lane];
        r.y = smm[i * S + lane];
        r.yl = __dmul_rn(__fma_rn(-r.d, r.y, 1.0), r.y);
        const unsigned e = ((unsigned)__double2hiint(r.d) >> 20) & 0x7ffu;
        r.ok = e - 963u < 121u;
        const double dj = sd[i * S + lane];
        x = div_recip(j0 + i == N - 1 ? dj : sub_rn(dj, mul_rn(sc[i * SG + lane], x)), r);
        if (!first && same_bits(x, sa[i * SG + lane])) {
          merged = true;
          break;
        }
        sa[i * SG + lane] = x;
      }
      if (!merged) out = x;
    }
    first = false;
    const double nb = neighbour(out, +1);
    act = n > 0 && j1 < N && !same_bits(nb, in);
    in = nb;
    if (!any(act)) break;
  }
  sync();
  // ---- out, coalesced over j -----------------------------------------------------
  if constexpr (WIDE) {
    for (int j = lane; j < N; j += T) fr[j] = sa[(j % L) * SG + j / L];
  } else {
    for (int r = 0; r < rows_per; ++r) {
      const int rr = blockIdx.x * rows_per + r;
      if (rr >= g.nrows || (g.nudt_row && g.nudt_row[rr] == 0.0)) continue;
      for (int j = lane; j < N; j += 32) g.f[(size_t)rr * N + j] = sa[(j % L) * SG + r * T + j / L];
    }
  }
}

namespace {

template <int L>
cudaError_t chunks(const ThomasArgs& a, cudaStream_t s) {
  int T = div_up(a.nv, L);
  const bool wide = T > 32;
  if (wide) T = div_up(T, 32) * 32;
  else
    for (int q = 1;; q <<= 1)
      if (q >= T) {
        T = q;
        break;
      }
  const int S = (wide ? T : 32) | 1;
  const bool gac = a.nv > THOMAS_SMEM_NV;
  const size_t smem = (size_t)(gac ? 3 : 5) * L * S * sizeof(double);
  const int blocks = wide ? a.nrows : div_up(a.nrows, 32 / T);
  const void* k = !wide ? (const void*)k_thomas_chunks<L, false, false>
                 : gac  ? (const void*)k_thomas_chunks<L, true, true>
                        : (const void*)k_thomas_chunks<L, true, false>;
  cudaError_t err = ensure_smem(k, smem);
  if (err != cudaSuccess) return err;
  if (!wide) k_thomas_chunks<L, false, false><<<blocks, 32, smem, s>>>(a, T);
  else if (gac) k_thomas_chunks<L, true, true><<<blocks, T, smem, s>>>(a, T);
  else k_thomas_chunks<L, true, false><<<blocks, T, smem, s>>>(a, T);
  return cudaGetLastError();
}

}  // namespace

double thomas_root_most(double root, const double* v, int nv) {
  double vmax = 0.0;
  for (int j = 0; j < nv; ++j) vmax = std::max(vmax, std::fabs(v[j]));
  return 2.0 * root * vmax;
}

cudaError_t launch_thomas_f64(double* f, int nrows, int nv, const double* v, const double* mom, int mstride,
                              int vbar_col, int vth_col, int dougherty, double nudt, const double* nudt_row,
                              double root_most, double dv, double dv_sq, double* scratch, cudaStream_t s) {
  ThomasArgs a = {f, nrows, nv, v, mom, mstride, vbar_col, vth_col, dougherty, nudt, nudt_row, dv, dv_sq,
                  scratch, false, 0.f};
  if (nv > THOMAS_CHUNK_NV || nv < 16 || nrows >= THOMAS_SERIAL_ROWS) {
    k_thomas_serial<<<div_up(nrows, 64), 64, 0, s>>>(a);
    return cudaGetLastError();
  }
  // Rows of strong collisions (c = nudt vth / dv^2) forget a guess over some 20 sqrt(c)
  // elements, so the sweeps over a full chip's rows cost 4e-5 us a cell and sqrt(c),
  // where one thread a row takes 1.6 us an element whatever c.  They meet near sqrt(c)
  // = 40000 / rows: 2048 x 4096 at c = 320 (6.8 ms; 45 ms in chunks at c = 1e5), 2048 x
  // 1024 at 340, 8192 x 1024 at 31, 11000 x 512 at 16.  Below a million cells the
  // chunks fit the chip and are never the slower (1024 x 1024: 1.8 against 1.6 ms at c
  // = 1e5; 300 x 2048: 2.2 against 3.1), except for the longest rows, one of which
  // fills an SM (4 x 4096 meets at 2e4, 64 x 8192 at 6e4).  vth is only known on the
  // device: both kernels are launched and one of them returns (an idle launch is 2 us).
  // The mean of sqrt(c) decides for all rows: the serial kernel takes as long for a few.
  // Where root_most, from the largest vth that a density of four or less has on the
  // grid, is below the line, the serial kernel is not launched.
  const long long cells = (long long)nrows * nv;
  double root = 40000.0 / nrows;
  if (cells < (1 << 20) || (nv >= 4096 && root > 200.0)) root = 200.0;
  root *= std::sqrt(dv_sq);
  a.either = thomas_either(nrows, nv) && !(root_most < root);
  a.stiff = (float)(32.0 * root);
  // The shortest chunk that still gives every scheduler at most two warps: a lane's share of the parallel work falls with L, while the
  // elements swept again do not depend on it, so once the schedulers are full
  // longer chunks waste less (32: five arrays of a warp's chunks take 42 KB, and
  // four warps must fit an SM)
  const cudaError_t err = nv <= 4096 && cells < 32LL * 8 * (8 * GB300_SMS) ? chunks<8>(a, s)
                          : cells < 32LL * 16 * (8 * GB300_SMS)            ? chunks<16>(a, s)
                                                                : chunks<32>(a, s);
  if (err != cudaSuccess || !a.either) return err;
  k_thomas_serial<<<div_up(nrows, 64), 64, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace vg
