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
// so there are never more sweeps than lanes; contraction makes it two to five
// (the pivots forget their start by a factor a c / p^2 per element, below 0.6
// for c = nu dt vth / dv^2 up to 13).  Measured: 64 x 1024 from 1.59 to 0.09 ms,
// 2048 x 4096 from 6.4 to 1.2 ms, against one thread per row.
//
// Divisions that share a divisor (by 2 dv, by a pivot) go through its
// correctly rounded reciprocal y and remainder term yl: q = n y + n yl is
// within an ulp of n / d, r = n - q d is exact, and q + r y rounds to the IEEE
// quotient (P. Markstein, Computation of elementary functions on the IBM RISC
// System/6000 processor, IBM J. Res. Dev. 34, 1990): four FP64 instructions
// instead of about eight.  Operands near the ends of the exponent range take
// the IEEE division itself.
#include "vg_internal.cuh"
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
};

__global__ void k_thomas_serial(ThomasArgs a) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
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
// pivots p, m (then the pivots' reciprocals), d.  GLOBAL_AC: a and c in the
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
  auto drift = [&](int j) { return div_recip(g.dougherty ? sub_rn(g.v[j], vbar) : g.v[j], two_dv); };

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

  // ---- pivots: p_0 = b, m_j = a[j-1] / p_{j-1}, p_j = b - m_j c[j-1] ----------
  double in;
  {
    // the map's fixed point with this chunk's coefficients, in FP32
    const float af = n > 0 ? (float)sa[lane] : 0.f, cf = (float)c_in, bf = (float)b;
    in = (double)(0.5f * (bf + sqrtf(fmaxf(bf * bf - 4.f * af * cf, 0.f))));
  }
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
  in = 0.0;
  if (n > 0 && t > 0) in = (double)((float)fr[j0 - 1] / (1.f + (float)smm[lane]));
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
        i = 1;
      }
      bool merged = false;
      for (; i < n; ++i) {
        dp = sub_rn(fr[j0 + i], mul_rn(smm[i * S + lane], dp));
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
  in = j1 < N && n > 0 ? fr[j1] : 0.0;  // the step moves f little: its old value next door
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

cudaError_t launch_thomas_f64(double* f, int nrows, int nv, const double* v, const double* mom, int mstride,
                              int vbar_col, int vth_col, int dougherty, double nudt, const double* nudt_row, double dv,
                              double dv_sq, double* scratch, cudaStream_t s) {
  const ThomasArgs a = {f, nrows, nv, v, mom, mstride, vbar_col, vth_col, dougherty, nudt, nudt_row, dv, dv_sq,
                        scratch};
  if (nv > THOMAS_CHUNK_NV || nv < 16 || nrows >= THOMAS_SERIAL_ROWS) {
    k_thomas_serial<<<div_up(nrows, 64), 64, 0, s>>>(a);
    return cudaGetLastError();
  }
  // The shortest chunk that still gives every scheduler at most two warps (152
  // x 8 = 1216): a lane's share of the parallel work falls with L, while the
  // elements swept again do not depend on it, so once the schedulers are full
  // longer chunks waste less (32: five arrays of a warp's chunks take 42 KB, and
  // four warps must fit an SM)
  const long long cells = (long long)nrows * nv;
  if (nv <= 4096 && cells < 32LL * 8 * 1216) return chunks<8>(a, s);
  if (cells < 32LL * 16 * 1216) return chunks<16>(a, s);
  return chunks<32>(a, s);
}

}  // namespace vg
