// Fixed-point v-advection of the FP64 mode (vlapy/core/vlasov.py:113-140): f <-
// Re IFFT_v(exp(-i kv e dt) FFT_v f) on row pairs, and the host side of the
// fixed-point tables.
//
// One group of N / 8 threads (N / 16 at 8192) owns a pair of rows as one complex
// sequence; f is read once and written once.
//
// Measured against the transforms in doubles (FP64 pipe 84 % busy), smooth rows:
// 4096 x 8192 4.44 -> 0.88 ms, 2048 x 4096 1.02 -> 0.24 ms, 64 x 1024 70 -> 16 us one
// launch after another (25 with cold caches).  Rows that go through doubles after all
// (vg_fx.cuh): 2048 x 4096 of noise 1.01 ms.  Bound by
// integer issue: a complex product is 12 wide multiplies at a quarter of the
// add rate.  Radix 16 (3 passes instead of 4 at 4096) takes 0.21 ms there but
// 34 us at 64 x 1024, where half as many threads carry the latency.  RMS error
// against 128-bit FFTs: 1.1e-16 of the line's RMS at 1024 and 2.7e-16 at 8192
// (smooth lines), in doubles 3.0e-16 and 3.2e-16.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "vg_advect_fx.cuh"
#include "vg_dd.cuh"
#include "vg_internal.cuh"

namespace vg {

namespace {

__host__ __device__ constexpr int fx_row_block(int n) { return fx_threads(n) > 256 ? fx_threads(n) : 256; }

template <int N>
__global__ void __launch_bounds__(fx_row_block(N), fx_row_block(N) > 256 ? 1 : 2)
    k_edfdv_fx(double* __restrict__ f, int nrows, const double* __restrict__ e, FxTurn turn,
               const float* __restrict__ rest, const fxw* __restrict__ tw, const cx<double>* __restrict__ tw64) {
  constexpr int R = fx_radix(N), G = fx_threads(N);
  constexpr int DOWN = ilog2(N) - fx_shift<N>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 red[G > 32 ? fx_row_block(N) / 32 : 1];
  __shared__ FxNorms nred[G > 32 ? fx_row_block(N) / 32 : 1];
  const int g = threadIdx.x / G, t = threadIdx.x - g * G;
  fx* s = reinterpret_cast<fx*>(smem_raw) + (size_t)g * sp_len<double>(N);
  const int ra = 2 * (blockIdx.x * (blockDim.x / G) + g), rb = ra + 1;
  if (ra >= nrows) return;  // the whole group; its barrier is its own
  const GroupSync sync = GroupSync::of(g, G);
  const unsigned mask = G < 32 ? sync.mask : 0xffffffffu;
  const bool vb = rb < nrows;
  double* fa = f + (size_t)ra * N;
  double* fb = f + (size_t)(vb ? rb : ra) * N;
  const double ea = e[ra], eb = vb ? e[rb] : 0.0;
  fx io[R];
  int Ea, Eb;
  bool bad_a, bad_b, zero_a, zero_b;
  {
    double da[R], db[R];
    unsigned ma = 0, mb = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      da[i] = fa[t + i * G];
      db[i] = vb ? fb[t + i * G] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      ma = max(ma, fx_exp_bits(da[i]));
      mb = max(mb, fx_exp_bits(db[i]));
    }
    ma = __reduce_max_sync(mask, ma);
    mb = __reduce_max_sync(mask, mb);
    if constexpr (G > 32) {
      if ((t & 31) == 0) red[threadIdx.x >> 5] = make_uint2(ma, mb);
      sync();
#pragma unroll
      for (int w = 0; w < G / 32; ++w) {
        ma = max(ma, red[g * (G / 32) + w].x);
        mb = max(mb, red[g * (G / 32) + w].y);
      }
    }
    zero_a = ma == 0;
    zero_b = mb == 0;
    Ea = fx_exp(ma);
    Eb = fx_exp(mb);
    bad_a = Ea == FX_NONFINITE || !isfinite(ea);
    bad_b = Eb == FX_NONFINITE || !isfinite(eb);
#pragma unroll
    for (int i = 0; i < R; ++i)
      io[i] = {bad_a ? 0 : fx_from_double(da[i], Ea), bad_b ? 0 : fx_from_double(db[i], Eb)};
  }
  fx_fft<N, false, true, false>(s, t, tw, sync, io);
  const unsigned long long ta = fx_turn(turn, bad_a ? 0.0 : ea), tb = fx_turn(turn, bad_b ? 0.0 : eb);
  const bool own = N >= FX_OWN_N && (fx_has_own(turn, ea) || fx_has_own(turn, eb));
  float oa = 0.f, ob = 0.f;
  if (own) {
    oa = bad_a ? 0.f : turn.own * (float)ea;
    ob = bad_b ? 0.f : turn.own * (float)eb;
  }
  FxNorms n = fx_rotate<N, DOWN>(s, t, ta, tb, own, oa, ob, rest, tw);
  n.l1 = __reduce_add_sync(mask, n.l1);
  n.a2 = __reduce_add_sync(mask, n.a2);
  n.b2 = __reduce_add_sync(mask, n.b2);
  if constexpr (G > 32) {
    if ((t & 31) == 0) nred[threadIdx.x >> 5] = n;
  }
  sync();
  if constexpr (G > 32) {
    n = nred[g * (G / 32)];
#pragma unroll
    for (int w = 1; w < G / 32; ++w) {
      const FxNorms q = nred[g * (G / 32) + w];
      n.l1 += q.l1;
      n.a2 += q.a2;
      n.b2 += q.b2;
    }
  }
  // (E <= 1: a line of zeros, or of values that small)
  const int h = fx_shift_back<N>(n, bad_a || Ea <= 1, bad_b || Eb <= 1);
  if (h < 0) {
    sync();
    fx_pair_f64<N>({fa, ta, oa, fx_up(Ea, n.a2), true, bad_a}, {fb, tb, ob, fx_up(Eb, n.b2), vb, bad_b}, 1,
                   reinterpret_cast<cx<double>*>(s), t, rest, tw, tw64, sync);
    return;
  }
  fx_fft<N, true, false, true>(s, t, tw, sync, io, h);
  // lines of zeros stay so: the partner's rounding does not reach them
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const bool set_a = bad_a || zero_a, set_b = bad_b || zero_b;
  const double val_a = bad_a ? nan : 0.0, val_b = bad_b ? nan : 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    fa[t + i * G] = set_a ? val_a : fx_to_double(io[i].x, Ea - FX_SCALE + h);
    if (vb) fb[t + i * G] = set_b ? val_b : fx_to_double(io[i].y, Eb - FX_SCALE + h);
  }
}

template <int N>
cudaError_t edfdv_fx_n(double* f, int nrows, const double* e, FxTurn turn, const float* rest, const fxw* tw,
                       const cx<double>* tw64, cudaStream_t s) {
  constexpr int G = fx_threads(N);
  const int pairs = (nrows + 1) / 2;
  // groups per CTA: fewer when the pairs would not give every SM two CTAs
  // (a scheduler runs the integer work of one CTA's warps with gaps), whole warps
  int P = fx_row_block(N) / G;
  while (P > 1 && (P / 2) * G >= 32 && div_up(pairs, P) < 2 * GB300_SMS) P /= 2;
  const size_t smem = (size_t)P * sp_len<double>(N) * sizeof(fx);
  cudaError_t err = ensure_smem((const void*)k_edfdv_fx<N>, smem);
  if (err != cudaSuccess) return err;
  k_edfdv_fx<N><<<div_up(pairs, P), P * G, smem, s>>>(f, nrows, e, turn, rest, tw, tw64);
  return cudaGetLastError();
}

// ---- host tables -------------------------------------------------------------
const dd kPi = {3.141592653589793116, 1.2246467991473532072e-16};
const dd kInv2Pi = {0.15915494309189534561, -9.8393383375912127e-18};

// cos and sin of pi j / 4096 for j <= 1024 (an eighth of the circle) by their Taylor series
void dd_cos_sin(int j, dd* c, dd* s) {
  const dd x = dd_mul(kPi, {(double)j / 4096.0, 0.0}), x2 = dd_mul(x, x);
  dd tc = {1.0, 0.0}, ts = x;
  *c = tc;
  *s = ts;
  for (int n = 1; n < 16; ++n) {
    const dd pc = dd_mul(tc, x2), ps = dd_mul(ts, x2);
    const double dc = -(2.0 * n - 1.0) * (2.0 * n), ds = -(2.0 * n) * (2.0 * n + 1.0);
    tc = dd_div(pc, dc);
    ts = dd_div(ps, ds);
    *c = dd_add(*c, tc);
    *s = dd_add(*s, ts);
  }
}
long long q62(dd a) {
  return (long long)std::llrint(std::ldexp(a.h, 62)) + (long long)std::llrint(std::ldexp(a.l, 62));
}

std::vector<fxw> build_table() {
  std::vector<long long> c(FX_NMAX), s(FX_NMAX);
  for (int j = 0; j <= FX_NMAX / 8; ++j) {
    dd cj, sj;
    dd_cos_sin(j, &cj, &sj);
    const long long C = q62(cj), S = q62(sj);
    const int h = FX_NMAX / 4, n = FX_NMAX;
    // the eight angles +-j, h +- j, 2h +- j, 3h +- j
    auto put = [&](int k, long long cc, long long ss) {
      c[(k + n) % n] = cc;
      s[(k + n) % n] = ss;
    };
    put(j, C, S);
    put(-j, C, -S);
    put(h - j, S, C);
    put(h + j, -S, C);
    put(2 * h - j, -C, S);
    put(2 * h + j, -C, -S);
    put(3 * h - j, -S, -C);
    put(3 * h + j, S, -C);
  }
  std::vector<fxw> out(FX_TABLE);
  for (int L = 2; L <= FX_NMAX; L *= 2)
    for (int q = 0; q < L; ++q) {
      const int k = q * (FX_NMAX / L);
      out[L - 2 + q] = fx_mult(c[k], -s[k]);
    }
  return out;
}

// both tables as they lie on the device, so that they go in one copy
const std::vector<unsigned char>& tables_host() {
  static const std::vector<unsigned char> bytes = [] {
    const std::vector<fxw> tw = build_table();
    std::vector<unsigned char> b(tw.size() * sizeof(fxw) + FX_LOG_ENTRIES * sizeof(FxLogEntry));
    std::memcpy(b.data(), tw.data(), tw.size() * sizeof(fxw));
    std::memcpy(b.data() + tw.size() * sizeof(fxw), fx_log_host(), FX_LOG_ENTRIES * sizeof(FxLogEntry));
    return b;
  }();
  return bytes;
}

std::mutex tables_mu;
std::vector<FxTables*> tables_held;  // one per device in use

}  // namespace

cudaError_t fx_tables_acquire(FxTables** out) {
  *out = nullptr;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  std::lock_guard<std::mutex> lk(tables_mu);
  for (FxTables* t : tables_held)
    if (t->device == dev) {
      ++t->refs;
      *out = t;
      return cudaSuccess;
    }
  FxTables t = {dev, 1, nullptr, nullptr};
  const std::vector<unsigned char>& host = tables_host();
  err = cudaMalloc(&t.tw, host.size());
  if (err != cudaSuccess) return err;
  t.log = reinterpret_cast<FxLogEntry*>(t.tw + FX_TABLE);
  err = cudaMemcpy(t.tw, host.data(), host.size(), cudaMemcpyHostToDevice);
  if (err != cudaSuccess) {
    cudaFree(t.tw);
    return err;
  }
  tables_held.push_back(new FxTables(t));
  *out = tables_held.back();
  return cudaSuccess;
}

void fx_tables_release(FxTables* t) {
  if (!t) return;
  std::lock_guard<std::mutex> lk(tables_mu);
  if (--t->refs > 0) return;
  tables_held.erase(std::find(tables_held.begin(), tables_held.end(), t));
  cudaFree(t->tw);
  delete t;
}

bool fx_make_turn(FxStep k1, double dt, FxTurn* out) {
  const double p = k1.h * dt;
  if (!std::isfinite(p) || std::fabs(p) > 1e280 || (p != 0.0 && std::fabs(p) < 1e-280)) return false;
  const dd a = dd_mul(dd_norm(p, std::fma(k1.h, dt, -p) + k1.l * dt), kInv2Pi);
  int e = 0;
  const double m = std::frexp(a.h, &e);
  out->am = -((long long)std::ldexp(m, 62) + (long long)std::llrint(std::ldexp(a.l, 62 - e)));
  out->ae = e - 62;
  out->own = (float)(-6.283185307179586 * dt);
  // |c| < 2^(e - 1022): own |c| times the largest rest above the least that counts
  const double most = std::fabs(k1.own * 6.283185307179586 * dt);
  out->own_e = most > 0.0 ? std::max(0, 1023 + std::ilogb(FX_OWN_LEAST / most)) : 4096;
  return true;
}

bool fx_uniform(const double* k, int n, FxStep* k1) {
  *k1 = {k[n > 1 ? 1 : 0], 0.0, 0.f};
  for (int m = 0; m <= n / 2; ++m) {
    const double want = m * k[n > 1 ? 1 : 0], tol = 1e-15 * std::fabs(want);
    if (!(std::fabs(std::fabs(k[m % n]) - std::fabs(want)) <= tol)) return false;
    if (2 * m != n && m > 0 && want != 0.0 && (k[m] < 0.0) != (want < 0.0)) return false;
  }
  // sum m k[m] / sum m^2 (the Nyquist bin's sign is the other way round)
  dd num = {0.0, 0.0};
  double den = 0.0;
  for (int m = 1; m <= n / 2; ++m) {
    const double km = std::copysign(k[m], k1->h), p = m * km;
    num = dd_add(num, {p, std::fma((double)m, km, -p)});
    den += (double)m * m;
  }
  // (far from the ends of the range, where the parts are doubles)
  if (std::fabs(num.h) > 1e-250 && std::fabs(num.h) < 1e250) {
    const dd s = dd_div(num, den);
    *k1 = {s.h, s.l, 0.f};
  }
  return true;
}

std::vector<float> fx_step_rest(const double* k, int n, FxStep* k1) {
  std::vector<float> r(n / 2 + 1, 0.f);
  for (int m = 1; m <= n / 2; ++m) {
    r[m] = (float)((std::fma(-(double)m, k1->h, std::copysign(k[m], k1->h)) - m * k1->l) * std::ldexp(kInv2Pi.h, 64));
    k1->own = std::max(k1->own, std::fabs(r[m]));
  }
  return r;
}

#define VG_FX_CASES(M) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13)

cudaError_t launch_edfdv_fx(double* f, int nrows, int nv, const double* e, FxTurn turn, const float* rest,
                            const fxw* tw, const cx<double>* tw64, cudaStream_t s) {
  switch (ilog2(nv)) {
#define CASE(L) \
  case L: return edfdv_fx_n<(1 << L)>(f, nrows, e, turn, rest, tw, tw64, s);
    VG_FX_CASES(CASE)
#undef CASE
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vg
