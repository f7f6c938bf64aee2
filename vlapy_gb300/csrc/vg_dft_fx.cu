// Fixed-point exponential advection of lines whose length N is not a power of
// two (the reference's scipy.fft takes any length): the line's DFT by its
// definition, on 64-bit integers.
//
// In doubles the direct DFT was 4 N^2 FP64 instructions a line at 64 cycles each
// and scheduler, one CTA per line: 708 us for 48 rows of 720.  Here
//  * a real line is folded, E_n = x_n + x_{N-n} and O_n = x_n - x_{N-n}, so that a
//    bin is sum E_n cos + i sum -O_n sin over half the points, and likewise on the
//    way back two points share their sums over the bins: N^2 products a line in
//    all instead of 4 N^2;
//  * a product is three wide multiplies and two adds;
//  * the bins (then the points) of a line are spread over CTAs: 32 a CTA, four
//    lanes to each, two lines at a time (one load of an angle serves both).
// A line is scaled so that the sum of its moduli, which bounds every bin, fills the
// 64 bits of the accumulators, and so are its bins on the way back (they go
// through scratch between the two kernels).  A step of 48 x 720 (two half kicks, a
// drift) went from 1.45 to 0.07 ms; the errors stay within twice the bound of a
// power-of-two transform in doubles where the direct sums in doubles were at
// several times it.
#include <algorithm>

#include "vg_advect_fx.cuh"
#include "vg_internal.cuh"

namespace vg {

namespace {

constexpr int DFT_LINES = 2;  // (lanes pick their line's sums by it)
constexpr int DFT_OUT = 32;  // bins or points of a CTA
constexpr int DFT_BLOCK = 4 * DFT_OUT;

__host__ __device__ constexpr int dft_bins(int n) { return n / 2 + 1; }
constexpr int DFT_BAD = 0x7fffffff;  // a line's scale when it is not finite
// (|re| + |im|) / 2^42, rounded up
__device__ __forceinline__ unsigned mod42(long long a) { return ((unsigned)abs((int)(a >> 32)) >> 10) + 1; }

__global__ void k_dft_table(int N, const fxw* __restrict__ tw, fxw* __restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= N) return;
  // q / N turns in units of 2^-64, by two 32-bit steps of long division
  const unsigned long long a = ((unsigned long long)q << 32) / (unsigned)N, r = ((unsigned long long)q << 32) % (unsigned)N;
  const unsigned long long b = ((r << 32) + (unsigned)N / 2) / (unsigned)N;
  out[q] = fx_mult(fx_sincos((a << 32) + b, tw));
}

// a product with its accumulator: s += a w / 2^64 for a in signed halves
__device__ __forceinline__ void mac(long long& s, int2 a, int wh, int wl) {
  const long long t = 0x80000000ll + wide(a.y, wh) + wide(a.x, wl);
  s += wide(a.x, wh) + (t >> 32);
}
__device__ __forceinline__ int2 halves(long long a) { return make_int2(fx_hi(a), fx_lo(a)); }
// sums over the four lanes of an output
__device__ __forceinline__ long long quad_sum(long long s) {
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s + __shfl_xor_sync(0xffffffffu, s, 2);
}

// E_n and O_n of a line as signed halves
struct __align__(16) Fold {
  int2 e, o;
};

template <int B>
using DftSums = unsigned[DFT_LINES][B / 32];

// by CTAs of B threads, B / 4 bins or points each
// forward: bins blockIdx.x B / 4 .. of lines l0, l0 + 1, rotated, into G[0 ..
// 1][bins], and the lines' scales into scale[0 .. 1].  ang: the N angles, fold: room
// for [lines][bins], both in shared memory
template <int B>
__device__ __forceinline__ void dft_fwd(const double* __restrict__ f, int N, int n_lines, long long es, long long ls,
                                        const double* __restrict__ c, FxTurn turn, const float* __restrict__ rest, float dt,
                                        const fxw* __restrict__ tw, const fxw* __restrict__ angles, fx* G, int* scale,
                                        int l0, fxw* ang, Fold* fold, DftSums<B>& red) {
  const int K = dft_bins(N);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int q = threadIdx.x; q < N; q += B) ang[q] = angles[q];
  int E[DFT_LINES];
  bool bad[DFT_LINES];
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    unsigned mx = 0;
    if (l0 + u < n_lines)
      for (int n = threadIdx.x; n < N; n += B) mx = max(mx, fx_exp_bits(f[(l0 + u) * ls + n * es]));
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) red[u][w] = mx;
  }
  __syncthreads();
  unsigned l1s[DFT_LINES];
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    unsigned mx = 0;
    for (int q = 0; q < B / 32; ++q) mx = max(mx, red[u][q]);
    E[u] = fx_exp(mx);
    const bool on = l0 + u < n_lines;
    bad[u] = E[u] == FX_NONFINITE || !isfinite(on ? c[l0 + u] : 0.0);
    unsigned l1 = 0;
    if (on && !bad[u])
      for (int n = threadIdx.x; n < N; n += B) l1 += mod42(fx_from_double(f[(l0 + u) * ls + n * es], E[u]));
    l1s[u] = __reduce_add_sync(0xffffffffu, l1);
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u)
    if (lane == 0) red[u][w] = l1s[u];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    // sum |x| 2^-g <= 2^64: the products are a quarter of that; |E_n| <= 2^60.5 2^-g <= 2^62
    unsigned l1 = 0;
    for (int q = 0; q < B / 32; ++q) l1 += red[u][q];
    int g = -1;
    while (g < 9 && (g < 0 ? l1 > (1u << 21) : (l1 >> g) >= (1u << 22))) ++g;
    E[u] += g;
    const bool on = l0 + u < n_lines;
    if (on && blockIdx.x == 0 && threadIdx.x == 0) scale[u] = bad[u] ? DFT_BAD : E[u];
    const double* fl = f + (l0 + u) * ls;
    for (int n = threadIdx.x; n < K; n += B) {
      const int m = n == 0 ? 0 : N - n;
      const long long x = on && !bad[u] ? fx_from_double(fl[n * es], E[u]) : 0;
      const long long y = on && !bad[u] && m != n && n > 0 ? fx_from_double(fl[m * es], E[u]) : 0;
      // (the points 0 and N / 2 have no partner: their sine is zero)
      fold[u * K + n] = {halves(x + y), halves(x - y)};
    }
  }
  const int k = blockIdx.x * (B / 4) + (threadIdx.x >> 2), part = threadIdx.x & 3;
  // lane u of an output's four rotates line u: its phase, while the sums wait for nothing
  const bool rot = part < DFT_LINES && k < K && l0 + part < n_lines;
  fxw p = {};
  if (rot) {
    const double cl = (part ? bad[1] : bad[0]) ? 0.0 : c[l0 + part];
    // (the wavenumber's own rounding, some 2^-53 of the phase, in FP32)
    const long long own = __float2ll_rn(-rest[k] * dt * (float)cl);
    p = fx_mult(fx_sincos((unsigned long long)k * fx_turn(turn, cl) + (unsigned long long)own, tw));
  }
  __syncthreads();
  long long re[DFT_LINES] = {}, im[DFT_LINES] = {};
  if (k < K) {
    int q = (k * part) % N;
    const int step = (4 * k) % N;
#pragma unroll 2
    for (int n = part; n < K; n += 4) {
      const fxw a = ang[q];
#pragma unroll
      for (int u = 0; u < DFT_LINES; ++u) {
        const Fold x = fold[u * K + n];
        mac(re[u], x.e, a.xh, a.xl);
        mac(im[u], x.o, a.yh, a.yl);
      }
      q += step;
      if (q >= N) q -= N;
    }
  }
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    re[u] = quad_sum(re[u]);
    im[u] = quad_sum(im[u]);
  }
  if (!rot) return;
  fx z = fx_cmul<0, false>({part ? re[1] : re[0], -(part ? im[1] : im[0])}, p);
  // half weight for the bins that have no mirror image
  if (k == 0 || 2 * k == N) z = fx_down<1>(z);
  G[part * K + k] = z;
}

// back: points blockIdx.x B / 4 .. and N minus these of lines l0, l0 + 1 from their
// bins (re and im as a Fold, in shared memory)
template <int B>
__device__ __forceinline__ void dft_inv(double* __restrict__ f, int N, int n_lines, long long es, long long ls,
                                        const fx* G, const int* scale, int l0, double inv, const fxw* ang, Fold* bins, DftSums<B>& red) {
  const int K = dft_bins(N);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // the sum of |re| + |im| over the bins (in units of 2^42, rounded up) bounds every sum
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    unsigned l1 = 0;
    if (l0 + u < n_lines)
      for (int k = threadIdx.x; k < K; k += B) {
        const fx z = G[u * K + k];
        l1 += mod42(z.x) + mod42(z.y);
      }
    l1 = __reduce_add_sync(0xffffffffu, l1);
    if (lane == 0) red[u][w] = l1;
  }
  __syncthreads();
  int up[DFT_LINES];
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    unsigned l1 = 0;
    for (int q = 0; q < B / 32; ++q) l1 += red[u][q];
    // up to two bits up (bins <= 2^60), or as many down as the sums need: l1 2^up <= 2^22
    int s = 2;
    while (s > -10 && (s >= 0 ? l1 > ((1u << 22) >> s) : (l1 >> -s) >= (1u << 22))) --s;
    up[u] = s;
    if (l0 + u < n_lines)
      for (int k = threadIdx.x; k < K; k += B) {
        fx z = G[u * K + k];
        if (s >= 0) {
          z.x = (long long)((unsigned long long)z.x << s);
          z.y = (long long)((unsigned long long)z.y << s);
        } else {
          z.x = (z.x + (1ll << (-s - 1))) >> -s;
          z.y = (z.y + (1ll << (-s - 1))) >> -s;
        }
        bins[u * K + k] = {halves(z.x), halves(z.y)};
      }
    else
      for (int k = threadIdx.x; k < K; k += B) bins[u * K + k] = {};
  }
  __syncthreads();
  const int n = blockIdx.x * (B / 4) + (threadIdx.x >> 2), part = threadIdx.x & 3;
  long long pc[DFT_LINES] = {}, ps[DFT_LINES] = {};
  if (n < K) {
    int q = (n * part) % N;
    const int step = (4 * n) % N;
#pragma unroll 2
    for (int k = part; k < K; k += 4) {
      const fxw a = ang[q];
#pragma unroll
      for (int u = 0; u < DFT_LINES; ++u) {
        const Fold z = bins[u * K + k];
        mac(pc[u], z.e, a.xh, a.xl);
        mac(ps[u], z.o, a.yh, a.yl);
      }
      q += step;
      if (q >= N) q -= N;
    }
  }
#pragma unroll
  for (int u = 0; u < DFT_LINES; ++u) {
    pc[u] = quad_sum(pc[u]);
    ps[u] = quad_sum(ps[u]);
  }
  // lanes 2 u and 2 u + 1 of the four write points n and N - n of line u
  const int u = part >> 1, m = (part & 1) ? N - n : n;
  if (n >= K || l0 + u >= n_lines || ((part & 1) && (n == 0 || 2 * n == N))) return;
  const int E = scale[u];
  const long long c = u ? pc[1] : pc[0], o = u ? ps[1] : ps[0], v = (part & 1) ? c + o : c - o;
  // forward x 2^(FX_SCALE - E) / 4 / 4, back / 4 and 2^up, halved weights
  f[(l0 + u) * ls + (long long)m * es] =
      E == DFT_BAD ? __longlong_as_double(0x7ff8000000000000ll) : fx_to_double(v, E - FX_SCALE + 7 - (u ? up[1] : up[0])) * inv;
}

__global__ void __launch_bounds__(DFT_BLOCK) k_dft_fwd_fx(const double* __restrict__ f, int N, int n_lines, long long es,
                                                          long long ls, const double* __restrict__ c, FxTurn turn,
                                                          const float* __restrict__ rest, float dt,
                                                          const fxw* __restrict__ tw, const fxw* __restrict__ angles,
                                                          fx* __restrict__ G, int* __restrict__ scale) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ DftSums<DFT_BLOCK> red;
  fxw* ang = reinterpret_cast<fxw*>(smem_raw);
  const int l0 = blockIdx.y * DFT_LINES;
  dft_fwd<DFT_BLOCK>(f, N, n_lines, es, ls, c, turn, rest, dt, tw, angles, G + (long long)l0 * dft_bins(N), scale + l0, l0, ang,
          reinterpret_cast<Fold*>(ang + N), red);
}
__global__ void __launch_bounds__(DFT_BLOCK) k_dft_inv_fx(double* __restrict__ f, int N, int n_lines, long long es,
                                                          long long ls, const fxw* __restrict__ angles,
                                                          const fx* __restrict__ G, const int* __restrict__ scale,
                                                          double inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ DftSums<DFT_BLOCK> red;
  fxw* ang = reinterpret_cast<fxw*>(smem_raw);
  for (int q = threadIdx.x; q < N; q += DFT_BLOCK) ang[q] = angles[q];
  const int l0 = blockIdx.y * DFT_LINES;
  dft_inv<DFT_BLOCK>(f, N, n_lines, es, ls, G + (long long)l0 * dft_bins(N), scale + l0, l0, inv, ang, reinterpret_cast<Fold*>(ang + N),
                     red);
}
// Short lines, all of whose bins one CTA holds (N < B / 2): both ways in one launch, the
// bins in shared memory.  The same operations, so the same bits.  One warp for N < 16,
// where the barriers are most of the time: 9 points take 8 us, 12 in two launches.
template <int B>
__global__ void __launch_bounds__(B) k_dft_short_fx(double* __restrict__ f, int N, int n_lines, long long es, long long ls,
                                                    const double* __restrict__ c, FxTurn turn, const float* __restrict__ rest,
                                                    float dt, double inv, const fxw* __restrict__ tw,
                                                    const fxw* __restrict__ angles) {
  __shared__ DftSums<B> red;
  __shared__ fxw ang[B / 2];
  __shared__ Fold fold[DFT_LINES * B / 4];
  __shared__ fx bins[DFT_LINES * B / 4];
  __shared__ int scale[DFT_LINES];
  const int l0 = blockIdx.y * DFT_LINES;
  dft_fwd<B>(f, N, n_lines, es, ls, c, turn, rest, dt, tw, angles, bins, scale, l0, ang, fold, red);
  __syncthreads();
  dft_inv<B>(f, N, n_lines, es, ls, bins, scale, l0, inv, ang, fold, red);
}

}  // namespace

size_t dft_fx_scratch(int nx, int nv, bool x, bool v) {
  size_t need = 0;
  if (v) need = (size_t)nx * (dft_bins(nv) * sizeof(fx) + sizeof(int));
  if (x) need = std::max(need, (size_t)nv * (dft_bins(nx) * sizeof(fx) + sizeof(int)));
  return need;
}

cudaError_t build_dft_table(int N, const fxw* tw, fxw* out, cudaStream_t s) {
  k_dft_table<<<div_up(N, 128), 128, 0, s>>>(N, tw, out);
  return cudaGetLastError();
}

cudaError_t launch_dft_fx(double* f, int N, int n_lines, long long es, long long ls, const double* c, FxTurn turn,
                          const float* rest, double dt, const fxw* tw, const fxw* angles, void* scratch, cudaStream_t s) {
  const int K = dft_bins(N);
  const size_t smem = (size_t)N * sizeof(fxw) + (size_t)DFT_LINES * K * sizeof(Fold);
  cudaError_t err = ensure_smem((const void*)k_dft_fwd_fx, smem);
  if (err == cudaSuccess) err = ensure_smem((const void*)k_dft_inv_fx, smem);
  if (err != cudaSuccess) return err;
  fx* G = static_cast<fx*>(scratch);
  int* scale = reinterpret_cast<int*>(G + (size_t)n_lines * K);
  const int tiles = div_up(K, DFT_OUT);
  const double inv = 1.0 / N;
  // grid.y holds at most 65535 line pairs
  for (int l0 = 0; l0 < n_lines; l0 += 2 * 65535) {
    const int n = std::min(n_lines - l0, 2 * 65535);
    const dim3 grid(tiles, div_up(n, DFT_LINES));
    double* fl = f + (long long)l0 * ls;
    if (tiles == 1) {
      if (N < 16) k_dft_short_fx<32><<<grid, 32, 0, s>>>(fl, N, n, es, ls, c + l0, turn, rest, (float)dt, inv, tw, angles);
      else k_dft_short_fx<DFT_BLOCK><<<grid, DFT_BLOCK, 0, s>>>(fl, N, n, es, ls, c + l0, turn, rest, (float)dt, inv, tw, angles);
      err = cudaGetLastError();
      if (err != cudaSuccess) return err;
      continue;
    }
    k_dft_fwd_fx<<<grid, DFT_BLOCK, smem, s>>>(fl, N, n, es, ls, c + l0, turn, rest, (float)dt, tw, angles, G + (size_t)l0 * K,
                                               scale + l0);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    k_dft_inv_fx<<<grid, DFT_BLOCK, smem, s>>>(fl, N, n, es, ls, angles, G + (size_t)l0 * K, scale + l0, inv);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

}  // namespace vg
