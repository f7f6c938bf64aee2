// The spectral Poisson solve e = Re IFFT(i / kx FFT(rho)) of vlapy/core/field.py:39-49
// as what it is for a real rho, a circular sum with a fixed kernel:
//   e_n = sum_j G[(n - j) mod N] rho_j,  G_n = -(1/N) sum_k inv_kx[k] sin(2 pi k n / N).
//
// The transform in doubles ran on one CTA of N / 8 threads, 64 cycles per FP64
// instruction: 38 us for a driven 64-point run, 60 us at 2048, 187 us by direct
// DFT at 48.  The sum is N^2 products, but on 64-bit integers (rho scaled by its
// largest value, G in Q62, sums kept in 96 bits) a product is some 20 ordinary
// instructions, every CTA takes 32 points, and the result is exact but for G's
// own rounding (a few 2^-53 of its largest value).  The driver's sines are
// evaluated by one warp meanwhile, one point a lane.
#include "vg_f64_body.cuh"
#include "vg_internal.cuh"
#include "vg_poisson_fx.cuh"

namespace vg {

namespace {

// double-double h + l += p + pe
__device__ __forceinline__ void dd_acc(double& h, double& l, double p, double pe) {
  const double t = h + p, z = t - h;
  l += ((h - (t - z)) + (p - z)) + pe;
  h = t;
}
// sin(2 pi q / nx), q < nx (in k_green itself they were most of its time: 0.3 ms at
// 4095)
__global__ void __launch_bounds__(128) k_sines(int nx, double* __restrict__ out) {
  const int q = blockIdx.x * 128 + threadIdx.x;
  if (q < nx) out[q] = sinpi(2.0 * (double)q / (double)nx);
}
// G of run blockIdx.y at n = the warp: the lanes' double-double sums over every
// 32nd bin, added across the warp and rounded to double
__global__ void __launch_bounds__(128) k_green(const double* __restrict__ inv_kx, const double* __restrict__ sines, int nx,
                                               double* __restrict__ out) {
  const int n = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (n > nx / 2) return;
  const double* inv = inv_kx + (size_t)blockIdx.y * nx;
  double h = 0.0, l = 0.0;
  int q = (int)(((long long)n * (lane + 1)) % nx);
  const int step = (int)(((long long)n * 32) % nx);
  for (int k = lane + 1; 2 * k < nx; k += 32) {
    // sin is odd in k: the bins k and nx - k together
    const double c = inv[k] - inv[nx - k], s = sines[q];
    const double p = c * s;
    dd_acc(h, l, p, fma(c, s, -p));
    q += step;
    if (q >= nx) q -= nx;
  }
  for (int m = 16; m > 0; m >>= 1) {
    const double oh = __shfl_down_sync(0xffffffffu, h, m), ol = __shfl_down_sync(0xffffffffu, l, m);
    dd_acc(h, l, oh, ol);
  }
  if (lane != 0) return;
  // (the bins 0 and nx / 2 of a real rho do not act, unless they are no numbers)
  const double g = -(h + l) / (double)nx + 0.0 * (inv[0] + (nx % 2 ? 0.0 : inv[nx / 2]));
  double* o = out + (size_t)blockIdx.y * nx;
  o[n] = g;
  if (n > 0 && 2 * n != nx) o[nx - n] = -g;
}

// the table of run blockIdx.x from its doubles
__global__ void __launch_bounds__(256) k_green_fx(const double* __restrict__ work, int nx, int2* __restrict__ g,
                                                  int* __restrict__ e) {
  __shared__ unsigned red[8];
  const double* w = work + (size_t)blockIdx.x * nx;
  unsigned mx = 0;
  for (int n = threadIdx.x; n < nx; n += blockDim.x) mx = max(mx, fx_exp_bits(w[n]));
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  for (int q = 0; q < 8; ++q) mx = max(mx, red[q]);
  // |G| < 2^ee: the largest exponent field plus one, less the bias
  const int ee = (int)(mx >> 20) - 1022;
  if (threadIdx.x == 0) e[blockIdx.x] = (mx >> 20) == 0x7ff ? 0x7ff : ee;
  for (int n = threadIdx.x; n < nx; n += blockDim.x) {
    const long long q = (mx >> 20) == 0x7ff ? 0 : __double2ll_rn(ldexp(w[n], 62 - ee));
    g[(size_t)blockIdx.x * nx + n] = make_int2(fx_hi(q), fx_lo(q));
  }
}

}  // namespace

cudaError_t build_poisson_fx(const double* inv_kx, int nx, int n_runs, int2* g, int* e, double* work, cudaStream_t s) {
  double* sines = work + (size_t)n_runs * nx;
  k_sines<<<div_up(nx, 128), 128, 0, s>>>(nx, sines);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  k_green<<<dim3(div_up(nx / 2 + 1, 4), n_runs), 128, 0, s>>>(inv_kx, sines, nx, work);
  err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  k_green_fx<<<n_runs, 256, 0, s>>>(work, nx, g, e);
  return cudaGetLastError();
}

// points n0 .. n0 + 31 of one run by the CTA's 256 threads; smem: nx + 1 int2
__device__ __forceinline__ void poisson_fx_tile(const double* __restrict__ dens, int is_density, int nx, int n0,
                                                const int2* __restrict__ g, int eg,
                                                const double* __restrict__ driver, int use_pulses,
                                                const vg_pulse* __restrict__ P, int np, const double* __restrict__ x,
                                                const FieldTimeDev& ft, double* __restrict__ e, int2* rho, int* flags) {
  __shared__ unsigned red[8];
  __shared__ Acc96 part[8][32];
  __shared__ double drv[32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = n0 + lane;
  // rho as integers, eight times the scale of vg_fx.cuh, each split in signed halves
  unsigned mx = 0;
  for (int j = threadIdx.x; j < nx; j += 256)
    mx = max(mx, fx_exp_bits(is_density ? sub_rn(1.0, dens[j]) : dens[j]));
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) red[w] = mx;
  __syncthreads();
  for (int q = 0; q < 8; ++q) mx = max(mx, red[q]);
  const int E = fx_exp(mx);
  const bool bad = E == FX_NONFINITE || eg == 0x7ff;
  for (int j = threadIdx.x; j < nx; j += 256) {
    const long long r = bad ? 0 : fx_from_double(is_density ? sub_rn(1.0, dens[j]) : dens[j], E) << 3;
    rho[j] = make_int2(fx_hi(r), fx_lo(r));
  }
  __syncthreads();
  if (w == 7) drv[lane] = n < nx ? driver_value(driver, use_pulses, P, np, field_time(ft), x, n) : 0.0;
  Acc96 s = {0, 0};
  if (n < nx) {
    int k = n - w;  // (n - j) mod nx
    if (k < 0) k += nx;
#pragma unroll 4
    for (int j = w; j < nx; j += 8) {
      const int2 r = rho[j], c = g[k];
      const long long t = 0x80000000ll + wide(r.y, c.x) + wide(r.x, c.y);
      acc_add(s, wide(r.x, c.x) + (t >> 32));
      k -= 8;
      if (k < 0) k += nx;
      if (k < 0) k += nx;  // nx < 8
    }
  }
  part[w][lane] = s;
  __syncthreads();
  if (w != 0 || n >= nx) return;
  for (int q = 1; q < 8; ++q) acc_add96(s, part[q][lane]);
  // rho G 2^(FX_SCALE - E + 62 - eg + 3 - 64)
  const double self = bad ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(acc_to_double(s), E - FX_SCALE + eg - 1);
  const double en = add_rn(drv[lane], self);
  e[n] = en;
  if (flags && !isfinite(en)) atomicOr(flags, VG_FLAG_NONFINITE);
}

__global__ void __launch_bounds__(256) k_poisson_fx(const double* __restrict__ dens, int is_density, int nx, PoissonFx t,
                                                    const double* __restrict__ driver, int use_pulses,
                                                    const vg_pulse* __restrict__ P, int np,
                                                    const double* __restrict__ x, FieldTimeDev ft,
                                                    double* __restrict__ e, int* flags) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  poisson_fx_tile(dens, is_density, nx, blockIdx.x * 32, t.g, *t.e, driver, use_pulses, P, np, x, ft, e,
                  reinterpret_cast<int2*>(smem_raw), flags);
}

// (run, tile) items of one nx, no driver
__global__ void __launch_bounds__(256) k_poisson_fx_runs(const int* __restrict__ x_off, const double* __restrict__ dens,
                                                         int nx, PoissonFx t, double* __restrict__ e, int* flags) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int r = blockIdx.y, off = x_off[r];
  const FieldTimeDev ft = {};
  poisson_fx_tile(dens + off, 1, nx, blockIdx.x * 32, t.g + (size_t)r * nx, t.e[r], nullptr, 0, nullptr, 0, nullptr, ft,
                  e + off, reinterpret_cast<int2*>(smem_raw), flags);
}

cudaError_t launch_poisson_fx(const vg_plan& p, const double* dens, int is_density, const double* driver,
                              const FieldTimeDev& ft, int use_pulses, double* e, cudaStream_t s) {
  const size_t smem = (size_t)p.nx * sizeof(int2);
  cudaError_t err = ensure_smem((const void*)k_poisson_fx, smem);
  if (err != cudaSuccess) return err;
  k_poisson_fx<<<div_up(p.nx, 32), 256, smem, s>>>(dens, is_density, p.nx, {p.green, p.green_e}, driver, use_pulses,
                                                   p.pulses, p.n_pulses, p.x, ft, e, p.flags);
  return cudaGetLastError();
}

cudaError_t launch_poisson_fx_runs(const int* x_off, int n_runs, const double* dens, int nx, const PoissonFx& t,
                                   double* e, int* flags, cudaStream_t s) {
  const size_t smem = (size_t)nx * sizeof(int2);
  cudaError_t err = ensure_smem((const void*)k_poisson_fx_runs, smem);
  if (err != cudaSuccess) return err;
  for (int r0 = 0; r0 < n_runs; r0 += 65535) {
    const int n = n_runs - r0 < 65535 ? n_runs - r0 : 65535;
    k_poisson_fx_runs<<<dim3(div_up(nx, 32), n), 256, smem, s>>>(x_off + r0, dens, nx, {t.g + (size_t)r0 * nx, t.e + r0},
                                                                 e, flags);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

}  // namespace vg
