// FP64 reductions, field solve and storage step.
//
// The density, the collision operators' moments and every mean over x are evaluated
// with NumPy's pairwise summation tree (a table built at plan creation): leaves of <= 128 terms are
// summed with eight interleaved accumulators (one thread per accumulator chain
// in the row moments), and one thread per moment replays the post-order
// combine program.  Products use
// explicitly rounded intrinsics so nvcc cannot contract them into FMAs.  With
// f equal, they are then bit-identical to the reference's np.trapz and np.mean
// (vlapy/core/field.py:36, vlapy/core/collisions.py, vlapy/core/step.py:174-229).
// The moments that a step stores are nearer to the exact sums than np.trapz's, and
// not its bits (vg_moments_fx.cu).
#include "vg_internal.cuh"
#include "vg_f64_body.cuh"

namespace vg {


// One CTA per row.  The work of a NumPy pairwise sum is spread over the
// threads without changing a single rounding: (A) the integrand products of a
// group of qg moments are formed once per element into shared memory; (B)
// every leaf of <= 128 terms is NumPy's eight interleaved accumulators, each
// a serial chain that one thread runs; (C) one thread per leaf adds the eight
// in NumPy's order plus the tail terms; then one thread per moment replays
// the combine program over the leaves.  Moments of the second phase
// (MOM_DG2) use the vbar the first phase produced.
__global__ void k_row_moments_f64(const double* __restrict__ f, int nv, const double* __restrict__ v,
                                  const double* __restrict__ v_pow, MomSpec spec,
                                  const int* __restrict__ table, double dv,
                                  double* __restrict__ out, int ostride, int qg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nl = table[0];
  double* prod = reinterpret_cast<double*>(smem_raw);  // [qg][nv]
  double* acc = prod + (size_t)qg * nv;               // [qg][nl][8]
  double* leaf = acc + (size_t)qg * nl * 8;           // [nm][nl]
  __shared__ double res[MOM_STRIDE];
  const size_t r = blockIdx.x;
  const double* fr = f + r * nv;
  const int* leaves = table + 2;
  const int nm = spec.nm;
  for (int phase = 0; phase < 2; ++phase) {
    for (int q0 = 0; q0 < nm; q0 += qg) {
      auto active = [&](int q) { return q < nm && (spec.kind[q] == MOM_DG2) == (phase == 1); };
      // (A) products p_q(j)
      for (int idx = threadIdx.x; idx < qg * nv; idx += blockDim.x) {
        const int qq = idx / nv, j = idx - qq * nv, q = q0 + qq;
        if (!active(q)) continue;
        const int kind = spec.kind[q], arg = spec.arg[q];
        const double vbar = kind == MOM_DG2 ? res[arg] : 0.0;
        prod[idx] = mom_product(kind, arg, fr[j], j, v, v_pow, nv, vbar);
      }
      __syncthreads();
      // trapz term j: (dv * (p(j + 1) + p(j))) / 2
      auto term = [&](const double* pq, int j) { return mul_rn(dv, add_rn(pq[j + 1], pq[j])) * 0.5; };
      // (B) the accumulator chains
      for (int idx = threadIdx.x; idx < qg * nl * 8; idx += blockDim.x) {
        const int qq = idx / (nl * 8), rem = idx - qq * nl * 8, L = rem >> 3, a = rem & 7;
        if (!active(q0 + qq) || nv < 2) continue;
        const double* pq = prod + (size_t)qq * nv;
        const int st = leaves[2 * L], len = leaves[2 * L + 1];
        if (len < 8) {
          if (a == 0) {
            double x = 0.0;
            for (int i = 0; i < len; ++i) x = add_rn(x, term(pq, st + i));
            acc[(size_t)qq * nl * 8 + L * 8] = x;
          }
          continue;
        }
        const int stop = len - (len % 8);
        double x = term(pq, st + a);
        for (int i = 8 + a; i < stop; i += 8) x = add_rn(x, term(pq, st + i));
        acc[(size_t)qq * nl * 8 + L * 8 + a] = x;
      }
      __syncthreads();
      // (C) the leaves
      for (int idx = threadIdx.x; idx < qg * nl; idx += blockDim.x) {
        const int qq = idx / nl, L = idx - qq * nl, q = q0 + qq;
        if (!active(q) || nv < 2) continue;
        const double* pq = prod + (size_t)qq * nv;
        const double* ac = acc + (size_t)qq * nl * 8 + L * 8;
        const int st = leaves[2 * L], len = leaves[2 * L + 1];
        double x;
        if (len < 8) {
          x = ac[0];
        } else {
          x = add_rn(add_rn(add_rn(ac[0], ac[1]), add_rn(ac[2], ac[3])), add_rn(add_rn(ac[4], ac[5]), add_rn(ac[6], ac[7])));
          for (int i = len - (len % 8); i < len; ++i) x = add_rn(x, term(pq, st + i));
        }
        leaf[(size_t)q * nl + L] = x;
      }
      __syncthreads();
    }
    for (int q = threadIdx.x; q < nm; q += blockDim.x) {
      if ((spec.kind[q] == MOM_DG2) != (phase == 1)) continue;
      const double val = nv > 1 ? combine_leaves(table, leaf + (size_t)q * nl) : 0.0;
      res[q] = val;
      out[r * ostride + q] = val;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// the density and the collision operator's moments, NumPy's sums bit for bit
// ---------------------------------------------------------------------------

// sum of the nv - 1 trapz terms dv (p_{j+1} + p_j) / 2 of the products p in NumPy's
// order, in every thread.  All threads form the terms; eight lanes then run a
// leaf's eight accumulators, and one thread the combine program, its stack in
// place of the leaves it has taken.  The halving is left to the end (exact; a
// factor of two commutes with every rounding above the subnormal range).
// p: nv products in shared memory, or the row itself in global memory.
__device__ __forceinline__ double trapz_exact(const double* p, int nv, double dv, const int* __restrict__ table,
                                              int by_level, double* term, double* leaf, double* result) {
  for (int j = threadIdx.x; j < nv - 1; j += blockDim.x) term[j] = mul_rn(dv, add_rn(p[j + 1], p[j]));
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nl = table[0], np = table[1];
  const int* leaves = table + 2;
  const int a = lane & 7;
  for (int L0 = 4 * w; L0 < nl; L0 += 4 * (blockDim.x >> 5)) {
    const int L = L0 + (lane >> 3);
    const int st = L < nl ? leaves[2 * L] : 0, len = L < nl ? leaves[2 * L + 1] : 0;
    const int stop = len - (len % 8);
    double x = 0.0;
    if (len < 8) {
      if (a == 0)
        for (int i = 0; i < len; ++i) x = add_rn(x, term[st + i]);
    } else {
      x = term[st + a];
      for (int i = 8 + a; i < stop; i += 8) x = add_rn(x, term[st + i]);
    }
    double r = x;
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) {
      const double o = __shfl_down_sync(0xffffffffu, r, m, 8);
      r = add_rn(r, o);
    }
    if (a == 0 && L < nl) {
      if (len < 8) r = x;
      else
        for (int i = stop; i < len; ++i) r = add_rn(r, term[st + i]);
      leaf[L] = r;
    }
  }
  __syncthreads();
  const int* prog = leaves + 2 * nl;
  if (by_level) {
    // the tree's additions level by level, side by side (one thread running the
    // program waited some 10,000 cycles for 31 leaves: density 77 -> 66 us, DG moments
    // 261 -> 234 us at 2048 x 4096)
    if (w == 0) {
      const int* lv = prog + np;
      const int levels = *lv++;
      for (int l = 0; l < levels; ++l) {
        const int n = *lv++;
        for (int i = lane; i < n; i += 32) {
          const int dst = lv[2 * i], src = lv[2 * i + 1];
          leaf[dst] = add_rn(leaf[dst], leaf[src]);
        }
        lv += 2 * n;
        __syncwarp();
      }
      if (lane == 0) *result = nv > 1 ? leaf[0] * 0.5 : 0.0;
    }
  } else if (threadIdx.x == 0) {
    int sp = 0;
    for (int i = 0; i < np; ++i) {
      const int op = prog[i];
      if (op >= 0) {
        leaf[sp++] = leaf[op];  // op >= sp: the stack never passes the leaves taken
      } else {
        --sp;
        leaf[sp - 1] = add_rn(leaf[sp - 1], leaf[sp]);
      }
    }
    *result = nv > 1 ? leaf[0] * 0.5 : 0.0;
  }
  __syncthreads();
  return *result;
}

// One CTA per row.  DENSITY: out[0] = trapz f.  DG: out[0] = vbar = trapz(f v),
// out[1] = trapz(f (v - vbar)^2).  LB: out[1] = trapz(f v^2.0).  Three FP64
// instructions per cell for the sum and one or three for the product; the
// general kernel above spends one more per moment and leaves the terms to the
// chains' few threads (2048 x 4096: density 137 -> 79 us, DG 353 -> 260 us;
// 64 x 1024: DG 19 -> 13 us).
template <int OP>
__global__ void __launch_bounds__(256) k_trapz_f64(const double* __restrict__ f, int nv, const double* __restrict__ v,
                                                   const double* __restrict__ v2, const int* __restrict__ table,
                                                   int by_level, double dv, double* __restrict__ out, int stride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double res[2];
  double* term = reinterpret_cast<double*>(smem_raw);  // [nv]
  double* leaf = term + nv;                            // [n_leaves]
  double* prod = leaf + table[0];                      // [nv] (DG, LB)
  const double* fr = f + (size_t)blockIdx.x * nv;
  double* o = out + (size_t)blockIdx.x * stride;
  if constexpr (OP == TRAPZ_DENSITY) {
    const double n = trapz_exact(fr, nv, dv, table, by_level, term, leaf, &res[0]);
    if (threadIdx.x == 0) o[0] = n;
  } else if constexpr (OP == TRAPZ_LB) {
    for (int j = threadIdx.x; j < nv; j += blockDim.x) prod[j] = mul_rn(fr[j], v2[j]);
    __syncthreads();
    const double t = trapz_exact(prod, nv, dv, table, by_level, term, leaf, &res[0]);
    if (threadIdx.x == 0) o[1] = t;
  } else {
    for (int j = threadIdx.x; j < nv; j += blockDim.x) prod[j] = mul_rn(fr[j], v[j]);
    __syncthreads();
    const double vbar = trapz_exact(prod, nv, dv, table, by_level, term, leaf, &res[0]);
    for (int j = threadIdx.x; j < nv; j += blockDim.x) {
      const double d = sub_rn(v[j], vbar);
      prod[j] = mul_rn(fr[j], mul_rn(d, d));
    }
    __syncthreads();
    const double t = trapz_exact(prod, nv, dv, table, by_level, term, leaf, &res[1]);
    if (threadIdx.x == 0) {
      o[0] = vbar;
      o[1] = t;
    }
  }
}

cudaError_t launch_trapz_f64(const vg_plan& p, int op, const double* f, double* out, int stride, cudaStream_t s) {
  const size_t smem = ((op == TRAPZ_DENSITY ? 1 : 2) * (size_t)p.nv + (size_t)p.pw_v_leaves) * sizeof(double);
  if (smem > ((size_t)220 << 10)) {
    // longer rows: the general kernel
    MomSpec spec = {};
    spec.nm = op == TRAPZ_DENSITY ? 1 : 2;
    spec.kind[0] = op == TRAPZ_DG ? MOM_V : MOM_ONE;
    spec.kind[1] = op == TRAPZ_DG ? MOM_DG2 : MOM_W;
    return launch_row_moments_f64(p, f, spec, out, stride, s);
  }
  const void* k = op == TRAPZ_DENSITY ? (const void*)k_trapz_f64<TRAPZ_DENSITY>
                : op == TRAPZ_DG      ? (const void*)k_trapz_f64<TRAPZ_DG>
                                      : (const void*)k_trapz_f64<TRAPZ_LB>;
  cudaError_t err = ensure_smem(k, smem);
  if (err != cudaSuccess) return err;
  const int block = p.nv >= 1024 ? 256 : p.nv >= 512 ? 128 : 64;
  if (op == TRAPZ_DENSITY)
    k_trapz_f64<TRAPZ_DENSITY><<<p.nx, block, smem, s>>>(f, p.nv, p.v, p.v_pow, p.pw_v, p.pw_v_levels, p.dv, out, stride);
  else if (op == TRAPZ_DG)
    k_trapz_f64<TRAPZ_DG><<<p.nx, block, smem, s>>>(f, p.nv, p.v, p.v_pow, p.pw_v, p.pw_v_levels, p.dv, out, stride);
  else
    k_trapz_f64<TRAPZ_LB><<<p.nx, block, smem, s>>>(f, p.nv, p.v, p.v_pow, p.pw_v, p.pw_v_levels, p.dv, out, stride);
  return cudaGetLastError();
}

cudaError_t launch_row_moments_f64(const vg_plan& p, const double* f, const MomSpec& spec,
                                   double* out, int out_stride, cudaStream_t s) {
  // products of as many moments at once as fit in 64 KB (at least one)
  const int nm = spec.nm;
  int qg = (int)(65536 / ((size_t)p.nv * sizeof(double)));
  qg = qg < 1 ? 1 : (qg > nm ? nm : qg);
  const size_t nl = (size_t)p.pw_v_leaves;
  const size_t smem = ((size_t)qg * p.nv + (size_t)qg * nl * 8 + (size_t)nm * nl) * sizeof(double);
  cudaError_t err = ensure_smem((const void*)k_row_moments_f64, smem);
  if (err != cudaSuccess) return err;
  k_row_moments_f64<<<p.nx, 256, smem, s>>>(f, p.nv, p.v, p.v_pow, spec, p.pw_v, p.dv, out, out_stride, qg);
  return cudaGetLastError();
}


__global__ void k_driver(const vg_pulse* __restrict__ P, int np, const double* __restrict__ x, int nx,
                         FieldTimeDev ft, double* __restrict__ out) {
  const double t = field_time(ft);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x)
    out[i] = pulse_sum(P, np, t, x[i]);
}

static FieldTimeDev to_dev(const FieldTime& ft) {
  FieldTimeDev d;
  d.t_ptr = ft.t_ptr;
  d.t_host = ft.t_host;
  d.nadd = ft.nadd;
  for (int i = 0; i < 6; ++i) d.add[i] = ft.add[i];
  return d;
}

cudaError_t launch_driver(const vg_plan& p, const FieldTime& ft, double* out, cudaStream_t s) {
  k_driver<<<div_up(p.nx, 256), 256, 0, s>>>(p.pulses, p.n_pulses, p.x, p.nx, to_dev(ft), out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// spectral Poisson, vlapy/core/field.py:39-88
// ---------------------------------------------------------------------------


template <int NX>
__global__ void __launch_bounds__(fft_threads<double>(NX)) k_poisson_fft_f64(
    const double* __restrict__ dens, int is_density, const double* __restrict__ inv_kx,
    const double* __restrict__ driver, int use_pulses, const vg_pulse* __restrict__ P, int np,
    const double* __restrict__ x, FieldTimeDev ft, const cx<double>* __restrict__ tw,
    double* __restrict__ e, int* flags) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  poisson_fft_body<NX>(dens, is_density, inv_kx, driver, use_pulses, P, np, x, ft, tw, e,
                       reinterpret_cast<cx<double>*>(smem_raw), threadIdx.x, flags);
}

// Direct DFT for the other lengths past the Green's function's (O(nx^2), one CTA).
__global__ void k_poisson_dft_f64(const double* __restrict__ dens, int is_density, int nx,
                                  const double* __restrict__ inv_kx, const double* __restrict__ driver,
                                  int use_pulses, const vg_pulse* __restrict__ P, int np,
                                  const double* __restrict__ x, FieldTimeDev ft,
                                  double* __restrict__ work, double* __restrict__ e, int* flags) {
  // work: [nx] rho, then [2*nx] spectrum
  double* rho = work;
  cx<double>* Y = reinterpret_cast<cx<double>*>(work + nx + (nx & 1));
  for (int n = threadIdx.x; n < nx; n += blockDim.x) rho[n] = is_density ? sub_rn(1.0, dens[n]) : dens[n];
  __syncthreads();
  for (int k = threadIdx.x; k < nx; k += blockDim.x) {
    double zr = 0.0, zi = 0.0;
    for (int n = 0; n < nx; ++n) {
      const long long q = ((long long)n * k) % nx;
      double sn, cs;
      sincospi(2.0 * (double)q / (double)nx, &sn, &cs);
      zr += rho[n] * cs;
      zi -= rho[n] * sn;
    }
    const double ik = inv_kx[k];
    Y[k] = {-ik * zi, ik * zr};
  }
  __syncthreads();
  const double tt = field_time(ft);
  for (int n = threadIdx.x; n < nx; n += blockDim.x) {
    double acc = 0.0;
    for (int k = 0; k < nx; ++k) {
      const long long q = ((long long)n * k) % nx;
      double sn, cs;
      sincospi(2.0 * (double)q / (double)nx, &sn, &cs);
      acc += Y[k].x * cs - Y[k].y * sn;
    }
    const double en = driver_value(driver, use_pulses, P, np, tt, x, n) + acc / nx;
    e[n] = en;
    if (flags && !isfinite(en)) atomicOr(flags, VG_FLAG_NONFINITE);
  }
}

namespace {
template <int NX>
cudaError_t poisson_n(const vg_plan& p, const double* dens, int is_density, const double* driver,
                      const FieldTime& ft, double* e, cudaStream_t s) {
  constexpr int G = fft_threads<double>(NX);
  const size_t smem = (size_t)sp_len<double>(NX) * sizeof(cx<double>);
  cudaError_t err = ensure_smem((const void*)k_poisson_fft_f64<NX>, smem);
  if (err != cudaSuccess) return err;
  k_poisson_fft_f64<NX><<<1, G, smem, s>>>(dens, is_density, p.inv_kx, driver, ft.use_pulses, p.pulses,
                                           p.n_pulses, p.x, to_dev(ft), p.tw64, e, p.flags);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_poisson_f64(const vg_plan& p, const double* dens, int is_density, const double* driver,
                               const FieldTime& ft, double* e, cudaStream_t s) {
  // (transforms: nx = 8192, and the solve without allocation, which has no table)
  if (p.green) return launch_poisson_fx(p, dens, is_density, driver, to_dev(ft), ft.use_pulses, e, s);
  if (p.nx_pow2 && p.nx <= 8192) {
    switch (ilog2(p.nx)) {
      case 1: return poisson_n<2>(p, dens, is_density, driver, ft, e, s);
      case 2: return poisson_n<4>(p, dens, is_density, driver, ft, e, s);
      case 3: return poisson_n<8>(p, dens, is_density, driver, ft, e, s);
      case 4: return poisson_n<16>(p, dens, is_density, driver, ft, e, s);
      case 5: return poisson_n<32>(p, dens, is_density, driver, ft, e, s);
      case 6: return poisson_n<64>(p, dens, is_density, driver, ft, e, s);
      case 7: return poisson_n<128>(p, dens, is_density, driver, ft, e, s);
      case 8: return poisson_n<256>(p, dens, is_density, driver, ft, e, s);
      case 9: return poisson_n<512>(p, dens, is_density, driver, ft, e, s);
      case 10: return poisson_n<1024>(p, dens, is_density, driver, ft, e, s);
      case 11: return poisson_n<2048>(p, dens, is_density, driver, ft, e, s);
      case 12: return poisson_n<4096>(p, dens, is_density, driver, ft, e, s);
      case 13: return poisson_n<8192>(p, dens, is_density, driver, ft, e, s);
      default: break;
    }
  }
  k_poisson_dft_f64<<<1, 256, 0, s>>>(dens, is_density, p.nx, p.inv_kx, driver, ft.use_pulses, p.pulses,
                                      p.n_pulses, p.x, to_dev(ft), p.etmp, e, p.flags);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// storage step, vlapy/core/step.py:116-283
// ---------------------------------------------------------------------------

// fields[.][i] and the seven x-means; mom holds n, j, T, q, fv4, vN, f^2, f log f
// per row.  One warp per series (lanes that took different series ran one after
// the other, 25 us at nx = 64 against 8), the eighth copies the fields.
__global__ void __launch_bounds__(256) k_fields_series_f64(const double* __restrict__ mom, const double* __restrict__ e,
                                                           const double* __restrict__ de, int nx, int i, vg_history h,
                                                           const int* __restrict__ table) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nl = table[0];
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t off = (size_t)i * nx;
  for (int idx = threadIdx.x; idx < 8 * nx; idx += blockDim.x) {
    const int k = idx / nx, n = idx - k * nx;
    if (h.fields[k]) h.fields[k][off + n] = k == 0 ? e[n] : k == 1 ? (de ? de[n] : 0.0) : mom[(size_t)n * MOM_STRIDE + k - 2];
  }
  // series sources: n, j, T, e^2, de^2, f^2, flogf
  if (q >= 7 || !h.series[q]) return;
  double* leaf = reinterpret_cast<double*>(smem_raw) + q * nl;
  if (q == 3) {
    warp_leaf_sums(table, lane, leaf, [&](int n) { return mul_rn(e[n], e[n]); });
  } else if (q == 4) {
    warp_leaf_sums(table, lane, leaf, [&](int n) { return de ? mul_rn(de[n], de[n]) : 0.0; });
  } else {
    const double* m = mom + (q < 3 ? q : q + 1);
    warp_leaf_sums(table, lane, leaf, [&](int n) { return m[(size_t)n * MOM_STRIDE]; });
  }
  __syncwarp();
  if (lane == 0) h.series[q][i] = __ddiv_rn(combine_leaves(table, leaf), (double)nx);
}

// stored_f[i][slot][v] = complex64(sum_x f[x][v] exp(-2 pi i m x / nx)).  A CTA
// takes 32 columns; its sixteen warps take every sixteenth row, eight loads in
// flight, and the partial sums are added in warp order.  MODES_AT_ONCE modes share one pass over f (their
// cosines and sines come from a table of the nx angles in shared memory, or, for
// long columns, straight from the plan's table or sincospi).  One thread per
// column had run 32 CTAs of serial loops: 2.01 ms at 2048 x 4096 with two modes,
// 136 us with eight warps and four loads, now 60 (the three FP64 operations a
// cell take 47).
constexpr int MODES_AT_ONCE = 2;
constexpr int MODES_TABLE_NX = 4096;
__device__ __forceinline__ cx<double> mode_angle(int q, int nx, int nx_pow2, const cx<double>* __restrict__ tw) {
  if (q == 0) return {1.0, 0.0};
  if (nx_pow2) {
    // exp(-2 pi i q / nx) from the span-ordered table; q >= nx/2 is the negated
    // entry q - nx/2
    const bool hi = 2 * q >= nx;
    const cx<double> w = tw[tw_index(nx, hi ? q - nx / 2 : q)];
    return hi ? cx<double>{-w.x, -w.y} : w;
  }
  double sn, cs;
  sincospi(2.0 * (double)q / (double)nx, &sn, &cs);
  return {cs, -sn};
}
constexpr int MODES_WARPS = 16;
__global__ void __launch_bounds__(32 * MODES_WARPS) k_store_modes_f64(const double* __restrict__ f, int nx, int nv, int n_modes,
                                                         int n_slots, int nx_pow2, const cx<double>* __restrict__ tw,
                                                         int i, cx<float>* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double part[2 * MODES_AT_ONCE][MODES_WARPS][32];
  cx<double>* angles = reinterpret_cast<cx<double>*>(smem_raw);
  const bool table = nx <= MODES_TABLE_NX && n_modes > 1;
  if (table)
    for (int q = threadIdx.x; q < nx; q += blockDim.x) angles[q] = mode_angle(q, nx, nx_pow2, tw);
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x * 32 + lane;
  cx<float>* dst = out + (size_t)i * n_slots * nv;
  const int nm = min(n_modes, n_slots);
  for (int m0 = 0; m0 < nm; m0 += MODES_AT_ONCE) {
    double zr[MODES_AT_ONCE], zi[MODES_AT_ONCE];
    int at[MODES_AT_ONCE], step[MODES_AT_ONCE];
#pragma unroll
    for (int u = 0; u < MODES_AT_ONCE; ++u) {
      zr[u] = zi[u] = 0.0;
      at[u] = (int)(((long long)(m0 + u) * w) % nx);
      step[u] = (int)(((long long)(m0 + u) * MODES_WARPS) % nx);
    }
    if (j < nv) {
      auto add = [&](double fv) {
#pragma unroll
        for (int u = 0; u < MODES_AT_ONCE; ++u) {
          if (m0 + u >= nm) continue;
          if (m0 + u == 0) {
            zr[u] += fv;
          } else {
            const cx<double> c = table ? angles[at[u]] : mode_angle(at[u], nx, nx_pow2, tw);
            zr[u] = fma(fv, c.x, zr[u]);
            zi[u] = fma(fv, c.y, zi[u]);
          }
          at[u] += step[u];
          if (at[u] >= nx) at[u] -= nx;
        }
      };
      int x = w;
      for (; x + 7 * MODES_WARPS < nx; x += 8 * MODES_WARPS) {
        double fv[8];  // eight loads in flight
#pragma unroll
        for (int u = 0; u < 8; ++u) fv[u] = f[(size_t)(x + u * MODES_WARPS) * nv + j];
#pragma unroll
        for (int u = 0; u < 8; ++u) add(fv[u]);
      }
      for (; x < nx; x += MODES_WARPS) add(f[(size_t)x * nv + j]);
    }
#pragma unroll
    for (int u = 0; u < MODES_AT_ONCE; ++u) {
      part[2 * u][w][lane] = zr[u];
      part[2 * u + 1][w][lane] = zi[u];
    }
    __syncthreads();
    if (w < 2 * MODES_AT_ONCE && m0 + w / 2 < nm && j < nv) {
      double z = part[w][0][lane];
      for (int q = 1; q < MODES_WARPS; ++q) z += part[w][q][lane];
      const float zf = __double2float_rn(z);
      const int m = m0 + w / 2;
      for (int sl = n_modes == 1 ? 0 : m; sl < (n_modes == 1 ? n_slots : m + 1); ++sl)
        reinterpret_cast<float*>(dst + (size_t)sl * nv + j)[w & 1] = zf;
    }
    __syncthreads();
  }
}

cudaError_t launch_storage_moments_f64(const vg_plan& p, const double* f, double* out, int stride, bool full,
                                       cudaStream_t s) {
  if (p.fx_pw.drop)
    return launch_moments_fx(f, p.nx, p.nv, p.v, p.v_pow, p.fx_pw, p.fx_log, p.dv, out, stride, full, s);
  MomSpec spec;
  const int kinds[8] = {MOM_ONE, MOM_V, MOM_W, MOM_W, MOM_W, MOM_W, MOM_SQ, MOM_FLOGF};
  const int args[8] = {0, 0, 1, 2, 3, 4, 0, 0};
  spec.nm = 0;
  for (int q = 0; q < 8; ++q) {
    if (!full && q >= 3 && q < 6) continue;
    spec.kind[spec.nm] = kinds[q];
    spec.arg[spec.nm++] = args[q];
  }
  return launch_row_moments_f64(p, f, spec, out, stride, s);
}

cudaError_t launch_storage_f64(const vg_plan& p, const double* f, const double* e, const double* de,
                               const vg_history& h, int i, cudaStream_t s) {
  cudaError_t err = launch_storage_moments_f64(p, f, p.mom, MOM_STRIDE, true, s);
  if (err != cudaSuccess) return err;
  const size_t smem = (size_t)7 * p.pw_x_leaves * sizeof(double);
  k_fields_series_f64<<<1, 256, smem, s>>>(p.mom, e, de, p.nx, i, h, p.pw_x);
  err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  if (h.stored_f) {
    if (h.store_all) {
      err = cudaMemcpyAsync(static_cast<double*>(h.stored_f) + (size_t)i * p.nx * p.nv, f,
                            (size_t)p.nx * p.nv * sizeof(double), cudaMemcpyDeviceToDevice, s);
    } else {
      const size_t tab = p.nx <= MODES_TABLE_NX && h.n_modes > 1 ? (size_t)p.nx * sizeof(cx<double>) : 0;
      err = ensure_smem((const void*)k_store_modes_f64, tab);
      if (err != cudaSuccess) return err;
      k_store_modes_f64<<<div_up(p.nv, 32), 32 * MODES_WARPS, tab, s>>>(f, p.nx, p.nv, h.n_modes, h.n_slots,
                                                           p.nx_pow2 && p.nx <= FFT_NMAX, p.tw64, i,
                                                           static_cast<cx<float>*>(h.stored_f));
      err = cudaGetLastError();
    }
  }
  return err;
}

// ---------------------------------------------------------------------------
// twiddle tables
// ---------------------------------------------------------------------------

__global__ void k_twiddles(cx<double>* __restrict__ t64, cx<float>* __restrict__ t32) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= FFT_NMAX) return;
  int k, h;
  tw_entry(q, k, h);
  double sn, cs;
  sincospi((double)k / (double)h, &sn, &cs);
  t64[q] = {cs, -sn};
  if (t32) t32[q] = {(float)cs, (float)-sn};
}

cudaError_t launch_twiddles(vg_plan& p, cudaStream_t s) {
  k_twiddles<<<div_up(FFT_NMAX, 256), 256, 0, s>>>(p.tw64, p.tw32);
  return cudaGetLastError();
}

}  // namespace vg
