// Fixed-point x-advection of the FP64 mode (vlapy/core/vlasov.py:83-110): f <-
// Re IFFT_x(exp(-i kx v dt) FFT_x f) on column pairs, for one run or for the
// (run, tile) items of a batch.
//
// A CTA owns S adjacent column pairs: thread (t, p) of the nx / 8 x S threads
// takes the elements x = t + i nx / 8 of pair p, so that the S lanes of equal t
// read one row segment of 16 S bytes; every element goes from global memory to
// registers and back once, and shared memory carries only the passes between.
//
// Measured against the transforms in doubles, smooth columns: 4096 x 8192 4.26 ->
// 1.04 ms, 2048 x 4096 0.98 -> 0.23 ms, 64 x 1024 57 -> 14 us one launch after another
// (17 with cold caches); of noise 2048 x 4096 0.96 ms.  Bound as the v-advection
// (vg_edfdv_fx.cu); 128-bit check: 0.8e-16 of the column's RMS at nx = 1024, in
// doubles 2.6e-16.
#include <algorithm>

#include "vg_advect_fx.cuh"
#include "vg_f64_body.cuh"
#include "vg_internal.cuh"

namespace vg {

namespace {

constexpr int FX_COL_BLOCK = 256;
__host__ __device__ constexpr int fx_col_max_pairs(int nx) {
  return FX_COL_BLOCK / fx_threads(nx) >= 2 ? FX_COL_BLOCK / fx_threads(nx) : (2 * fx_threads(nx) <= 512 ? 2 : 1);
}
__host__ __device__ constexpr int fx_col_block(int nx) { return fx_col_max_pairs(nx) * fx_threads(nx); }
// stride of the pairs' sequences in elements: eight 16-byte accesses of a
// phase are 8 / S consecutive t of S pairs (S < 8), or eight pairs
__host__ __device__ constexpr int fx_col_ld(int nx, int S) {
  const int want = S >= 8 ? 1 : S == 4 ? 2 : S == 2 ? 4 : 0;
  int ld = fx_len(nx);
  if (S >= 8) return ld | 1;
  if (S == 1) return ld;
  return ld + ((want - ld % 8) + 8) % 8;
}

template <int NX>
__global__ void __launch_bounds__(fx_col_block(NX), fx_col_block(NX) > 256 ? 1 : 2)
    k_vdfdx_fx(double* __restrict__ f, const FxColRun* __restrict__ runs, const int2* __restrict__ items, FxColRun one,
               int s_log, int ld, const fxw* __restrict__ tw, const cx<double>* __restrict__ tw64) {
  constexpr int R = fx_radix(NX), G = fx_threads(NX);
  constexpr int DOWN = ilog2(NX) - fx_shift<NX>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int S = 1 << s_log;
  const int p = threadIdx.x & (S - 1), t = threadIdx.x >> s_log;
  fx* s = reinterpret_cast<fx*>(smem_raw) + (size_t)p * ld;
  unsigned* red = reinterpret_cast<unsigned*>(smem_raw + (size_t)S * ld * sizeof(fx));  // [S][5]
  const int2 it = items ? items[blockIdx.x] : make_int2(0, blockIdx.x);
  const FxColRun r = items ? runs[it.x] : one;
  const int nv = r.nv;
  const int col = 2 * (it.y * S + p);
  const bool va = col < nv, vb = col + 1 < nv;
  double* fc = f + r.f_off + (va ? col : 0);
  // both columns in one 16-byte access where every row keeps the alignment
  const bool vec = vb && (nv & 1) == 0 && (reinterpret_cast<uintptr_t>(fc) & 15) == 0;
  if (t == 0)
    for (int q = 0; q < 5; ++q) red[5 * p + q] = 0;
  const double ca = va ? r.v[col] : 0.0, cb = vb ? r.v[col + 1] : 0.0;
  fx io[R];
  int Ea, Eb;
  bool bad_a, bad_b, zero_a, zero_b;
  {
    double da[R], db[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const double* q = fc + (size_t)(t + i * G) * nv;
      if (vec) {
        const double2 z = *reinterpret_cast<const double2*>(q);
        da[i] = z.x;
        db[i] = z.y;
      } else {
        da[i] = va ? q[0] : 0.0;
        db[i] = vb ? q[1] : 0.0;
      }
    }
    __syncthreads();
    unsigned ma = 0, mb = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      ma = max(ma, fx_exp_bits(da[i]));
      mb = max(mb, fx_exp_bits(db[i]));
    }
    if constexpr (G > 1) {
      atomicMax(&red[5 * p], ma);
      atomicMax(&red[5 * p + 1], mb);
      __syncthreads();
      ma = red[5 * p];
      mb = red[5 * p + 1];
    }
    zero_a = ma == 0;
    zero_b = mb == 0;
    Ea = fx_exp(ma);
    Eb = fx_exp(mb);
    bad_a = Ea == FX_NONFINITE || !isfinite(ca);
    bad_b = Eb == FX_NONFINITE || !isfinite(cb);
#pragma unroll
    for (int i = 0; i < R; ++i)
      io[i] = {bad_a ? 0 : fx_from_double(da[i], Ea), bad_b ? 0 : fx_from_double(db[i], Eb)};
  }
  const CtaSync sync;
  fx_fft<NX, false, true, false>(s, t, tw, sync, io);
  const unsigned long long ta = fx_turn(r.turn, bad_a ? 0.0 : ca), tb = fx_turn(r.turn, bad_b ? 0.0 : cb);
  const bool own = NX >= FX_OWN_N && (fx_has_own(r.turn, ca) || fx_has_own(r.turn, cb));
  float oa = 0.f, ob = 0.f;
  if (own) {
    oa = bad_a ? 0.f : r.turn.own * (float)ca;
    ob = bad_b ? 0.f : r.turn.own * (float)cb;
  }
  FxNorms n = fx_rotate<NX, DOWN>(s, t, ta, tb, own, oa, ob, r.rest, tw);
  if constexpr (G > 1) {
    atomicAdd(&red[5 * p + 2], n.l1);
    atomicAdd(&red[5 * p + 3], n.a2);
    atomicAdd(&red[5 * p + 4], n.b2);
    __syncthreads();
    n = {red[5 * p + 2], red[5 * p + 3], red[5 * p + 4]};
  }
  // (E <= 1: a column of zeros, or of values that small)
  const int h = fx_shift_back<NX>(n, bad_a || Ea <= 1, bad_b || Eb <= 1);
  // Pairs that fixed point is not exact enough for go through doubles, pair by pair: a
  // column comes out the same whatever its tile holds (a batch and a single run have
  // different tiles).  The tile's other pairs go along with nothing to load or store,
  // for the barriers.
  const bool turned = h < 0;
  const int n_turned = __syncthreads_count(turned);  // threads
  auto in_doubles = [&]() {
    cx<double>* sd = reinterpret_cast<cx<double>*>(smem_raw) + (size_t)p * (sp_len<double>(NX) + COL_PAD);
    fx_pair_f64<NX>({fc, ta, oa, fx_up(Ea, n.a2), va && turned, bad_a}, {fc + 1, tb, ob, fx_up(Eb, n.b2), vb && turned, bad_b},
                    nv, sd, t, r.rest, tw, tw64, sync);
  };
  // (short columns are hardly ever turned away, and a second copy of the call is 2 us of
  // a cold launch)
  if constexpr (NX >= 256) {
    if (n_turned == (int)blockDim.x) {
      in_doubles();
      return;
    }
  }
  fx_fft<NX, true, false, true>(s, t, tw, sync, io, turned ? 16 : h);
  // lines of zeros stay so: the partner's rounding does not reach them
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const bool set_a = bad_a || zero_a, set_b = bad_b || zero_b;
  const double val_a = bad_a ? nan : 0.0, val_b = bad_b ? nan : 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (turned) break;
    double* q = fc + (size_t)(t + i * G) * nv;
    const double xa = set_a ? val_a : fx_to_double(io[i].x, Ea - FX_SCALE + h);
    const double xb = set_b ? val_b : fx_to_double(io[i].y, Eb - FX_SCALE + h);
    if (vec) {
      *reinterpret_cast<double2*>(q) = make_double2(xa, xb);
    } else {
      if (va) q[0] = xa;
      if (vb) q[1] = xb;
    }
  }
  if (n_turned > 0) {
    __syncthreads();
    in_doubles();
  }
}

template <int NX>
cudaError_t vdfdx_fx_n(double* f, const FxColRun* runs, const int2* items, int n_items, const FxColRun& one, int S,
                       const fxw* tw, const cx<double>* tw64, cudaStream_t s) {
  constexpr int G = fx_threads(NX);
  const int ld = fx_col_ld(NX, S);
  const size_t smem = std::max((size_t)S * ld * sizeof(fx) + (size_t)S * 5 * sizeof(unsigned),
                               (size_t)S * (sp_len<double>(NX) + COL_PAD) * sizeof(cx<double>));
  cudaError_t err = ensure_smem((const void*)k_vdfdx_fx<NX>, smem);
  if (err != cudaSuccess) return err;
  const int blocks = items ? n_items : div_up((one.nv + 1) / 2, S);
  k_vdfdx_fx<NX><<<blocks, S * G, smem, s>>>(f, runs, items, one, ilog2(S), ld, tw, tw64);
  return cudaGetLastError();
}

template <int NX>
int col_pairs_n(long long pairs) {
  int S = fx_col_max_pairs(NX);
  while (S > 1 && (S / 2) * fx_threads(NX) >= 32 && (pairs + S - 1) / S < 2 * GB300_SMS) S /= 2;
  return S;
}

}  // namespace

#define VG_FX_CASES(M) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13)

int fx_col_pairs(int nx, long long pairs) {
  switch (ilog2(nx)) {
#define CASE(L) \
  case L: return col_pairs_n<(1 << L)>(pairs);
    VG_FX_CASES(CASE)
#undef CASE
    default: return 1;
  }
}

cudaError_t launch_vdfdx_fx(double* f, int nx, const FxColRun* runs, const int2* items, int n_items, FxColRun one, int S,
                            const fxw* tw, const cx<double>* tw64, cudaStream_t s) {
  switch (ilog2(nx)) {
#define CASE(L) \
  case L: return vdfdx_fx_n<(1 << L)>(f, runs, items, n_items, one, S, tw, tw64, s);
    VG_FX_CASES(CASE)
#undef CASE
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vg
