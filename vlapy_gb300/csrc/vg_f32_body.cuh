// Device bodies of the FP32 delta-f step shared by the single-run kernels
// (vg_step_f32.cu) and the batched sweep (vg_sweep.cu): one column tile of
// the x-drift, and one row-pair group of the row pass (kick, collide,
// measure, kick).
#pragma once

#include "vg_f32.cuh"
#include "vg_f32_plan.cuh"
#include "vg_internal.cuh"

namespace vg {

// Shape of a column tile of the single-run x-drift: S column pairs by G threads
// each, laid out so that L neighbouring lanes hold neighbouring pairs of one row
// (8 L contiguous bytes), the rows following.  The sequences start 16 / L elements
// apart modulo the banks (a row of 16 lanes then covers all of them), at least one.
template <int NX, int R>
struct Col32 {
  static constexpr int G = NX / R;
  static constexpr int S = col32_seqs(NX, R);
  static constexpr int L = S < 32 ? S : 32;
  static constexpr int SETS = S / L;
  static constexpr int LD = (sp_len<float>(NX) + 15) / 16 * 16 + (L < 16 ? 16 / L : 1);
  static constexpr size_t smem =
      (size_t)S * LD * sizeof(cx<float>) + (size_t)NX * sizeof(df32) + (SETS > 1 ? (size_t)SETS * NX * sizeof(float) : 0);
};

// One column tile at column c0: x-drift by exp(i m (-dkx dt) v_col) and the tile's
// trapz-weighted density partials added into dacc[x].  Columns past nv (the tile is
// wider than a short row) are zeros that nothing reads.  vec: g is 8-byte aligned.
//
// The elements t + i G of a pair go from global memory into the first pass's
// registers and from the last pass's back; both transforms run the same code
// (exchanged parts, as in kick_io).  A pass over 4096 x 8192 took 229 us by way of
// shared memory at either end, with each transform written out; now 155.
template <int NX, int R>
__device__ __forceinline__ void col_tile(float* __restrict__ g, int nv, int c0, bool vec, float2 kdt,
                                         const float2* __restrict__ vhl, const cx<float>* __restrict__ tw,
                                         cx<float>* smem, float* dset, df32* dacc) {
  using C = Col32<NX, R>;
  constexpr int G = C::G, L = C::L;
  const int lane = threadIdx.x & 31;
  const int slot = threadIdx.x / L;
  const int t = slot & (G - 1), set = slot / G;
  const int grp = (threadIdx.x & (L - 1)) + L * set;
  cx<float>* sg = smem + (size_t)grp * C::LD;
  const int c = c0 + 2 * grp;
  const bool valid = c < nv;
  float* gc = g + c;
  const CtaSync sync;
  cx<float> io[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float* q = gc + (size_t)(t + i * G) * nv;
    if (!valid) io[i] = {0.f, 0.f};
    else if (vec) io[i] = *reinterpret_cast<const cx<float>*>(q);
    else io[i] = {q[0], q[1]};
  }
#pragma unroll 1
  for (int inverse = 0; inverse < 2; ++inverse) {
    block_fft_io<float, NX, false, R, 3>(sg, t, tw, sync, io);
    if (inverse) break;
    sync();
#pragma unroll
    for (int i = 0; i < R; ++i) sg[sp<float>(t + i * G)] = io[i];
    sync();
    // theta(m) = m * (-dkx dt) v_col (kx = m dkx on the bins m <= NX/2); the angle
    // per unit m is the double-float product of kdt = -dkx dt and v (both split)
    const Ang aa = mul_angle(kdt, vhl[valid ? c : 0]);
    const Ang ab = mul_angle(kdt, vhl[valid ? c + 1 : 0]);
    const float scale = 1.f / NX;
    // phases exp(i m a) for this thread's bins m = t, t+G, ...: one sincos for
    // the start, one for the step, complex products in between
    float sa, ca, sb, cb, sga, cga, sgb, cgb;
    sincos_m((float)t, aa, sa, ca);
    sincos_m((float)t, ab, sb, cb);
    sincos_m((float)G, aa, sga, cga);
    sincos_m((float)G, ab, sgb, cgb);
    two_real_rotate<float, true>(sg, NX, t, G, [&](int, float& pca, float& psa, float& pcb, float& psb) {
      pca = ca * scale;
      psa = sa * scale;
      pcb = cb * scale;
      psb = sb * scale;
      const float na = sa * cga + ca * sga, nca = ca * cga - sa * sga;
      const float nb = sb * cgb + cb * sgb, ncb = cb * cgb - sb * sgb;
      sa = na;
      ca = nca;
      sb = nb;
      cb = ncb;
    });
    sync();
#pragma unroll
    for (int i = 0; i < R; ++i) io[i] = sg[sp<float>(t + i * G)];
  }
  // column c is in the imaginary parts now, c + 1 in the real ones.  Density
  // partials with trapz weights: 1/2 at the two v end points
  float d[R];
  const float wa = c == 0 ? 0.5f : 1.f, wb = c + 1 == nv - 1 ? 0.5f : 1.f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    float* q = gc + (size_t)(t + i * G) * nv;
    if (valid && vec) {
      *reinterpret_cast<cx<float>*>(q) = {io[i].y, io[i].x};
    } else if (valid) {
      q[0] = io[i].y;
      q[1] = io[i].x;
    }
    d[i] = fmaf(wb, io[i].x, wa * io[i].y);
  }
  int idx;
  bool writer;
  lane_transpose_sum<R, L>(d, lane, idx, writer);
  if (writer) {
#pragma unroll
    for (int q = 0; q < (R > L ? R / L : 1); ++q) {
      const int x = t + (idx + q) * G;
      if constexpr (C::SETS == 1) dacc[x] = df_add(dacc[x], {d[q], 0.f});
      else dset[set * NX + x] = d[q];
    }
  }
  if constexpr (C::SETS > 1) {
    sync();
    for (int x = threadIdx.x; x < NX; x += C::S * G) {
      float acc = 0.f;
      for (int q = 0; q < C::SETS; ++q) acc += dset[q * NX + x];
      dacc[x] = df_add(dacc[x], {acc, 0.f});
    }
  }
}

// Moment slot q of one row (0..5: n, j, T, q, fv4, vN; 6: trapz(f^2);
// 7: trapz(f log f)) from the raw double-float sums the row pass leaves in
// its [8]-double slots: dv * sum + the background's share, in FP64.
__device__ __forceinline__ double row_moment(const double* __restrict__ slots, int q, const RowConsts& rc) {
  const df32 m = reinterpret_cast<const df32*>(slots)[q];
  const double sum = (double)m.hi + (double)m.lo;
  return q < 7 ? rc.dv * sum + rc.f0m[q] : rc.dv * sum;
}

// the same without the background's share (slot 7 has none apart) in double-float (7e-15
// relative), off the FP64 pipe
__device__ __forceinline__ df32 row_deviation_df(const double* __restrict__ slots, int q, const RowConsts& rc) {
  return df_mul({rc.dv2f.x, rc.dv2f.y}, reinterpret_cast<const df32*>(slots)[q]);
}

// rotation of one packed row pair with the delta-f background term; the 1/N of
// the inverse transform is folded in.  ha/hb: half-angle per kv index.  The
// result is left with real and imaginary parts exchanged, for kick_io.
template <int N, int PS = pad_shift<float>()>
__device__ __forceinline__ void kick_rotate(cx<float>* s, int t, int G, Ang ha, Ang hb,
                                            const cx<float>* __restrict__ F0) {
  const float sc = 1.f / N;
  // half-angle rotations h(k) = exp(i k a / 2) for this thread's bins k = t, t+G, ...
  // by one sincos for the start and one for the step, then complex products
  float sa, ca, sb, cb, sga, cga, sgb, cgb;
  sincos_m((float)t, ha, sa, ca);
  sincos_m((float)t, hb, sb, cb);
  sincos_m((float)G, ha, sga, cga);
  sincos_m((float)G, hb, sgb, cgb);
  for (int k = t; k <= N / 2; k += G) {
    // P = (1 - 2 sin^2, 2 sin cos) of the half angle; P - 1 = (-2 sin^2, 2 sin cos)
    const float pa_m1r = -2.f * sa * sa, pa_i = 2.f * sa * ca, pa_r = 1.f + pa_m1r;
    const float pb_m1r = -2.f * sb * sb, pb_i = 2.f * sb * cb, pb_r = 1.f + pb_m1r;
    const cx<float> f0 = F0[k];
    if (k == 0 || 2 * k == N) {
      const cx<float> z = s[sp<float, PS>(k)];
      // real bins: only Re(P) survives
      s[sp<float, PS>(k)] = {(pb_r * z.y + pb_m1r * f0.x) * sc, (pa_r * z.x + pa_m1r * f0.x) * sc};
    } else {
      const cx<float> zk = s[sp<float, PS>(k)], zm = s[sp<float, PS>(N - k)];
      const cx<float> hs = mul2({0.5f, 0.5f}, zk + zm), hd = mul2({0.5f, 0.5f}, zk - zm);
      const cx<float> fa = {hs.x, hd.y}, fb = {hs.y, -hd.x};
      const cx<float> ga = {(pa_r * fa.x - pa_i * fa.y + pa_m1r * f0.x - pa_i * f0.y) * sc,
                            (pa_r * fa.y + pa_i * fa.x + pa_m1r * f0.y + pa_i * f0.x) * sc};
      const cx<float> gb = {(pb_r * fb.x - pb_i * fb.y + pb_m1r * f0.x - pb_i * f0.y) * sc,
                            (pb_r * fb.y + pb_i * fb.x + pb_m1r * f0.y + pb_i * f0.x) * sc};
      s[sp<float, PS>(k)] = {ga.y + gb.x, ga.x - gb.y};
      s[sp<float, PS>(N - k)] = {gb.x - ga.y, ga.x + gb.y};
    }
    const float na = sa * cga + ca * sga, nca = ca * cga - sa * sga;
    const float nb = sb * cgb + cb * sgb, ncb = cb * cgb - sb * sgb;
    sa = na;
    ca = nca;
    sb = nb;
    cb = ncb;
  }
}

// The kick of a row pair whose elements t + i G are in registers, before and after.
// Both transforms run the same code: with real and imaginary parts exchanged at
// either end, the forward transform is the inverse one.
template <int N, int R, typename Sync>
__device__ __forceinline__ void kick_io(cx<float>* s, int t, float hk, float ea, float eb,
                                        const cx<float>* __restrict__ F0, const cx<float>* __restrict__ tw,
                                        const Sync& sync, cx<float> (&io)[R]) {
  constexpr int G = N / R;
  constexpr int PS = row_pad_shift(R);
#pragma unroll 1
  for (int inverse = 0; inverse < 2; ++inverse) {
    block_fft_io<float, N, false, R, 3, Sync, PS>(s, t, tw, sync, io);
    if (inverse) break;
    sync();
#pragma unroll
    for (int i = 0; i < R; ++i) s[sp<float, PS>(t + i * G)] = io[i];
    sync();
    // theta(k) = -kv_k dt e = k * (-dkv dt e); hk = -dkv dt / 2 gives the half
    // angle for P - 1.  The kick angle stays O(10) rad, so an FP32 product is
    // accurate to ~1e-6 rad here
    kick_rotate<N, PS>(s, t, G, {hk * ea, 0.f}, {hk * eb, 0.f}, F0);
    sync();
#pragma unroll
    for (int i = 0; i < R; ++i) io[i] = s[sp<float, PS>(t + i * G)];
  }
#pragma unroll
  for (int i = 0; i < R; ++i) io[i] = {io[i].y, io[i].x};
}

// Per-row collision scalars from the row's raw moment sums (sum w g v^p,
// p = 0, 1, 2), in double-float; each FP32 coefficient is rounded once:
// out = {-vth/dv^2, 1 + 2 nudt vth/dv^2, vbar, nudt vth, nudt vbar}.
__device__ __forceinline__ void collision_scalars(const RowConsts& rc, float2 nudt2, int dougherty, df32 s0,
                                                  df32 s1, df32 s2, float* out) {
  const df32 dv = {rc.dv2f.x, rc.dv2f.y};
  const df32 M0 = df_add(df_mul(dv, s0), {rc.f0m2f[0].x, rc.f0m2f[0].y});
  const df32 M1 = df_add(df_mul(dv, s1), {rc.f0m2f[1].x, rc.f0m2f[1].y});
  const df32 M2 = df_add(df_mul(dv, s2), {rc.f0m2f[2].x, rc.f0m2f[2].y});
  // DG: vbar = trapz(f v), v0t^2 = trapz(f (v - vbar)^2) = M2 + vbar^2 (M0 - 2)
  // LB: v0t^2 = trapz(f v^2), no drift
  const df32 vbar = dougherty ? M1 : df32{0.f, 0.f};
  const df32 vth = dougherty ? df_add(M2, df_mul(df_mul(vbar, vbar), df_add(M0, {-2.f, 0.f}))) : M2;
  const df32 nd = {nudt2.x, nudt2.y};
  const df32 a = df_mul(vth, {rc.idv2f.x, rc.idv2f.y});  // vth / dv^2
  const df32 na = df_mul(nd, a);
  out[0] = -df_round(a);
  out[1] = df_round(df_add({1.f, 0.f}, {2.f * na.hi, 2.f * na.lo}));
  out[2] = df_round(vbar);
  out[3] = df_round(df_mul(nd, vth));
  out[4] = df_round(df_mul(nd, vbar));
}

// Fokker-Planck step, in delta-f form, of both rows of a packed pair (row a
// in the real parts of s, row b in the imaginary parts).  The moments and the
// right-hand sides of the two rows share one pass over the pair (one 8-byte
// access per element, one load of each constant) and one reduction; the two
// tridiagonal solves run one after the other, in one copy of the code.
//
// What bounds the row pass is the instruction cache, before FP32 issue: a row pair
// walks through all of its code once, and two CTAs do so at different places.  With
// the transforms of a kick, the two solves and the loops over a thread's R elements
// all written out, a third to a half of the stalls were for instructions (nv = 8192:
// 555 us a pass over 4096 rows, now 430) and the time changed by 15 % with whatever
// else the library held.  So each of them is there once, in loops that stay rolled,
// and the passes over shared memory are unrolled by ROW_UNROLL (2: 8 % slower over
// the whole step at 4096 x 8192, 4: 2 %, 16: as fast; a sweep of 64 runs 7 %, 2 %,
// 0 %).
constexpr int ROW_UNROLL = 8;
template <int N, int R, typename Sync = CtaSync>
__device__ __forceinline__ void collide_pair(cx<float>* s, int t, const RowConsts& rc, float2 nudt2, float nudt_f,
                                             int dougherty, df32* red, float* pcr, const Sync& sync = Sync()) {
  constexpr int G = N / R;
  // moments of g: sum w g, sum w g v, sum w g v^2 of each row.  The
  // elementwise parts give consecutive threads consecutive j, so the constant
  // vectors load coalesced; only the tridiagonal solves work on chunks
  df32 mv[6];
  {
    // (both rows in one packed operation)
    cx<float> m[3] = {};
#pragma unroll ROW_UNROLL
    for (int i = 0; i < R; ++i) {
      const int j = t + i * G;
      const float w = (j == 0 || j == N - 1) ? 0.5f : 1.f;
      const float vj = rc.v[j];
      const cx<float> vv = {vj, vj};
      const cx<float> z = mul2({w, w}, s[sp<float, row_pad_shift(R)>(j)]);
      m[0] = add2(m[0], z);
      m[1] = fma2(z, vv, m[1]);
      m[2] = fma2(mul2(z, vv), vv, m[2]);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      mv[q] = {m[q].x, 0.f};
      mv[3 + q] = {m[q].y, 0.f};
    }
  }
  // per-row scalars in double-float, each row's by one thread; the group reads them back
  float* sc = reinterpret_cast<float*>(red);
  if constexpr (G >= 32) {
    df32 s0 = group_df_sum_lanes<6>(mv, reinterpret_cast<df32*>(pcr), G, t, sync);
    if (t < 32) {
      const df32 s1 = df_shfl_down(s0, 1), s2 = df_shfl_down(s0, 2);
      if (t == 0 || t == 3) collision_scalars(rc, nudt2, dougherty, s0, s1, s2, sc + (t ? 5 : 0));
    }
  } else {
    group_df_sum<6, true>(mv, red, G, t, sync);
    for (int q = t; q < 2; q += G)
      collision_scalars(rc, nudt2, dougherty, q ? mv[3] : mv[0], q ? mv[4] : mv[1], q ? mv[5] : mv[2], sc + 5 * q);
  }
  sync();
  float sa[5], sb[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    sa[q] = sc[q];
    sb[q] = sc[5 + q];
  }
  const float nu = nudt_f;
  const float cm = nu;
  const float i2dv = rc.i2dv;
  sync();
  // right-hand sides: g - (A - I) f0 with (A - I) f0 = nudt (-vth S + Mv - vbar D)
#pragma unroll ROW_UNROLL
  for (int i = 0; i < R; ++i) {
    const int j = t + i * G;
    const float S = rc.S[j], Mv = rc.Mv[j], D = rc.D[j];
    const cx<float> z = s[sp<float, row_pad_shift(R)>(j)];
    // (the three terms nearly cancel: their sum first)
    const float cM = -cm * Mv;
    const cx<float> u = fma2({sa[4], sb[4]}, {D, D}, fma2({sa[3], sb[3]}, {S, S}, {cM, cM}));
    s[sp<float, row_pad_shift(R)>(j)] = add2(z, u);
  }
  sync();
  // off-diagonals at v[j -+ 1] of the uniform grid v[j] = v[0] + j dv, formed in
  // registers
  const float v0 = rc.v0f, dvf = rc.dvf;
#pragma unroll 1
  for (int row = 0; row < 2; ++row) {
    const float Af = row ? sb[0] : sa[0], diag = row ? sb[1] : sa[1], vb = row ? sb[2] : sa[2];
    // l(j) = nu (Af + (v[j - 1] - vb) / 2 dv), u(j) = nu (Af - (v[j + 1] - vb) / 2 dv)
    const float ls = nu * (Af + (fmaf((float)(t * R - 1), dvf, v0) - vb) * i2dv);
    const float us = nu * (Af - (fmaf((float)(t * R + 1), dvf, v0) - vb) * i2dv);
    const float dl = nu * (dvf * i2dv);
    partition_solve<R, G>(reinterpret_cast<float*>(s) + row, t, diag, ls, dl, us, -dl, pcr, sync);
  }
}

// One row-pair group of the row pass: load, [kick dt1], [collide], [moments
// and x-mode partials], [kick dt2], store.  grp_base: this group's shared
// memory (row32_group_bytes); macc: the CTA's mode accumulators [n_modes][N].
// NPOW: how many power moments sum w g v^p (p < NPOW) the storage needs (6:
// n, j, T, q, fv4, vN; the batched sweep's series need only p < 3); the
// slots of the others are left unwritten.  KICK_ONLY: the leading half kick
// of a step sequence alone (registers in from global memory, out to it).
template <int N, int R, typename Sync = CtaSync, int NPOW = 6, bool KICK_ONLY = false>
__device__ __forceinline__ void row_pair(const RowArgs& a, int pair, unsigned char* grp_base, cx<float>* macc,
                                         int P, int grp, int t, const Sync& sync = Sync()) {
  constexpr int G = N / R;
  cx<float>* s = reinterpret_cast<cx<float>*>(grp_base);
  constexpr size_t seq_bytes = row32_seq_bytes(N, R);
  static_assert(seq_bytes % 16 == 0 && row32_group_bytes(N, R) % 16 == 0 &&
                    seq_bytes + 8 * G * sizeof(float) + round16((G / 32 + 1) * 9 * sizeof(df32)) ==
                        row32_group_bytes(N, R),
                "row-pair group layout and its host-side size disagree");
  float* pcr = reinterpret_cast<float*>(grp_base + seq_bytes);
  df32* red = reinterpret_cast<df32*>(grp_base + seq_bytes + 8 * G * sizeof(float));
  const int nm = a.n_modes;
  const int ra = 2 * pair, rb = ra + 1;
  const bool va = ra < a.nx, vb = rb < a.nx;
  float* ga = a.g + (size_t)ra * N;
  float* gbp = a.g + (size_t)rb * N;
  const bool kicks = a.hk1 != 0.f || a.hk2 != 0.f;
  const float ea = (kicks && va) ? a.e32[ra] : 0.f, eb = (kicks && vb) ? a.e32[rb] : 0.f;
  if constexpr (KICK_ONLY) {
    cx<float> io[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int n = t + i * G;
      io[i] = {va ? ga[n] : 0.f, vb ? gbp[n] : 0.f};
    }
    if (a.hk1 != 0.f) kick_io<N, R>(s, t, a.hk1, ea, eb, a.F0, a.tw, sync, io);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int n = t + i * G;
      if (va) ga[n] = io[i].x;
      if (vb) gbp[n] = io[i].y;
    }
    sync();
  } else {
  // both kicks run the same code (registers in, registers out), once each in
  // a loop the compiler keeps rolled, so the kernel holds one copy of the
  // kick's FFTs instead of four differently specialised ones (instruction-
  // cache pressure); the collision and the moments sit between the two
#pragma unroll 1
  for (int kpass = 0; kpass < 2; ++kpass) {
    const float hk = kpass == 0 ? a.hk1 : a.hk2;
    // the pair's elements t + i G, exactly what the first FFT pass reads: from
    // global memory before the first kick, from shared memory before the
    // second (io is defined afresh in every pass, so it is dead in between)
    cx<float> io[R];
    if (kpass == 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int n = t + i * G;
        io[i] = {va ? ga[n] : 0.f, vb ? gbp[n] : 0.f};
      }
    } else {
#pragma unroll
      for (int i = 0; i < R; ++i) io[i] = s[sp<float, row_pad_shift(R)>(t + i * G)];
    }
    if (hk != 0.f) {
      kick_io<N, R>(s, t, hk, ea, eb, a.F0, a.tw, sync, io);
    }
    if (kpass == 1) {
      // the last FFT pass left elements t + i G in registers: the store
      // pattern, so they go straight back to global memory
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int n = t + i * G;
        if (va) ga[n] = io[i].x;
        if (vb) gbp[n] = io[i].y;
      }
      break;
    }
    // the pair into shared memory for the collision and the moments (after
    // every thread's last kick pass has read it)
    sync();
#pragma unroll
    for (int i = 0; i < R; ++i) s[sp<float, row_pad_shift(R)>(t + i * G)] = io[i];
    sync();
    if (a.fp) {
      collide_pair<N, R>(s, t, *a.rc, a.nudt2, a.nudt_f, a.dougherty, red, pcr, sync);
    }
    if (a.want_mom) {
      // sums of w g v^p (p < NPOW), sum w g^2, sum w g f0, sum w f log f for
      // both rows: [0, NQ) row a, [NQ, 2 NQ) row b
      static_assert(NPOW >= 1 && NPOW <= 6, "power moments");
      constexpr int NQ = NPOW + 3;
      cx<float> sum[NQ] = {};  // (row a, row b), packed
  #pragma unroll ROW_UNROLL
      for (int i = 0; i < R; ++i) {
        const int j = t + i * G;  // consecutive threads, consecutive j: coalesced loads
        const float w = (j == 0 || j == N - 1) ? 0.5f : 1.f;
        const float vj = a.rc->v[j], f0j = a.rc->f0[j];
        const cx<float> z = s[sp<float, row_pad_shift(R)>(j)], vv = {vj, vj}, f0 = {f0j, f0j}, ww = {w, w};
        const cx<float> wz = mul2(ww, z);
        cx<float> pw = wz;
  #pragma unroll
        for (int p = 0; p < NPOW; ++p) {
          sum[p] = add2(sum[p], pw);
          if (p + 1 < NPOW) pw = mul2(pw, vv);
        }
        sum[NPOW] = fma2(wz, z, sum[NPOW]);
        sum[NPOW + 1] = fma2(wz, f0, sum[NPOW + 1]);
        // f log f by the fast logarithm (3 ulp; NaN for f < 0 as in FP64)
        const cx<float> f = add2(z, f0);
        sum[NPOW + 2] = fma2(mul2(ww, f), {__logf(f.x), __logf(f.y)}, sum[NPOW + 2]);
      }
      df32 m2[2 * NQ];
  #pragma unroll
      for (int q = 0; q < NQ; ++q) {
        m2[q] = {sum[q].x, 0.f};
        m2[NQ + q] = {sum[q].y, 0.f};
      }
      // raw sums; the storage kernels form dv * sum + trapz(f0 ...) in FP64: slots
      // 0 .. NPOW - 1 the powers, 6 sum w (g^2 + 2 g f0), 7 sum w f log f
      if constexpr (G >= 32) {
        const df32 tot = group_df_sum_lanes<2 * NQ>(m2, reinterpret_cast<df32*>(pcr), G, t, sync);
        if (t < 32) {
          const df32 nx1 = df_shfl_down(tot, 1);
          const int q = t < NQ ? t : t - NQ, row = t < NQ ? ra : rb;
          if (t < 2 * NQ && row < a.nx && q != NPOW + 1) {
            df32* out = reinterpret_cast<df32*>(a.mom + (size_t)row * MOM_STRIDE);
            if (q < NPOW) out[q] = tot;
            else if (q == NPOW) out[6] = df_add(tot, {2.f * nx1.hi, 2.f * nx1.lo});
            else out[7] = tot;
          }
        }
      } else {
        group_df_sum<2 * NQ, true>(m2, red, G, t, sync);
        if (t == 0) {
          // each array is indexed by constants only, so it stays in registers
          auto put = [&](int o, int row) {
            df32* out = reinterpret_cast<df32*>(a.mom + (size_t)row * MOM_STRIDE);
  #pragma unroll
            for (int p = 0; p < NPOW; ++p) out[p] = m2[o + p];
            out[6] = df_add(m2[o + NPOW], {2.f * m2[o + NPOW + 1].hi, 2.f * m2[o + NPOW + 1].lo});
            out[7] = m2[o + NPOW + 2];
          };
          if (va) put(0, ra);
          if (vb) put(NQ, rb);
        }
      }
      // x-Fourier modes of f (the f0 part of mode 0 is added in the reduction);
      // the groups of a CTA hold different rows but add into the same bins,
      // so they take turns
      // (only with a CTA-wide sync: the turns are CTA barriers)
      if (Sync::cta_wide && nm > 0) {
        for (int gq = 0; gq < P; ++gq) {
          if (gq == grp) {
            for (int mq = 0; mq < nm; ++mq) {
              float swa = 0.f, cwa = 0.f, swb = 0.f, cwb = 0.f;
              if (va) sincospif(-2.f * (float)((mq * ra) % a.nx) / (float)a.nx, &swa, &cwa);
              if (vb) sincospif(-2.f * (float)((mq * rb) % a.nx) / (float)a.nx, &swb, &cwb);
              // in batches: reads first, so that a batch waits once.  Accumulators in
              // global memory are added to in L2, whence nothing returns to wait for
              // (a bin is one thread's at a time, so the order is fixed)
              constexpr int U = R < ROW_UNROLL ? R : ROW_UNROLL;
              cx<float>* m0 = macc + (size_t)mq * N + t;
              for (int i0 = 0; i0 < R; i0 += U) {
                cx<float> z[U];
  #pragma unroll
                for (int u = 0; u < U; ++u) {
                  const cx<float> q = s[sp<float, row_pad_shift(R)>(t + (i0 + u) * G)];
                  z[u] = {q.x * cwa + q.y * cwb, q.x * swa + q.y * swb};
                }
                if (a.macc_global) {
  #pragma unroll
                  for (int u = 0; u < U; ++u)
                    atomicAdd(reinterpret_cast<float2*>(m0 + (i0 + u) * G), make_float2(z[u].x, z[u].y));
                } else {
                  cx<float> acc[U];
  #pragma unroll
                  for (int u = 0; u < U; ++u) acc[u] = m0[(i0 + u) * G];
  #pragma unroll
                  for (int u = 0; u < U; ++u) m0[(i0 + u) * G] = {acc[u].x + z[u].x, acc[u].y + z[u].y};
                }
              }
            }
          }
          __syncthreads();
        }
      }
    }
  }
  sync();
  }
}


}  // namespace vg
