// Fixed-point transforms for the FP64 advection: complex 64-bit integers in
// place of complex doubles.
//
// Why.  GB300 issues one FP64 warp instruction per 64 cycles and scheduler (19
// cycles per SM with all four busy), so the exponential integrators were bound
// by their FP64 instruction count (84 % of that pipe, 2 % of the HBM rate).  A
// 64-bit integer add is two ordinary instructions and a 64 x 64 -> high 64
// product four or five, on a pipe 32 times as wide, so the same transforms in
// fixed point cost a small part of the time.
//
// Precision.  A line is scaled by its own power of two so that its largest
// element is below 2^59.5 and every operation rounds at one unit of that fixed
// scale (a double's own rounding is 2^-53 of each element).
//  * Forward, a factor 1/4 is given up per radix-4 stage, since the sum of four
//    values of modulus <= M has modulus <= 4 M: the bins come out divided by the
//    length, each rounded a few times at 2^-59 of the line's maximum.
//  * Back, nothing is given up: every partial sum is at most the sum of the bins'
//    moduli, which the rotation adds up on the way.  Where that sum (times 2^h)
//    still fits, the bins are used as they are (shifted by h).  A distribution
//    function's spectrum is compact: h is 0 or 1.
//  * The error of the result is then about 0.6 sqrt(N) 2^h units, and the lines
//    for which that is more than the error of a transform in doubles are
//    transformed in doubles instead, inside the same kernel, so that the error
//    is at or below that of the doubles on every input (measured against 128-bit
//    arithmetic).  These are the lines whose RMS is below 0.002 to 0.005 sqrt(N)
//    of their maximum, by the maximum's mantissa: of Maxwellians on |v| < 8, at N =
//    1024 some of vth 0.1, at 4096 half of vth 0.3 (a third of vth 1 on |v| < 16), at
//    8192 a fifth of vth 1 (two thirds on |v| < 16); and lines whose spectrum is
//    broad (h > 0): noise from N = 256 on, filaments and fronts of the longest grids.
// Lines that hold a NaN or infinity come out as NaN, as from a transform in
// doubles.
//
// A line pair a + i b is transformed as one complex sequence; since the
// separation of the two is linear, each of the two has its own scale.
#pragma once

#include "vg_common.cuh"
#include "vg_fft.cuh"

namespace vg {

struct __align__(16) fx {
  long long x, y;
};
__device__ __forceinline__ fx operator+(fx a, fx b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fx operator-(fx a, fx b) { return {a.x - b.x, a.y - b.y}; }

// A multiplier in Q62, each component as h 2^32 + l with l signed, so that all
// partial products are signed 32 x 32 -> 64
struct __align__(16) fxw {
  int xh, xl, yh, yl;
};
__host__ __device__ constexpr int fx_lo(long long a) { return (int)(unsigned)(unsigned long long)a; }
__host__ __device__ constexpr int fx_hi(long long a) {
  return (int)((a + 0x80000000ll) >> 32);
}
__host__ __device__ __forceinline__ fxw fx_mult(long long c, long long s) {
  return {fx_hi(c), fx_lo(c), fx_hi(s), fx_lo(s)};
}
__device__ __forceinline__ long long wide(int a, int b) { return (long long)a * b; }

// a * w / 2^(64 - SH) for a real a, |a| 2^SH < 2^63, rounded (the product of the
// two low words, below a quarter unit, is dropped)
template <int SH>
__device__ __forceinline__ long long fx_rmul(long long a, int wh, int wl) {
  a = (long long)((unsigned long long)a << SH);
  const int ah = fx_hi(a), al = fx_lo(a);
  const long long t = 0x80000000ll + wide(al, wh) + wide(ah, wl);
  return wide(ah, wh) + (t >> 32);
}
// a * w / 2^(2 - SH) for a Q62 multiplier w of modulus <= 1 (CONJ: its
// conjugate).  SH < 2: |a| 2^SH <= 2^62, so that the four middle products add up
// in 64 bits; SH = 2 keeps them in two sums and takes |a| < 2^61
template <int SH, bool CONJ>
__device__ __forceinline__ fx fx_cmul(fx a, const fxw& w) {
  const long long ax = (long long)((unsigned long long)a.x << SH), ay = (long long)((unsigned long long)a.y << SH);
  const int axh = fx_hi(ax), axl = fx_lo(ax), ayh = fx_hi(ay), ayl = fx_lo(ay);
  const int yh = CONJ ? -w.yh : w.yh, yl = CONJ ? -w.yl : w.yl;
  const int nh = CONJ ? w.yh : -w.yh, nl = CONJ ? w.yl : -w.yl;
  const long long tr = 0x80000000ll + wide(axl, w.xh) + wide(axh, w.xl);
  const long long ti = 0x80000000ll + wide(axl, yh) + wide(axh, yl);
  if constexpr (SH < 2) {
    const long long t2r = tr + wide(ayl, nh) + wide(ayh, nl), t2i = ti + wide(ayl, w.xh) + wide(ayh, w.xl);
    return {(t2r >> 32) + wide(axh, w.xh) + wide(ayh, nh), (t2i >> 32) + wide(axh, yh) + wide(ayh, w.xh)};
  } else {
    const long long ur = 0x80000000ll + wide(ayl, nh) + wide(ayh, nl);
    const long long ui = 0x80000000ll + wide(ayl, w.xh) + wide(ayh, w.xl);
    return {(tr >> 32) + (ur >> 32) + wide(axh, w.xh) + wide(ayh, nh),
            (ti >> 32) + (ui >> 32) + wide(axh, yh) + wide(ayh, w.xh)};
  }
}
// a / 2^D, rounded half to even: with D of one or two bits a half is common, and
// rounding it up would add the same bias to every bin, which the transform
// back collects in one element
template <int D>
__device__ __forceinline__ long long fx_down(long long a) {
  if constexpr (D == 0) return a;
  else return (a + ((1ll << (D - 1)) - 1) + (long long)(((unsigned)a >> D) & 1u)) >> D;
}
template <int D>
__device__ __forceinline__ fx fx_down(fx a) {
  return {fx_down<D>(a.x), fx_down<D>(a.y)};
}

// A sum in 96 bits, so that products near 2^61 add up exactly
struct Acc96 {
  unsigned long long lo;
  int hi;
};
__device__ __forceinline__ void acc_add(Acc96& s, long long x) {
  asm("add.cc.u64 %0, %0, %2;\n\taddc.s32 %1, %1, %3;" : "+l"(s.lo), "+r"(s.hi) : "l"(x), "r"((int)(x >> 63)));
}
__device__ __forceinline__ void acc_add96(Acc96& s, const Acc96& o) {
  asm("add.cc.u64 %0, %0, %2;\n\taddc.s32 %1, %1, %3;" : "+l"(s.lo), "+r"(s.hi) : "l"(o.lo), "r"(o.hi));
}
// rounded once: the sum in two parts of 48 bits
__device__ __forceinline__ double acc_to_double(const Acc96& s) {
  const long long up = ((long long)s.hi << 16) | (long long)(s.lo >> 48);
  return fma((double)up, 281474976710656.0, (double)(long long)(s.lo & 0xffffffffffffull));  // 2^48
}

// cos(2 pi j / 16), j = 0..4, in Q62
constexpr long long FX_ONE = 1ll << 62;
constexpr long long FX_C1 = 4260642322793532497ll;   // cos(pi / 8)
constexpr long long FX_C2 = 3260954456333195553ll;   // cos(pi / 4)
constexpr long long FX_C3 = 1764815834521887442ll;   // cos(3 pi / 8)

// multiply by exp(-+ 2 pi i K / 16) (forward sign '-' unless INV) and divide by 2^(2 - SH)
template <int K, bool INV, int SH>
__device__ __forceinline__ fx fx_rot16(fx a) {
  if constexpr (K == 0) return fx_down<2 - SH>(a);
  else if constexpr (K == 4) return fx_down<2 - SH>(INV ? fx{-a.y, a.x} : fx{a.y, -a.x});
  else if constexpr (K == 2 || K == 6) {
    // c (1 -+ i) and c (-1 -+ i), c = cos(pi / 4); for SH = 2 in Q63 (the sums'
    // moduli reach 2^61.5)
    constexpr long long c = SH == 2 ? 2 * FX_C2 : FX_C2;
    constexpr int sh = SH == 2 ? 1 : SH;
    const long long p = fx_rmul<sh>(a.x + a.y, fx_hi(c), fx_lo(c));
    const long long m = fx_rmul<sh>(a.y - a.x, fx_hi(c), fx_lo(c));
    if constexpr (K == 2) return INV ? fx{-m, p} : fx{p, m};
    else return INV ? fx{-p, -m} : fx{m, -p};
  } else {
    constexpr long long c = K == 1 ? FX_C1 : K == 3 ? FX_C3 : -FX_C1;  // K = 9: cos = -C1
    constexpr long long s = K == 1 ? FX_C3 : K == 3 ? FX_C1 : -FX_C3;
    static_assert(K == 1 || K == 3 || K == 9, "rotations of the 4 x 4 butterfly");
    constexpr fxw w = {fx_hi(c), fx_lo(c), fx_hi(-s), fx_lo(-s)};
    return fx_cmul<SH, INV>(a, w);
  }
}

template <bool INV>
__device__ __forceinline__ void fx_dft4(fx& a0, fx& a1, fx& a2, fx& a3) {
  const fx s02 = a0 + a2, d02 = a0 - a2, s13 = a1 + a3, d13 = a1 - a3;
  const fx r = INV ? fx{-d13.y, d13.x} : fx{d13.y, -d13.x};
  a0 = s02 + s13;
  a2 = s02 - s13;
  a1 = d02 + r;
  a3 = d02 - r;
}

// In-register DFT of R values, natural order out.  Forward, R = 16 gives up 2
// bits at its inner rotations and R = 8 one (it starts with a radix-2 stage).
template <int R, bool INV>
struct FxDft;
template <bool INV>
struct FxDft<2, INV> {
  static __device__ __forceinline__ void run(fx (&a)[2]) {
    const fx t = a[0];
    a[0] = t + a[1];
    a[1] = t - a[1];
  }
};
template <bool INV>
struct FxDft<4, INV> {
  static __device__ __forceinline__ void run(fx (&a)[4]) { fx_dft4<INV>(a[0], a[1], a[2], a[3]); }
};
template <bool INV>
struct FxDft<8, INV> {
  static constexpr int SH = INV ? 2 : 1;
  // radix 2 over (i, i + 4), rotation by i k / 8, radix 4 over i
  static __device__ __forceinline__ void run(fx (&a)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const fx t = a[i];
      a[i] = t + a[i + 4];
      a[i + 4] = t - a[i + 4];
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) a[i] = fx_down<2 - SH>(a[i]);
    a[5] = fx_rot16<2, INV, SH>(a[5]);
    a[6] = fx_rot16<4, INV, SH>(a[6]);
    a[7] = fx_rot16<6, INV, SH>(a[7]);
    fx_dft4<INV>(a[0], a[1], a[2], a[3]);  // even outputs 0, 2, 4, 6
    fx_dft4<INV>(a[4], a[5], a[6], a[7]);  // odd outputs 1, 3, 5, 7
    const fx b1 = a[1], b2 = a[2], b3 = a[3], b4 = a[4], b5 = a[5], b6 = a[6];
    a[1] = b4;
    a[2] = b1;
    a[3] = b5;
    a[4] = b2;
    a[5] = b6;
    a[6] = b3;
  }
};
template <bool INV>
struct FxDft<16, INV> {
  static constexpr int SH = INV ? 2 : 0;
  // radix 4 over (i, i + 4, i + 8, i + 12), rotation by i k / 16, radix 4 over i
  static __device__ __forceinline__ void run(fx (&a)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) fx_dft4<INV>(a[i], a[i + 4], a[i + 8], a[i + 12]);
    a[0] = fx_down<2 - SH>(a[0]);
    a[1] = fx_down<2 - SH>(a[1]);
    a[2] = fx_down<2 - SH>(a[2]);
    a[3] = fx_down<2 - SH>(a[3]);
    a[4] = fx_down<2 - SH>(a[4]);
    a[5] = fx_rot16<1, INV, SH>(a[5]);
    a[6] = fx_rot16<2, INV, SH>(a[6]);
    a[7] = fx_rot16<3, INV, SH>(a[7]);
    a[8] = fx_down<2 - SH>(a[8]);
    a[9] = fx_rot16<2, INV, SH>(a[9]);
    a[10] = fx_rot16<4, INV, SH>(a[10]);
    a[11] = fx_rot16<6, INV, SH>(a[11]);
    a[12] = fx_down<2 - SH>(a[12]);
    a[13] = fx_rot16<3, INV, SH>(a[13]);
    a[14] = fx_rot16<6, INV, SH>(a[14]);
    a[15] = fx_rot16<9, INV, SH>(a[15]);
#pragma unroll
    for (int k = 0; k < 4; ++k) fx_dft4<INV>(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
    // output 4 q + k sits at a[4 k + q]: transpose
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = k + 1; q < 4; ++q) {
        const fx t = a[4 * k + q];
        a[4 * k + q] = a[4 * q + k];
        a[4 * q + k] = t;
      }
  }
};

// elements per thread of a length-N transform, and its threads
// (radix 8: 32 data registers; radix 16 with its 15 twiddles spills 1 to 2 KB a
// thread, and is used only where radix 8 would need 1024 threads a sequence)
__host__ __device__ constexpr int fx_radix(int n) { return n < 8 ? n : (n <= 4096 ? 8 : 16); }
__host__ __device__ constexpr int fx_threads(int n) { return n / fx_radix(n); }
// padded index: one pad element per 16 (the first pass's stride-16 stores then
// step 17, and eight 16-byte accesses of a phase fall in distinct banks)
__host__ __device__ constexpr int fx_sp(int i) { return i + (i >> 4); }
__host__ __device__ constexpr int fx_len(int n) { return n + (n >> 4); }

// The twiddle table: for every span L = 2 .. FX_NMAX the full circle
// exp(-2 pi i q / L), q = 0 .. L - 1, at L - 2 + q
constexpr int FX_NMAX = 8192;
constexpr int FX_TABLE = 2 * FX_NMAX - 2;

// Bits given up by the whole forward transform of length N (its value is the
// unnormalised transform divided by 2^shift)
template <int N>
constexpr int fx_shift(int ns = 1) {
  constexpr int R = fx_radix(N);
  int s = 0;
  while (ns < N) {
    const int r = (N / ns < R) ? N / ns : R;
    if (ns > 1) s += 2;
    s += r == 16 ? 2 : r == 8 ? 1 : 0;
    ns *= r;
  }
  return s;
}

// a twiddle, loaded where it is used (an ordinary load is hoisted together with
// the pass's others, which costs their registers)
__device__ __forceinline__ fxw fx_tw(const fxw* __restrict__ p) {
  fxw w;
  asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(w.xh), "=r"(w.xl), "=r"(w.yh), "=r"(w.yl) : "l"(p));
  return w;
}

// One Stockham pass (vg_fft.cuh) at span ns on r elements a butterfly: loads from s
// (FIRST: from io), twiddles, butterflies, results in a.  The transform back first
// divides its bins by 2^h.
template <int N, bool INV, int r, bool FIRST>
__device__ __forceinline__ void fx_pass(const fx* s, int t, const fxw* __restrict__ tw, int ns, int h,
                                        const fx (&io)[fx_radix(N)], fx (&a)[fx_radix(N)]) {
  constexpr int R = fx_radix(N), G = N / R, BPT = R / r;
#pragma unroll
  for (int b = 0; b < BPT; ++b) {
    const int j = t + b * G;
    fx v[r];
#pragma unroll
    for (int m = 0; m < r; ++m) {
      if constexpr (FIRST) v[m] = io[m];
      else v[m] = s[fx_sp(j + m * (N / r))];
    }
    if constexpr (!FIRST) {
      const int k = j & (ns - 1);
      const fxw* span = tw + (ns * r - 2);
      if constexpr (!INV) v[0] = fx_down<2>(v[0]);
#pragma unroll
      for (int m = 1; m < r; ++m) v[m] = fx_cmul<INV ? 2 : 0, INV>(v[m], fx_tw(span + m * k));
    } else if constexpr (INV) {
      if (h > 0) {
#pragma unroll
        for (int m = 0; m < r; ++m) {
          v[m].x = (v[m].x + (1ll << (h - 1))) >> h;
          v[m].y = (v[m].y + (1ll << (h - 1))) >> h;
        }
      }
    }
    FxDft<r, INV>::run(v);
#pragma unroll
    for (int m = 0; m < r; ++m) a[b * r + m] = v[m];
  }
}
template <int N, int r>
__device__ __forceinline__ void fx_scatter(fx* s, int t, int ns, const fx (&a)[fx_radix(N)]) {
  constexpr int R = fx_radix(N), G = N / R;
#pragma unroll
  for (int b = 0; b < R / r; ++b) {
    const int j = t + b * G;
    const int k = j & (ns - 1);
    const int base = (j - k) * r + k;
#pragma unroll
    for (int m = 0; m < r; ++m) s[fx_sp(base + m * ns)] = a[b * r + m];
  }
}

// The transform of a sequence: element i of thread t is t + i N / R.  IN_REGS: the
// input is in io, else in s; OUT_REGS: the output ends in io, else in s.  The passes
// of full radix after the first share their code, in a loop that stays rolled: a
// small run is bound by instruction fetches (five of eight stall cycles at 64 x 1024
// with every pass written out, 37 us a launch with cold caches, now 24).
template <int N, bool INV, bool IN_REGS, bool OUT_REGS, typename Sync>
__device__ __forceinline__ void fx_fft(fx* s, int t, const fxw* __restrict__ tw, const Sync& sync,
                                       fx (&io)[fx_radix(N)], int h = 0) {
  constexpr int R = fx_radix(N), G = N / R;
  constexpr int FULL = ilog2(N) / ilog2(R);          // passes of radix R
  constexpr int REST = N >> (FULL * ilog2(R));       // radix of the last one, or 1
  fx a[R];
  if constexpr (!IN_REGS) {
#pragma unroll
    for (int i = 0; i < R; ++i) io[i] = s[fx_sp(t + i * G)];
  }
  fx_pass<N, INV, R, true>(s, t, tw, 1, h, io, a);
  int ns = 1;
#pragma unroll 1
  for (int q = 1; q < FULL; ++q) {
    sync();
    fx_scatter<N, R>(s, t, ns, a);
    sync();
    ns *= R;
    fx_pass<N, INV, R, false>(s, t, tw, ns, h, io, a);
  }
  if constexpr (REST > 1) {
    sync();
    fx_scatter<N, R>(s, t, ns, a);
    sync();
    fx_pass<N, INV, REST, false>(s, t, tw, N / REST, h, io, a);
  }
  constexpr int r = REST > 1 ? REST : R;
  if constexpr (OUT_REGS) {
    // butterfly b of thread t holds elements t + G (b + m R / r)
#pragma unroll
    for (int b = 0; b < R / r; ++b)
#pragma unroll
      for (int m = 0; m < r; ++m) io[b + m * (R / r)] = a[b * r + m];
  } else {
    sync();
    fx_scatter<N, r>(s, t, N / r, a);
    sync();
  }
}

// ---- doubles to fixed point and back ------------------------------------------
// The largest element of a line decides its scale: element f -> f 2^(1081 - E)
// with E the exponent field, or one less where the largest mantissa is below
// sqrt(2), so that the largest value is in [2^58.5, 2^59.5) (zero and below for
// lines of subnormal values).
// (0 for a zero alone)
__device__ __forceinline__ unsigned fx_exp_bits(double f) {
  return max((unsigned)__double2hiint(f) & 0x7fffffffu, (unsigned)(__double2loint(f) != 0));
}
__device__ __forceinline__ int fx_exp(unsigned max_hi) {
  const int e = (int)(max_hi >> 20);
  if (e == 0x7ff) return e;
  if (e == 0) return max_hi ? __clz(max_hi) == 31 ? -19 : 12 - __clz(max_hi) : 1;  // subnormal: its own leading bit
  return e == 1 ? 1 : e - ((max_hi & 0xfffff) < 0x6a09e ? 1 : 0);
}
constexpr int FX_SCALE = 1081;
constexpr int FX_NONFINITE = 0x7ff;  // fx_exp of a line with a NaN or infinity

__device__ __forceinline__ long long fx_from_double(double f, int E) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(f);
  const int e = (int)((u >> 52) & 0x7ff);
  long long m = (long long)(u & 0xfffffffffffffull);
  if (e) m |= 1ll << 52;
  // f = m 2^(max(e, 1) - 1075); scaled to m 2^(max(e, 1) - E + 6)
  const int sh = (e < 1 ? 1 : e) - E + 6;
  m <<= (sh > 0 ? sh : 0);
  const int dn = sh < 0 ? (sh < -62 ? 62 : -sh) : 0;
  if (dn) m = (m + (1ll << (dn - 1))) >> dn;
  return (long long)u < 0 ? -m : m;
}

// (out of line, as are the other rare or repeated pieces: instruction fetches are what
// a small run waits for)
inline __device__ __noinline__ double fx_to_double_far(long long v, int k) { return ldexp(__ll2double_rn(v), k); }
// v 2^k as a double, rounded to nearest even
__device__ __forceinline__ double fx_to_double(long long v, int k) {
  if (v == 0) return 0.0;
  const unsigned long long sign = (unsigned long long)v & 0x8000000000000000ull;
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int z = __clzll((long long)a);
  const unsigned long long n = a << z;               // top bit at 63
  const unsigned long long m = n >> 11;              // 53 bits
  const unsigned long long rem = n & 0x7ff;
  const int e = 63 - z + k + 1023;                   // exponent field
  if (e < 1 || e > 2045) return fx_to_double_far(v, k);
  // the implicit bit of m adds one to the exponent field; a carry of the rounding runs into it
  unsigned long long r = ((unsigned long long)(e - 1) << 52) + m;
  r += (rem > 0x400 || (rem == 0x400 && (m & 1))) ? 1 : 0;
  return __longlong_as_double((long long)(sign | r));
}

// ---- phases -----------------------------------------------------------------------
// Turns per index of a line: frac(A c) 2^64 for the double c and the constant
// A = am 2^ae turns per unit of c (am a signed 64-bit integer), exact up to the
// last of the 64 bits.  Counted in whole turns the phase of index k is k times
// this, modulo 2^64.
struct FxTurn {
  long long am;
  int ae;
  float own;  // what fx_step_rest's are to be multiplied with, besides c, for fx_own
  int own_e;  // from which exponent of c on that is worth while
};
__device__ __forceinline__ unsigned long long fx_turn(FxTurn A, double c) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(c);
  const int e = (int)((u >> 52) & 0x7ff);
  long long m = (long long)(u & 0xfffffffffffffull);
  if (e) m |= 1ll << 52;
  if ((long long)u < 0) m = -m;
  // product p = am m (117 bits), value p 2^(ae + ee); in units of 2^-64: p 2^sh
  const int sh = A.ae + (e < 1 ? 1 : e) - 1075 + 64;
  const long long hi = __mul64hi(A.am, m);
  const unsigned long long lo = (unsigned long long)A.am * (unsigned long long)m;
  if (sh >= 64) return 0;  // whole turns
  if (sh >= 0) return lo << sh;
  const int d = -sh;
  if (d >= 128) return 0;
  if (d >= 64) return (unsigned long long)((d == 64 ? hi : hi >> (d - 64)) +
                                           (long long)(d == 64 ? lo >> 63 : ((unsigned long long)hi >> (d - 65)) & 1));
  return (((unsigned long long)hi << (64 - d)) | (lo >> d)) + ((lo >> (d - 1)) & 1);
}

struct fxc {
  long long c, s;  // Q62
};
__device__ __forceinline__ fxw fx_mult(fxc p) {
  return {fx_hi(p.c), fx_lo(p.c), fx_hi(p.s), fx_lo(p.s)};
}
// cos and sin of 2 pi tau / 2^64: the nearest of 8192 table angles, and the
// rest (|x| < 3.9e-4) by the Taylor terms to x^4
__device__ __forceinline__ fxc fx_sincos(unsigned long long tau, const fxw* __restrict__ tw) {
  const unsigned q = (unsigned)((tau + (1ull << 50)) >> 51) & (FX_NMAX - 1);
  const long long d = (long long)(tau - ((unsigned long long)q << 51));
  // X = x 2^73, V = x^2 2^82
  const long long X = __mul64hi(d << 13, 7244019458077122842ll);  // 2 pi 2^60
  const long long V = __mul64hi(X, X);
  const int w4 = (int)(__mul64hi(V, V) >> 32);                    // x^4 2^68
  const long long cm1 = -(V >> 21) + (long long)(((unsigned long long)(unsigned)w4 * 2796203ull) >> 32);
  const long long s1 = (X >> 11) - (__mul64hi(__mul64hi(X, V), 3074457345618258603ll) >> 29);
  const fxw w = tw[FX_NMAX - 2 + q];  // (cos, -sin) of the table angle
  // (c0 + i s0)(1 + cm1 + i s1) - (c0 + i s0)
  const fx p = fx_cmul<2, true>({cm1, s1}, w);
  const long long c0 = ((long long)w.xh << 32) + w.xl, n0 = ((long long)w.yh << 32) + w.yl;
  return {c0 + p.x, p.y - n0};
}
inline __device__ __noinline__ fxc fx_sincos_call(unsigned long long tau, const fxw* tw) { return fx_sincos(tau, tw); }
// the product of two unit rotations
__device__ __forceinline__ fxc fx_turn_by(fxc a, const fxw& w) {
  const fx p = fx_cmul<0, false>({a.c, a.s}, w);
  return {(long long)((unsigned long long)p.x << 2), (long long)((unsigned long long)p.y << 2)};
}

// A grid's wavenumbers are m k1 to their own rounding only, which is some 2^-53 of the
// phase: what wavenumber m is off by (rest of fx_step_rest, here in FP32) times -2 pi
// dt c, a small angle in Q64, is turned on top of the m steps.  (Without it the
// phases' errors are those of the doubles ((-k) dt) c, twice to thirty times the
// transform's on lines with all wavenumbers in them.)  It is 3 % of the x-drift; below
// 2^-51, what the wavenumbers' rounding makes of phases of ten radians or so, it is left
// out: the transform's own error is as large.
// (by its exponent: a conversion takes as long as some thirty other instructions)
__device__ __forceinline__ bool fx_has_own(const FxTurn& t, double c) {
  return ((__double2hiint(c) >> 20) & 0x7ff) >= t.own_e;
}
__device__ __forceinline__ fxc fx_own(fxc p, float own) {
  const int d = __float2int_rn(own);
  return {p.c - __mulhi((int)(p.s >> 32), d), p.s + __mulhi((int)(p.c >> 32), d)};
}
constexpr double FX_OWN_LEAST = 8192.0;  // 2^-51 in Q64
// (shorter lines hardly have such phases: the code is left out for the cold launches' sake)
constexpr int FX_OWN_N = 128;

// What the rotation learns about the bins it leaves: an upper bound of the sum
// of their moduli in units of 2^38, and the sums of the squares of line a's and
// b's bins in units of 2^88, rounded down (by Parseval's theorem a sum is the line's
// mean square, below 2^31 units)
struct FxNorms {
  unsigned l1, a2, b2;
};
__device__ __forceinline__ unsigned fx_abs_hi(long long a) { return (unsigned)abs((int)(a >> 32)); }
// |z| <= max + (sqrt(2) - 1) min of |re|, |im|, in units of 2^38, rounded up
__device__ __forceinline__ unsigned fx_mod(fx z) {
  const unsigned x = (fx_abs_hi(z.x) >> 6) + 1, y = (fx_abs_hi(z.y) >> 6) + 1;
  const unsigned lo = min(x, y);
  return max(x, y) + lo - (lo >> 1) - (lo >> 4);  // (1 - 1/2 - 1/16) lo
}
__device__ __forceinline__ unsigned fx_sq(long long a) {
  const unsigned q = fx_abs_hi(a) >> 12;
  return q * q;
}

// Rotation of a packed line pair in the bins (two_real_rotate of vg_fft.cuh):
// the sequence in s is the transform of a + i b, still to be divided by 2^DOWN;
// bin k of a is multiplied by exp(2 pi i k fa / 2^64) and, if own, turned by rest[k]
// oa, of b likewise.  The G threads of the sequence take the bins t, t + G, ... <= N/2.
template <int N, int DOWN>
__device__ __forceinline__ FxNorms fx_rotate(fx* s, int t, unsigned long long fa, unsigned long long fb, bool own,
                                             float oa, float ob, const float* __restrict__ rest,
                                             const fxw* __restrict__ tw) {
  constexpr int G = fx_threads(N);
  FxNorms n = {0, 0, 0};
  fxc pa = fx_sincos_call((unsigned long long)t * fa, tw), pb = fx_sincos_call((unsigned long long)t * fb, tw);
  const fxw ga = fx_mult(fx_sincos_call((unsigned long long)G * fa, tw));
  const fxw gb = fx_mult(fx_sincos_call((unsigned long long)G * fb, tw));
  for (int k = t; k <= N / 2; k += G) {
    fxc qa = pa, qb = pb;
    if (own) {
      const float r = rest[k];
      qa = fx_own(pa, r * oa);
      qb = fx_own(pb, r * ob);
    }
    const fxw wa = fx_mult(qa), wb = fx_mult(qb);
    const fx zk = fx_down<DOWN>(s[fx_sp(k)]);
    if (k == 0 || 2 * k == N) {
      // the bins of both lines are real: only the real part of the rotation acts
      const fx z = {fx_rmul<2>(zk.x, wa.xh, wa.xl), fx_rmul<2>(zk.y, wb.xh, wb.xl)};
      s[fx_sp(k)] = z;
      n.l1 += fx_mod(z);
      n.a2 += fx_sq(zk.x);
      n.b2 += fx_sq(zk.y);
    } else {
      const fx zm = fx_down<DOWN>(s[fx_sp(N - k)]);
      // 2 A = zk + conj(zm), 2 i B = zk - conj(zm)
      const fx A = fx_cmul<1, false>({zk.x + zm.x, zk.y - zm.y}, wa);
      const fx B = fx_cmul<1, false>({zk.y + zm.y, zm.x - zk.x}, wb);
      const fx u = {A.x - B.y, A.y + B.x}, v = {A.x + B.y, B.x - A.y};
      s[fx_sp(k)] = u;
      s[fx_sp(N - k)] = v;
      n.l1 += fx_mod(u) + fx_mod(v);
      n.a2 += 2 * (fx_sq(A.x) + fx_sq(A.y));
      n.b2 += 2 * (fx_sq(B.x) + fx_sq(B.y));
    }
    pa = fx_turn_by(pa, ga);
    pb = fx_turn_by(pb, gb);
  }
  return n;
}

// The shift of the bins of a sequence with these norms (its partial sums then
// stay below 2^60.9, where neither the butterflies nor the products of
// fx_cmul<2> overflow), or -1 where the error of the result, FX_NOISE sqrt(N)
// 2^h units, exceeds that of the transform in doubles, 1e-16 (1 + log2(N) / 5)
// of a line's RMS.  A line that is zero (no_a, no_b) has no error to speak of.
constexpr float FX_NOISE = 0.6f;
template <int N>
__device__ __forceinline__ int fx_shift_back(const FxNorms& n, bool no_a, bool no_b) {
  constexpr unsigned lim = 7827145u;  // 2^22.9
  int h = 0;
  while (h < 16 && (n.l1 >> h) >= lim) ++h;
  constexpr float dbl = 1e-16f * (1.f + 0.2f * ilog2(N));
  // rms^2 = q 2^88 >= N (FX_NOISE 2^h / dbl)^2
  const float need = FX_NOISE * (float)(1 << h) / (dbl * 17592186044416.f);  // 2^44
  const float least = (float)N * need * need;
  if ((!no_a && (float)n.a2 < least) || (!no_b && (float)n.b2 < least)) return -1;
  return h;
}

inline __device__ __noinline__ double fx_scale_far(double x, int k) { return ldexp(x, k); }
// x 2^k without an FP64 instruction where x and the result are ordinary
__device__ __forceinline__ double fx_scale(double x, int k) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  if ((unsigned)(e - 1) < 2046u && (unsigned)(e + k - 1) < 2046u) return __hiloint2double(hi + (k << 20), __double2loint(x));
  return x == 0.0 ? x : fx_scale_far(x, k);
}

// One line of a pair and its phase: elements f[n es], the power of two that brings
// it to an RMS of order one, its turns per index and what its fx_own angles are the
// rest's multiples of; bad: it comes out as NaN
struct FxLine {
  double* f;
  unsigned long long turn;
  float own;
  int up;
  bool on, bad;
};
// that power of two for a line of scale E whose bins' squares add up to q (FxNorms).
__device__ __forceinline__ int fx_up(int E, unsigned q) { return FX_SCALE - 44 - E - (32 - __clz((int)q)) / 2; }
// The pair in doubles, for the lines that fx_shift_back turns away.  Each line is
// brought to the same RMS by its own power of two (exact): what one of them rounds at
// reaches the other, which must not take more than its own.  (Brought to the same
// maximum, a spike beside a smooth line took five times the error it has alone at 2048.)
// The phases are the fixed-point ones (their sines were a quarter of the FP64
// instructions) and the scaling moves exponents, since the pair has paid for the
// fixed-point forward transform as well: a half kick of 2048 x 4096 of noise takes 1.01
// ms, 1.23 with sines and products in doubles, 1.02 with no fixed point at all (0.24 for
// smooth rows); 4096 x 4096 columns 2.17, 2.55, 2.13.
// Out of line: it must not take registers from the fixed-point path.
template <int N, typename Sync>
__device__ __noinline__ void fx_pair_f64(FxLine a, FxLine b, long long es, cx<double>* s, int t,
                                         const float* __restrict__ rest, const fxw* __restrict__ angles,
                                         const cx<double>* __restrict__ tw, Sync sync) {
  constexpr int R = fx_radix(N), G = fx_threads(N);
  const bool use_a = a.on && !a.bad, use_b = b.on && !b.bad;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const long long n = (long long)(t + i * G) * es;
    s[sp<double>(t + i * G)] = {use_a ? fx_scale(a.f[n], a.up) : 0.0, use_b ? fx_scale(b.f[n], b.up) : 0.0};
  }
  sync();
  block_fft<double, N, false, R>(s, t, tw, sync);
  fxc pa = fx_sincos_call((unsigned long long)t * a.turn, angles), pb = fx_sincos_call((unsigned long long)t * b.turn, angles);
  const fxw ga = fx_mult(fx_sincos_call((unsigned long long)G * a.turn, angles));
  const fxw gb = fx_mult(fx_sincos_call((unsigned long long)G * b.turn, angles));
  two_real_rotate<double>(s, N, t, G, [&](int k, double& ca, double& sa, double& cb, double& sb) {
    const float own = rest[k];
    const fxc qa = fx_own(pa, own * a.own), qb = fx_own(pb, own * b.own);
    ca = fx_to_double(qa.c, -62);
    sa = fx_to_double(qa.s, -62);
    cb = fx_to_double(qb.c, -62);
    sb = fx_to_double(qb.s, -62);
    pa = fx_turn_by(pa, ga);
    pb = fx_turn_by(pb, gb);
  });
  sync();
  block_fft<double, N, true, R>(s, t, tw, sync);
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const long long n = (long long)(t + i * G) * es;
    const cx<double> z = s[sp<double>(t + i * G)];
    if (a.on) a.f[n] = a.bad ? nan : fx_scale(z.x, -a.up - ilog2(N));
    if (b.on) b.f[n] = b.bad ? nan : fx_scale(z.y, -b.up - ilog2(N));
  }
}

}  // namespace vg
