// 64-bit block fixed point for the transforms of the FP64 form.
//
// GB300 issues 2 FP64 instructions per clock and SM against 32 widening
// 32 x 32 + 64 bit integer multiply-adds and about 60 64-bit integer adds, so
// an FP64 transform is cheaper in integers: a line is scaled by one power of
// two to integers below 2^K, every pass of the transform runs in integers, and
// between passes the tile is shifted back below 2^K (the largest magnitude
// says by how much).  K leaves room for the growth of one pass, so no sum can
// overflow: fx_bits and fx_pad_bits by the pass's radix, and a tile one bit
// short of it stays as it is, so the unit is 2^-56 (radices 9 to 16) to 2^-61
// of the tile's largest value.  (A tile holds one to four lines, which share the
// exponent.)  FP64 rounds at 2^-53 of each value instead: small values beside
// large ones keep fewer digits here, but the error of a transform relative to
// its tile is below that of the FP64 transform it replaced on random-phase
// spectra from white to k^-2 (against long double; tests/test_gpu_kernels.py and
// test_gpu_fixed_point.py).
//
// Constants and twiddles are 62-bit fractions split into 32-bit halves with a
// signed low half.  A product keeps the three larger partial products (the
// low x low one is below one unit) and is rounded to nearest.
#pragma once
#include <cuda_runtime.h>

#include "pal_consts.h"

namespace pal {

using fxc = longlong2;  // complex fixed point; the exponent belongs to the tile

struct FxHalves {
  int h, l;
};
__device__ __forceinline__ FxHalves fx_split(long long v) {
  const unsigned lo = (unsigned)v;
  return {(int)(v >> 32) + (int)(lo >> 31), (int)lo};
}
// a b + c as one widening multiply-add (spelled out: the compiler's own choice
// for the C expression ran the twiddle product at 0.76 clk per SM, this at 0.50)
__device__ __forceinline__ long long fx_mad(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
__device__ __forceinline__ long long fx_wide(int a, int b) {
  long long r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
// (acc 2^32 + cross) / 2^30, cross already holding the rounding half
__device__ __forceinline__ long long fx_join(long long acc, long long cross) { return (acc << 2) + (cross >> 30); }
constexpr long long kFxHalf = 1LL << 29;

// x * (c + i s), or x * (c - i s) with CONJ; w = {c.h, c.l, s.h, s.l}.  |x|
// (modulus) below 2^62.8 keeps every sum inside 64 bits.
template <bool CONJ>
__device__ __forceinline__ fxc fx_cmul(fxc x, int4 w) {
  const FxHalves X = fx_split(x.x), Y = fx_split(x.y);
  const int nh = -w.z, nl = -w.w;
  const int rh = CONJ ? w.z : nh, rl = CONJ ? w.w : nl;  // re = x c + y r
  const int ih = CONJ ? nh : w.z, il = CONJ ? nl : w.w;  // im = x i + y c
  long long kr = fx_mad(X.h, w.y, kFxHalf), ki = fx_mad(X.h, il, kFxHalf);
  kr = fx_mad(Y.h, rl, kr);
  ki = fx_mad(Y.h, w.y, ki);
  kr = fx_mad(X.l, w.x, kr);
  ki = fx_mad(X.l, ih, ki);
  kr = fx_mad(Y.l, rh, kr);
  ki = fx_mad(Y.l, w.x, ki);
  const long long ar = fx_mad(X.h, w.x, fx_wide(Y.h, rh)), ai = fx_mad(X.h, ih, fx_wide(Y.h, w.x));
  return fxc{fx_join(ar, kr), fx_join(ai, ki)};
}
// The same divided by 4: the halves' weights then line up with whole words, so
// the carry joins through the accumulators (18 instructions for 28).  A pass
// multiplies by its run-time twiddles this way; the factor 1/4 takes back the
// growth of a radix-16 butterfly on uncorrelated data.
template <bool CONJ>
__device__ __forceinline__ fxc fx_cmul4(fxc x, int4 w) {
  const FxHalves X = fx_split(x.x), Y = fx_split(x.y);
  const int nh = -w.z, nl = -w.w;
  const int rh = CONJ ? w.z : nh, rl = CONJ ? w.w : nl;
  const int ih = CONJ ? nh : w.z, il = CONJ ? nl : w.w;
  constexpr long long half = 1LL << 31;
  long long kr = fx_mad(X.h, w.y, half), ki = fx_mad(X.h, il, half);
  kr = fx_mad(Y.h, rl, kr);
  ki = fx_mad(Y.h, w.y, ki);
  kr = fx_mad(X.l, w.x, kr);
  ki = fx_mad(X.l, ih, ki);
  kr = fx_mad(Y.l, rh, kr);
  ki = fx_mad(Y.l, w.x, ki);
  return fxc{fx_mad(Y.h, rh, fx_mad(X.h, w.x, kr >> 32)), fx_mad(Y.h, w.x, fx_mad(X.h, ih, ki >> 32))};
}
// x * c for a constant c = {h, l}
__device__ __forceinline__ long long fx_mulc(long long x, int h, int l) {
  const FxHalves X = fx_split(x);
  return fx_join(fx_wide(X.h, h), fx_mad(X.h, l, fx_mad(X.l, h, kFxHalf)));
}
// x y / 2^64 for |x|, |y| below 2^62
__device__ __forceinline__ long long fx_mul(long long x, long long y) {
  const FxHalves X = fx_split(x), Y = fx_split(y);
  return fx_mad(X.h, Y.h, fx_mad(X.h, Y.l, fx_mad(X.l, Y.h, 1LL << 31)) >> 32);
}

// Halves of a constant known at compile time.
__host__ __device__ constexpr int fx_hi(long long v) { return (int)((v + (1LL << 31)) >> 32); }
__host__ __device__ constexpr int fx_lo(long long v) { return (int)(v - ((long long)fx_hi(v) << 32)); }

// Bits of the largest input component of a pass of radix R: a component below
// 2^K has a modulus below 2^(K + 1/2), R of them add up to less than 2^62.6.
__host__ __device__ constexpr int fx_bits(int R) {
  return R <= 2 ? 61 : R <= 4 ? 60 : R <= 8 ? 59 : R <= 16 ? 58 : 57;
}
// The same for the first pass over a line with the 3/2 pad: a butterfly of a
// radix R divisible by 3 has R / 3 zeros among its inputs (the middle third, in
// natural order for the first radix and in digit-reversed for the last).
__host__ __device__ constexpr int fx_pad_bits(int R) { return fx_bits(R % 3 == 0 ? 2 * R / 3 : R); }

// Multiply by W_R^(SIGN*E), all compile time (the integer counterpart of twc).
template <int R, int E, int SIGN>
__device__ __forceinline__ fxc fx_twc(fxc a) {
  constexpr int e = ((E % R) + R) % R;
  if constexpr (e == 0) {
    return a;
  } else if constexpr ((4 * e) % R == 0) {
    constexpr int q = 4 * e / R;  // quarter turns
    if constexpr (q == 2) {
      return fxc{-a.x, -a.y};
    } else if constexpr ((q == 1) == (SIGN > 0)) {
      return fxc{-a.y, a.x};
    } else {
      return fxc{a.y, -a.x};
    }
  } else if constexpr ((8 * e) % R == 0) {
    constexpr int q = 8 * e / R;  // odd multiple of pi/4: sums first, two products
    constexpr long long h = TrigQ<8>::c[1];
    constexpr bool cn = !(q == 1 || q == 7);
    constexpr bool sn = (q == 1 || q == 3) != (SIGN > 0);
    const long long cx = cn ? -a.x : a.x, cy = cn ? -a.y : a.y, sx = sn ? -a.x : a.x, sy = sn ? -a.y : a.y;
    return fxc{fx_mulc(cx - sy, fx_hi(h), fx_lo(h)), fx_mulc(sx + cy, fx_hi(h), fx_lo(h))};
  } else {
    constexpr long long c = TrigQ<R>::c[e], s = TrigQ<R>::s[e];
    return fx_cmul<(SIGN < 0)>(a, make_int4(fx_hi(c), fx_lo(c), fx_hi(s), fx_lo(s)));
  }
}
// x / 2, halves rounded up and down in turn (no bias)
__device__ __forceinline__ long long fx_half(long long x) { return (x + ((x >> 1) & 1)) >> 1; }

// Range of the high words seen by a thread; fx_top_word is the largest
// magnitude's high word (for a maximum over the tile).
struct FxRange {
  int hi = 0, lo = 0;
  __device__ __forceinline__ void add(fxc x) {
    const int a = (int)(x.x >> 32), b = (int)(x.y >> 32);
    hi = __vimax3_s32(hi, a, b);
    lo = __vimin3_s32(lo, a, b);
  }
  __device__ __forceinline__ unsigned word() const { return (unsigned)max(hi, ~lo); }
};
// Left shift (negative: right) that brings a tile with this largest word to K
// bits; a tile at most one bit short stays as it is (its shifts would cost more
// than the bit is worth).
__device__ __forceinline__ int fx_shift_exact(unsigned word, int K) { return K - 64 + __clz((int)word); }
__device__ __forceinline__ int fx_shift(unsigned word, int K) {
  const int s = fx_shift_exact(word, K);
  return s == 1 ? 0 : s;
}

template <int R>
__device__ __forceinline__ void fx_rescale(fxc (&x)[R], int s) {
  if (s > 0) {
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = fxc{x[k].x << s, x[k].y << s};
  } else if (s < 0) {
    const long long half = 1LL << (-s - 1);
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = fxc{(x[k].x + half) >> -s, (x[k].y + half) >> -s};
  }
}

// FP64 -> fixed point: d 2^(K + 1022 - emax), truncated (toward zero, so without
// bias), for a tile whose largest biased exponent is emax (at least 1): the
// result is below 2^K.
template <int K>
__device__ __forceinline__ long long fx_from_double(double d, int emax) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const int e = (int)(hi >> 20) & 0x7ff;
  // the significand with its leading bit in bit 63; a subnormal (e = 0) has no
  // leading one and the exponent of e = 1
  unsigned long long m = ((unsigned long long)((hi << 11) | 0x80000000u | (lo >> 21)) << 32) | (lo << 11);
  if (e == 0) m <<= 1;
  const int sh = emax - e + (64 - K);
  const long long q = sh > 63 ? 0 : (long long)(m >> sh), sg = (int)hi >> 31;
  return (q ^ sg) - sg;
}
// Exponent E of the fixed-point value of fx_from_double: value = q 2^E.
__device__ __forceinline__ int fx_exponent(int emax, int K) { return emax - 1022 - K; }

// q 2^E in FP64, rounded to nearest (ties away from zero); E in
// [-1020, 950], or any E through fx_scalbn.
__device__ __forceinline__ double fx_to_double(long long q, int E) {
  const long long sg = q >> 63;
  unsigned long long u = (unsigned long long)((q ^ sg) - sg);
  int lz = __clz((int)(u >> 32));
  if (lz == 32) {  // below 2^32
    if (u == 0) return 0.0;
    lz = __clzll((long long)u);
  }
  u <<= lz;
  const unsigned long long m = (u >> 11) + ((u >> 10) & 1);  // 2^52 <= m <= 2^53
  const int hi = (int)(m >> 32) + ((E + 1085 - lz) << 20);
  return __hiloint2double(hi | ((int)sg & (int)0x80000000), (int)(unsigned)m);
}
// An integer of at most 24 bits in FP64 without the FP64 pipe: through float,
// whose bits are those of the double, rebiased.
__device__ __forceinline__ double fx_small(int i) {
  const unsigned b = __float_as_uint((float)i);
  const unsigned hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20));
  return i == 0 ? 0.0 : __hiloint2double((int)hi, (int)(b << 29));
}
__device__ __forceinline__ bool fx_normal(int E) { return E >= -1020 && E <= 950; }
__device__ __noinline__ static double fx_scalbn(long long q, int E) { return scalbn(fx_to_double(q, 0), E); }

// 1 / d by two steps of Newton's iteration from the hardware's reciprocal
// estimate (about 20 bits: each step doubles them).  d is finite and at least 1.
__device__ __forceinline__ double newton_rcp(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(r, fma(-d, r, 1.0), r);
  return fma(r, fma(-d, r, 1.0), r);
}

// cos and sin of pi/4 * r / M (0 <= r <= M) as 63-bit fractions, by their Taylor
// series in integers (eleven terms: below 2^-63 for arguments up to pi/4).
__device__ __forceinline__ unsigned long long fx_mul63(unsigned long long a, unsigned long long b) {
  return (__umul64hi(a, b) << 1) | ((a * b) >> 63);
}
__device__ inline void fx_cossin(unsigned r, unsigned M, unsigned long long* c, unsigned long long* s) {
  const unsigned long long p4 = 0xC90FDAA22168C234ull;  // pi/4 as a 64-bit fraction
  const unsigned long long one = 1ull << 63;
  const unsigned long long x = ((p4 / M) * r + ((p4 % M) * r) / M) >> 1;
  const unsigned long long t = fx_mul63(x, x);
  unsigned long long cs = one, sn = one;
  for (int k = 11; k >= 1; --k) {
    cs = one - fx_mul63(t, cs) / (unsigned)((2 * k - 1) * (2 * k));
    sn = one - fx_mul63(t, sn) / (unsigned)((2 * k) * (2 * k + 1));
  }
  *c = cs;
  *s = fx_mul63(x, sn);
}
// exp(-2 pi i a / M), 0 <= a < M, as {c.h, c.l, s.h, s.l} of c + i s.
__device__ inline int4 fx_root(int a, int M) {
  const int o = (8 * a) / M, r = 8 * a - o * M;
  unsigned long long c63, s63;
  fx_cossin((o & 1) ? M - r : r, M, &c63, &s63);
  const long long c = (long long)((c63 + 1) >> 1), s = (long long)((s63 + 1) >> 1);
  long long re, im;  // of exp(+2 pi i a / M)
  switch (o) {
    case 0: re = c, im = s; break;
    case 1: re = s, im = c; break;
    case 2: re = -s, im = c; break;
    case 3: re = -c, im = s; break;
    case 4: re = -c, im = -s; break;
    case 5: re = -s, im = -c; break;
    case 6: re = s, im = -c; break;
    default: re = c, im = -s; break;
  }
  im = -im;
  if ((int)re == (int)0x80000000) ++re;  // no low half of -2^31: fx_cmul negates it
  if ((int)im == (int)0x80000000) ++im;
  const FxHalves a0 = fx_split(re), a1 = fx_split(im);
  return make_int4(a0.h, a0.l, a1.h, a1.l);
}

}  // namespace pal
