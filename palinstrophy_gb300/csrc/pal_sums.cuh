// Sums of squares for the diagnostics, in plain C++ so that a host program can
// run the same arithmetic.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

namespace pal {

template <class To, class From>
__host__ __device__ __forceinline__ To bits_as(From f) {
  static_assert(sizeof(To) == sizeof(From), "same size");
  To t;
  memcpy(&t, &f, sizeof t);
  return t;
}

// Compensated FP64 summation: s + c carries the running sum, c the exact
// rounding errors of the additions into s (TwoSum, which needs no ordering of
// the operands' magnitudes).
__host__ __device__ __forceinline__ void csum_add(double& s, double& c, double x) {
  const double t = s + x;
  const double bp = t - s;
  c += (s - (t - bp)) + (x - bp);
  s = t;
}

// csum_add for s, x >= 0 (no NaN ordering is needed: a NaN stays one): the
// larger operand is found on the bit patterns, and then Fast2Sum's four FP64
// instructions do what TwoSum needs seven for.
__host__ __device__ __forceinline__ void csum_add_pos(double& s, double& c, double x) {
  const long long is = bits_as<long long>(s), ix = bits_as<long long>(x);
  const double hi = bits_as<double>(is > ix ? is : ix), lo = bits_as<double>(is > ix ? ix : is);
  s = hi + lo;
  c += lo - (s - hi);
}

// u^2 + v^2 of an FP64 point added to a compensated sum.
__host__ __device__ __forceinline__ void add_point(double u, double v, double& acc, double& comp) {
  csum_add_pos(acc, comp, fma(u, u, v * v));
}

// u 2^e in FP64 without the FP64 pipe, rounded to nearest (halves up); the
// result is normal or zero.
__host__ __device__ __forceinline__ double scaled_u64(unsigned long long u, int e) {
  if (u == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)u);
#else
  const int lz = __builtin_clzll(u);
#endif
  u <<= lz;
  const unsigned long long m = (u >> 11) + ((u >> 10) & 1);  // 2^52 <= m <= 2^53, value m 2^(e + 11 - lz)
  return bits_as<double>(((unsigned long long)(e + 11 - lz + 52 + 1022) << 52) + m);
}

// u^2 + v^2 of G FP32 points added to a compensated sum.  Every square is an
// exact integer (24-bit mantissas) and they are added at the exponent E of the
// group's largest value: the whole units of 2^(2 (E - 150)) in one word, the
// fractions they leave when shifted down to it, 60 bits, in another.  Only
// squares that lie 2^62 and more below are left out, so the group's sum is off
// by less than 2^-56 of it (a sum of rounded points by up to 2^-53).
//
// Bound by issue: the FP64 pipe, which gives a warp one instruction in 64
// cycles, has five of them a group; fused multiply-adds on the widened values
// took 3 a point.  The diagnostic k_phys of N=2048 takes 81 us (72 with the
// fractions cut off, 173 with fused multiply-adds, 295 with a TwoSum a point).
template <int G>
__host__ __device__ __forceinline__ void add_squares(const float2 (&x)[G], double& acc, double& comp) {
  static_assert(G <= 8, "2 G squares below 2^48 in 53 bits, 2 G fractions below 2^60 in 64");
  constexpr unsigned MAG = 0x7fffffffu, FRAC = 0x7fffffu;
  unsigned top = 0;
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const unsigned bx = bits_as<unsigned>(x[i].x) & MAG, by = bits_as<unsigned>(x[i].y) & MAG;
    top = top > bx ? top : bx;
    top = top > by ? top : by;
  }
  if (top > MAG - (FRAC + 1)) {  // an infinity or NaN
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < G; ++i) s = fma(double(x[i].x), double(x[i].x), fma(double(x[i].y), double(x[i].y), s));
    csum_add_pos(acc, comp, s);
    return;
  }
  // subnormals have exponent 1 and no leading bit
  const int E = (int)(top >> 23) > 1 ? (int)(top >> 23) : 1;
  unsigned long long whole = 0, part = 0;  // sum = whole + part 2^-60
  auto add = [&](float f) {
    const unsigned b = bits_as<unsigned>(f) & MAG, e = b >> 23;
    int d = 2 * (E - (e > 1 ? (int)e : 1));
    const unsigned m = d > 60 ? 0u : (b & FRAC) | (e != 0 ? FRAC + 1 : 0u);
    d = d > 60 ? 60 : d;
    const unsigned long long sq = (unsigned long long)m * m;
    whole += sq >> d;
    part += (sq << (60 - d)) & ((1ull << 60) - 1);
  };
#pragma unroll
  for (int i = 0; i < G; ++i) {
    add(x[i].x);
    add(x[i].y);
  }
  whole += part >> 60;
  csum_add_pos(acc, comp, scaled_u64(whole, 2 * (E - 150)));  // at most 53 bits: exact
  comp += scaled_u64(part & ((1ull << 60) - 1), 2 * (E - 150) - 60);
}

}  // namespace pal
