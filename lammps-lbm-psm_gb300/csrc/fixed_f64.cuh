// fixed_f64.cuh -- IEEE double additions and some products of the collide step on
// the integer units, bit for bit.
//
// This GPU issues 1.68 FP64 operations per clock and multiprocessor against
// about 100 integer ones, and both at once, so an addition whose rounding
// position is known can be had for a dozen integer instructions beside the
// FP64 pipe.  Near rest it is known: populations, their sums and the factors
// 1 + 3 e.u + ... of the equilibria keep to a few binades.  The values are held
// as 64-bit integers in units of 2^-61 (density and momentum sums) or 2^-62 (the
// factors, equilibria and their differences from the populations); each result
// is rounded to 53 significant bits, ties to even, as the IEEE operation it
// stands for.  Products by the constants 3, 4.5 and 1.5 and of a density with a
// factor are formed the same way.  Every function states the range it needs;
// the ranges are checked (populations and density in macro_sums, velocity
// components below 5/64 by the caller) and the FP64 expressions taken otherwise.
// A suspension whose spheres move at 0.04 stays inside.
//
// Host compilable: the functions are compared with IEEE arithmetic on the CPU.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define LBMPSM_HD __host__ __device__ __forceinline__
#else
#define LBMPSM_HD inline
#endif

namespace lbmpsm {
namespace fx {

typedef unsigned long long u64;
typedef long long i64;

LBMPSM_HD u64 bits_of(double x) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(x);
#else
  u64 b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
LBMPSM_HD double of_bits(u64 b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((i64)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
LBMPSM_HD int clz32(unsigned x) {  // x != 0
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return __builtin_clz(x);
#endif
}
LBMPSM_HD int clz64(u64 x) {  // x != 0
#ifdef __CUDA_ARCH__
  return __clzll((i64)x);
#else
  return __builtin_clzll(x);
#endif
}

// f in units of 2^-61; f in [2^-7, 1), else bad becomes non-zero.  The result
// is a multiple of 4.
LBMPSM_HD u64 to61(double f, unsigned& bad) {
  const u64 b = bits_of(f);
  const unsigned hi = (unsigned)(b >> 32);
  const unsigned s = (hi >> 20) - (1023u - 7u);  // 0..6; sign, small, large, inf, NaN: beyond
  bad |= s > 6u ? 1u : 0u;
  const u64 m = ((u64)((hi & 0xFFFFFu) | 0x100000u) << 32) | (b & 0xFFFFFFFFull);
  return m << ((s + 2u) & 15u);
}

// t rounded to a multiple of 2^sh, ties to even (t >= 0)
LBMPSM_HD u64 rne(u64 t, int sh) {
  return (t + ((1ull << (sh - 1)) - 1ull) + ((t >> sh) & 1ull)) & ~((1ull << sh) - 1ull);
}

// t >= 0 in units of 2^-61, rounded to 53 bits: t in [2^(59+k0), 2^(61+k0))
// where k0 = 0 (t in [1/4, 1)) or 1 (t in [1/2, 2))
LBMPSM_HD u64 rne53_of2(u64 t, int k0) {
  const unsigned c = (unsigned)(t >> (60 + k0)) & 1u;
  const int sh = 7 + k0 + (int)c;
  const u64 half = 64ull << (k0 + (int)c);
  return (t + (half - 1ull) + ((t >> sh) & 1ull)) & ~(2ull * half - 1ull);
}

// high word of |t| (of |t| - 1 for negative t)
LBMPSM_HD unsigned abs_hi(i64 t) { return (unsigned)((u64)t >> 32) ^ (unsigned)(t >> 63); }

// t (a multiple of 4, |t| < 2^62) rounded to 53 bits: multiples of 4 below
// 2^55 are held exactly (and left alone by the rounding to 2^2)
LBMPSM_HD i64 rne53_signed(i64 t) {
  const int sh = 2 + (9 - clz32(abs_hi(t) | 0x400000u));
  const unsigned m = (1u << sh) - 1u;
  const u64 inc = (u64)((m >> 1) + (((unsigned)t >> sh) & 1u));
  return (i64)(((u64)t + inc) & ~(u64)m);
}

// the double t * 2^-61 (t with at most 53 significant bits)
LBMPSM_HD double from61(i64 t) {
  const u64 sg = (u64)t & 0x8000000000000000ull;
  const u64 a = t < 0 ? (u64)0 - (u64)t : (u64)t;
  if (a == 0) return 0.0;
  const int lz = clz64(a);
  const u64 m = (a << lz) >> 11;  // 53 bits, the leading one at bit 52
  return of_bits(sg | (m + ((u64)(1024 - lz) << 52)));
}

// the double t * 2^-61 for a 53-bit t in [1/2, 2)
LBMPSM_HD double from61_near1(u64 t) {
  const unsigned c = (unsigned)(t >> 61);
  return of_bits((t >> (8 + c)) + ((u64)(1021u + c) << 52));
}

// |x * K / 2^H| rounded as a double, in units of 2^-62 (K/2^H = 3, 4.5 or 1.5;
// |x| <= 5/32): the 53 bits of the product are formed with the significand's
// multiple; bits below the unit are kept as a set lowest bit ("sticky"), which
// rounds like them at any position above bit 1.  (A product in the denormal
// range is all sticky.)
template <int K, int H>
LBMPSM_HD u64 times62(double x) {
  static_assert(K == 3 || K == 9, "");
  const u64 b = bits_of(x);
  const unsigned e = (unsigned)(b >> 52) & 0x7FFu;
  u64 m = (b & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull);
  m = K == 3 ? m + (m << 1) : m + (m << 3);  // the leading bit at 53 or 54 (K = 9: 55 or 56)
  const unsigned c = (unsigned)(m >> (K == 3 ? 54 : 56)) & 1u;
  const int sh = (K == 3 ? 1 : 3) + (int)c;
  const u64 half = (K == 3 ? 1ull : 4ull) << c;
  m = ((m + (half - 1ull) + ((m >> sh) & 1ull)) & ~(2ull * half - 1ull)) << 7;
  const unsigned r0 = 1020u + H - e;
  const unsigned r = r0 < 63u ? r0 : 63u;
  const u64 a = m >> r;
  return (a << r) != m ? (a | 1ull) : a;
}

constexpr u64 ONE62 = 1ull << 62;

// s >= 0 in units of 2^-62 rounded to 53 bits: s in [1/2, 2)
LBMPSM_HD u64 rne53_62(u64 s) {
  const unsigned c = (unsigned)(s >> 62);
  const int sh = 9 + (int)c;
  const u64 half = 256ull << c;
  return (s + (half - 1ull) + ((s >> sh) & 1ull)) & ~(2ull * half - 1ull);
}

// ((1 + 3 e) + 4.5 ee) - u and ((1 - 3 e) + 4.5 ee) - u in units of 2^-62, each
// operation rounded, for |e| <= 5/32, ee = e*e rounded and 0 <= u < 1/24 (u
// aligned already): the first stays in [1 - u, 3/2 + u], the second in
// [3/5 - u, 1] (e >= 0; the other way round below)
LBMPSM_HD void factors(double e, double ee, u64 u62, u64& plus, u64& minus) {
  const u64 A = times62<3, 0>(e), B = times62<9, 1>(ee);
  u64 p = rne(ONE62 + A, 10);          // in [1, 3/2): units of 2^-52
  u64 m = rne(ONE62 - A, 9);           // in (1/2, 1]: units of 2^-53
  p = rne53_62(rne(p + B, 10) - u62);  // (in [1, 2) before the subtraction)
  m = rne53_62(rne53_62(m + B) - u62);
  const bool neg = (i64)bits_of(e) < 0;
  plus = neg ? m : p;
  minus = neg ? p : m;
}

// 1 - u, rounded (u aligned, below 1/24), in units of 2^-62
LBMPSM_HD u64 one_minus(u64 u62) { return rne(ONE62 - u62, 9); }

// x in [2^-7, 1) in units of 2^-64 and of 2^-62
LBMPSM_HD u64 to64(double x) {
  const u64 b = bits_of(x);
  return (((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11) >> ((1022u - (unsigned)(b >> 52)) & 63u);
}
LBMPSM_HD u64 to62(double x) {
  const u64 b = bits_of(x);
  return ((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << (((unsigned)(b >> 52) - 1013u) & 63u);
}

// the product of r (units of 2^-64) and s (units of 2^-62), rounded to 53 bits,
// in units of 2^-62: from 2^-7 to 2, so that at least three bits of the unit
// lie below the last place.  (An equilibrium rho*w*factor is at least 0.0094:
// macro_sums lets densities of 0.609375 (D3Q19) and 0.5546875 (D2Q9) through at
// the lowest, w is 1/36 at the lowest, and with velocity components below 5/64 a
// factor is above 0.613 = 1 - 3 (5/32) + 4.5 (5/32)^2 - 1.5 * 3 (5/64)^2.)
LBMPSM_HD u64 product62(u64 r, u64 s) {
  const unsigned __int128 x = (unsigned __int128)r * s;
  const u64 t = (u64)(x >> 64) | ((u64)x != 0 ? 1ull : 0ull);
  const int sh = 11 - clz32((unsigned)(t >> 32));
  const u64 m = (1ull << sh) - 1ull;
  return (t + (m >> 1) + ((t >> sh) & 1ull)) & ~m;
}

// a - b rounded, as a double (units of 2^-62, both multiples of 8 below 2^63).
// Multiples of 8 below 2^56 in size need no rounding.
LBMPSM_HD double difference62(u64 a, u64 b) {
  i64 t = (i64)(a - b);
  if (abs_hi(t) >> 24) {
    const int sh = 11 - clz32(abs_hi(t));
    const u64 m = (1ull << sh) - 1ull;
    t = (i64)(((u64)t + (m >> 1) + (((u64)t >> sh) & 1ull)) & ~m);
  }
  const u64 sg = (u64)t & 0x8000000000000000ull;
  const u64 v = t < 0 ? (u64)0 - (u64)t : (u64)t;
  const unsigned hi = (unsigned)(v >> 32);
  const int lz = clz32(hi ? hi : ((unsigned)v | 1u)) + (hi ? 0 : 32);
  const u64 d = sg | (((v << lz) >> 11) + ((u64)(1023 - lz) << 52));
  return v == 0 ? 0.0 : of_bits(d);
}

// Density and momentum sums of compute_macro_values
// (src/LBM_PSM_BGK_dynamics.cpp:48-77), each addition rounded in its place:
// rho = ((f0 + f1) + f2) + ..., j_a the signed sum over the directions with a
// component along a.  Returns whether every range held (else the outputs are
// not to be used): populations in [2^-7, 1), the sum of the first two (D3Q19:
// the first two in [1/4, 1/2), the first three below 1/2; the first five) at
// least 1/2, the density below 2, the partial sums of j below 1/4.  With the other
// populations at 2^-7 at least, the density is 1/2 + 14/128 = 0.609375 (D3Q19) or
// 1/2 + 7/128 = 0.5546875 (D2Q9) at the lowest.
template <class L>
LBMPSM_HD bool macro_sums(const double* f, double& rho, double (&j)[3]) {
  constexpr int Q = L::Q;
  u64 F[Q];
  unsigned bad = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) F[q] = to61(f[q], bad);
  u64 t = F[0];
#pragma unroll
  for (int q = 1; q < Q; ++q) {
    t += F[q];
    if (Q == 19) {
      // at rest 7/18, 8/18 | 1/2 | 5/9 .. 1
      if (q == 1) bad |= t < (1ull << 59) ? 1u : 0u;
      if (q == 2) bad |= t >= (1ull << 60) ? 1u : 0u;
      if (q == 4) bad |= t < (1ull << 60) || t >= (1ull << 61) ? 1u : 0u;
      t = q <= 2 ? rne(t, 7) : rne53_of2(t, q == 3 ? 0 : 1);
    } else {
      // at rest 5/9 .. 1
      if (q == 1) bad |= t < (1ull << 60) ? 1u : 0u;
      t = rne53_of2(t, 1);
    }
  }
  bad |= t >= (1ull << 62) ? 1u : 0u;
  rho = from61_near1(t);
  unsigned over = 0;  // high words of the partial sums
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    j[a] = 0.0;
    if (a == 2 && Q == 9) continue;
    i64 s = 0;
    int terms = 0;
#pragma unroll
    for (int q = 1; q < Q; ++q) {
      const int c = a == 0 ? L::ex(q) : (a == 1 ? L::ey(q) : L::ez(q));
      if (c == 0) continue;
      s = c > 0 ? s + (i64)F[q] : s - (i64)F[q];
      if (++terms == 1) continue;  // one population: exact
      over |= abs_hi(s);
      s = rne53_signed(s);
    }
    j[a] = from61(s);
  }
  return (bad | (over >> 27)) == 0;
}

// |x| < 5/64 (false for inf and NaN)
LBMPSM_HD bool slow(double x) { return ((unsigned)(bits_of(x) >> 32) & 0x7FFFFFFFu) < 0x3FB40000u; }

}  // namespace fx
}  // namespace lbmpsm
