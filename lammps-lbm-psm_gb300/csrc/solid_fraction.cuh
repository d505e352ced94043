// solid_fraction.cuh -- the sub-cell count of calcSolidFraction
// (src/LBM_PSM_exchangeParticleData.cpp:116-169) for one node and one sphere:
// FP32 decisions with proven margins, the reference's FP64 expressions for
// the few sub-cells that FP32 leaves open.  The counts are the reference's.
// The FP64 expressions use explicitly rounded intrinsics, so they are the
// same in units built with and without multiply-add contraction.
#pragma once

#include "lbmpsm_internal.cuh"

namespace lbmpsm {

// A sphere as the count needs it (Img holds the same fields).
struct SphereRec {
  double xl[3];  // lattice-local centre; xl = xi + xf exactly up to the rounding of xf
  int xi[3];
  float xf[3];
  double r, rP2, rM2;
  float rP2f, rM2f, rSqf;
};

// xl = xi + xfrac exactly (the fractional part of a double is exact)
static __device__ __forceinline__ void split_centre(double xl, int& xi, float& xf) {
  const bool small = fabs(xl) < 1.0e9;
  const double fl = small ? floor(xl) : 0.0;
  xi = (int)fl;
  xf = (float)(xl - fl);
}

// Early-out part of calcSolidFraction for one node, decided in FP32 with a
// proven margin, else in FP64 with the reference's expressions.  Returns a
// code (0 or SF_ONE) or -1 for a shell node whose sub-cells must be counted.
//
// Offsets dx = (double)h - xl are formed as (h - xi) - xfrac with xl = xi + xfrac
// split exactly, so |dxf - dx| <= u(|dx| + 1), u = 2^-24, and the FP32 squared
// distance obeys |d32 - dist| <= u(5 dist + 2 sum|d|).  The margin m is 16x that.
template <class Sphere>
static __device__ __forceinline__ int classify_node(int hi, int hj, int hk, const Sphere& im,
                                                    float& dxf, float& dyf, float& dzf) {
  const float u = 5.9604644775390625e-08f;  // 2^-24
  dxf = small_int_to_float(hi - im.xi[0]) - im.xf[0];
  dyf = small_int_to_float(hj - im.xi[1]) - im.xf[1];
  dzf = small_int_to_float(hk - im.xi[2]) - im.xf[2];
  const float d32 = dxf * dxf + dyf * dyf + dzf * dzf;
  const float ad = fabsf(dxf) + fabsf(dyf) + fabsf(dzf);
  const float m = 16.0f * u * (5.0f * d32 + 2.0f * ad + 1.0f + im.rP2f);
  if (d32 > im.rP2f + m) return 0;
  const bool nearP = d32 >= im.rP2f - m;
  const bool nearM = d32 >= im.rM2f - m && d32 <= im.rM2f + m;
  if (nearP || nearM) {
    const double dx = (double)hi - im.xl[0];
    const double dy = (double)hj - im.xl[1];
    const double dz = (double)hk - im.xl[2];
    const double dist =
        __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    if (dist > im.rP2) return 0;
    if (dist < im.rM2) return SF_ONE;
    return -1;
  }
  if (d32 < im.rM2f) return SF_ONE;  // below rM^2 - m: inside for certain
  return -1;
}

// Exact double of a small non-negative integer without the conversion unit.
static __device__ __forceinline__ double small_int_to_double(int k) {
  return __hiloint2double(0x43300000, k) - 4503599627370496.0;  // 2^52 + k - 2^52
}

static __device__ __forceinline__ float sub_offset(int k) {
  return -0.45f + 0.1f * small_int_to_float(k);  // within 1.7u of the reference's delta_k
}

// One sub-cell with the reference's FP64 expressions
// (src/LBM_PSM_exchangeParticleData.cpp:144-168): index i[d] along axis d.
template <class Sphere>
static __device__ __noinline__ bool sub_cell_inside(int dim, const Sphere& im, int hx, int hy, int hz,
                                                    int i0, int i1, int i2) {
  const double width = 1.0 / ((double)10);
  const int h[3] = {hx, hy, hz}, i[3] = {i0, i1, i2};
  double sum = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (d >= dim) break;
    const double delta = __dadd_rn(-0.5, __dmul_rn(small_int_to_double(i[d]) + 0.5, width));
    const double t = __dadd_rn(__dadd_rn(small_int_to_double(h[d]), -im.xl[d]), delta);
    const double sq = __dmul_rn(t, t);
    sum = d == 0 ? sq : __dadd_rn(sum, sq);
  }
  return sum < __dmul_rn(im.r, im.r);
}

// Number of sub-cell centres inside the sphere for a shell node at offset
// (dxf, dyf, dzf) from its centre (classify_node's FP32 offsets).
//
// Rows of ten sub-cells run along the axis c of the largest |offset|, where
// the surface cuts them most steeply.  With the sign turned so that dc > 0
// every centre of a row has t_k = dc - 0.45 + 0.1 k > 0, so the ones inside
// are those with t_k < h, h = sqrt(r^2 - s_ab): the row's count is the
// integer nearest to v = 10 (h - dc + 0.5), kept in [0, 10] -- one square root,
// one saturating add, two fused multiply-adds per row, no branch (the
// saturation also sends the NaN of a negative radicand to 0).  v is certain
// when it is not within eps of a half-integer:
//   |s_ab error| <= M = 8u (Ea^2 + Eb^2 + r^2), E = |d| + 2: the terms carry at
//   most 5u(|t|+1/2)^2 each, r^2 and the two subtractions 4u r^2;
//   so h is off by at most M / t_0 near any threshold (M <= t_0^2, sqrt being
//   within 2^-23 of its argument's root), and eps = 10 (M / t_0) + 2u (40 dc +
//   200) also bounds the roundings of h - dc + 0.5 and of the products.
// A row that is not certain has exactly one open sub-cell (eps < 1/2), which
// the reference's FP64 expressions decide.  Nodes closer to the centre than
// 0.75 along every axis (radii below 2.2 nodes only), and radii so large that
// eps would reach 1/4, compare each sub-cell with the FP32 margin instead.
//
// Bound by issue and the square roots (16 per clock and multiprocessor): 100
// rows of 8 instructions per node in 3-D.
template <class Sphere>
static __device__ int shell_count(int dim, const Sphere& im, int hx, int hy, int hz, float dxf,
                                  float dyf, float dzf) {
  const float u = 5.9604644775390625e-08f;  // 2^-24
  const float rSqf = im.rSqf;
  const float ax = fabsf(dxf), ay = fabsf(dyf), az = dim == 3 ? fabsf(dzf) : -1.0f;
  // c: largest |offset|; a, b the others (2-D: one row axis b only, a unused)
  float da, db, dc;
  int pc;
  if (az >= ax && az >= ay) {
    pc = 2; dc = dzf; da = dxf; db = dyf;
  } else if (ay >= ax) {
    pc = 1; dc = dyf; da = dzf; db = dxf;
  } else {
    pc = 0; dc = dxf; da = dzf; db = dyf;
  }
  const int pb = pc == 0 ? 1 : (pc == 1 ? 0 : 1), pa = 3 - pc - pb;
  const bool flip = dc < 0.0f;
  const float dca = fabsf(dc);
  const float Ea = fabsf(da) + 2.0f, Eb = fabsf(db) + 2.0f;
  const float M = 8.0f * u * ((dim == 3 ? Ea * Ea : 0.0f) + Eb * Eb + rSqf);
  const float t0 = dca - 0.45f;
  const float eps = 10.0f * (M / t0) + 2.0f * u * (40.0f * dca + 200.0f);
  const int na = dim == 3 ? 10 : 1;
  auto decide = [&](int a, int b, int k) {  // sub-cell (a, b, k-th along c from the centre side)
    const int kc = flip ? 9 - k : k;
    const int i0 = pa == 0 ? a : (pb == 0 ? b : kc);
    const int i1 = pa == 1 ? a : (pb == 1 ? b : kc);
    const int i2 = pa == 2 ? a : (pb == 2 ? b : kc);
    return sub_cell_inside(dim, im, hx, hy, hz, i0, i1, i2) ? 1 : 0;
  };
  if (!(dca >= 0.75f) || !(eps < 0.25f)) {
    // every sub-cell against the surface with the FP32 margin of a whole sum
    const float Ec = dca + 2.0f;
    const float M3 = 16.0f * u * ((dim == 3 ? Ea * Ea : 0.0f) + Eb * Eb + Ec * Ec + rSqf);
    const float lo = rSqf - M3, hi = rSqf + M3;
    int n = 0;
    for (int a = 0; a < na; ++a) {
      const float ta = da + sub_offset(a);
      const float sa = dim == 3 ? ta * ta : 0.0f;
      for (int b = 0; b < 10; ++b) {
        const float tb = db + sub_offset(b);
        const float sab = sa + tb * tb;
#pragma unroll 1
        for (int k = 0; k < 10; ++k) {
          const float t = dca + sub_offset(k);
          const float s = sab + t * t;
          if (s < lo)
            ++n;
          else if (s <= hi)
            n += decide(a, b, k);
        }
      }
    }
    return n;
  }
  constexpr float MAGIC = 12582912.0f;  // 1.5 * 2^23: adding it rounds to the nearest integer
  const float K = 0.5f - dca;
  const float open = 0.5f - eps;
  float sb[10];
#pragma unroll
  for (int b = 0; b < 10; ++b) {
    const float tb = db + sub_offset(b);
    sb[b] = tb * tb;
  }
  auto row = [&](float x, float s, float& n) {  // its count; returns the distance from it
    float h;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(h) : "f"(x - s));
    const float w = __saturatef(h + K);
    n = __fmaf_rn(w, 10.0f, MAGIC) - MAGIC;
    return fabsf(__fmaf_rn(w, 10.0f, -n));
  };
  float total = 0.0f;
#pragma unroll 1
  for (int a = 0; a < na; ++a) {
    const float ta = da + sub_offset(a);
    const float x = dim == 3 ? rSqf - ta * ta : rSqf;
    float cnt = 0.0f, far = 0.0f;
#pragma unroll
    for (int b = 0; b < 10; ++b) {
      float n;
      far = fmaxf(far, row(x, sb[b], n));
      cnt += n;
    }
    if (far >= open) {  // an open row in this slab (about one slab in 2000): its rows again
      cnt = 0.0f;
#pragma unroll 1
      for (int b = 0; b < 10; ++b) {
        const float tb = db + sub_offset(b);
        const float s = tb * tb;
        float n;
        const float e = row(x, s, n);
        if (e >= open) {
          float h;
          asm("sqrt.approx.f32 %0, %1;" : "=f"(h) : "f"(x - s));
          const float w = __saturatef(h + K);
          // v = k + 1/2 up to eps: sub-cells below k are inside, above k outside
          const int k = __float2int_rd(__fmul_rn(w, 10.0f));
          n = (float)(k + decide(a, b, k));
        }
        cnt += n;
      }
    }
    total += cnt;
  }
  return (int)total;
}

}  // namespace lbmpsm
