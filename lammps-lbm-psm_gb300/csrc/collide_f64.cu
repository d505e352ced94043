// collide_f64.cu -- FP64 "plain" path: fused macro / BGK-PSM collision /
// A-A streaming kernel and the Zou-He face kernel, keeping the reference's
// operand order so that results match the reference CPU code bit for bit.
// Compiled with -fmad=false (no contraction of a*b+c).
//
// Reference: LBMPSMBGKDynamics::compute_macro_values
// (src/LBM_PSM_BGK_dynamics.cpp:48-77), collisionAndStream
// (src/LBM_PSM_BGK_dynamics.h:40-114), feq / F_iq
// (src/LBM_PSM_dynamics.h:43-116), add_Fhyd (src/LBM_PSM_lattice.cpp:355-363),
// macroCollideStream (src/LBM_PSM_BGK_dynamics.cpp:81-109), ZouHeBC
// (src/LBM_PSM_zou_he_BC.cpp:25-398).
#include "fixed_f64.cuh"
#include "lbmpsm_internal.cuh"

namespace lbmpsm {

constexpr int F64_THREADS = 128;
// Blocks per multiprocessor: of the columns without a body force five (four 2%
// slower, six spill and gain 0.6% at most), with one four (five 1% slower).
constexpr int f64_blocks(bool force) { return force ? 4 : 5; }

// Opposite directions in pairs (q, o = opp(q)), q the one whose first non-zero
// component is +1: e_q = +1 on axis i1, s2 on axis i2 (axis pairs: s2 = 0, i2 = i1).
// g[a] is the index of component a of e_q in 0, +1, -1 (0, 1, 2).
struct PairDesc {
  int q, o, i1, i2, s2, g[3];
};
__constant__ PairDesc c_pairs19[9] = {
    {1, 2, 0, 0, 0, {1, 0, 0}},   {3, 4, 1, 1, 0, {0, 1, 0}},    {5, 6, 2, 2, 0, {0, 0, 1}},
    {7, 8, 0, 1, 1, {1, 1, 0}},   {9, 10, 0, 2, 1, {1, 0, 1}},   {11, 12, 1, 2, 1, {0, 1, 1}},
    {13, 14, 0, 1, -1, {1, 2, 0}}, {15, 16, 0, 2, -1, {1, 0, 2}}, {17, 18, 1, 2, -1, {0, 1, 2}}};
__constant__ PairDesc c_pairs9[4] = {{1, 3, 0, 0, 0, {1, 0, 0}},
                                     {2, 4, 1, 1, 0, {0, 1, 0}},
                                     {5, 7, 0, 1, 1, {1, 1, 0}},
                                     {8, 6, 0, 1, -1, {1, 2, 0}}};
template <class L>
__device__ __forceinline__ const PairDesc& pair_desc(int k) {
  return L::Q == 19 ? c_pairs19[k] : c_pairs9[k];
}

// x with its sign turned where neg (exact)
__device__ __forceinline__ double turned(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}

// a / b for three numerators: one correctly rounded reciprocal y, then per
// quotient two corrections with exact remainders (Markstein, IBM J. Res. Dev.
// 34 (1990): if y = RN(1/b) and q is faithful, RN(q + y RN(a - b q)) is the
// correctly rounded quotient; the first correction makes q faithful).  Out of
// the range where no intermediate under- or overflows (zero numerators but
// b > 0 excepted), plain divisions.
__device__ __forceinline__ bool is_zero(double a) {
  return ((__double2hiint(a) & 0x7fffffff) | __double2loint(a)) == 0;
}
__device__ __forceinline__ bool div_range(double a) {
  const int e = (__double2hiint(a) >> 20) & 0x7ff;
  return (e > 523 && e < 1523) || is_zero(a);
}
__device__ __forceinline__ double div_by(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  const double t = __fma_rn(__fma_rn(-b, q, a), y, q);
  return is_zero(a) ? a : t;
}
__device__ __noinline__ double div_plain(double a, double b) { return a / b; }
__device__ __forceinline__ void div3(const double (&a)[3], double b, double (&q)[3]) {
  const int e = __double2hiint(b) >> 20;  // sign and exponent: b within 2^+-100 and positive
  if (e > 923 && e < 1123 && div_range(a[0]) && div_range(a[1]) && div_range(a[2])) {
    const double y = __drcp_rn(b);
#pragma unroll
    for (int c = 0; c < 3; ++c) q[c] = div_by(a[c], b, y);
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) q[c] = div_plain(a[c], b);
  }
}

// The values of a block's nodes that the loop over direction pairs indexes:
// one column per thread, so no barrier and no bank conflict.  Kept in shared
// memory so that the loop stays rolled: unrolled over 19 directions with two
// slots the step is 60 KB of instructions, and its warps waited for
// instruction fetches half of the time.
template <class L, bool FORCE>
struct NodeCols {
  double f[L::Q][F64_THREADS];       // populations, replaced pair by pair
  double u[L::DIM][F64_THREADS];     // fluid velocity
  double us[2][L::DIM][F64_THREADS]; // slot velocities
  double F[2][L::DIM][F64_THREADS];  // slot forces
  double t[L::Q == 9 ? 2 : 1][L::Q == 9 ? 9 : 1][F64_THREADS];  // B*Omega_s of every direction (D2Q9)
  // (c - u_a)*F_a at 3a + (0: c = 0, 1: c = 1, 2: c = -1); of a force along one
  // axis only that axis's, times invCs2, at 0 to 2
  double g[FORCE ? 9 : 1][F64_THREADS];
};

// What the directions of one node share besides.
struct NodeF64 {
  double vv[3];  // v.v of the fluid and of the slots
  double rw[3];  // rho*w of the rest, axis and diagonal weights
  double B[2], oneMinusBtot;
  double uz;  // (D2Q9's columns hold no third component)
  int axis;   // of the body force if it has one non-zero component, else -1
};

// e.v of a pair's first direction, from a velocity's columns
__device__ __forceinline__ double pair_dot(const PairDesc& d, const double (*v)[F64_THREADS], int t) {
  const double x = v[d.i1][t];
  return d.s2 == 0 ? x : x + turned(v[d.i2][t], d.s2 < 0);
}

// The equilibria rw*(1 +- 3 e.v + 4.5 (e.v)^2 - 1.5 v.v) of a pair minus its
// populations: e.v, its multiple and its square are formed once, the opposite
// direction taking them with the sign turned (negation is exact, so both round
// as when formed alone; 0.5*invCs4 is exact).
__device__ __forceinline__ double2 pair_diff(double ev, const CollideParams& p, double half, double rw,
                                             double fp, double fm) {
  const double a = ev * p.invCs2, b = ev * ev * (0.5 * p.invCs4);
  return make_double2(rw * ((1.0 + a) + b - half) - fp, rw * ((1.0 - a) + b - half) - fm);
}

// The same on the integer units (fixed_f64.cuh), but for one product: the
// constants are 3 and 4.5 exactly.  One copy of the code, called by the fluid's
// and the slots' loops: inlined, warps of the different loops on one
// multiprocessor waited for instruction fetches (128 x 96 x 160 nodes with 230
// spheres: 920 us a step, called 845).
static_assert(1.0 / (1.0 / 3.0) == 3.0 && 1.0 / ((1.0 / 3.0) * (1.0 / 3.0)) == 9.0, "");
__device__ __noinline__ double2 pair_diff62(double ev, fx::u64 half, fx::u64 rw, fx::u64 fp,
                                            fx::u64 fm) {
  fx::u64 plus, minus;
  fx::factors(ev, ev * ev, half, plus, minus);
  return make_double2(fx::difference62(fx::product62(rw, plus), fp),
                      fx::difference62(fx::product62(rw, minus), fm));
}

// fi after collision (collisionAndStream, src/LBM_PSM_BGK_dynamics.h:40-114)
// with NS slots (0: plain BGK); d and ds: feq - fi of the fluid and of the slot
// velocities; t: B*Omega_s per slot.
template <int NS>
__device__ __forceinline__ double relaxed(double fi, double d, const double (&ds)[2],
                                          const NodeF64& nd, double omega, double omo,
                                          double (&t)[2]) {
  if (NS == 0) return fi + d * omega;
  const double od = omo * d;  // one_minus_omega*(fi - feq) is -od bit for bit
  double r = fi + nd.oneMinusBtot * d * omega;
#pragma unroll
  for (int n = 0; n < NS; ++n) {
    t[n] = nd.B[n] * (ds[n] - od);
    r = r + t[n];
  }
  return r;
}

// All directions of a node.  Guo forcing (src/LBM_PSM_dynamics.h:102-116):
// pref*(w*(((e - u).F)*invCs2 + (e.u)*invCs4*(e.F))).
template <class L, bool FORCE, int NS, bool FX>
__device__ __forceinline__ void collide_dirs(NodeCols<L, FORCE>& s, int t, const NodeF64& nd,
                                             const CollideParams& p, const BoxParams& bp,
                                             bool has_force) {
  const double pref = bp.guo_pref, omega = bp.omega, omo = bp.one_minus_omega;
  const double invCs2 = p.invCs2, invCs4 = p.invCs4;
  double half[1 + NS];  // 0.5*v.v*invCs2 of the fluid and of the slots
  fx::u64 half62[1 + NS], rw62[3];
#pragma unroll
  for (int n = 0; n <= NS; ++n) {
    if (FX)
      half62[n] = fx::times62<3, 1>(nd.vv[n]);
    else
      half[n] = 0.5 * nd.vv[n] * invCs2;
  }
  if (FX) {
#pragma unroll
    for (int c = 0; c < 3; ++c) rw62[c] = fx::to64(nd.rw[c]);
  }
  // A force along one axis (the usual one): the other axes' terms are zeros, and
  // directions without a component along the axis share one value per weight.
  // The sums round as with the zeros added.  (Nodes of a forced fluid spent more
  // FP64 operations on the force than on the rest: 24 steps forward and back of
  // 56^3 took 10.7 ms, with this 9.3.)
  const bool single = FORCE && FX && nd.axis >= 0;
  double still[2] = {0.0, 0.0};  // those values, axis and diagonal directions
  if (FORCE) {
    if (single) {
      const double Fa = bp.F[nd.axis], ua = s.u[nd.axis][t];
      const double g0 = (0.0 - ua) * Fa * invCs2;
      s.g[0][t] = g0;
      s.g[1][t] = (1.0 - ua) * Fa * invCs2;
      s.g[2][t] = (-1.0 - ua) * Fa * invCs2;
      still[0] = pref * (L::w(1) * g0);
      still[1] = pref * (L::w(L::Q - 1) * g0);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double Fc = has_force ? bp.F[c] : 0.0;
        const double uc = c < L::DIM ? s.u[c < L::DIM ? c : 0][t] : nd.uz;
        s.g[3 * c][t] = (0.0 - uc) * Fc;
        s.g[3 * c + 1][t] = (1.0 - uc) * Fc;
        s.g[3 * c + 2][t] = (-1.0 - uc) * Fc;
      }
    }
  }
  auto guo = [&](int g0, int g1, int g2, double w, double last) {
    if (single) return pref * (w * s.g[0][t]);  // (the rest direction)
    const double a = s.g[g0][t] + s.g[3 + g1][t] + s.g[6 + g2][t];
    return pref * (w * (a * invCs2 + last));
  };
  {  // the rest population
    const double fi = s.f[0][t];
    double d[1 + NS], ds[2] = {0.0, 0.0}, bo[2];
#pragma unroll
    for (int n = 0; n <= NS; ++n)
      d[n] = FX ? fx::difference62(fx::product62(rw62[0], fx::one_minus(half62[n])), fx::to62(fi))
                : nd.rw[0] * (1.0 - half[n]) - fi;
#pragma unroll
    for (int n = 0; n < NS; ++n) ds[n] = d[1 + n];
    double r = relaxed<NS>(fi, d[0], ds, nd, omega, omo, bo);
    if (FORCE) r = r + guo(0, 0, 0, L::w(0), 0.0);
    s.f[0][t] = r;
  }
#pragma unroll 1
  for (int k = 0; k < (L::Q - 1) / 2; ++k) {
    const PairDesc& d = pair_desc<L>(k);
    const double eu = pair_dot(d, s.u, t);
    const double fi = s.f[d.q][t], fo = s.f[d.o][t];
    double2 dd[1 + NS];  // feq - f of both directions, the fluid's and the slots' velocities
    double sp[2] = {0.0, 0.0}, sm[2] = {0.0, 0.0}, tp[2], tm[2];
    if (FX) {
      const fx::u64 fi62 = fx::to62(fi), fo62 = fx::to62(fo), rw = d.s2 == 0 ? rw62[1] : rw62[2];
#pragma unroll
      for (int n = 0; n <= NS; ++n)  // feq(iq, rho, uSolid) (src/LBM_PSM_dynamics.h:72-85)
        dd[n] = pair_diff62(n == 0 ? eu : pair_dot(d, s.us[n > 0 ? n - 1 : 0], t), half62[n], rw, fi62, fo62);
    } else {
      const double rw = d.s2 == 0 ? nd.rw[1] : nd.rw[2];
#pragma unroll
      for (int n = 0; n <= NS; ++n)
        dd[n] = pair_diff(n == 0 ? eu : pair_dot(d, s.us[n > 0 ? n - 1 : 0], t), p, half[n], rw, fi, fo);
    }
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      sp[n] = dd[1 + n].x;
      sm[n] = dd[1 + n].y;
    }
    double fp = relaxed<NS>(fi, dd[0].x, sp, nd, omega, omo, tp);
    double fm = relaxed<NS>(fo, dd[0].y, sm, nd, omega, omo, tm);
    if (FORCE) {
      const int c = single ? d.g[nd.axis] : -1;
      if (c == 0) {
        const double gs = d.s2 == 0 ? still[0] : still[1];
        fp = fp + gs;
        fm = fm + gs;
      } else {
        const double w = d.s2 == 0 ? L::w(1) : L::w(L::Q - 1);
        const double eF = has_force ? bp.eF[(L::Q == 9 ? 9 : 0) + k] : 0.0;
        const double last = (eu * invCs4) * eF;  // both signs turn: the same for the opposite
        if (single) {
          fp = fp + pref * (w * (s.g[c][t] + last));
          fm = fm + pref * (w * (s.g[3 - c][t] + last));
        } else {
          fp = fp + guo(d.g[0], d.g[1], d.g[2], w, last);
          fm = fm + guo(d.g[0] ? 3 - d.g[0] : 0, d.g[1] ? 3 - d.g[1] : 0, d.g[2] ? 3 - d.g[2] : 0, w, last);
        }
      }
    }
    s.f[d.q][t] = fp;
    s.f[d.o][t] = fm;
    // node force on the particles (add_Fhyd): F += -B*Omega_s*e, in direction order
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      if (L::Q == 19) {  // (the pairs are in that order)
        s.F[n][d.i1][t] = (s.F[n][d.i1][t] - tp[n]) + tm[n];
        if (d.s2 != 0)
          s.F[n][d.i2][t] = (s.F[n][d.i2][t] - turned(tp[n], d.s2 < 0)) + turned(tm[n], d.s2 < 0);
      } else {
        s.t[n][d.q][t] = tp[n];
        s.t[n][d.o][t] = tm[n];
      }
    }
  }
  if (L::Q == 9) {
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      double F[2] = {0.0, 0.0};
#pragma unroll
      for (int q = 1; q < L::Q; ++q) {
        const double b = s.t[n][q][t];
        if (L::ex(q)) F[0] = L::ex(q) > 0 ? F[0] - b : F[0] + b;
        if (L::ey(q)) F[1] = L::ey(q) > 0 ? F[1] - b : F[1] + b;
      }
      s.F[n][0][t] = F[0];
      s.F[n][1][t] = F[1];
    }
  }
}

// One node of the FP64 collide + A-A stream step.
//
// Bound by the FP64 pipe (1.68 operations per clock and multiprocessor) and,
// with the work split, as much by the integer units (both 50 to 65% busy; DRAM
// 11%), so: sums and equilibria near rest run on the integer units
// (fixed_f64.cuh), what directions share is formed once (pair_diff), three
// quotients share one reciprocal (div3), the body force is
// a template argument, and a warp takes the plain loop when none of its nodes
// is a PSM node, the one-slot loop when none holds two particles -- an unused
// slot has B = 0 and adds zeros, and a node without any has 1 - B = 1, so the
// longer loops leave its populations bit for bit as the shorter ones.
template <class L, bool ODD, bool FORCE>
__device__ __forceinline__ void collide_f64_node(NodeCols<L, FORCE>& s, const CollideParams& p,
                                                 int sx, int sy, int sz) {
  constexpr int Q = L::Q;
  const int t = threadIdx.x;
  const Geom& g = p.g;
  const long long n = node_index(g, sx, sy, sz);
  const Nbr nb = make_nbr(g, sx, sy, sz);
  const BoxParams& bp = p.box[box_of_z(g, sz)];
  double* F = static_cast<double*>(p.f);
  // in place unless a separate source is given (recomputation of stored states)
  const double* Fin = p.fsrc ? static_cast<const double*>(p.fsrc) : F;
  const long long Np = g.Np;
  const unsigned act = __activemask();

  const uint8_t flag = p.tab.flag[n];
  double rho, j[3];
  bool near;
  {
    double f[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
      // incoming population q comes from the node at -e_q
      const bool ok = nbr_ok(nb, -cx, -cy, -cz);
      if (!ODD) {
        f[q] = ok ? Fin[q * Np + n] : L::w(q);
      } else {
        const int o = nbr_off(nb, -cx, -cy, -cz);
        f[q] = ok ? Fin[L::opp(q) * Np + n + o] : L::w(q);
      }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) s.f[q][t] = f[q];
    // macro values (src/LBM_PSM_BGK_dynamics.cpp:48-77): on the integer units
    // where every node of the warp is near rest, else in FP64
    near = fx::macro_sums<L>(f, rho, j);
    if (!__all_sync(act, near)) {
      near = false;
      rho = f[0];
#pragma unroll
      for (int q = 1; q < Q; ++q) rho = rho + f[q];
      // (each sum's first term is a +e direction, taken as it is instead of 0 + f)
      j[0] = f[1];
      j[1] = f[Q == 19 ? 3 : 2];
      j[2] = Q == 19 ? f[5] : 0.0;
#pragma unroll
      for (int q = 2; q < Q; ++q) {
        const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
        if (cx) j[0] = cx > 0 ? j[0] + f[q] : j[0] - f[q];
        if (cy && q > (Q == 19 ? 3 : 2)) j[1] = cy > 0 ? j[1] + f[q] : j[1] - f[q];
        if (cz && q > 5) j[2] = cz > 0 ? j[2] + f[q] : j[2] - f[q];
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)  // (|F|^2 of a non-zero F may underflow to "no force")
    if (FORCE || !is_zero(bp.F[c])) j[c] = j[c] + bp.F[c] * 0.5;
  double u[3];
  div3(j, rho, u);
  if (p.store_macro) {
    p.rho_out[n] = rho;
#pragma unroll
    for (int c = 0; c < 3; ++c) p.u_out[3 * n + c] = u[c];
  }
  NodeF64 nd;
  nd.vv[0] = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    near = near && fx::slow(u[c]);
    if (c < L::DIM) s.u[c][t] = u[c];
    nd.rw[c] = rho * L::w(c == 0 ? 0 : (c == 1 ? 1 : Q - 1));
  }
  const bool has_force = FORCE && bp.has_force != 0;  // (a box of an ensemble may have none)
  nd.uz = u[2];
  nd.axis = -1;
  if (has_force) {
    // (an out-of-plane force has its part in D2Q9 too, through u_z)
    const bool z0 = is_zero(bp.F[0]), z1 = is_zero(bp.F[1]), z2 = is_zero(bp.F[2]);
    if (z1 && z2) nd.axis = 0;
    if (z0 && z2) nd.axis = 1;
    if (L::DIM == 3 && z0 && z1) nd.axis = 2;
  }

  const bool psm = flag != 0;
  if (!__any_sync(act, psm)) {
    if (__all_sync(act, near))
      collide_dirs<L, FORCE, 0, true>(s, t, nd, p, bp, has_force);
    else
      collide_dirs<L, FORCE, 0, false>(s, t, nd, p, bp, has_force);
  } else {
    int2 id = make_int2(0, 0);
    double2 e = make_double2(0.0, 0.0);
    if (psm) {
      id = p.tab.ids[n];
      e = p.tab.eps[n];
    }
    const bool has[2] = {id.x > 0, id.y > 0};
    double B1 = has[0] ? e.x : 0.0;
    double B2 = has[1] ? e.y : 0.0;
    if (p.weighting == 1) {  // Noble-Torczynski weighting (opt-in)
      const double tm = bp.tau - 0.5;
      if (has[0]) B1 = B1 * tm / ((1.0 - B1) + tm);
      if (has[1]) B2 = B2 * tm / ((1.0 - B2) + tm);
    }
    double Btot = B1 + B2;
    if (Btot > 1.0) {
      B1 = B1 / Btot;
      B2 = B2 / Btot;
      Btot = 1.0;
    }
    nd.B[0] = B1;
    nd.B[1] = B2;
    nd.oneMinusBtot = 1.0 - Btot;
    const double* us = p.tab.us + 6 * n;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      double v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[c] = has[k] ? us[3 * k + c] : 0.0;
        if (c < L::DIM) {
          s.us[k][c][t] = v[c];
          s.F[k][c][t] = 0.0;
        }
        near = near && fx::slow(v[c]);
      }
      nd.vv[1 + k] = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    }
    const bool one = !__any_sync(act, (flag & 2) != 0);
    if (__all_sync(act, near)) {
      if (one)
        collide_dirs<L, FORCE, 1, true>(s, t, nd, p, bp, has_force);
      else
        collide_dirs<L, FORCE, 2, true>(s, t, nd, p, bp, has_force);
    } else {
      if (one)
        collide_dirs<L, FORCE, 1, false>(s, t, nd, p, bp, has_force);
      else
        collide_dirs<L, FORCE, 2, false>(s, t, nd, p, bp, has_force);
    }
    if (psm) {
      double* nf = static_cast<double*>(p.tab.nodeF) + 6 * n;
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) nf[3 * k + c] = c < L::DIM ? s.F[k][c < L::DIM ? c : 0][t] : 0.0;
    }
  }

#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
    if (!ODD) {
      F[L::opp(q) * Np + n] = s.f[q][t];
    } else {
      if (nbr_ok(nb, cx, cy, cz)) F[q * Np + n + nbr_off(nb, cx, cy, cz)] = s.f[q][t];
    }
  }
}

// Deals the nodes of block b to its threads (every thread of the block calls):
// those of two particles first, those of one, then the fluid.  A node of a
// sphere costs more than twice a fluid one and a warp takes the loop of its
// dearest node; spheres cut most rows, so that with nodes in order 42% of the
// warps took the PSM loop where 17% of the nodes needed it, dealt out 23%
// (128 x 96 x 160 nodes, 230 spheres: 1190 -> 1000 us a step).  The accesses stay
// within the block's cache lines, and no other node reads or writes a node's
// slots.
__device__ __forceinline__ bool dealt_node(const CollideParams& p, unsigned b, int& sx, int& sy,
                                           int& sz) {
  constexpr int W = F64_THREADS / 32;
  __shared__ unsigned char order[F64_THREADS];
  __shared__ int count[3][W];
  const int t = threadIdx.x, w = t >> 5;
  const bool in = node_of_block<F64_THREADS>(p.g, b, sx, sy, sz);
  const unsigned flag = in ? p.tab.flag[node_index(p.g, sx, sy, sz)] : 0u;
  if (!__syncthreads_or(flag != 0u)) return in;
  const int cls = !in ? 3 : ((flag & 2u) ? 0 : (flag ? 1 : 2));
  int before = 0;  // nodes of the class in the warp's lower lanes
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const unsigned m = __ballot_sync(0xffffffffu, cls == c);
    if ((t & 31) == 0) count[c][w] = __popc(m);
    if (cls == c) before = __popc(m & ((1u << (t & 31)) - 1u));
  }
  __syncthreads();
  int total = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int m = count[c][k];
      if (c < cls || (c == cls && k < w)) before += m;
      total += m;
    }
  if (in) order[before] = (unsigned char)t;
  __syncthreads();
  if (t >= total) return false;
  return node_of_block<F64_THREADS>(p.g, b, sx, sy, sz, order[t]);
}

template <class L, bool ODD, bool FORCE>
__global__ void __launch_bounds__(F64_THREADS, f64_blocks(FORCE)) collide_f64_kernel(CollideParams p) {
  __shared__ NodeCols<L, FORCE> s;
  int sx, sy, sz;
  if (!dealt_node(p, blockIdx.x, sx, sy, sz)) return;
  collide_f64_node<L, ODD, FORCE>(s, p, sx, sy, sz);
}

// The members of a group in one launch: member m owns blocks
// [first[m], first[m+1]), laid out as its own kernel's; every node runs the
// same code as above, so the results are the members'.
template <class L, bool ODD, bool FORCE>
__global__ void __launch_bounds__(F64_THREADS, f64_blocks(FORCE)) collide_f64_multi_kernel(MultiCollide mc) {
  __shared__ NodeCols<L, FORCE> s;
  const int b = blockIdx.x;
  int m = 0;
  while (m + 1 < mc.nm && b >= mc.first[m + 1]) ++m;
  const CollideParams& p = mc.m[m].p;
  int sx, sy, sz;
  if (!dealt_node(p, (unsigned)(b - mc.first[m]), sx, sy, sz)) return;
  collide_f64_node<L, ODD, FORCE>(s, p, sx, sy, sz);
}

long long collide_f64_blocks(const Geom& g) {
  return ((long long)g.S[0] * g.S[1] * g.S[2] + F64_THREADS - 1) / F64_THREADS;
}

cudaError_t launch_collide_f64_multi(const MultiCollide& mc, int odd, cudaStream_t st) {
  const unsigned grid = (unsigned)mc.first[mc.nm];
  if (grid == 0) return cudaSuccess;
  if (mc.any_force) {
    if (odd)
      collide_f64_multi_kernel<D3Q19, true, true><<<grid, F64_THREADS, 0, st>>>(mc);
    else
      collide_f64_multi_kernel<D3Q19, false, true><<<grid, F64_THREADS, 0, st>>>(mc);
  } else {
    if (odd)
      collide_f64_multi_kernel<D3Q19, true, false><<<grid, F64_THREADS, 0, st>>>(mc);
    else
      collide_f64_multi_kernel<D3Q19, false, false><<<grid, F64_THREADS, 0, st>>>(mc);
  }
  return cudaGetLastError();
}

template <class L>
static cudaError_t launch_collide_impl(const CollideParams& p, int odd, cudaStream_t st) {
  const unsigned grid = (unsigned)collide_f64_blocks(p.g);
  if (p.has_force) {
    if (odd)
      collide_f64_kernel<L, true, true><<<grid, F64_THREADS, 0, st>>>(p);
    else
      collide_f64_kernel<L, false, true><<<grid, F64_THREADS, 0, st>>>(p);
  } else {
    if (odd)
      collide_f64_kernel<L, true, false><<<grid, F64_THREADS, 0, st>>>(p);
    else
      collide_f64_kernel<L, false, false><<<grid, F64_THREADS, 0, st>>>(p);
  }
  return cudaGetLastError();
}

cudaError_t launch_collide_f64(const CollideParams& p, int odd, cudaStream_t st) {
  return p.g.dim == 2 ? launch_collide_impl<D2Q9>(p, odd, st)
                      : launch_collide_impl<D3Q19>(p, odd, st);
}

// ------------------------------------------------------------------ Zou-He
// Exact restatements of the ZouHeBC members on one node's populations f[].
__device__ void zh_apply_f64(int kind, double* f, double p0) {
  const double o3 = 1.0 / 3.0, o6 = 1.0 / 6.0, t3 = 2.0 / 3.0;
  switch (kind) {
    case FACE_VEL2_XN: {  // :25-40
      const double ux = p0;
      double rho = 1.0 / (1.0 - ux) * (f[0] + f[2] + f[4] + 2.0 * (f[3] + f[6] + f[7]));
      f[5] = f[7] + 0.5 * (f[4] - f[2]) + rho * ux * o6;
      f[8] = f[6] + 0.5 * (f[2] - f[4]) + rho * ux * o6;
      f[1] = f[3] + t3 * rho * ux;
    } break;
    case FACE_VEL2_XP: {  // :43-58
      const double ux = p0;
      double rho = 1.0 / (1.0 - ux) * (f[0] + f[2] + f[4] + 2.0 * (f[1] + f[5] + f[8]));
      f[7] = f[5] + 0.5 * (f[2] - f[4]) - rho * ux * o6;
      f[6] = f[8] + 0.5 * (f[4] - f[2]) - rho * ux * o6;
      f[3] = f[1] - t3 * rho * ux;
    } break;
    case FACE_DENS2_XP: {  // :61-76
      const double rb = p0;
      double ux = -1.0 + 1.0 / rb * (f[0] + f[2] + f[4] + 2.0 * (f[1] + f[5] + f[8]));
      f[6] = f[8] + 0.5 * (f[4] - f[2]) - rb * ux * o6;
      f[7] = f[5] + 0.5 * (f[2] - f[4]) - rb * ux * o6;
      f[3] = f[1] - t3 * rb * ux;
    } break;
    case FACE_VEL2_YN: {  // :79-94
      const double ux = p0;
      double rho = f[0] + f[3] + f[1] + 2.0 * (f[8] + f[4] + f[7]);
      f[6] = f[8] + 0.5 * (f[1] - f[3]) - rho * ux * 0.5;
      f[5] = f[7] + 0.5 * (f[3] - f[1]) + rho * ux * 0.5;
      f[2] = f[4];
    } break;
    case FACE_VEL2_YP: {  // :97-112
      const double ux = p0;
      double rho = f[0] + f[3] + f[1] + 2.0 * (f[6] + f[2] + f[5]);
      f[7] = f[5] + 0.5 * (f[1] - f[3]) - rho * ux * 0.5;
      f[8] = f[6] + 0.5 * (f[3] - f[1]) + rho * ux * 0.5;
      f[4] = f[2];
    } break;
    case FACE_VEL3_XN: {  // :153-185 (uy = uz = 0 at every call site)
      const double ux = p0, uy = 0.0, uz = 0.0;
      double rho = 1.0 / (1.0 - ux) *
                   (f[0] + f[3] + f[4] + f[5] + f[6] + f[11] + f[17] + f[18] + f[12] +
                    2.0 * (f[2] + f[14] + f[8] + f[16] + f[10]));
      double Nyx = 0.5 * (f[3] + f[11] + f[17] - (f[4] + f[18] + f[12])) - o3 * rho * uy;
      double Nzx = 0.5 * (f[5] + f[18] + f[11] - (f[6] + f[17] + f[12])) - o3 * rho * uz;
      f[1] = f[2] + o3 * rho * ux;
      f[13] = f[14] + rho * o6 * (ux - uy) + Nyx;
      f[7] = f[8] + rho * o6 * (ux + uy) - Nyx;
      f[9] = f[10] + rho * o6 * (ux + uz) - Nzx;
      f[15] = f[16] + rho * o6 * (ux - uz) + Nzx;
    } break;
    case FACE_VEL3_XP: {  // :189-221
      const double ux = p0, uy = 0.0, uz = 0.0;
      double rho = 1.0 / (1.0 + ux) *
                   (f[0] + f[3] + f[4] + f[5] + f[6] + f[11] + f[17] + f[18] + f[12] +
                    2.0 * (f[1] + f[7] + f[13] + f[9] + f[15]));
      double Nyx = 0.5 * (f[3] + f[11] + f[17] - (f[4] + f[18] + f[12])) - o3 * rho * uy;
      double Nzx = 0.5 * (f[5] + f[18] + f[11] - (f[6] + f[17] + f[12])) - o3 * rho * uz;
      f[2] = f[1] - o3 * rho * ux;
      f[14] = f[13] + rho * o6 * (-ux + uy) - Nyx;
      f[8] = f[7] + rho * o6 * (-ux - uy) + Nyx;
      f[10] = f[9] + rho * o6 * (-ux - uz) + Nzx;
      f[16] = f[15] + rho * o6 * (-ux + uz) - Nzx;
    } break;
    case FACE_DENS3_XP: {  // :225-257
      const double rb = p0, uy = 0.0, uz = 0.0;
      double ux = -1.0 + 1.0 / rb *
                             (f[0] + f[3] + f[4] + f[5] + f[6] + f[11] + f[17] + f[18] + f[12] +
                              2.0 * (f[1] + f[7] + f[13] + f[9] + f[15]));
      double Nyx = 0.5 * (f[3] + f[11] + f[17] - (f[4] + f[18] + f[12])) - o3 * rb * uy;
      double Nzx = 0.5 * (f[5] + f[18] + f[11] - (f[6] + f[17] + f[12])) - o3 * rb * uz;
      f[2] = f[1] - o3 * rb * ux;
      f[14] = f[13] + rb * o6 * (-ux + uy) - Nyx;
      f[8] = f[7] + rb * o6 * (-ux - uy) + Nyx;
      f[10] = f[9] + rb * o6 * (-ux - uz) + Nzx;
      f[16] = f[15] + rb * o6 * (-ux + uz) - Nzx;
    } break;
    case FACE_VEL3_YN: {  // :261-293
      const double ux = p0, uy = 0.0, uz = 0.0;
      double rho = 1.0 / (1.0 - uy) *
                   (f[0] + f[1] + f[2] + f[5] + f[6] + f[9] + f[15] + f[16] + f[10] +
                    2.0 * (f[4] + f[13] + f[8] + f[18] + f[12]));
      double Nxy = 0.5 * (f[1] + f[9] + f[15] - (f[2] + f[16] + f[10])) - o3 * rho * ux;
      double Nzy = 0.5 * (f[5] + f[9] + f[16] - (f[6] + f[15] + f[10])) - o3 * rho * uz;
      f[3] = f[4] + o3 * rho * uy;
      f[7] = f[8] + rho * o6 * (uy + ux) - Nxy;
      f[14] = f[13] + rho * o6 * (uy - ux) + Nxy;
      f[11] = f[12] + rho * o6 * (uy + uz) - Nzy;
      f[17] = f[18] + rho * o6 * (uy - uz) + Nzy;
    } break;
    case FACE_VEL3_YP: {  // :296-328
      const double ux = p0, uy = 0.0, uz = 0.0;
      double rho = 1.0 / (1.0 + uy) *
                   (f[0] + f[1] + f[2] + f[5] + f[6] + f[9] + f[15] + f[16] + f[10] +
                    2.0 * (f[3] + f[7] + f[14] + f[11] + f[17]));
      double Nxy = 0.5 * (f[1] + f[9] + f[15] - (f[2] + f[16] + f[10])) - o3 * rho * ux;
      double Nzy = 0.5 * (f[5] + f[9] + f[16] - (f[6] + f[15] + f[10])) - o3 * rho * uz;
      f[4] = f[3] - o3 * rho * uy;
      f[8] = f[7] + rho * o6 * (-uy - ux) + Nxy;
      f[13] = f[14] + rho * o6 * (-uy + ux) - Nxy;
      f[12] = f[11] + rho * o6 * (-uy - uz) + Nzy;
      f[18] = f[17] + rho * o6 * (-uy + uz) - Nzy;
    } break;
    case FACE_VEL3_ZN: {  // :331-363
      const double ux = p0, uy = 0.0, uz = 0.0;
      double rho = 1.0 / (1.0 - uz) *
                   (f[0] + f[1] + f[2] + f[3] + f[4] + f[7] + f[13] + f[14] + f[8] +
                    2.0 * (f[6] + f[15] + f[10] + f[17] + f[12]));
      double Nxz = 0.5 * (f[1] + f[7] + f[13] - (f[2] + f[14] + f[8])) - o3 * rho * ux;
      double Nyz = 0.5 * (f[3] + f[7] + f[14] - (f[4] + f[13] + f[8])) - o3 * rho * uy;
      f[5] = f[6] + o3 * rho * uz;
      f[9] = f[10] + rho * o6 * (uz + ux) - Nxz;
      f[16] = f[15] + rho * o6 * (uz - ux) + Nxz;
      f[11] = f[12] + rho * o6 * (uz + uy) - Nyz;
      f[18] = f[17] + rho * o6 * (uz - uy) + Nyz;
    } break;
    case FACE_VEL3_ZP: {  // :366-398
      const double ux = p0, uy = 0.0, uz = 0.0;
      double rho = 1.0 / (1.0 + uz) *
                   (f[0] + f[1] + f[2] + f[3] + f[4] + f[7] + f[14] + f[8] + f[13] +
                    2.0 * (f[5] + f[9] + f[16] + f[11] + f[18]));
      double Nxz = 0.5 * (f[1] + f[7] + f[13] - (f[2] + f[14] + f[8])) - o3 * rho * ux;
      double Nyz = 0.5 * (f[3] + f[7] + f[14] - (f[4] + f[13] + f[8])) - o3 * rho * uy;
      f[6] = f[5] - o3 * rho * uz;
      f[15] = f[16] + rho * o6 * (-uz + ux) - Nxz;
      f[10] = f[9] + rho * o6 * (-uz - ux) + Nxz;
      f[17] = f[18] + rho * o6 * (-uz + uy) - Nyz;
      f[12] = f[11] + rho * o6 * (-uz - uy) + Nyz;
    } break;
    default:
      break;
  }
}

__device__ __forceinline__ bool face_contains(const Face& fc, int sx, int sy, int sz) {
  return sx >= fc.lo[0] && sx <= fc.hi[0] && sy >= fc.lo[1] && sy <= fc.hi[1] &&
         sz >= fc.lo[2] && sz <= fc.hi[2];
}

// Location of the post-stream population q of node n: after an even step it
// sits in the upstream node's opposite slot, after an odd step in the node's
// own slot.  Returns -1 when the upstream node does not exist (constant).
template <class L>
__device__ __forceinline__ long long post_stream_loc(const Geom& g, const Nbr& nb, long long n,
                                                     int q, int after_odd) {
  const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
  if (!nbr_ok(nb, -cx, -cy, -cz)) return -1;
  if (after_odd) return (long long)q * g.Np + n;
  return (long long)L::opp(q) * g.Np + n + nbr_off(nb, -cx, -cy, -cz);
}

// One thread per (face, node of the face); the node is processed by the
// first face of the list that contains it, which then applies every face
// containing the node in list order (the reference applies whole faces one
// after another, and each face call touches only the node's own populations).
template <class L>
__global__ void bc_f64_kernel(BCParams p) {
  constexpr int Q = L::Q;
  const int fi = blockIdx.y;
  const Face& fc = p.face[fi];
  const int na = fc.hi[0] - fc.lo[0] + 1, nb_ = fc.hi[1] - fc.lo[1] + 1,
            nc = fc.hi[2] - fc.lo[2] + 1;
  const long long total = (long long)na * nb_ * nc;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int sx = fc.lo[0] + (int)(t % na);
  const int sy = fc.lo[1] + (int)((t / na) % nb_);
  const int sz = fc.lo[2] + (int)(t / ((long long)na * nb_));
  for (int k = 0; k < fi; ++k)
    if (face_contains(p.face[k], sx, sy, sz)) return;
  const Geom& g = p.g;
  const Nbr nb = make_nbr(g, sx, sy, sz);
  const long long n = node_index(g, sx, sy, sz);
  double* F = static_cast<double*>(p.f);
  double f[Q];
  long long loc[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    loc[q] = post_stream_loc<L>(g, nb, n, q, p.after_odd);
    f[q] = loc[q] >= 0 ? F[loc[q]] : L::w(q);
  }
  for (int k = fi; k < p.nfaces; ++k)
    if (face_contains(p.face[k], sx, sy, sz)) zh_apply_f64(p.face[k].kind, f, p.face[k].p0);
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (loc[q] >= 0) F[loc[q]] = f[q];
}

cudaError_t launch_bc_f64(const BCParams& p, cudaStream_t st) {
  if (p.nfaces == 0) return cudaSuccess;
  long long maxn = 0;
  for (int k = 0; k < p.nfaces; ++k) {
    const Face& fc = p.face[k];
    long long c = (long long)(fc.hi[0] - fc.lo[0] + 1) * (fc.hi[1] - fc.lo[1] + 1) *
                  (fc.hi[2] - fc.lo[2] + 1);
    if (c > maxn) maxn = c;
  }
  if (maxn <= 0) return cudaSuccess;
  dim3 block(128);
  dim3 grid((unsigned)((maxn + 127) / 128), (unsigned)p.nfaces);
  if (p.g.dim == 2)
    bc_f64_kernel<D2Q9><<<grid, block, 0, st>>>(p);
  else
    bc_f64_kernel<D3Q19><<<grid, block, 0, st>>>(p);
  return cudaGetLastError();
}

}  // namespace lbmpsm
