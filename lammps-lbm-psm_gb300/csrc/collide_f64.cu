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
#include "lbmpsm_internal.cuh"

namespace lbmpsm {

// signed sum of the non-zero components of e (each in {-1,0,1}) times v, in
// axis order; equal to the reference's ex*vx + ey*vy + ez*vz for these e.
template <int cx, int cy, int cz>
__device__ __forceinline__ double edot(double vx, double vy, double vz) {
  double s = 0.0;
  bool first = true;
  if (cx != 0) {
    s = cx > 0 ? vx : -vx;
    first = false;
  }
  if (cy != 0) {
    if (first) {
      s = cy > 0 ? vy : -vy;
      first = false;
    } else {
      s = cy > 0 ? s + vy : s - vy;
    }
  }
  if (cz != 0) {
    if (first) {
      s = cz > 0 ? vz : -vz;
      first = false;
    } else {
      s = cz > 0 ? s + vz : s - vz;
    }
  }
  return s;
}

// The lattice's directions as opposite pairs (q, opp(q)), q the lower index.
template <class L>
struct Pairs {
  static constexpr int N = (L::Q - 1) / 2;
  __host__ __device__ static constexpr int q(int k) {
    return L::Q == 19 ? 2 * k + 1 : (k < 2 ? k + 1 : k + 3);
  }
};

// a / b for three numerators: one correctly rounded reciprocal y, then per
// quotient two corrections with exact remainders (Markstein, IBM J. Res. Dev.
// 34 (1990): if y = RN(1/b) and q is faithful, RN(q + y RN(a - b q)) is the
// correctly rounded quotient; the first correction makes q faithful).  Out of
// the range where no intermediate under- or overflows (zero numerators but
// b > 0 excepted), plain divisions.
__device__ __forceinline__ bool div_range(double a) {
  const int e = (__double2hiint(a) >> 20) & 0x7ff;
  return (e > 523 && e < 1523) || a == 0.0;
}
__device__ __forceinline__ double div_by(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  const double t = __fma_rn(__fma_rn(-b, q, a), y, q);
  return a == 0.0 ? a : t;
}
__device__ __forceinline__ void div3(double a0, double a1, double a2, double b, double& q0,
                                     double& q1, double& q2) {
  const int e = __double2hiint(b) >> 20;  // sign and exponent: b within 2^+-100 and positive
  if (e > 923 && e < 1123 && div_range(a0) && div_range(a1) && div_range(a2)) {
    const double y = __drcp_rn(b);
    q0 = div_by(a0, b, y);
    q1 = div_by(a1, b, y);
    q2 = div_by(a2, b, y);
  } else {
    q0 = a0 / b;
    q1 = a1 / b;
    q2 = a2 / b;
  }
}

// One slot of a PSM node.
struct Slot {
  double B, us[3], half;  // half = 0.5*|us|^2*invCs2
  double F[3];            // add_Fhyd: F += -B*Omega_s*e
};

// What the directions of one node share.  gF[a][c] = (c - u_a)*F_a for c = 0, 1
// and, at index 2, -1: the products of the Guo term.
struct NodeF64 {
  double u[3], usq_half, rw[3];  // rw: rho*w of the rest, axis and diagonal weights
  double gF[3][3], F[3];
  double oneMinusBtot;
};

template <class L>
__device__ __forceinline__ constexpr int weight_class(int q) {
  return q == 0 ? 0 : (L::ex(q) * L::ex(q) + L::ey(q) * L::ey(q) + L::ez(q) * L::ez(q) == 1 ? 1 : 2);
}

// Guo forcing of direction q (src/LBM_PSM_dynamics.h:102-116), scaled by
// (1 - omega/2); g4 = (e.u)*invCs4
template <class L, int q>
__device__ __forceinline__ double guo_q(const NodeF64& nd, double g4, double invCs2, double pref) {
  constexpr int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
  const double a = nd.gF[0][cx < 0 ? 2 : cx] + nd.gF[1][cy < 0 ? 2 : cy] + nd.gF[2][cz < 0 ? 2 : cz];
  const double w = L::w(q);
  if (q == 0) return pref * (w * (a * invCs2 + 0.0));
  const double eF = edot<cx, cy, cz>(nd.F[0], nd.F[1], nd.F[2]);
  return pref * (w * (a * invCs2 + (g4 * eF)));
}

// f after collision of direction q and its node force contributions
// (collisionAndStream, src/LBM_PSM_BGK_dynamics.h:40-114), from feq and the
// slots' solid equilibria f0s; NS slots (0: plain BGK).
template <class L, int q, bool FORCE, int NS>
__device__ __forceinline__ void relax_q(double& fq, double feq, double f0s0, double f0s1, double Fq,
                                        const NodeF64& nd, double omega, double omo,
                                        Slot (&sl)[2], double (&t)[2]) {
  const double fi = fq;
  const double d = feq - fi;
  if (NS == 0) {
    fq = FORCE ? fi + d * omega + Fq : fi + d * omega;
    return;
  }
  // one_minus_omega*(fi - feq) is -(omo*d) bit for bit
  const double od = omo * d;
  double r = fi + nd.oneMinusBtot * d * omega;
  t[0] = sl[0].B * ((f0s0 - fi) - od);
  r = r + t[0];
  if (NS == 2) {
    t[1] = sl[1].B * ((f0s1 - fi) - od);
    r = r + t[1];
  }
  fq = FORCE ? r + Fq : r;
}

template <class L, int q>
__device__ __forceinline__ void add_force(double (&F)[3], double t) {  // F += -t*e_q
  constexpr int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
  if (cx) F[0] = cx > 0 ? F[0] - t : F[0] + t;
  if (cy) F[1] = cy > 0 ? F[1] - t : F[1] + t;
  if (cz) F[2] = cz > 0 ? F[2] - t : F[2] + t;
}

// The pair k = (q, opp q): e.u, its multiple and its square are formed once,
// the opposite direction taking them with the sign turned (negation is exact,
// so both directions round as when formed alone); 0.5*invCs4 is exact.
template <class L, int k, bool FORCE, int NS>
struct CollidePairs {
  __device__ __forceinline__ static void run(double (&f)[L::Q], const NodeF64& nd, double invCs2,
                                             double invCs4, double omega, double omo, double pref,
                                             Slot (&sl)[2], double (&t)[L::Q][2]) {
    constexpr int q = Pairs<L>::q(k), o = L::opp(q);
    constexpr int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
    const double rw = nd.rw[weight_class<L>(q)];
    const double eu = edot<cx, cy, cz>(nd.u[0], nd.u[1], nd.u[2]);
    const double a = eu * invCs2, b = eu * eu * (0.5 * invCs4);
    const double ep = rw * ((1.0 + a) + b - nd.usq_half), em = rw * ((1.0 - a) + b - nd.usq_half);
    double sp[2] = {0.0, 0.0}, sm[2] = {0.0, 0.0};
#pragma unroll
    for (int n = 0; n < NS; ++n) {  // feq(iq, rho, uSolid) (src/LBM_PSM_dynamics.h:72-85)
      const double es = edot<cx, cy, cz>(sl[n].us[0], sl[n].us[1], sl[n].us[2]);
      const double as = es * invCs2, bs = es * es * (0.5 * invCs4);
      sp[n] = rw * ((1.0 + as) + bs - sl[n].half);
      sm[n] = rw * ((1.0 - as) + bs - sl[n].half);
    }
    const double g4 = FORCE ? eu * invCs4 : 0.0;
    const double Fp = FORCE ? guo_q<L, q>(nd, g4, invCs2, pref) : 0.0;
    const double Fm = FORCE ? guo_q<L, o>(nd, -g4, invCs2, pref) : 0.0;
    relax_q<L, q, FORCE, NS>(f[q], ep, sp[0], sp[1], Fp, nd, omega, omo, sl, t[q]);
    relax_q<L, o, FORCE, NS>(f[o], em, sm[0], sm[1], Fm, nd, omega, omo, sl, t[o]);
    if (L::Q == 19) {  // the pairs are in direction order: add as the reference does
#pragma unroll
      for (int n = 0; n < NS; ++n) {
        add_force<L, q>(sl[n].F, t[q][n]);
        add_force<L, o>(sl[n].F, t[o][n]);
      }
    }
    CollidePairs<L, k + 1, FORCE, NS>::run(f, nd, invCs2, invCs4, omega, omo, pref, sl, t);
  }
};
template <class L, bool FORCE, int NS>
struct CollidePairs<L, Pairs<L>::N, FORCE, NS> {
  __device__ __forceinline__ static void run(double (&)[L::Q], const NodeF64&, double, double, double,
                                             double, double, Slot (&)[2], double (&)[L::Q][2]) {}
};
template <class L, int q>
struct ForceUnroll {  // in direction order, as the reference adds them
  __device__ __forceinline__ static void run(double (&F)[3], const double (&t)[L::Q][2], int n) {
    add_force<L, q>(F, t[q][n]);
    ForceUnroll<L, q + 1>::run(F, t, n);
  }
};
template <class L>
struct ForceUnroll<L, L::Q> {
  __device__ __forceinline__ static void run(double (&)[3], const double (&)[L::Q][2], int) {}
};

template <class L, bool FORCE, int NS>
__device__ __forceinline__ void collide_dirs(double (&f)[L::Q], const NodeF64& nd,
                                             const CollideParams& p, const BoxParams& bp,
                                             Slot (&sl)[2]) {
  double t[L::Q][2];
  const double pref = bp.guo_pref, omega = bp.omega, omo = bp.one_minus_omega;
  const double f0 = nd.rw[0] * (1.0 - nd.usq_half);
  double s0[2] = {0.0, 0.0};
#pragma unroll
  for (int n = 0; n < NS; ++n) s0[n] = nd.rw[0] * (1.0 - sl[n].half);
  const double F0 = FORCE ? guo_q<L, 0>(nd, 0.0, p.invCs2, pref) : 0.0;
  relax_q<L, 0, FORCE, NS>(f[0], f0, s0[0], s0[1], F0, nd, omega, omo, sl, t[0]);
  CollidePairs<L, 0, FORCE, NS>::run(f, nd, p.invCs2, p.invCs4, omega, omo, pref, sl, t);
  if (L::Q != 19) {
#pragma unroll
    for (int n = 0; n < NS; ++n) ForceUnroll<L, 1>::run(sl[n].F, t, n);
  }
}

// One node of the FP64 collide + A-A stream step.
//
// Bound by the FP64 pipe (1.68 operations per clock and multiprocessor, the
// memory system at a few per cent): so what directions share is formed once
// (CollidePairs), three quotients share one reciprocal (div3), the body force
// is a template argument, and a warp takes the plain loop when none of its
// nodes is a PSM node, the one-slot loop when none holds two particles -- an
// unused slot has B = 0 and adds zeros, and a node without any has 1 - B = 1,
// so the longer loops leave its populations bit for bit as the shorter ones.
template <class L, bool ODD, bool FORCE>
__device__ __forceinline__ void collide_f64_node(const CollideParams& p, int sx, int sy, int sz) {
  constexpr int Q = L::Q;
  const Geom& g = p.g;
  const long long n = node_index(g, sx, sy, sz);
  const Nbr nb = make_nbr(g, sx, sy, sz);
  const BoxParams& bp = p.box[box_of_z(g, sz)];
  double* F = static_cast<double*>(p.f);
  // in place unless a separate source is given (recomputation of stored states)
  const double* Fin = p.fsrc ? static_cast<const double*>(p.fsrc) : F;
  const long long Np = g.Np;

  const uint8_t flag = p.tab.flag[n];
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

  // macro values (src/LBM_PSM_BGK_dynamics.cpp:48-77)
  double rho = f[0];
#pragma unroll
  for (int q = 1; q < Q; ++q) rho = rho + f[q];
  // (each sum's first term is a +e direction, taken as it is instead of 0 + f)
  double j[3] = {f[1], f[L::Q == 19 ? 3 : 2], L::Q == 19 ? f[5] : 0.0};
#pragma unroll
  for (int q = 2; q < Q; ++q) {
    const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
    if (cx) j[0] = cx > 0 ? j[0] + f[q] : j[0] - f[q];
    if (cy && q > (L::Q == 19 ? 3 : 2)) j[1] = cy > 0 ? j[1] + f[q] : j[1] - f[q];
    if (cz && q > 5) j[2] = cz > 0 ? j[2] + f[q] : j[2] - f[q];
  }
  NodeF64 nd;
  if (FORCE) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      j[c] = j[c] + bp.F[c] * 0.5;
      nd.F[c] = bp.has_force ? bp.F[c] : 0.0;  // (a box of an ensemble may have none)
    }
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c)  // (|F|^2 of a non-zero F may underflow to "no force")
      if ((__double_as_longlong(bp.F[c]) << 1) != 0ll) j[c] = j[c] + bp.F[c] * 0.5;
  }
  div3(j[0], j[1], j[2], rho, nd.u[0], nd.u[1], nd.u[2]);
  if (p.store_macro) {
    p.rho_out[n] = rho;
#pragma unroll
    for (int c = 0; c < 3; ++c) p.u_out[3 * n + c] = nd.u[c];
  }
  nd.usq_half = 0.5 * (nd.u[0] * nd.u[0] + nd.u[1] * nd.u[1] + nd.u[2] * nd.u[2]) * p.invCs2;
#pragma unroll
  for (int c = 0; c < 3; ++c) nd.rw[c] = rho * L::w(c == 0 ? 0 : (c == 1 ? 1 : Q - 1));
  if (FORCE) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      nd.gF[c][0] = (0.0 - nd.u[c]) * nd.F[c];
      nd.gF[c][1] = (1.0 - nd.u[c]) * nd.F[c];
      nd.gF[c][2] = (-1.0 - nd.u[c]) * nd.F[c];
    }
  }
  nd.oneMinusBtot = 1.0;

  const unsigned act = __activemask();
  const bool psm = flag != 0;
  Slot sl[2];
  if (!__any_sync(act, psm)) {
    collide_dirs<L, FORCE, 0>(f, nd, p, bp, sl);
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      sl[k].B = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) sl[k].us[c] = sl[k].F[c] = 0.0;
      sl[k].half = 0.0;
    }
    if (psm) {
      const int2 id = p.tab.ids[n];
      const double2 e = p.tab.eps[n];
      const double* us = p.tab.us + 6 * n;
      const bool has1 = id.x > 0, has2 = id.y > 0;
      double B1 = has1 ? e.x : 0.0;
      double B2 = has2 ? e.y : 0.0;
      if (p.weighting == 1) {  // Noble-Torczynski weighting (opt-in)
        const double tm = bp.tau - 0.5;
        if (has1) B1 = B1 * tm / ((1.0 - B1) + tm);
        if (has2) B2 = B2 * tm / ((1.0 - B2) + tm);
      }
      double Btot = B1 + B2;
      if (Btot > 1.0) {
        B1 = B1 / Btot;
        B2 = B2 / Btot;
        Btot = 1.0;
      }
      sl[0].B = B1;
      sl[1].B = B2;
      nd.oneMinusBtot = 1.0 - Btot;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (has1) sl[0].us[c] = us[c];
        if (has2) sl[1].us[c] = us[3 + c];
      }
#pragma unroll
      for (int k = 0; k < 2; ++k)
        sl[k].half = 0.5 *
                     (sl[k].us[0] * sl[k].us[0] + sl[k].us[1] * sl[k].us[1] + sl[k].us[2] * sl[k].us[2]) *
                     p.invCs2;
    }
    if (!__any_sync(act, (flag & 2) != 0))
      collide_dirs<L, FORCE, 1>(f, nd, p, bp, sl);
    else
      collide_dirs<L, FORCE, 2>(f, nd, p, bp, sl);
    if (psm) {
      double* nf = static_cast<double*>(p.tab.nodeF) + 6 * n;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        nf[c] = sl[0].F[c];
        nf[3 + c] = sl[1].F[c];
      }
    }
  }

#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
    if (!ODD) {
      F[L::opp(q) * Np + n] = f[q];
    } else {
      if (nbr_ok(nb, cx, cy, cz)) F[q * Np + n + nbr_off(nb, cx, cy, cz)] = f[q];
    }
  }
}

// Node of thread t of block b when the stored nodes (x fastest, without the
// rows' padding) are dealt out 128 to a block: rows shorter than a block, or
// not a multiple of a warp, leave no lane of the FP64 pipe idle.
constexpr int F64_THREADS = 128;
__device__ __forceinline__ bool node_of(const Geom& g, unsigned b, int& sx, int& sy, int& sz) {
  const unsigned S0 = (unsigned)g.S[0];
  const unsigned first = b * (unsigned)F64_THREADS;  // the node count stays below 2^32 (memory)
  unsigned row = first / S0;
  unsigned x = first - row * S0 + threadIdx.x;
  const unsigned up = x / S0;
  x -= up * S0;
  row += up;
  const unsigned z = row / (unsigned)g.S[1];
  sx = (int)x;
  sy = (int)(row - z * (unsigned)g.S[1]);
  sz = (int)z;
  return z < (unsigned)g.S[2];
}

template <class L, bool ODD, bool FORCE>
__global__ void __launch_bounds__(F64_THREADS) collide_f64_kernel(CollideParams p) {
  int sx, sy, sz;
  if (!node_of(p.g, blockIdx.x, sx, sy, sz)) return;
  collide_f64_node<L, ODD, FORCE>(p, sx, sy, sz);
}

// The members of a group in one launch: member m owns blocks
// [first[m], first[m+1]), laid out as its own kernel's; every node runs the
// same code as above, so the results are the members'.
template <class L, bool ODD, bool FORCE>
__global__ void __launch_bounds__(F64_THREADS) collide_f64_multi_kernel(MultiCollide mc) {
  const int b = blockIdx.x;
  int m = 0;
  while (m + 1 < mc.nm && b >= mc.first[m + 1]) ++m;
  const CollideParams& p = mc.m[m].p;
  int sx, sy, sz;
  if (!node_of(p.g, (unsigned)(b - mc.first[m]), sx, sy, sz)) return;
  collide_f64_node<L, ODD, FORCE>(p, sx, sy, sz);
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
