// adjoint.cu -- discrete adjoint and tangent of the FP64 collide-stream-PSM
// step on a fully periodic lattice with the particles held in place.
//
// Forward step (one node, pre-collision populations f, table weights B_s and
// solid velocities us_s; compute_macro_values + collisionAndStream,
// src/LBM_PSM_BGK_dynamics.cpp:48-109, src/LBM_PSM_BGK_dynamics.h:40-114,
// feq / F_iq src/LBM_PSM_dynamics.h:43-116), in exact arithmetic:
//
//   rho = sum f, m = sum f e, j = m + F/2, u = j / rho
//   C_q = (1-w) f_q + (w - Bt) feq_q(rho, u) + sum_s B_s feq_q(rho, us_s) + (1 - w/2) g_q(u)
//   g_q = w_q [3 (e_q - u).F + 9 (e_q.u)(e_q.F)]             (unscaled Guo term)
//   f_{t+1, q}(x + e_q) = C_q(x)                              (streaming)
//   slot force (add_Fhyd, src/LBM_PSM_lattice.cpp:355-363):
//   -B_s sum_q Omega_s,q e_q = B_s (m + (1-w) F/2 - rho us_s)
//
// Objective: J = sum_t c_t sum_nodes sum_s cw_s d . (slot force), where cw_s
// counts the images of the slot's particle whose reduction box holds the
// node (calculateHydrodynamicInteractions, src/LBM_PSM_exchangeParticleData.cpp:172-244)
// and c_t = forceFactor / M inside the averaging window, 0 outside.
//
// The reverse step pulls the adjoint of the next step's pre-collision
// populations, mu_q(x) = lambda_{t+1,q}(x + e_q), and applies the transposed
// node Jacobian through moments of w_q mu_q (M0, M1_a, M2_ab), so that every
// contraction sum_q mu_q dC_q/d(.) costs a few FP64 operations per node.
// The tangent step pushes dC along a direction (dtau, dF, dx).  Centre
// derivatives enter through the solid fractions: the central difference of
// calcSolidFraction's sub-cell count (src/LBM_PSM_exchangeParticleData.cpp:116-169)
// at step h, computed exactly with the reference's FP64 operations.
#include "lbmpsm_internal.cuh"
#include "solid_fraction.cuh"

namespace lbmpsm {

namespace {

constexpr int ADJ_THREADS = 128;

// Weights of the two slots and their derivatives (BGK weighting B = eps, or
// Noble-Torczynski B = eps (tau-1/2) / ((1-eps) + tau-1/2); renormalised to
// sum 1 when the sum exceeds 1, as in collisionAndStream :90-95).
struct SlotWeights {
  double B[2];
  double dBde[2][2];  // dB_r / deps_k
  double dBdtau[2];
};

__device__ __forceinline__ void slot_weights(double e0, double e1, bool occ0, bool occ1,
                                             int weighting, double tau, SlotWeights& w) {
  const double e[2] = {occ0 ? e0 : 0.0, occ1 ? e1 : 0.0};
  double b[2], db[2], dbt[2];
  const double tm = tau - 0.5;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (weighting == 1) {
      const double den = (1.0 - e[k]) + tm;
      b[k] = e[k] * tm / den;
      db[k] = tm * (1.0 + tm) / (den * den);
      dbt[k] = e[k] * (1.0 - e[k]) / (den * den);
    } else {
      b[k] = e[k];
      db[k] = 1.0;
      dbt[k] = 0.0;
    }
  }
  const double s = b[0] + b[1];
  double J[2][2];
  if (s > 1.0) {
    const double is2 = 1.0 / (s * s);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      w.B[r] = b[r] / s;
#pragma unroll
      for (int k = 0; k < 2; ++k) J[r][k] = ((r == k ? s : 0.0) - b[r]) * is2;
    }
  } else {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      w.B[r] = b[r];
#pragma unroll
      for (int k = 0; k < 2; ++k) J[r][k] = r == k ? 1.0 : 0.0;
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    w.dBde[r][0] = J[r][0] * db[0];
    w.dBde[r][1] = J[r][1] * db[1];
    w.dBdtau[r] = J[r][0] * dbt[0] + J[r][1] * dbt[1];
  }
}

// The lattice's directions as opposite pairs (q(k), o(k)), e_q = +1 on its
// first axis.
template <class L>
struct PairOf {
  static constexpr int N = (L::Q - 1) / 2;
  __host__ __device__ static constexpr int q(int k) {
    return L::Q == 19 ? 2 * k + 1 : (k == 0 ? 1 : (k == 1 ? 2 : (k == 2 ? 5 : 8)));
  }
  __host__ __device__ static constexpr int o(int k) { return L::opp(q(k)); }
};

// Moments of v_q = w_q mu_q: M0 = sum v, M1_a = sum v e_a,
// M2 = sum v e_a e_b in the order xx, yy, zz, xy, xz, yz, from the sums and
// differences of opposite directions (the weights applied to their totals).
template <class L>
__device__ __forceinline__ void moments(const double* mu, double& M0, double M1[3],
                                        double M2[6]) {
  double s0[2] = {0.0, 0.0}, s1[2][3], s2[2][6];  // [axis | diagonal directions]
#pragma unroll
  for (int c = 0; c < 2; ++c) {
#pragma unroll
    for (int a = 0; a < 3; ++a) s1[c][a] = 0.0;
#pragma unroll
    for (int a = 0; a < 6; ++a) s2[c][a] = 0.0;
  }
#pragma unroll
  for (int k = 0; k < PairOf<L>::N; ++k) {
    const int q = PairOf<L>::q(k);
    const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
    const int c = cx * cx + cy * cy + cz * cz == 1 ? 0 : 1;
    const double s = mu[q] + mu[PairOf<L>::o(k)], d = mu[q] - mu[PairOf<L>::o(k)];
    s0[c] += s;
    if (cx) s1[c][0] += cx > 0 ? d : -d;
    if (cy) s1[c][1] += cy > 0 ? d : -d;
    if (cz) s1[c][2] += cz > 0 ? d : -d;
    if (cx) s2[c][0] += s;
    if (cy) s2[c][1] += s;
    if (cz) s2[c][2] += s;
    if (cx && cy) s2[c][3] += cx * cy > 0 ? s : -s;
    if (cx && cz) s2[c][4] += cx * cz > 0 ? s : -s;
    if (cy && cz) s2[c][5] += cy * cz > 0 ? s : -s;
  }
  const double wa = L::w(1), wd = L::w(L::Q - 1);
  M0 = L::w(0) * mu[0] + wa * s0[0] + wd * s0[1];
#pragma unroll
  for (int a = 0; a < 3; ++a) M1[a] = wa * s1[0][a] + wd * s1[1][a];
#pragma unroll
  for (int a = 0; a < 6; ++a) M2[a] = a < 3 ? wa * s2[0][a] + wd * s2[1][a] : wd * s2[1][a];
}

__device__ __forceinline__ void m2_times(const double M2[6], const double a[3], double out[3]) {
  out[0] = M2[0] * a[0] + M2[3] * a[1] + M2[4] * a[2];
  out[1] = M2[3] * a[0] + M2[1] * a[1] + M2[5] * a[2];
  out[2] = M2[4] * a[0] + M2[5] * a[1] + M2[2] * a[2];
}

__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

template <class L, int q>
__device__ __forceinline__ double edot_c(const double v[3]) {
  // (-0 is the identity of IEEE addition: the leading term costs nothing)
  double s = -0.0;
  if (L::ex(q)) s += L::ex(q) > 0 ? v[0] : -v[0];
  if (L::ey(q)) s += L::ey(q) > 0 ? v[1] : -v[1];
  if (L::ez(q)) s += L::ez(q) > 0 ? v[2] : -v[2];
  return s;
}

template <class L, int k>
struct UnrollPairs {
  template <class Fn>
  __device__ __forceinline__ static void run(Fn& fn) {
    fn.template apply<k>();
    UnrollPairs<L, k + 1>::run(fn);
  }
};
template <class L>
struct UnrollPairs<L, PairOf<L>::N> {
  template <class Fn>
  __device__ __forceinline__ static void run(Fn&) {}
};

// rho = sum f and m = sum f e, from the sums and differences of opposite directions
template <class L>
__device__ __forceinline__ void density_momentum(const double* f, double& rho, double m[3]) {
  rho = f[0];
  m[0] = m[1] = m[2] = -0.0;
#pragma unroll
  for (int k = 0; k < PairOf<L>::N; ++k) {
    const int q = PairOf<L>::q(k);
    const double d = f[q] - f[PairOf<L>::o(k)];
    rho += f[q] + f[PairOf<L>::o(k)];
    if (L::ex(q)) m[0] += L::ex(q) > 0 ? d : -d;
    if (L::ey(q)) m[1] += L::ey(q) > 0 ? d : -d;
    if (L::ez(q)) m[2] += L::ez(q) > 0 ? d : -d;
  }
}

// the pre-collision populations of node n in A-A storage, as the FP64
// collide kernel reads them
template <class L>
__device__ __forceinline__ void load_state(const double* F, long long Np, long long n,
                                           const Nbr& nb, int odd, double* f) {
#pragma unroll
  for (int q = 0; q < L::Q; ++q) {
    const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
    if (!odd)
      f[q] = F[q * Np + n];
    else
      f[q] = F[L::opp(q) * Np + n + nbr_off(nb, -cx, -cy, -cz)];
  }
}

// One node's slots as the sweeps see them.
struct NodeSlots {
  bool live[2];     // slot has a particle (table) or an entering one (band)
  bool band;
  double B[2];
  double us[2][3];
  double cw[2];
  SlotWeights w;
};

__device__ __forceinline__ void node_slots(const AdjParams& p, long long n, NodeSlots& s) {
  const uint8_t flag = p.tab.flag[n];
  const uint8_t band = p.an.band[n];
  s.band = band != 0;
  s.live[0] = s.live[1] = false;
  s.B[0] = s.B[1] = 0.0;
  s.cw[0] = s.cw[1] = 0.0;
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) s.us[k][c] = 0.0;
#pragma unroll
  for (int k = 0; k < 2; ++k) s.w.B[k] = s.w.dBde[k][0] = s.w.dBde[k][1] = s.w.dBdtau[k] = 0.0;
  if (!flag && !band) return;
  int2 id = make_int2(0, 0);
  double2 e = make_double2(0.0, 0.0);
  if (flag) {
    id = p.tab.ids[n];
    e = p.tab.eps[n];
  }
  const bool occ0 = id.x > 0, occ1 = id.y > 0;
  slot_weights(e.x, e.y, occ0, occ1, p.weighting, p.bp.tau, s.w);
  const int2 cw = p.an.cw[n];
  const int2 et = band ? p.an.tag[n] : make_int2(0, 0);
  const bool occ[2] = {occ0, occ1};
  const int etag[2] = {et.x, et.y};
  const int cwk[2] = {cw.x, cw.y};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (occ[k]) {
      s.live[k] = true;
      s.B[k] = s.w.B[k];
#pragma unroll
      for (int c = 0; c < 3; ++c) s.us[k][c] = p.tab.us[6 * n + 3 * k + c];
      s.cw[k] = (double)cwk[k];
    } else if (etag[k] > 0) {
      s.live[k] = true;
#pragma unroll
      for (int c = 0; c < 3; ++c) s.us[k][c] = p.an.us[6 * n + 3 * k + c];
      s.cw[k] = (double)cwk[k];
    }
  }
}

// deterministic block sum of the first N of ADJ_PART values into this block's
// slot: within a warp the first levels halve the values each lane carries
// (9 FP64 additions for five values, 5 for one)
template <int N>
__device__ __forceinline__ void block_accumulate(const double (&v)[ADJ_PART], double* part) {
  __shared__ double red[ADJ_THREADS / 32][ADJ_PART];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (N == 1) {
    double x = v[0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[wid][0] = x;
  } else {
    static_assert(ADJ_PART <= 8, "values");
    double w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = k < ADJ_PART ? v[k < ADJ_PART ? k : 0] : 0.0;
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {  // lane bits 16, 8, 4 choose value bits 4, 2, 1
      const bool up = (lane & (4 * h)) != 0;
#pragma unroll
      for (int k = 0; k < h; ++k) {
        const double keep = up ? w[k + h] : w[k], send = up ? w[k] : w[k + h];
        w[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * h);
      }
    }
    double x = w[0];
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    const int k = lane >> 2;
    if ((lane & 3) == 0 && k < ADJ_PART) red[wid][k] = x;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double x = 0.0;
#pragma unroll
    for (int w = 0; w < ADJ_THREADS / 32; ++w) x += red[w][threadIdx.x];
    part[(long long)blockIdx.x * ADJ_PART + threadIdx.x] += x;
  }
}

// ------------------------------------------------------------ reverse step
// out_q = (1 - omega) mu_q + base + e_q.V, e.V once per pair of directions
template <class L>
struct AdjPairs {
  const double* mu;
  double omw, base;
  const double* V;
  double* out;
  template <int k>
  __device__ __forceinline__ void apply() {
    constexpr int q = PairOf<L>::q(k), o = PairOf<L>::o(k);
    const double eV = edot_c<L, q>(V);
    out[q] = omw * mu[q] + base + eV;
    out[o] = omw * mu[o] + base - eV;
  }
};

// Bound by the FP64 pipe, as the collide: moments from the sums and
// differences of opposite directions, the per-direction terms gathered into
// one vector, nodes dealt out to blocks without regard to rows (56^3: 117 us a
// step; every direction on its own and rows of 56 nodes to a block: 197 us);
// factors of the body force from the host, drag terms only where a particle is
// (24 steps forward and back 8.72 -> 8.55 ms).
template <class L>
__global__ void __launch_bounds__(ADJ_THREADS) adj_step_kernel(AdjParams p) {
  constexpr int Q = L::Q;
  const Geom& g = p.g;
  int sx, sy, sz;
  double acc[ADJ_PART] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (node_of_block<ADJ_THREADS>(g, blockIdx.x, sx, sy, sz)) {
    const long long n = node_index(g, sx, sy, sz);
    const Nbr nb = make_nbr(g, sx, sy, sz);
    const long long Np = g.Np;
    const BoxParams& bp = p.bp;
    const double omega = bp.omega;
    const double F[3] = {bp.F[0], bp.F[1], bp.F[2]};
    double f[Q], mu[Q];
    load_state<L>(p.state, Np, n, nb, p.odd, f);
#pragma unroll
    for (int q = 0; q < Q; ++q)
      mu[q] = p.lin[q * Np + n + nbr_off(nb, L::ex(q), L::ey(q), L::ez(q))];
    double rho, m[3], smf = mu[0] * f[0];
    density_momentum<L>(f, rho, m);
#pragma unroll
    for (int q = 1; q < Q; ++q) smf += mu[q] * f[q];
    const double inv_rho = 1.0 / rho;
    double u[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = (m[a] + 0.5 * F[a]) * inv_rho;
    double M0, M1[3], M2[6];
    moments<L>(mu, M0, M1, M2);
    const double usq = dot3(u, u);
    // F3 = 3 F and F9 = 9 F come with the parameters: an operation on values all
    // nodes share costs the FP64 pipe as much as one on the node's own
    const double F3[3] = {p.F3[0], p.F3[1], p.F3[2]}, F9[3] = {p.F9[0], p.F9[1], p.F9[2]};
    double M2u[3], M2F[3];  // (of 9 F)
    m2_times(M2, u, M2u);
    m2_times(M2, F9, M2F);
    const double uM2u = dot3(u, M2u);
    const double smfeq = rho * (M0 * (1.0 - 1.5 * usq) + 3.0 * dot3(u, M1) + 4.5 * uM2u);
    const double A_rho = M0 * (1.0 + 1.5 * usq) - 4.5 * uM2u;
    double Aj[3], Au[3];  // a third of A_j; A_u without its factor gp
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      Aj[a] = M1[a] + 3.0 * M2u[a] - u[a] * M0;
      Au[a] = M2F[a] - F3[a] * M0;
    }
    const double smg = dot3(M1, F3) - M0 * dot3(u, F3) + dot3(u, M2F);

    NodeSlots sl;
    node_slots(p, n, sl);
    const bool slots = sl.live[0] || sl.live[1];
    double sumBAs = 0.0, coef = 0.0, dconst = 0.0, Bt = 0.0, sum_cB = 0.0, gtauB = 0.0;
    double beta[2] = {0.0, 0.0}, d[3] = {0.0, 0.0, 0.0}, dm = 0.0, dF = 0.0;
    if (slots) {
#pragma unroll
      for (int a = 0; a < 3; ++a) d[a] = p.d[a];
      dm = dot3(d, m);
      dF = dot3(d, F);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (!sl.live[k]) continue;
      const double* vs = sl.us[k];
      double M2v[3];
      m2_times(M2, vs, M2v);
      const double As = M0 * (1.0 - 1.5 * dot3(vs, vs)) + 3.0 * dot3(vs, M1) + 4.5 * dot3(vs, M2v);
      const double dvs = dot3(d, vs);
      const double cB = p.c * sl.cw[k] * sl.B[k];
      sumBAs += sl.B[k] * As;
      Bt += sl.B[k];
      coef += cB;
      dconst -= cB * dvs;
      sum_cB += cB;
      beta[k] = rho * As - smfeq +
                p.c * sl.cw[k] * (dm + (1.0 - omega) * dF * 0.5 - rho * dvs);
    }
    if (p.weighting == 1) gtauB = beta[0] * sl.w.dBdtau[0] + beta[1] * sl.w.dBdtau[1];
    if (sl.band) {
      p.an.sigma[2 * n] += beta[0];
      p.an.sigma[2 * n + 1] += beta[1];
    }
    const double gp = 1.0 - 0.5 * omega, gi = gp * inv_rho, ob = omega - Bt, ob3 = 3.0 * ob;
    double V[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) V[a] = ob3 * Aj[a] + Au[a] * gi;
    AdjPairs<L> fn;
    fn.mu = mu;
    fn.omw = 1.0 - omega;
    fn.base = ob * A_rho - dot3(u, Au) * gi;
    if (slots) {
#pragma unroll
      for (int a = 0; a < 3; ++a) V[a] += coef * d[a];
      fn.base += sumBAs + dconst;
    }
    fn.V = V;
    double out[Q];
    fn.out = out;
    out[0] = fn.omw * mu[0] + fn.base;
    UnrollPairs<L, 0>::run(fn);
#pragma unroll
    for (int q = 0; q < Q; ++q) p.lout[q * Np + n] = out[q];

    acc[0] = smfeq - smf - 0.5 * smg;
    acc[1] = gtauB;
    const double cj = 0.5 * ob3 + 3.0 * gp, cu = 0.5 * gi;
#pragma unroll
    for (int a = 0; a < 3; ++a) acc[2 + a] = cj * Aj[a] + cu * Au[a];
    if (slots) {
      acc[0] -= sum_cB * dF * 0.5;
#pragma unroll
      for (int a = 0; a < 3; ++a) acc[2 + a] += sum_cB * (1.0 - omega) * d[a] * 0.5;
    }
  }
  block_accumulate<ADJ_PART>(acc, p.part);
}

// ------------------------------------------------------------ tangent step
// The tangent of direction q, dC_q, has a part even in e and one odd in e:
//   even: w [K + (e.u)(e.W1) + (e.F)(e.W2) + sum_k (e.us_k)(e.Y_k)]
//   odd : w e.V
// with K, V, W1, W2, Y_k sums over the node, so that a pair of opposite
// directions shares everything but the last addition (48^3: 96 us a step; every
// direction on its own and rows of 48 nodes to a block: 326 us).  The force terms
// all nodes share come from the host, the drag terms are formed only where a
// particle is (16 steps 3.67 -> 3.59 ms).
template <class L>
struct TanPairs {
  const double *u, *F, *V, *W1, *W2, (*us)[3], (*Y)[3];
  double K, omw, domega;
  bool slots;
  const double *f, *fd;
  double* out;
  template <int k>
  __device__ __forceinline__ void apply() {
    constexpr int q = PairOf<L>::q(k), o = PairOf<L>::o(k);
    double even = K + edot_c<L, q>(u) * edot_c<L, q>(W1) + edot_c<L, q>(F) * edot_c<L, q>(W2);
    if (slots)
      even += edot_c<L, q>(us[0]) * edot_c<L, q>(Y[0]) + edot_c<L, q>(us[1]) * edot_c<L, q>(Y[1]);
    const double odd = edot_c<L, q>(V), w = L::w(q);
    out[q] = omw * fd[q] - domega * f[q] + w * (even + odd);
    out[o] = omw * fd[o] - domega * f[o] + w * (even - odd);
  }
};

template <class L>
__global__ void __launch_bounds__(ADJ_THREADS) tan_step_kernel(AdjParams p) {
  constexpr int Q = L::Q;
  const Geom& g = p.g;
  int sx, sy, sz;
  double acc[ADJ_PART] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (node_of_block<ADJ_THREADS>(g, blockIdx.x, sx, sy, sz)) {
    const long long n = node_index(g, sx, sy, sz);
    const Nbr nb = make_nbr(g, sx, sy, sz);
    const long long Np = g.Np;
    const BoxParams& bp = p.bp;
    const double omega = bp.omega, domega = p.domega;
    const double F[3] = {bp.F[0], bp.F[1], bp.F[2]};
    const double dFv[3] = {p.dF[0], p.dF[1], p.dF[2]};
    double f[Q], fd[Q];
    load_state<L>(p.state, Np, n, nb, p.odd, f);
#pragma unroll
    for (int q = 0; q < Q; ++q) fd[q] = p.lin[q * Np + n];
    double rho, rhod, m[3], md[3];
    density_momentum<L>(f, rho, m);
    density_momentum<L>(fd, rhod, md);
    const double inv_rho = 1.0 / rho;
    double u[3], jd[3], ud[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      u[a] = (m[a] + 0.5 * F[a]) * inv_rho;
      jd[a] = md[a] + 0.5 * dFv[a];
      ud[a] = (jd[a] - u[a] * rhod) * inv_rho;
    }
    const double usq = dot3(u, u);
    const double uF = dot3(u, F), udF = dot3(u, dFv), ujd = dot3(u, jd), Fud = dot3(F, ud);

    NodeSlots sl;
    node_slots(p, n, sl);
    double Bd[2] = {0.0, 0.0};
    if (sl.live[0] || sl.live[1]) {
      const double ed0 = sl.band ? p.an.edot[2 * n] : 0.0;
      const double ed1 = sl.band ? p.an.edot[2 * n + 1] : 0.0;
#pragma unroll
      for (int k = 0; k < 2; ++k)
        Bd[k] = sl.w.dBde[k][0] * ed0 + sl.w.dBde[k][1] * ed1 + sl.w.dBdtau[k] * p.dtau;
    }
    const double Bt = sl.B[0] + sl.B[1], Btd = Bd[0] + Bd[1];
    const double gp = 1.0 - 0.5 * omega;
    const double rr = rhod * inv_rho;
    const double cf = domega - Btd, ob = omega - Bt;  // factors of feq and of its tangent
    TanPairs<L> fn;
    fn.K = cf * rho * (1.0 - 1.5 * usq) + ob * (rhod * (1.0 + 1.5 * usq) - 3.0 * ujd) +
           1.5 * domega * uF - 3.0 * gp * (Fud + udF);
    const double a1 = 4.5 * (cf * rho - ob * rhod);
    double V[3], W1[3], W2[3], Y[2][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double t = ob * jd[a] + p.force[a];
      V[a] = 3.0 * (cf * rho * u[a] + t);
      W1[a] = a1 * u[a] + 9.0 * t;
      W2[a] = 9.0 * gp * ud[a];
      Y[0][a] = Y[1][a] = 0.0;
    }
    fn.slots = sl.live[0] || sl.live[1];
    if (fn.slots) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (!sl.live[k]) continue;
        const double ck = rho * (Bd[k] + sl.B[k] * rr);
        fn.K += ck * (1.0 - 1.5 * dot3(sl.us[k], sl.us[k]));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          V[a] += 3.0 * ck * sl.us[k][a];
          Y[k][a] = 4.5 * ck * sl.us[k][a];
        }
      }
    }
    double out[Q];
    fn.u = u;
    fn.F = F;
    fn.V = V;
    fn.W1 = W1;
    fn.W2 = W2;
    fn.us = sl.us;
    fn.Y = Y;
    fn.omw = 1.0 - omega;
    fn.domega = domega;
    fn.f = f;
    fn.fd = fd;
    fn.out = out;
    out[0] = fn.omw * fd[0] - domega * f[0] + L::w(0) * fn.K;
    UnrollPairs<L, 0>::run(fn);
#pragma unroll
    for (int q = 0; q < Q; ++q)
      p.lout[q * Np + n + nbr_off(nb, L::ex(q), L::ey(q), L::ez(q))] = out[q];

    double d[3] = {0.0, 0.0, 0.0}, dm = 0.0, dmd = 0.0, dF = 0.0, ddF = 0.0;
    if (fn.slots) {
#pragma unroll
      for (int a = 0; a < 3; ++a) d[a] = p.d[a];
      dm = dot3(d, m);
      dmd = dot3(d, md);
      dF = dot3(d, F);
      ddF = dot3(d, dFv);
    }
    double dJ = 0.0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (!sl.live[k]) continue;
      const double dvs = dot3(d, sl.us[k]);
      const double base = dm + (1.0 - omega) * dF * 0.5 - rho * dvs;
      dJ += p.c * sl.cw[k] *
            (Bd[k] * base +
             sl.B[k] * (dmd - domega * dF * 0.5 + (1.0 - omega) * ddF * 0.5 - rhod * dvs));
    }
    acc[0] = dJ;
  }
  block_accumulate<1>(acc, p.part);
}

// ------------------------------------------------------- entries and weights
__global__ void adj_entries_kernel(AdjSetup s) {
  const Geom& g = s.g;
  const long long total = (long long)g.S[0] * g.S[1] * g.S[2];
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int sx = (int)(idx % g.S[0]);
  const int sy = (int)((idx / g.S[0]) % g.S[1]);
  const int sz = (int)(idx / ((long long)g.S[0] * g.S[1]));
  const long long n = node_index(g, sx, sy, sz);
  const int2 id = s.tab.ids[n];
  const bool occ[2] = {id.x > 0, id.y > 0};
  int tag[2] = {occ[0] ? id.x : 0, occ[1] ? id.y : 0};
  double us[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  bool band = false;
  int seen[4];
  int nseen = 0;
  int status = 0;
  const int hx = sx + g.off[0], hy = sy + g.off[1], hz = sz + g.off[2];
  const int cell = ((sz / s.cb[2]) * s.C[1] + sy / s.cb[1]) * s.C[0] + sx / s.cb[0];
  const int off = s.cell_off[cell], cnt = s.cell_count[cell];
  for (int k = 0; k < cnt; ++k) {
    const Img& im = s.img[s.list[off + k]];
    if (!im.valid) continue;
    if (sx < im.lo[0] || sx >= im.hi[0] || sy < im.lo[1] || sy >= im.hi[1] || sz < im.lo[2] ||
        sz >= im.hi[2])
      continue;
    const double dx = (double)hx - im.xl[0];
    const double dy = (double)hy - im.xl[1];
    const double dz = (double)hz - im.xl[2];
    const double dist = dx * dx + dy * dy + dz * dz;
    const double rl = fmax(im.r - s.h0 - 2.0 * s.hl, 0.0), rh = im.r + s.h0 + 2.0 * s.hl;
    if (dist < rl * rl || dist > rh * rh) continue;
    band = true;
    const int t = im.tag;
    for (int j = 0; j < nseen; ++j)
      if (seen[j] == t) status |= STATUS_ADJ_SAME_TAG;
    if (nseen < 4) seen[nseen++] = t;
    if ((occ[0] && tag[0] == t) || (occ[1] && tag[1] == t)) continue;
    // an entering particle takes the first empty slot (setParticle, src/LBM_PSM_lattice.cpp:257-330)
    int slot = -1;
    if (tag[0] == 0 || tag[0] == t) {
      slot = 0;
    } else if (tag[1] == 0 || tag[1] == t) {
      slot = 1;
    } else {
      status |= STATUS_ADJ_CROWDED;
    }
    if (slot >= 0 && tag[slot] == 0) {
      tag[slot] = t;
      // node velocity u = uT + omega x (node - x_l) (src/LBM_PSM_exchangeParticleData.cpp:83-89)
      us[3 * slot + 0] = im.uT[0] + im.om[1] * dz - im.om[2] * dy;
      us[3 * slot + 1] = im.uT[1] + im.om[2] * dx - im.om[0] * dz;
      us[3 * slot + 2] = im.uT[2] + im.om[0] * dy - im.om[1] * dx;
    }
  }
  int cw[2] = {0, 0};
  if (tag[0] > 0 || tag[1] > 0) {
    for (int k = 0; k < cnt; ++k) {
      const Img& im = s.img[s.list[off + k]];
      if (!im.valid) continue;
      if (hx < im.rlo[0] || hx >= im.rhi[0] || hy < im.rlo[1] || hy >= im.rhi[1] ||
          hz < im.rlo[2] || hz >= im.rhi[2])
        continue;
      // the reduction's tag match: slot 1 first, then slot 2
      if (im.tag == tag[0])
        ++cw[0];
      else if (im.tag == tag[1])
        ++cw[1];
    }
  }
  s.an.band[n] = band ? 1 : 0;
  s.an.tag[n] = make_int2(tag[0], tag[1]);
  s.an.cw[n] = make_int2(cw[0], cw[1]);
  if (band)
    for (int c = 0; c < 6; ++c) s.an.us[6 * n + c] = us[c];
  if (status) atomicOr(s.status, status);
}

// calcSolidFraction (src/LBM_PSM_exchangeParticleData.cpp:116-169): the early-out
// value or the reference's sub-cell count times 1/10^dim.
__device__ __forceinline__ double eps_of(int dim, int i, int j, int k, const SphereRec& sp) {
  float dx, dy, dz;
  const int c = classify_node(i, j, k, sp, dx, dy, dz);
  if (c >= 0) return c ? 1.0 : 0.0;
  const int n = shell_count(dim, sp, i, j, k, dx, dy, dz);
  return (dim == 3 ? 1.0 / 1000.0 : 1.0 / 100.0) * small_int_to_double(n);
}

// lattice-local centre on one rank (src/LBM_PSM_exchangeParticleData.cpp:31-37)
__device__ __forceinline__ double local_centre_of(double x, double origin, double dx) {
  const double g = (x - origin) / dx;
  return g - ((0 - ((double)0 * 2.0 * (double)1)) - 1);
}

constexpr int CEN_THREADS = 128;

// Central difference of the solid fraction of an image at every surface node
// of its map box, for each axis; the adjoint contracts it with the
// accumulated dJ/dB, the tangent stores the rate along xdot.
//
// Block (i, part) takes every gridDim.y-th run of nodes of image i's box; its
// warps gather surface nodes until 32 are at hand, so that every lane counts
// (an eighth of the box lies in the shell).  Six sub-cell counts per node in
// FP32 with the exact decision of open sub-cells (solid_fraction.cuh); in FP64
// throughout, one block per image, they took 10.97 ms for 7-16 images of
// diameter 12 whatever their number.  Partial sums of an image go to
// c.part, added in order by adj_centre_sum_kernel.
__global__ void __launch_bounds__(CEN_THREADS) adj_centre_kernel(AdjCentre c) {
  constexpr int NW = CEN_THREADS / 32;
  const int i = blockIdx.x;
  const Img& im = c.img[i];
  const Geom& g = c.g;
  __shared__ SphereRec sp[6];       // the image moved by +-h along each axis
  __shared__ int q_node[NW][64], q_slot[NW][64];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double acc[3] = {0.0, 0.0, 0.0};
  if (im.valid) {
    if (threadIdx.x < 6) {
      const int a = threadIdx.x >> 1;
      SphereRec s;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        s.xl[d] = im.xl[d];
        if (d == a)
          s.xl[d] = local_centre_of((threadIdx.x & 1) ? c.x[3 * i + d] - c.h : c.x[3 * i + d] + c.h,
                                    c.origin[d], c.dx);
        split_centre(s.xl[d], s.xi[d], s.xf[d]);
      }
      s.r = im.r;
      s.rP2 = im.rP2;
      s.rM2 = im.rM2;
      s.rP2f = im.rP2f;
      s.rM2f = im.rM2f;
      s.rSqf = im.rSqf;
      sp[threadIdx.x] = s;
    }
    __syncthreads();
    const int wx = im.box[0], wy = im.box[1];
    const int vol = wx * wy * im.box[2];
    const double inv2h = 1.0 / (2.0 * c.h);
    int qn = 0;  // surface nodes at hand (warp-uniform)
    auto take = [&](int k) {  // node k of this warp's queue
      const int li = q_node[wid][k], s = q_slot[wid][k];
      const int sx = im.lo[0] + li % wx;
      const int sy = im.lo[1] + (li / wx) % wy;
      const int sz = im.lo[2] + li / (wx * wy);
      const long long n = node_index(g, sx, sy, sz);
      const int hx = sx + g.off[0], hy = sy + g.off[1], hz = sz + g.off[2];
      double de[3];
#pragma unroll 1
      for (int a = 0; a < 3; ++a) {
        const double ep = eps_of(g.dim, hx, hy, hz, sp[2 * a]);
        const double em = eps_of(g.dim, hx, hy, hz, sp[2 * a + 1]);
        de[a] = (ep - em) * inv2h;
      }
      if (c.xdot) {
        c.an.edot[2 * n + s] =
            c.xdot[3 * i] * de[0] + c.xdot[3 * i + 1] * de[1] + c.xdot[3 * i + 2] * de[2];
      } else if (de[0] != 0.0 || de[1] != 0.0 || de[2] != 0.0) {
        const uint8_t flag = c.tab.flag[n];
        int2 id = make_int2(0, 0);
        double2 e = make_double2(0.0, 0.0);
        if (flag) {
          id = c.tab.ids[n];
          e = c.tab.eps[n];
        }
        SlotWeights w;
        slot_weights(e.x, e.y, id.x > 0, id.y > 0, c.weighting, c.tau, w);
        const double chain = c.an.sigma[2 * n] * w.dBde[0][s] + c.an.sigma[2 * n + 1] * w.dBde[1][s];
#pragma unroll
        for (int a = 0; a < 3; ++a) acc[a] += chain * de[a];
      }
    };
    for (int base = (blockIdx.y * NW + wid) * 32; base < vol; base += (int)gridDim.y * CEN_THREADS) {
      const int li = base + lane;
      int s = -1;
      if (li < vol) {
        const long long n = node_index(g, im.lo[0] + li % wx, im.lo[1] + (li / wx) % wy,
                                       im.lo[2] + li / (wx * wy));
        if (c.an.band[n]) {
          const int2 et = c.an.tag[n];
          s = et.x == im.tag ? 0 : (et.y == im.tag ? 1 : -1);
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, s >= 0);
      if (s >= 0) {
        const int k = qn + __popc(m & ((1u << lane) - 1u));
        q_node[wid][k] = li;
        q_slot[wid][k] = s;
      }
      qn += __popc(m);
      __syncwarp();
      if (qn >= 32) {
        take(lane);
        __syncwarp();
        const int rn = q_node[wid][32 + lane], rs = q_slot[wid][32 + lane];
        __syncwarp();
        q_node[wid][lane] = rn;
        q_slot[wid][lane] = rs;
        qn -= 32;
        __syncwarp();
      }
    }
    if (lane < qn) take(lane);
  }
  if (c.xdot) return;
  __shared__ double red[NW][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double x = acc[a];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[wid][a] = x;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double x = 0.0;
    for (int w = 0; w < NW; ++w) x += red[w][threadIdx.x];
    c.part[3 * ((long long)i * gridDim.y + blockIdx.y) + threadIdx.x] = x;
  }
}

__global__ void adj_centre_sum_kernel(const double* part, int n3, int parts, double* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;  // 3 * image + axis
  if (k >= n3) return;
  double x = 0.0;
  for (int p = 0; p < parts; ++p) x += part[3 * ((long long)(k / 3) * parts + p) + k % 3];
  out[k] = x;
}

// total drag of one step along d, summed over the images in their order
__global__ void adj_drag_kernel(const double* fh, int n, double d0, double d1, double d2,
                                double* out) {
  double s = 0.0;
  for (int i = 0; i < n; ++i) s += d0 * fh[3 * i] + d1 * fh[3 * i + 1] + d2 * fh[3 * i + 2];
  *out = s;
}

// sum of the per-block partials, fixed order
constexpr int SUM_THREADS = 256;
__global__ void __launch_bounds__(SUM_THREADS) adj_sum_kernel(const double* part,
                                                              long long nblocks, double* out) {
  __shared__ double red[SUM_THREADS][ADJ_PART];
  double acc[ADJ_PART] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (long long b = threadIdx.x; b < nblocks; b += SUM_THREADS)
#pragma unroll
    for (int k = 0; k < ADJ_PART; ++k) acc[k] += part[b * ADJ_PART + k];
#pragma unroll
  for (int k = 0; k < ADJ_PART; ++k) red[threadIdx.x][k] = acc[k];
  __syncthreads();
  for (int s = SUM_THREADS / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
#pragma unroll
      for (int k = 0; k < ADJ_PART; ++k) red[threadIdx.x][k] += red[threadIdx.x + s][k];
    __syncthreads();
  }
  if (threadIdx.x < ADJ_PART) out[threadIdx.x] = red[0][threadIdx.x];
}

}  // namespace

long long adj_blocks(const Geom& g) {
  return ((long long)g.S[0] * g.S[1] * g.S[2] + ADJ_THREADS - 1) / ADJ_THREADS;
}

cudaError_t launch_adj_entries(const AdjSetup& s, cudaStream_t st) {
  const long long total = (long long)s.g.S[0] * s.g.S[1] * s.g.S[2];
  adj_entries_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(s);
  return cudaGetLastError();
}

cudaError_t launch_adj_step(const AdjParams& p, int tangent, cudaStream_t st) {
  const unsigned grid = (unsigned)adj_blocks(p.g);
  if (p.g.dim == 2) {
    if (tangent)
      tan_step_kernel<D2Q9><<<grid, ADJ_THREADS, 0, st>>>(p);
    else
      adj_step_kernel<D2Q9><<<grid, ADJ_THREADS, 0, st>>>(p);
  } else {
    if (tangent)
      tan_step_kernel<D3Q19><<<grid, ADJ_THREADS, 0, st>>>(p);
    else
      adj_step_kernel<D3Q19><<<grid, ADJ_THREADS, 0, st>>>(p);
  }
  return cudaGetLastError();
}

cudaError_t launch_adj_centre(const AdjCentre& c, cudaStream_t st) {
  if (c.n <= 0) return cudaSuccess;
  adj_centre_kernel<<<dim3((unsigned)c.n, ADJ_CEN_PARTS), CEN_THREADS, 0, st>>>(c);
  if (!c.xdot)
    adj_centre_sum_kernel<<<(3 * c.n + 127) / 128, 128, 0, st>>>(c.part, 3 * c.n, ADJ_CEN_PARTS, c.out);
  return cudaGetLastError();
}

cudaError_t launch_adj_drag(const double* fh, int n, double d0, double d1, double d2,
                            double* out, cudaStream_t st) {
  adj_drag_kernel<<<1, 1, 0, st>>>(fh, n, d0, d1, d2, out);
  return cudaGetLastError();
}

cudaError_t launch_adj_sum(const double* part, long long nblocks, double* out, cudaStream_t st) {
  adj_sum_kernel<<<1, SUM_THREADS, 0, st>>>(part, nblocks, out);
  return cudaGetLastError();
}

}  // namespace lbmpsm
