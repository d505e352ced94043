// Compares the integer additions of fixed_f64.cuh with IEEE double arithmetic
// on random near-rest nodes; prints the number of differences per check.
#include <cmath>
#include <cstdio>
#include <random>

#include "fixed_f64.cuh"

using namespace lbmpsm;

static const int E19[19][3] = {{0, 0, 0}, {1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1},
                               {1, 1, 0}, {-1, -1, 0}, {1, 0, 1}, {-1, 0, -1}, {0, 1, 1}, {0, -1, -1},
                               {1, -1, 0}, {-1, 1, 0}, {1, 0, -1}, {-1, 0, 1}, {0, 1, -1}, {0, -1, 1}};
static const int E9[9][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {-1, 0, 0}, {0, -1, 0}, {1, 1, 0}, {-1, 1, 0},
                             {-1, -1, 0}, {1, -1, 0}};
struct D3 {
  static constexpr int Q = 19;
  static int e(int q, int a) { return E19[q][a]; }
  static int ex(int q) { return e(q, 0); }
  static int ey(int q) { return e(q, 1); }
  static int ez(int q) { return e(q, 2); }
  static double w(int q) { return q == 0 ? 1.0 / 3 : (q <= 6 ? 1.0 / 18 : 1.0 / 36); }
};
struct D2 {
  static constexpr int Q = 9;
  static int e(int q, int a) { return E9[q][a]; }
  static int ex(int q) { return e(q, 0); }
  static int ey(int q) { return e(q, 1); }
  static int ez(int q) { return e(q, 2); }
  static double w(int q) { return q == 0 ? 4.0 / 9 : (q <= 4 ? 1.0 / 9 : 1.0 / 36); }
};

static std::mt19937_64 gen(20261205);
static double uni(double a, double b) { return a + (b - a) * (double)(gen() >> 11) * 0x1p-53; }

template <class L>
static void sums(const char* name, long n) {
  long ok = 0, bad = 0;
  for (long it = 0; it < n; ++it) {
    const double um = std::pow(10.0, -uni(0.9, 6)), nm = it % 4 ? std::pow(10.0, -uni(1.5, 8)) : 0.0;
    const double u[3] = {uni(-um, um), uni(-um, um), L::Q == 9 ? 0.0 : uni(-um, um)};
    const double uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
    const double rho = it % 17 == 0 ? 1.0 : 1.0 + uni(-0.09, 0.3) * (it % 3 ? 0.1 : 1.0);
    double f[19];
    for (int q = 0; q < L::Q; ++q) {
      const double eu = L::ex(q) * u[0] + L::ey(q) * u[1] + L::ez(q) * u[2];
      f[q] = L::w(q) * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * uu) * (1 + uni(-nm, nm));
      if (it % 5 == 0) f[q] = std::ldexp(std::rint(std::ldexp(f[q], 56)), -56);  // many ties
      if (it % 19 == 0) f[q] = L::w(q);
    }
    if (it % 1001 == 0) f[it % L::Q] = it % 2 ? NAN : (it % 3 ? -f[0] : INFINITY);
    volatile double r = 0.0;
    for (int q = 0; q < L::Q; ++q) r = r + f[q];
    double J[3];
    for (int a = 0; a < 3; ++a) {
      volatile double s = 0.0;
      for (int q = 0; q < L::Q; ++q)
        if (L::e(q, a)) s = L::e(q, a) > 0 ? s + f[q] : s - f[q];
      J[a] = s;
    }
    double R, j[3];
    if (!fx::macro_sums<L>(f, R, j)) continue;
    ++ok;
    if (!(R == r) || !(j[0] == J[0]) || !(j[1] == J[1]) || !(j[2] == J[2])) ++bad;
  }
  std::printf("%s in_range %.3f different %ld\n", name, (double)ok / n, bad);
}

static void factors(long n) {
  long bad = 0, done = 0;
  for (long it = 0; it < n; ++it) {
    const double mag = it % 7 == 0 ? 0.0 : std::exp2(-uni(0, 70)), lim = 0.078125;
    double u[3] = {uni(-lim, lim) * (it % 3 ? 1 : mag), uni(-lim, lim) * (it % 5 ? 1 : mag), uni(-lim, lim) * mag};
    if (it % 11 == 0) u[0] = std::ldexp((double)((int)(gen() % 129) - 64), -11 - (int)(gen() % 40));
    if (it % 101 == 0) u[0] = std::ldexp(u[0], -1000 - (int)(gen() % 60));
    if (!fx::slow(u[0]) || !fx::slow(u[1])) continue;
    const double eu = it % 2 ? u[0] + u[1] : u[0], a = eu * 3.0, ee = eu * eu, b = ee * 4.5;
    const double vv = u[0] * u[0] + u[1] * u[1] + u[2] * u[2], uu = 0.5 * vv * 3.0;
    volatile double p = 1.0 + a, m = 1.0 - a, o = 1.0 - uu;
    p = p + b;
    p = p - uu;
    m = m + b;
    m = m - uu;
    // the equilibria and their differences from populations
    const double w[4] = {1.0 / 3, 1.0 / 18, 1.0 / 36, 4.0 / 9};
    const double rho = it % 13 == 0 ? 1.0 : uni(0.62, 1.9), rw = rho * w[it % 4];
    volatile double fe[3] = {rw * p, rw * m, rw * o};
    double fi = it % 3 ? fe[it % 3] * (1 + uni(-1, 1) * std::exp2(-uni(1, 50))) : uni(0.0079, 0.99);
    if (it % 23 == 0) fi = fe[it % 3];
    if (!(fi >= 0x1p-7 && fi < 1.0)) continue;
    ++done;
    volatile double d[3] = {fe[0] - fi, fe[1] - fi, fe[2] - fi};
    fx::u64 P, M;
    const fx::u64 u62 = fx::times62<3, 1>(vv), r64 = fx::to64(rw), f62 = fx::to62(fi), zero = 0;
    fx::factors(eu, ee, u62, P, M);
    const fx::u64 F[3] = {P, M, fx::one_minus(u62)};
    if (fx::difference62(P, zero) != p || fx::difference62(M, zero) != m || fx::difference62(F[2], zero) != o) ++bad;
    for (int k = 0; k < 3; ++k) {
      const fx::u64 e = fx::product62(r64, F[k]);
      if (fx::difference62(e, zero) != fe[k] || fx::difference62(e, f62) != d[k]) ++bad;
      if (std::signbit(fx::difference62(e, f62)) != std::signbit(d[k])) ++bad;
    }
  }
  std::printf("factors in_range %.3f different %ld\n", (double)done / n, bad);
}

int main() {
  sums<D3>("D3Q19", 1000000);
  sums<D2>("D2Q9", 1000000);
  factors(4000000);
  return 0;
}
