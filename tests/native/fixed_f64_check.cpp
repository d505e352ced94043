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
  long bad = 0;
  for (long it = 0; it < n; ++it) {
    const double mag = it % 7 == 0 ? 0.0 : std::exp2(-uni(0, 70)), lim = 0.078125;
    double u[3] = {uni(-lim, lim) * (it % 3 ? 1 : mag), uni(-lim, lim) * (it % 5 ? 1 : mag), uni(-lim, lim) * mag};
    if (it % 11 == 0) u[0] = std::ldexp((double)((int)(gen() % 129) - 64), -11 - (int)(gen() % 40));
    if (it % 101 == 0) u[0] = std::ldexp(u[0], -1000 - (int)(gen() % 60));
    if (!fx::slow(u[0]) || !fx::slow(u[1])) continue;
    const double eu = it % 2 ? u[0] + u[1] : u[0], a = eu * 3.0, b = eu * eu * 4.5;
    const double uu = 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]) * 3.0;
    volatile double p = 1.0 + a, m = 1.0 - a, o = 1.0 - uu;
    p = p + b;
    p = p - uu;
    m = m + b;
    m = m - uu;
    double P, M;
    const fx::u64 u62 = fx::align62(uu);
    fx::factors(a, b, u62, P, M);
    if (P != p || M != m || fx::one_minus(u62) != o) ++bad;
  }
  std::printf("factors in_range 1.000 different %ld\n", bad);
}

int main() {
  sums<D3>("D3Q19", 1000000);
  sums<D2>("D2Q9", 1000000);
  factors(4000000);
  return 0;
}
