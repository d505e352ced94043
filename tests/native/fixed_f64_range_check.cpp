// The lowest densities that macro_sums of fixed_f64.cuh lets through, and the
// equilibria and differences there, at the largest velocities: against IEEE
// double arithmetic.  Prints per lattice the lowest density seen, the lowest
// equilibrium and the number of differences.
#include <algorithm>
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
  static constexpr int Q = 19, FIRST = 5;  // populations whose sum is 1/2 at least
  static int ex(int q) { return E19[q][0]; }
  static int ey(int q) { return E19[q][1]; }
  static int ez(int q) { return E19[q][2]; }
  static constexpr double w[3] = {1.0 / 3, 1.0 / 18, 1.0 / 36};
};
struct D2 {
  static constexpr int Q = 9, FIRST = 2;
  static int ex(int q) { return E9[q][0]; }
  static int ey(int q) { return E9[q][1]; }
  static int ez(int q) { return E9[q][2]; }
  static constexpr double w[3] = {4.0 / 9, 1.0 / 9, 1.0 / 36};
};

static std::mt19937_64 gen(20261206);
static double uni(double a, double b) { return a + (b - a) * (double)(gen() >> 11) * 0x1p-53; }

template <class L>
static void range(const char* name, long n) {
  constexpr double LOW = 0.5 + (L::Q - L::FIRST) * 0x1p-7;  // the bound the header states
  long bad = 0;
  double least = 2.0, least_eq = 2.0;
  for (long it = 0; it < n; ++it) {
    // states at the border: the first populations sum to about 1/2, the others
    // are about 2^-7
    double f[19], part = 0.0;
    const double near = std::exp2(-uni(3, 50));
    for (int q = 0; q < L::Q; ++q) f[q] = 0x1p-7 * (1 + near * uni(it % 2 ? 0 : -0.2, 1));
    for (int q = 1; q < L::FIRST; ++q) f[q] = uni(0.02, 0.03);
    if (L::Q == 19) f[1] = 0.25 - (f[0] = uni(0.2, 0.24)) + 0.15;
    for (int q = 1; q < L::FIRST; ++q) part += f[q];
    f[0] = 0.5 * (1 + near * uni(it % 2 ? 0 : -0.2, 1)) - part;
    double rho, j[3];
    if (fx::macro_sums<L>(f, rho, j)) {
      least = std::min(least, rho);
      if (rho < LOW) ++bad;
    }
    // the equilibria at the lowest densities and the largest velocities
    const double r = it % 3 ? LOW * (1 + near * uni(0, 1)) : LOW;
    const double lim = std::nextafter(0x5p-6, 0.0);
    double u[3];
    for (double& c : u) c = (gen() & 1 ? 1 : -1) * (it % 5 ? lim * (1 - near * uni(0, 1)) : lim);
    if (!fx::slow(u[0]) || !fx::slow(u[1]) || !fx::slow(u[2])) ++bad;
    const double eu = it % 4 == 0 ? u[0] : u[0] + u[1], ee = eu * eu;
    const double a = eu * 3.0, b = ee * 4.5, vv = u[0] * u[0] + u[1] * u[1] + u[2] * u[2], uu = 0.5 * vv * 3.0;
    const double rw = r * L::w[it % 4 == 0 ? 1 : 2];
    const double fe[2] = {rw * ((1.0 + a) + b - uu), rw * ((1.0 - a) + b - uu)};
    fx::u64 P, M;
    fx::factors(eu, ee, fx::times62<3, 1>(vv), P, M);
    const fx::u64 F[2] = {P, M}, r64 = fx::to64(rw);
    for (int k = 0; k < 2; ++k) {
      least_eq = std::min(least_eq, fe[k]);
      const double fi = it % 3 == 0 ? 0x1p-7 : std::max(0x1p-7, fe[k] * (1 + near * uni(-1, 1)));
      const fx::u64 e = fx::product62(r64, F[k]);
      if (e % 8 != 0 || fx::difference62(e, 0) != fe[k] || fx::difference62(e, fx::to62(fi)) != fe[k] - fi) ++bad;
    }
  }
  std::printf("%s least_density %.7f least_equilibrium %.6f different %ld\n", name, least, least_eq, bad);
}

int main() {
  range<D3>("D3Q19", 2000000);
  range<D2>("D2Q9", 2000000);
  return 0;
}
