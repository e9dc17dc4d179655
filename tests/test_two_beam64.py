"""The FP64 path's two integrators (two_beam64.h, here on the host) against extended precision: fixed point is
taken only where it is no less precise than FP64, by the rule on the image and by each column's amplitude."""
from tests.test_field_plan import run

COMMON = r"""
#include "two_beam64.h"
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
using namespace stem;
typedef long double Real;
struct Sample { double x, y, rho; };
#define CHECK(c) do { if (!(c)) { std::printf("line %d: " #c "\n", __LINE__); return 1; } } while (0)
"""

COLUMNS = COMMON + r"""
Real exact(const std::vector<Sample>& s, double b0, double bg, double dz, double a) {
  const int Mz = (int)s.size();
  Real p[4] = {1, 0, 0, 0};
  auto deriv = [&](int z, const Real* q, Real* d) {
    const Sample& v = s[z < Mz ? z : 0];
    const Real c0 = (Real)b0 * v.rho, cr = (Real)bg * v.rho * v.x, ci = (Real)bg * v.rho * v.y, ca = c0 + a;
    d[0] = -(c0 * q[1] + ci * q[2] + cr * q[3]);
    d[1] = c0 * q[0] + cr * q[2] - ci * q[3];
    d[2] = -(ca * q[3] + cr * q[1] - ci * q[0]);
    d[3] = ca * q[2] + ci * q[1] + cr * q[0];
  };
  for (int z = 2; z <= Mz; z += 2) {
    Real k[4][4], q[4];
    deriv(z - 2, p, k[0]);
    for (int i = 0; i < 4; ++i) q[i] = p[i] + dz * k[0][i];
    deriv(z - 1, q, k[1]);
    for (int i = 0; i < 4; ++i) q[i] = p[i] + dz * k[1][i];
    deriv(z - 1, q, k[2]);
    for (int i = 0; i < 4; ++i) q[i] = p[i] + 2 * (Real)dz * k[2][i];
    deriv(z, q, k[3]);
    for (int i = 0; i < 4; ++i) p[i] += (Real)dz / 3 * (k[0][i] + 2 * k[1][i] + 2 * k[2][i] + k[3][i]);
  }
  const Real g = p[2] * p[2] + p[3] * p[3];
  return g / (g + p[0] * p[0] + p[1] * p[1]);
}
struct Source {
  const std::vector<Sample>& s;
  const FixedRule& R;
  long long a;
  struct Raw { double x, y, r; };
  Raw load(int z) const { return Raw{s[z].x * R.bg * s[z].rho, s[z].y * R.bg * s[z].rho, s[z].rho * R.b0}; }
  SFix coef(const Raw& q) const { return sfix(to60(q.r), to60(q.x), to60(q.y), a); }
};
int main() {
  std::mt19937_64 rng(1);
  auto U = [&](double lo, double hi) { return lo + (hi - lo) * (double)(rng() >> 11) * 0x1p-53; };
  double sum[2] = {0, 0}, strong = 0, weak_seen = 0;
  for (int t = 0; t < 6000; ++t) {
    const int Mz = (int)std::exp(U(std::log(16), std::log(3000)));
    const double bg = std::exp(U(std::log(1e-3), std::log(3e-2))), b0 = bg * std::exp(U(std::log(.1), std::log(300)));
    const double a = bg * U(-10, 10), dz = U(.3, 1.4);
    const FixedRule R = fixed_rule(dz, b0, bg, Mz, &a, 1);
    if (R.shift < 0) continue;
    const bool dens = rng() & 1;
    const double fill = std::exp(U(std::log(.002), 0)), amp = dens ? std::exp(U(std::log(1e-5), 0)) : 1;
    const int lo = (int)(U(0, 1 - fill) * Mz), hi = lo + (int)std::ceil(fill * Mz);
    std::vector<Sample> s(Mz);
    for (int z = 0; z < Mz; ++z) {
      const double ph = U(-.3, .3);
      const bool in = z >= lo && z < hi;
      s[z] = Sample{in ? std::cos(ph) : 0, in ? std::sin(ph) : 0, dens ? (in ? amp * U(.5, 1) : 0) : 1};
    }
    bool weak;
    const double f = column60(Mz, R.shift, Source{s, R, to60(a * R.a)}, weak);
    const double d = column64(Mz, dz, a, std::fabs(b0) + bg + std::fabs(a),
                              [&](int z) { return S64{b0 * s[z].rho, s[z].rho * s[z].x * bg, s[z].rho * s[z].y * bg}; });
    const Real e = exact(s, b0, bg, dz, a);
    CHECK(e > 0);
    if (weak) {
      CHECK(e < 0x1p-11);  // both parts below 2^-6
      ++weak_seen;
      continue;
    }
    const double ef = (double)((f - e) / e), ed = (double)((d - e) / e);
    sum[0] += ef * ef;
    sum[1] += ed * ed;
    ++strong;
  }
  CHECK(strong > 500 && weak_seen > 500);
  CHECK(sum[0] <= sum[1]);  // no less precise than FP64
  // a column without a field is exactly zero, and not weak
  std::vector<Sample> none(100, Sample{0, 0, 1});
  const double a = 0.02;
  const FixedRule R = fixed_rule(0.7, 0.03, 0.015, 100, &a, 1);
  bool weak = true;
  CHECK(R.shift >= 0 && column60(100, R.shift, Source{none, R, to60(a * R.a)}, weak) == 0.0 && !weak);
  std::puts("ok");
  return 0;
}
"""

RULE = COMMON + r"""
int main() {
  // just inside and just outside each condition
  auto shift = [](double dz, double b0, double bg, int Mz, double a) { return fixed_rule(dz, b0, bg, Mz, &a, 1).shift; };
  const double up = 1 + 1e-12, dn = 1 - 1e-12;
  CHECK(shift(0.5, 0.1, 0.1, 1000, 0.05 * dn) >= 0 && shift(0.5, 0.1, 0.1, 1000, 0.05 * up) < 0);   // step length
  CHECK(shift(0.5, 0.001, 0.001, 1000, 0.032 * dn) >= 0 && shift(0.5, 0.001, 0.001, 1000, -0.032 * up) < 0);
  CHECK(shift(0.5, 0.001, 0.00125 * up, 100, 0.0) >= 0 && shift(0.5, 0.001, 0.00125 * dn, 100, 0.0) < 0);  // thickness
  CHECK(shift(0.5, 0.01, 0.01, 50000, 0.0) >= 0 && shift(0.5, 0.01, 0.01, 50001, 0.0) < 0);
  CHECK(shift(0.5, 0.01, 0.01, 100, NAN) < 0 && shift(0.5, NAN, 0.01, 100, 0.0) < 0 && shift(0.5, 0.01, NAN, 100, 0.0) < 0);
  const double two[2] = {0.0, 0.16};
  CHECK(fixed_rule(0.5, 0.1, 0.1, 1000, two, 1).shift >= 0 && fixed_rule(0.5, 0.1, 0.1, 1000, two, 2).shift < 0);
  std::puts("ok");
  return 0;
}
"""


def test_fixed_point_is_no_less_precise(tmp_path):
    run(tmp_path, COLUMNS)


def test_both_sides_of_the_rule(tmp_path):
    run(tmp_path, RULE)
