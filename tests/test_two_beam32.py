"""The FP32 integration step (two_beam32.h, here on the host) against extended precision and against a step that adds
its four parts to phi one by one."""
from tests.test_field_plan import run

STEP = r"""
#include "two_beam32.h"
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
using namespace stem::field32;
typedef long double Real;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: " #c "\n", __LINE__); return 1; } } while (0)
template <typename D>
void four_parts(const Sample& s0, const Sample& s1, const Sample& s2, float a, float dz, float* ph, D deriv_of) {
  float d[4], p1[4], q[4];
  const float third = dz / 3.f, thirds = 2.f * dz / 3.f;
  deriv_of(s0, a, ph, d);
  for (int i = 0; i < 4; ++i) { p1[i] = fmaf(d[i], third, ph[i]); q[i] = fmaf(d[i], dz, ph[i]); }
  deriv_of(s1, a, q, d);
  for (int i = 0; i < 4; ++i) { q[i] = fmaf(d[i], dz, ph[i]); p1[i] = fmaf(d[i], thirds, p1[i]); }
  deriv_of(s1, a, q, d);
  for (int i = 0; i < 4; ++i) { q[i] = fmaf(d[i], 2.f * dz, ph[i]); p1[i] = fmaf(d[i], thirds, p1[i]); }
  deriv_of(s2, a, q, d);
  for (int i = 0; i < 4; ++i) ph[i] = fmaf(d[i], third, p1[i]);
}
// the same in extended precision; dz / 3 as the FP32 steps have it
void exact(const Sample& s0, const Sample& s1, const Sample& s2, Real a, float dz, Real* p) {
  auto deriv_of = [&](const Sample& s, const Real* q, Real* d) {
    const Real c0 = s.c0, cr = s.cgr, ci = s.cgi, ca = c0 + a;
    d[0] = -(c0 * q[1] + ci * q[2] + cr * q[3]);
    d[1] = c0 * q[0] + cr * q[2] - ci * q[3];
    d[2] = -(ca * q[3] + cr * q[1] - ci * q[0]);
    d[3] = ca * q[2] + ci * q[1] + cr * q[0];
  };
  Real k[4][4], q[4];
  deriv_of(s0, p, k[0]);
  for (int i = 0; i < 4; ++i) q[i] = p[i] + dz * k[0][i];
  deriv_of(s1, q, k[1]);
  for (int i = 0; i < 4; ++i) q[i] = p[i] + dz * k[1][i];
  deriv_of(s1, q, k[2]);
  for (int i = 0; i < 4; ++i) q[i] = p[i] + 2 * (Real)dz * k[2][i];
  deriv_of(s2, q, k[3]);
  for (int i = 0; i < 4; ++i) p[i] += (Real)(dz / 3.f) * (k[0][i] + 2 * (k[1][i] + k[2][i]) + k[3][i]);
}
int main() {
  std::mt19937_64 rng(2);
  auto U = [&](double lo, double hi) { return lo + (hi - lo) * (double)(rng() >> 11) * 0x1p-53; };
  double one = 0, four = 0;
  for (int t = 0; t < 2000; ++t) {
    const int steps = 100;
    const float bg = (float)U(.01, .03), b0 = (float)U(.01, .04), a = (float)U(-.02, .02), dz = .7f;
    std::vector<Sample> s(2 * steps + 1);
    for (Sample& v : s) { const double f = U(-.3, .3); v = Sample{b0, (float)(bg * std::cos(f)), (float)(bg * std::sin(f))}; }
    float x[4] = {1, 0, 0, 0}, y[4] = {1, 0, 0, 0};
    Real e[4] = {1, 0, 0, 0};
    for (int k = 0; k < steps; ++k) {
      rk4<float>(s[2 * k], s[2 * k + 1], s[2 * k + 2], a, dz, x);
      four_parts(s[2 * k], s[2 * k + 1], s[2 * k + 2], a, dz, y, deriv<float>);
      exact(s[2 * k], s[2 * k + 1], s[2 * k + 2], a, dz, e);
    }
    for (int i = 0; i < 4; ++i) {
      one += (double)((x[i] - e[i]) * (x[i] - e[i]));
      four += (double)((y[i] - e[i]) * (y[i] - e[i]));
    }
  }
  std::printf("rms %.2e %.2e\n", std::sqrt(one / 8000), std::sqrt(four / 8000));
  // phi is rounded once instead of four times a step: half the error, with room for the derivatives' own rounding
  CHECK(std::sqrt(one) <= 0.75 * std::sqrt(four));
  std::puts("ok");
  return 0;
}
"""


def test_a_step_rounds_phi_once(tmp_path):
    run(tmp_path, STEP)
