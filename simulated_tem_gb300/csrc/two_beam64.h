// The two-beam equations down a column (Lib_DynamicalTwoBeamImaging.f90:2316-2480) in FP64 and in fixed
// point, and the rule that chooses between them: the FP64 path's integrator (k_field64.cu).  The same
// code on the host and on the GPU.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define TB_HD __host__ __device__ __forceinline__
#else
#define TB_HD inline
#endif
#ifdef __CUDA_ARCH__
#define TB_MUL(a, b) __dmul_rn(a, b)
#define TB_ADD(a, b) __dadd_rn(a, b)
#define TB_FMA(a, b, c) __fma_rn(a, b, c)
#define TB_DIV(a, b) __ddiv_rn(a, b)
#define TB_RSQRT(a) rsqrt(a)
#else  // compiled without contraction
#define TB_MUL(a, b) ((a) * (b))
#define TB_ADD(a, b) ((a) + (b))
#define TB_FMA(a, b, c) fma(a, b, c)
#define TB_DIV(a, b) ((a) / (b))
#define TB_RSQRT(a) (1.0 / sqrt(a))
#endif

namespace stem {

// A fixed-point number as two limbs, h 2^29 + l or h 2^30 + l with 0 <= l: the product of two is three
// 32 x 32-bit multiply-adds.
struct alignas(8) Fixed {
  int h, l;
};

TB_HD long long wide(int a, int b) { return (long long)a * b; }

TB_HD int64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  int64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}

// ---- FP64

struct S64 {
  double c0, cgr, cgi;
};

// d/dz (phi_0, phi_g) of the two-beam equations (:2375-2380, 2393-2396), fused
TB_HD void deriv64(const S64& s, double ca, const double* ph, double* d) {
  d[0] = TB_FMA(-s.cgr, ph[3], TB_FMA(-s.cgi, ph[2], -TB_MUL(s.c0, ph[1])));
  d[1] = TB_FMA(-s.cgi, ph[3], TB_FMA(s.cgr, ph[2], TB_MUL(s.c0, ph[0])));
  d[2] = TB_FMA(-ca, ph[3], TB_FMA(-s.cgr, ph[1], TB_MUL(s.cgi, ph[0])));
  d[3] = TB_FMA(ca, ph[2], TB_FMA(s.cgi, ph[1], TB_MUL(s.cgr, ph[0])));
}

// One RK4 double step (:2389-2464): phi + dz/3 (k1 + 2 k2 + 2 k3 + k4), dz/3 in two parts so
// that its rounding does not add up along the column.
TB_HD void rk4_64(const S64& s0, const S64& s1, const S64& s2, double a, double dz, double dz3h, double dz3l,
                  double* ph) {
  double k1[4], k2[4], k[4], q[4];
  const double ca1 = TB_ADD(s1.c0, a);
  deriv64(s0, TB_ADD(s0.c0, a), ph, k1);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = TB_FMA(k1[i], dz, ph[i]);
  deriv64(s1, ca1, q, k2);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = TB_FMA(k2[i], dz, ph[i]);
  deriv64(s1, ca1, q, k);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    k2[i] = TB_ADD(k2[i], k[i]);
    q[i] = TB_FMA(k[i], 2.0 * dz, ph[i]);
  }
  deriv64(s2, TB_ADD(s2.c0, a), q, k);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double t = TB_FMA(2.0, k2[i], TB_ADD(k1[i], k[i]));
    ph[i] = TB_FMA(t, dz3h, TB_FMA(t, dz3l, ph[i]));
  }
}

// |phi_g|^2 of a column, its samples coef(z) = (b0 rho, bg rho x).  The equations being linear, the
// reference's renormalisation after every double step (:2466-2472) only scales phi: it is done every 8
// steps, and at the end through the quotient (every step when a step could grow phi by more than a
// small factor; `reach`: the largest |b0| + |bg| + |a|).
template <typename Coef>
TB_HD double column64(int Mz, double dz, double a, double reach, Coef coef) {
  const double dz3h = TB_DIV(dz, 3.0), dz3l = TB_DIV(TB_FMA(-3.0, dz3h, dz), 3.0);
  const int every = 2.0 * dz * reach < 1.0 ? 8 : 1;
  double ph[4] = {1.0, 0.0, 0.0, 0.0};
  S64 s0 = coef(0);
  int n = 0;
  for (int z = 2; z <= Mz; z += 2) {  // the last sample of an even column is the first (:1898-1899)
    const S64 s1 = coef(z - 1), s2 = coef(z < Mz ? z : 0);
    rk4_64(s0, s1, s2, a, dz, dz3h, dz3l, ph);
    s0 = s2;
    if (++n == every) {
      n = 0;
      const double inv =
          TB_RSQRT(TB_FMA(ph[3], ph[3], TB_FMA(ph[2], ph[2], TB_FMA(ph[1], ph[1], TB_MUL(ph[0], ph[0])))));
#pragma unroll
      for (int i = 0; i < 4; ++i) ph[i] = TB_MUL(ph[i], inv);
    }
  }
  const double ig = TB_FMA(ph[2], ph[2], TB_MUL(ph[3], ph[3]));
  return TB_DIV(ig, TB_FMA(ph[0], ph[0], TB_FMA(ph[1], ph[1], ig)));
}

// ---- fixed point, units of 2^-60

constexpr int kLimb60 = 30;

// x (|x| <= 1) in units of 2^-60, cut off
TB_HD long long to60(double x) {
  const int64_t b = bits_of(x);
  const int e = (int)(b >> 52) & 0x7FF, shift = 1023 - e;
  const long long m = (long long)(((b & ((1LL << 52) - 1)) | (1LL << 52)) << 8) >> (shift < 63 ? shift : 63);
  return b < 0 ? -m : m;
}

TB_HD Fixed split60(long long v) { return Fixed{(int)(v >> kLimb60), (int)v & ((1 << kLimb60) - 1)}; }

struct SFix {
  Fixed c0, ca, cgr, cgi, ngi;  // times dz 2^shift; ngi = -cgi
};

TB_HD SFix sfix(long long c0, long long cgr, long long cgi, long long a) {
  const Fixed gi = split60(cgi);
  return SFix{split60(c0), split60(c0 + a), split60(cgr), gi, Fixed{-gi.h, -gi.l}};
}

// (a x + b y + c z) 2^-shift, rounded (the low limbs' products, below one unit before the shift, left out)
TB_HD long long row60(const Fixed& a, const Fixed& x, const Fixed& b, const Fixed& y, const Fixed& c, const Fixed& z,
                      long long half, int shift) {
  long long hh = half, m = 0;
  hh += wide(a.h, x.h);
  hh += wide(b.h, y.h);
  hh += wide(c.h, z.h);
  m += wide(a.h, x.l);
  m += wide(a.l, x.h);
  m += wide(b.h, y.l);
  m += wide(b.l, y.h);
  m += wide(c.h, z.l);
  m += wide(c.l, z.h);
  return (hh + (m >> kLimb60)) >> shift;
}

// dz d/dz (phi_0, phi_g), as deriv64
TB_HD void deriv60(const SFix& s, const long long* v, long long half, int shift, long long* d) {
  Fixed p[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = split60(v[i]);
  d[0] = -row60(s.c0, p[1], s.cgi, p[2], s.cgr, p[3], half, shift);
  d[1] = row60(s.c0, p[0], s.cgr, p[2], s.ngi, p[3], half, shift);
  d[2] = -row60(s.ca, p[3], s.cgr, p[1], s.ngi, p[0], half, shift);
  d[3] = row60(s.ca, p[2], s.cgi, p[1], s.cgr, p[0], half, shift);
}

TB_HD void rk4_60(const SFix& s0, const SFix& s1, const SFix& s2, long long half, int shift, long long* ph) {
  long long k1[4], ks[4], k[4], q[4];
  deriv60(s0, ph, half, shift, k1);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = ph[i] + k1[i];
  deriv60(s1, q, half, shift, ks);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = ph[i] + ks[i];
  deriv60(s1, q, half, shift, k);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ks[i] += k[i];
    q[i] = ph[i] + 2 * k[i];
  }
  deriv60(s2, q, half, shift, k);
  const int third = 357913941;  // 2^60 / 3, both limbs
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const Fixed t = split60(k1[i] + k[i] + 2 * ks[i]);
    ph[i] += wide(t.h, third) + ((wide(t.h, third) + wide(t.l, third) + (3LL << (kLimb60 - 2))) >> kLimb60);
  }
}

// |phi_g|^2 of a column.  src.load(z) fetches a sample (the next double step's are loaded ahead),
// src.coef(sample) makes an SFix of it.  `weak`: the column has a field, but no |phi_g| on the way was
// 2^-kWeak: 2^-60 is then coarser than FP64 would be, and the caller takes column64.  Of random columns
// (16 to 3,000 slices, filled to 0.2 to 100 %), relative error of |phi_g|^2, root mean square: at |phi_g| 2^-2
// fixed 4.6e-16 and FP64 1.9e-15, at 2^-6 1.6e-15 and 3.0e-15, at 2^-8 3.5e-15 and 5.9e-15, at 2^-10 1.3e-14 and
// 1.6e-15, at 2^-20 1.2e-11 and 9.4e-16.
constexpr int kWeak = 6;
template <typename Src>
TB_HD double column60(int Mz, int shift, const Src& src, bool& weak) {
  const long long half = (1LL << shift) >> 1;
  long long ph[4] = {1LL << 60, 0, 0, 0};
  auto at = [&](int z) { return z < Mz ? z : 0; };
  SFix s0 = src.coef(src.load(0));
  auto x1 = src.load(at(1)), x2 = src.load(at(2));
  int most = 0;             // of the upper words of |phi_g|
  long long any = 0;
#pragma unroll 1
  for (int z = 2; z <= Mz; z += 2) {
    const SFix s1 = src.coef(x1), s2 = src.coef(x2);
    x1 = src.load(at(z + 1));
    x2 = src.load(at(z + 2));
    rk4_60(s0, s1, s2, half, shift, ph);
    s0 = s2;
    const int g2 = (int)(ph[2] >> 32), g3 = (int)(ph[3] >> 32);
    most |= (g2 ^ (g2 >> 31)) | (g3 ^ (g3 >> 31));
    any |= ph[2] | ph[3];
  }
  weak = any != 0 && most < 1 << (60 - 32 - kWeak);
  double v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (double)ph[i];
  const double ig = TB_FMA(v[2], v[2], TB_MUL(v[3], v[3]));
  return TB_DIV(ig, TB_FMA(v[0], v[0], TB_FMA(v[1], v[1], ig)));
}

// Whether an image's columns run in fixed point, and dz times 1, b0 and bg times 2^shift (shift < 0: FP64).
// Where it is no less precise than FP64: the double steps are short (no intermediate exceeds 1.3; a step
// loses less than 4e-6 of the norm, which the quotient at the end restores), and |phi_g| is not
// small against 1 in a full column, neither by a weak reflection (|phi_g| up to the thickness times bg) nor by
// excitation errors (up to bg / a).  The coefficients are scaled up, by the largest of them, to use their
// limbs; b0 far above bg leaves bg fewer bits, but costs FP64 more (b0 / bg of 300 to 3,000, 2,000 to 30,000 slices:
// 2e-15 and 6e-14).
struct FixedRule {
  int shift = -1;
  double a = 0.0, b0 = 0.0, bg = 0.0;
};
inline FixedRule fixed_rule(double dz, double b0, double bg, int Mz, const double* aa, int n_prec) {
  FixedRule r;
  double a = 0.0;
  for (int k = 0; k < n_prec; ++k) {
    if (!isfinite(aa[k])) return r;
    a = fmax(a, fabs(aa[k]));
  }
  const double c0 = fabs(b0), cg = fabs(bg);
  if (!(dz > 0.0) || !(2.0 * dz * (c0 + cg + a) <= 0.25) || !(cg * 32.0 >= a) ||
      !(Mz * dz * cg >= 1.0 / 16.0) || Mz > 50000)
    return r;
  int e = 0;
  frexp(dz * fmax(c0 + a, cg), &e);  // below 2^e <= 1/4
  if (e < -24) return r;
  r.shift = -e;
  r.a = ldexp(dz, -e);
  r.b0 = b0 * r.a;
  r.bg = bg * r.a;
  return r;
}

}  // namespace stem
