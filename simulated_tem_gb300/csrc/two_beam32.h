// The two-beam equations down a column (Lib_DynamicalTwoBeamImaging.f90:2316-2480) in FP32: one RK4 double step
// (k_field32.cu; the form for one angle also on the host).
#pragma once

#include <math.h>

#include "two_beam64.h"

namespace stem {
namespace field32 {

// The RK4 double step in explicitly rounded operations, on one precession angle
// (float) or two (float2: .x angle k, .y angle k + 1, one FP32x2 instruction per
// operation).  Both forms round every operation the same way, so an angle's result
// does not depend on how many angles share a thread.
#ifdef __CUDA_ARCH__
TB_HD float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
TB_HD float mul_(float a, float b) { return __fmul_rn(a, b); }
TB_HD float add_(float a, float b) { return __fadd_rn(a, b); }
TB_HD float rsq_(float a) { return rsqrtf(a); }
#else
TB_HD float fma_(float a, float b, float c) { return fmaf(a, b, c); }
TB_HD float mul_(float a, float b) { return a * b; }
TB_HD float add_(float a, float b) { return a + b; }
TB_HD float rsq_(float a) { return 1.f / sqrtf(a); }
#endif
TB_HD float neg_(float a) { return -a; }
template <typename T>
TB_HD T bc(float v);
template <>
TB_HD float bc<float>(float v) { return v; }
#ifdef __CUDACC__
__device__ __forceinline__ float2 fma_(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul_(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add_(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 neg_(float2 a) { return make_float2(-a.x, -a.y); }
template <>
__device__ __forceinline__ float2 bc<float2>(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 rsq_(float2 a) { return make_float2(rsqrtf(a.x), rsqrtf(a.y)); }
#endif

struct Sample {
  float c0, cgr, cgi;
};

// d/dz (phi_0, phi_g) of the reference's two-beam equations (:2375-2380), phases as
// (Re phi_0, Im phi_0, Re phi_g, Im phi_g)
template <typename T>
TB_HD void deriv(const Sample& s, T a, const T* ph, T* d) {
  const T c0 = bc<T>(s.c0), cgr = bc<T>(s.cgr), cgi = bc<T>(s.cgi), ca = add_(c0, a);
  d[0] = fma_(neg_(cgr), ph[3], fma_(neg_(cgi), ph[2], mul_(neg_(c0), ph[1])));
  d[1] = fma_(neg_(cgi), ph[3], fma_(cgr, ph[2], mul_(c0, ph[0])));
  d[2] = fma_(neg_(ca), ph[3], fma_(neg_(cgr), ph[1], mul_(cgi, ph[0])));
  d[3] = fma_(ca, ph[2], fma_(cgi, ph[1], mul_(cgr, ph[0])));
}

// One RK4 double step over samples (z-2, z-1, z): phi + dz/3 (k1 + 2 k2 + 2 k3 + k4) (:2389-2464), added to phi
// at once, so that a step rounds phi once (its four parts added one by one had twice the error).
template <typename T>
TB_HD void rk4(const Sample& s0, const Sample& s1, const Sample& s2, T a, float dzf, T* ph) {
  T k1[4], s[4], d[4], q[4];
  const T dz = bc<T>(dzf), dz3 = bc<T>(dzf / 3.f), dz2 = bc<T>(2.f * dzf);
  deriv(s0, a, ph, k1);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = fma_(k1[i], dz, ph[i]);
  deriv(s1, a, q, s);
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = fma_(s[i], dz, ph[i]);
  deriv(s1, a, q, d);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    s[i] = add_(s[i], d[i]);
    q[i] = fma_(d[i], dz2, ph[i]);
  }
  deriv(s2, a, q, d);
#pragma unroll
  for (int i = 0; i < 4; ++i) ph[i] = fma_(fma_(bc<T>(2.f), s[i], add_(k1[i], d[i])), dz3, ph[i]);
}

template <typename T>
TB_HD void renormalise(T* ph) {
  const T inv = rsq_(fma_(ph[3], ph[3], fma_(ph[2], ph[2], fma_(ph[1], ph[1], mul_(ph[0], ph[0])))));
#pragma unroll
  for (int i = 0; i < 4; ++i) ph[i] = mul_(ph[i], inv);
}

}  // namespace field32
}  // namespace stem
