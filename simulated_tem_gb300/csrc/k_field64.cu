// K2+K3, FP64: the voxel field of the plain FP64 path on the slab ring, and its column
// integrator.
//
// The pixel loop of computeD2BI_img (Lib_DynamicalTwoBeamImaging.f90:1870-1900) with the
// neighbour search of Lib_LinkCell3D.f90:1515-1605 (k_field64) and the integrator of
// :2316-2480 (k_integrate64).  The field samples of a column pass through device memory
// (16 bytes a voxel), so that the field kernel splits a column's depth over warps (an image
// of a few hundred patches still fills the GPU) and is computed once however many precession
// angles integrate over it.
//
// The field kernel: one warp per 8 x 4 pixel columns and range of slices, four slices per
// step (two where some image's steps of four do not fit the ring), the atoms of the link-cell
// slabs staged in warp-private shared memory and ordered by z bin (slab_ring.cuh).
//
// The FP64 pipe takes one warp instruction per 76 cycles and SM sub-partition (measured;
// predicated-off lanes, fully predicated-off instructions and FP64 <-> FP32 conversions cost the
// same), against 2 for an FP32 or integer instruction and 4 for a 32 x 32 -> 64-bit multiply-add,
// which run beside it.  So FP64 is spent only where the result needs it, and sums and products of
// bounded numbers are fixed-point:
// * The accept decision is the reference's, d.d <= (3 sigma)^2 in its rounded operations
//   (d_a = a_aa (f_a + (k_a - zi_frac_a)), the fractions f of the FP64 binning, the unwrapped
//   27-cell offsets k).  An FP32 distance decides every pair further than kGuard64 from the
//   cutoff; the others (2 % of the warp's atoms have one) are decided in FP64, so the accepted
//   set equals the reference's.
// * The weight is a product of three Gaussians, one per axis: exp(-d_x^2 / 2 sigma^2) depends on
//   the atom and one of the patch's 8 columns, the y factor on one of its 4 rows, the z factor
//   (times the phasor) on the slice.  The warp evaluates the values that an accepting lane needs
//   as one flat list of tasks over its lanes instead of one exp per lane.
// * The Gaussian itself is a table value times a short polynomial (gauss64): six FP64 operations
//   for the distance, the rest integers.
// * A lane then multiplies two 58-bit numbers per atom, and adds two products per slice, six
//   32 x 32-bit multiply-adds.  The sums do not round.  (FP64's spacing of an accepted weight, exp(-4.5) to 1,
//   is 2^-59 to 2^-53: 2^-58 is finer but for the smallest weights.)
// Now latency bounds it (12 warps per SM, limited by their staging; 0.45 instructions per cycle and
// sub-partition), and code size: with two copies of the consuming code, or two atoms per iteration, the
// instruction fetches cost 128k atoms with density a fifth.
// Measured (GB300, whole calls): 128k atoms with density 29.0 ms with one exp, the divisions of the
// reference's integrator and hypot in every lane, 7.2 with all of this in FP64, 4.35 now; 28k atoms
// 6.75, 0.83, 0.54; 16k atoms with six precession angles 13.6, 1.32, 0.71.  128k atoms: field 3.95 ms
// (a third of it the sums, a fifth the tests and the density's nearest atoms, a fifth the Gaussians),
// integrator 0.21.
//
// Precision: the Gaussians are within 2.4 units of 2^-53 of the exact value (root mean square 0.57;
// exp of the rounded d.d / 2 sigma^2, up to 4.5, is within 13.5, 2.1 in the mean square: the rounding of
// its argument).  Images against a 64-bit evaluation of the same sums: relative 2-norm 0.3 to 1.0e-15
// (before 0.5 to 1.6e-15).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "internal.h"
#include "slab_ring.cuh"
#include "two_beam64.h"

namespace stem {
namespace field64 {

using slab::Geo;
using slab::kBins;
using slab::kRing;
using slab::load_slab;

constexpr int kWarps = 4;
// Scaled r^2 (cutoff 6.49): the FP32 distance decides outside this distance of the cutoff.  Its
// error is below 8e-4 for the images that the host sends here (field64_eligible).
constexpr float kGuard64 = 1e-3f;

// A number in [-1, 1] in units of 2^-58, as two limbs of 29 bits.
constexpr int kLimb = 29, kLow = (1 << kLimb) - 1;
constexpr int kPass = 32;         // atoms per pass over the lanes
constexpr int kN = 64;            // step buffer: flushed at 32, before a round of 32 may add more
constexpr float kOff = -1e30f;    // hmax of a slice the slab does not serve

#define DM __dmul_rn
#define DA __dadd_rn
#define DS __dsub_rn
#define DF __fma_rn

template <int CAPS, int SL>
struct WarpSmem {
  static_assert(CAPS % 32 == 0, "the z sort holds CAPS / 32 atoms per lane");
  float4 p[kRing][CAPS];  // X', Y', z (scaled FP32), cell code
  int gi[kRing][CAPS];    // index of the kept atom
  int bin[kRing][kBins + 1];
  int count[kRing];
  alignas(16) float hm[kN][SL];  // per slice: the largest accepted in-plane r^2 (FP32, scaled)
  alignas(16) unsigned m[kPass][SL];  // of the pass's atoms, per slice: the lanes that accept
  int sel[kPass];         // their places in the step buffer
  float2 xy[kN];          // X', Y'
  int2 ref[kN];           // kept atom, cell code | slab number within the step << 16 | place in the slab << 18
  Fixed exy[kPass][12];   // the patch's 8 column and 4 row factors of the Gaussian
  int4 be[SL][kPass];     // per slice: z factor times (cos, sin); before that, the list of exy's tasks
  double off[12][3];      // k - zi_frac of the patch's columns and rows, k = -1, 0, 1
  double zoff[kRing][SL]; // the same for the step's slices, per slab
  float cx[12];           // X' of the columns, Y' of the rows
  int hc[12];             // their home cells in the atoms' cell code
};

__device__ __forceinline__ Fixed split58(long long v) { return Fixed{(int)(v >> kLimb), (int)v & kLow}; }

// A product of two fixed-point numbers.  The low limbs' product, 0 to 1 units, counts as a quarter.
__device__ __forceinline__ long long mul58(const Fixed& a, const Fixed& b) {
  return wide(a.h, b.h) + ((wide(a.h, b.l) + wide(a.l, b.h) + (3LL << (kLimb - 2))) >> kLimb);
}

// x (|x| <= 1) in units of 2^-58, cut off
__device__ __forceinline__ long long to58(double x) {
  const long long b = __double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7FF;
  const long long m = (((b & ((1LL << 52) - 1)) | (1LL << 52)) << 6) >> min(63, 1023 - e);
  return b < 0 ? -m : m;
}

// exp(-d^2 / 2 sigma^2) for d >= 0 in units of 2^-58, given jf = d / (sigma / 1024) to within about one
// unit: with d_c = j sigma / 1024 (exact: a power of two and an integer), d^2 - d_c^2 =
// (d - d_c)(d + d_c) is small, so its exponential is a polynomial, and exp(-d_c^2 / 2 sigma^2) does not
// depend on sigma: one table for every image, exact to half a unit of FP64.  |u| <= 0.003 where jf is
// rounded right: the degree-4 Taylor polynomial is within 2e-17.  (Table-driven evaluation after Tang,
// ACM TOMS 15 (1989) 144, here on the distance instead of the exponent.)  FP64 up to u; a sum with a
// large constant leaves u as an integer, and the rest is integer arithmetic.  A distance beyond the
// table's end (no accepted atom has one) gives a meaningless number.
__device__ __forceinline__ long long gauss64(double d, float jf, const long long* __restrict__ T, double s1024,
                                             double ni2s2) {
  jf = fminf(rintf(jf), (float)(kGauss64Size - 1));
  const int b = __float_as_int(jf);
  // the FP64 bits of an FP32 integer (a conversion instruction runs on the FP64 pipe); 0 becomes 2^-127
  const double jd = __hiloint2double((b >> 3) + 0x38000000, b << 29);
  const long long t = __ldg(T + (int)jf);
  const double del = DF(-jd, s1024, d);
  const double s = DF(2.0, d, -del);
  const double v = DF(DM(del, s), ni2s2, 0x1.8p-6);  // u + 3/128: |u| < 1/128, the last bit is 2^-58
  const long long u = __double_as_longlong(v) - __double_as_longlong(0x1.8p-6);
  const int uh = (int)(u >> 20), ul = (int)u & 0xFFFFF;                // 2^-38, 2^-58
  const long long u2 = wide(uh, uh) + (wide(uh, ul) >> 19);            // u^2, 2^-76
  const int u2h = (int)(u2 >> 30);                                     // 2^-46
  const int r = (int)((wide(uh, 357913941) + (wide(u2h, 89478485) >> 8)) >> 28);  // u/6 + u^2/24, 2^-41
  const long long E = u + ((u2 + (wide(u2h, r) >> 10) + (1 << 18)) >> 19);         // exp(u) - 1, 2^-58
  const int eh = (int)(E >> 20), el = (int)E & 0xFFFFF;
  const Fixed f = split58(t);
  return t + ((wide(f.h, eh) + (wide(f.l, eh) >> 29) + (wide(f.h, el) >> 20) + 256) >> 9);
}

// A sum of products of fixed-point numbers: kFold of them in hh (2^-58) and x (2^-87), then folded into
// 96 bits, so that no number of atoms overflows.
constexpr int kFold = 16;
struct Sum58 {
  long long hh, x;
  unsigned long long lo;
  int hi;
  __device__ __forceinline__ void clear() {
    hh = x = 0;
    lo = 0;
    hi = 0;
  }
  __device__ __forceinline__ void add(const Fixed& a, int h, int l) {
    hh += wide(a.h, h);
    x += wide(a.h, l);
    x += wide(a.l, h);
  }
  __device__ __forceinline__ void fold() {
    const long long v = hh + ((x + (1LL << (kLimb - 1))) >> kLimb);
    lo += (unsigned long long)v;
    hi += (int)(v >> 63) + (lo < (unsigned long long)v ? 1 : 0);
    hh = x = 0;
  }
};

// A folded sum times 2^58
__device__ __forceinline__ double value58(unsigned long long lo, int hi) {
  if (hi == (int)((long long)lo >> 63)) return __ll2double_rn((long long)lo);
  return DF((double)hi, 0x1p64, __ull2double_rn(lo));
}

// The sample of a voxel: f S / max(1e-16, |S|) (:1877-1892), the bits of an FP64 number or
// units of 2^-60; one copy of its code for all slices.
__device__ __noinline__ longlong2 sample(unsigned long long rl, int rh, unsigned long long il, int ih, double f,
                                         bool fixed) {
  const double sr = value58(rl, rh), si = value58(il, ih);
  const double inv = rsqrt(fmax(DF(sr, sr, DM(si, si)), 1e-32 * 0x1p116));
  const double x = DM(DM(sr, inv), f), y = DM(DM(si, inv), f);
  if (fixed) return make_longlong2(to60(x), to60(y));
  return make_longlong2(__double_as_longlong(x), __double_as_longlong(y));
}

template <int SL>
struct Acc {
  Sum58 sr[SL], si[SL];
  // density: the FP32 minimum of r^2 - cutoff^2 (scaled), the next one, and the minimum's atom
  float rm[SL], next[SL];
  int id[SL];
};

// Exact squared distance of kept atom gi (cell code `code`) and this lane's column at slice k of
// the step, in the reference's operations; +inf outside the lane's 27 cells.
template <int CAPS, int SL>
__device__ __noinline__ double exact_dd(const ColumnParams& p, const WarpSmem<CAPS, SL>& W, int gi, int code, int us,
                                           int k, int lane) {
  const int c = lane & 7, r = 8 + (lane >> 3);
  const int kx = (code & 255) - W.hc[c], ky = ((code >> 8) & 255) - W.hc[r];
  if (kx < -1 || kx > 1 || ky < -1 || ky > 1) return (double)INFINITY;
  const double4_32a f = p.f64[gi];
  const double d0 = DM(p.a11, DA(f.x, W.off[c][kx + 1]));
  const double d1 = DM(p.a22, DA(f.y, W.off[r][ky + 1]));
  const double d2 = DM(p.a33, DA(f.z, W.zoff[us][k]));
  return DA(DA(DM(d0, d0), DM(d1, d1)), DM(d2, d2));
}

// The buffered atoms: which lanes accept them, in passes of up to 32 that some lane accepts; their
// Gaussian factors (tasks over the lanes), where an accepting lane needs them; then every lane's sums.
template <int CAPS, int SL, bool kDens>
__device__ __forceinline__ void consume(const ColumnParams& p, WarpSmem<CAPS, SL>& W, int n, float Xv, float Yv,
                                        float cut2f, const long long* __restrict__ T, double s1024, double ni2s2,
                                        Acc<SL>& A, unsigned act, unsigned& n_acc, int lane) {
  constexpr float kGrid = 1.1774100225f * 1024.f;  // scaled length -> sigma / 1024
  __syncwarp();
  const int c = lane & 7, row = 8 + (lane >> 3);
  const unsigned bit = 1u << lane;
  for (int i = 0; i < n;) {
    int cnt = 0;
    for (; i < n && cnt < kPass; ++i) {
      const float2 q = W.xy[i];
      const float dx = q.x - Xv, dy = q.y - Yv;
      const float h = fmaf(dx, dx, dy * dy);
      bool acc[SL], near = false;
      float g[SL];
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        g[k] = h - W.hm[i][k];
        acc[k] = g[k] <= 0.f;
        near = near || fabsf(g[k]) <= kGuard64;
      }
      if (__any_sync(0xffffffffu, near)) {
        if (near) {
          const int2 r = W.ref[i];
#pragma unroll
          for (int k = 0; k < SL; ++k)
            if (fabsf(g[k]) <= kGuard64) acc[k] = exact_dd(p, W, r.x, r.y, (r.y >> 16) & 3, k, lane) <= p.cut2;
        }
        __syncwarp();
      }
      unsigned m[SL], any = 0;
      const int id = kDens ? W.ref[i].y >> 16 : 0;
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        m[k] = __ballot_sync(0xffffffffu, acc[k]);
        any |= m[k];
        if (kDens) {
          A.next[k] = fminf(A.next[k], fmaxf(g[k], A.rm[k]));
          if (g[k] < A.rm[k]) A.id[k] = id;
          A.rm[k] = fminf(A.rm[k], g[k]);
        }
      }
      if (any) {
        if (lane == 0) {
          W.sel[cnt] = i;
          if constexpr (SL == 4) *reinterpret_cast<uint4*>(W.m[cnt]) = make_uint4(m[0], m[1], m[2], m[3]);
          else *reinterpret_cast<uint2*>(W.m[cnt]) = make_uint2(m[0], m[1]);
        }
        ++cnt;
      }
    }
    if (cnt == 0) continue;
    __syncwarp();
    // the list of the columns and rows that some lane needs: place in the buffer, in the pass, column
    unsigned short* list = reinterpret_cast<unsigned short*>(&W.be[0][0]);
    int tasks;
    {
      unsigned need = 0;
      if (lane < cnt) {
        unsigned any = 0;
#pragma unroll
        for (int k = 0; k < SL; ++k) {
          any |= W.m[lane][k];
          n_acc += __popc(W.m[lane][k] & act);
        }
        need = (any | any >> 16);
        need = (need | need >> 8) & 255u;
#pragma unroll
        for (int r = 0; r < 4; ++r) need |= (any >> (8 * r) & 255u) ? 256u << r : 0u;
      }
      const int c0 = __popc(need);
      int incl = c0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      tasks = __shfl_sync(0xffffffffu, incl, 31);
      int at = incl - c0;
      const int e0 = lane << 4 | (lane < cnt ? W.sel[lane] << 9 : 0);
      for (unsigned b = need; b; b &= b - 1) list[at++] = (unsigned short)(e0 | (__ffs(b) - 1));
    }
    __syncwarp();
    for (int t = lane; t < tasks; t += 32) {
      const int e = list[t], j = (e >> 4) & 31, c = e & 15, i = e >> 9;
      const bool x = c < 8;
      const int2 r = W.ref[i];
      const int k = min(1, max(-1, (x ? r.y & 255 : (r.y >> 8) & 255) - W.hc[c]));
      const double f = reinterpret_cast<const double*>(p.f64 + r.x)[x ? 0 : 1];
      const float2 q = W.xy[i];
      const float df = fabsf((x ? q.x : q.y) - W.cx[c]);
      const double d = fabs(DM(x ? p.a11 : p.a22, DA(f, W.off[c][k + 1])));
      W.exy[j][c] = split58(gauss64(d, df * kGrid, T, s1024, ni2s2));
    }
    __syncwarp();
    for (int t = lane; t < SL * cnt; t += 32) {
      const int j = t / SL, k = t - SL * j, i = W.sel[j];
      const int2 r = W.ref[i];
      const double f = reinterpret_cast<const double*>(p.f64 + r.x)[2];
      const double2 cs = p.cs64[r.x];
      const float df = sqrtf(fmaxf(0.f, cut2f - W.hm[i][k]));
      const double d = fabs(DM(p.a33, DA(f, W.zoff[(r.y >> 16) & 3][k])));
      const Fixed e = split58(gauss64(d, df * kGrid, T, s1024, ni2s2));
      const Fixed re = split58(mul58(e, split58(to58(cs.x)))), im = split58(mul58(e, split58(to58(cs.y))));
      W.be[k][j] = make_int4(re.h, re.l, im.h, im.l);
    }
    __syncwarp();
    for (int j0 = 0; j0 < cnt; j0 += kFold) {
      const int j1 = min(cnt, j0 + kFold);
#pragma unroll 1
      for (int j = j0; j < j1; ++j) {
        // every load first: the products of w hide their latency
        const Fixed gx = W.exy[j][c], gy = W.exy[j][row];
        alignas(16) unsigned ms[SL];
        if constexpr (SL == 4) *reinterpret_cast<uint4*>(ms) = *reinterpret_cast<const uint4*>(W.m[j]);
        else *reinterpret_cast<uint2*>(ms) = *reinterpret_cast<const uint2*>(W.m[j]);
        int4 e[SL];
#pragma unroll
        for (int k = 0; k < SL; ++k) e[k] = W.be[k][j];
        const Fixed w = split58(mul58(gx, gy));
#pragma unroll
        for (int k = 0; k < SL; ++k)
          if (ms[k] & bit) {
            A.sr[k].add(w, e[k].x, e[k].y);
            A.si[k].add(w, e[k].z, e[k].w);
          }
      }
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        A.sr[k].fold();
        A.si[k].fold();
      }
    }
    __syncwarp();
  }
}

// rho of convertScaledRangeToRho (:1973-1994), the reference's operations.
__device__ __noinline__ double rho64(double r2min, double sig) {
  if (r2min < DM(sig, sig)) return 1.0;
  if (r2min > DM(DM(4.0, sig), sig)) return 0.0;
  const double xx = DS(__ddiv_rn(__dsqrt_rn(r2min), sig), 1.0);
  const double poly = DA(DS(10.0, DM(15.0, xx)), DM(DM(6.0, xx), xx));
  return DS(1.0, DM(DM(DM(xx, xx), xx), poly));
}

// The slices [z_lo, z_hi) of one patch (the 8 x 4 columns of warp tile `tile`): samples to `out`
// (slice z, lane at out[(z << 5) + lane]).  False when a slab overflows its staging.
template <int CAPS, int SL, bool kDens, bool kMasked>
__device__ __noinline__ bool field_tile(const ColumnParams& p, WarpSmem<CAPS, SL>& W, int tile, int z_lo, int z_hi,
                                        longlong2* __restrict__ out, long long* __restrict__ out_rho,
                                        const long long* __restrict__ T, int lane) {
  constexpr int TX = 8, TY = 4;
  const int Wd = p.ix1 - p.ix0;
  const int tiles_x = (Wd + TX - 1) / TX;
  const int tx = tile % tiles_x, ty = tile / tiles_x;
  const int ix = p.ix0 + tx * TX + (lane % TX);
  const int iy = p.iy0 + ty * TY + lane / TX;
  const bool active = ix < p.ix1 && iy < p.iy1;
  if constexpr (kMasked) {
    const bool wanted =
        active && (!p.tile_mask || p.tile_mask[(iy / p.mask_T) * p.mask_ntx + ix / p.mask_T] != 0);
    if (!__any_sync(0xffffffffu, wanted)) return true;
  }

  const double sd = sqrt(p.i2s2 * 1.4426950408889634);
  Geo G;
  G.scale = (float)sd;
  const int ixc = min(ix, p.ix1 - 1), iyc = min(iy, p.iy1 - 1);
  const int hx = p.xtab[ixc].x, hy = p.ytab[iyc].x;
  const double fvx = p.xfv[ixc], fvy = p.yfv[iyc];
  float Xv, Yv;
  slab::patch_frame(p, G, sd, active, hx, hy, fvx, fvy, Xv, Yv);
  const float cut2f = (float)(p.cut2 * sd * sd);
  const float r3 = sqrtf(cut2f) * 1.0001f + 1e-3f;  // z-window half width, rounded up
  G.pre2 = cut2f * 1.0002f + 1e-2f;
  const float inv_bin = kBins / G.a33s;
  const unsigned lt = (1u << lane) - 1;
  const double s1024 = p.sigma * (1.0 / 1024.0), ni2s2 = -p.i2s2;
  __syncwarp();  // a previous unit's reads of the tables are done
  if (lane < 8) {  // k - zi_frac for k = -1, 0, 1 (:1576-1588), per column ...
    W.cx[lane] = Xv;
    W.hc[lane] = hx - G.ux_ref + 8;
    for (int k = 0; k < 3; ++k) W.off[lane][k] = DS((double)(k - 1), fvx);
  }
  if ((lane & 7) == 0) {  // ... and row
    const int r = 8 + (lane >> 3);
    W.cx[r] = Yv;
    W.hc[r] = hy - G.uy_ref + 8;
    for (int k = 0; k < 3; ++k) W.off[r][k] = DS((double)(k - 1), fvy);
  }
  // rho changes between sigma and 2 sigma (scaled r^2 - cutoff^2; margins for the FP32 distance)
  const float sig2 = (float)(p.sigma * p.sigma * sd * sd);
  const float rm_lo = sig2 - cut2f - kGuard64, rm_hi = 4.f * sig2 - cut2f + kGuard64;

  int ring_lo = 1 << 30, ring_hi = (1 << 30) - 1;
  const unsigned act = __ballot_sync(0xffffffffu, active);
  unsigned n_acc = 0;  // accepted by the tile's columns, of the atoms that this lane counts
  unsigned long long n_tst = 0;
  for (int z0 = z_lo; z0 < z_hi; z0 += SL) {
    // the step's slices: home z cells, FP32 depths in the frame of home cell hz[0] (the
    // table gives each pair's from its even slice's home cell)
    int hz[SL];
    float zv[SL];
    bool has[SL];
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      has[k] = z0 + k < p.Mz;
      const int2 e = p.ztab[has[k] ? z0 + k : z0];
      hz[k] = has[k] ? e.x : hz[0];
      zv[k] = has[k] ? __int_as_float(e.y) : 0.f;
    }
#pragma unroll
    for (int k = 2; k < SL; ++k)
      if (has[k]) zv[k] = __fadd_rn(zv[k], __fmul_rn(G.a33s, (float)(hz[k & ~1] - hz[0])));
    int hz_last = hz[0];
#pragma unroll
    for (int k = 1; k < SL; ++k)
      if (has[k]) hz_last = hz[k];
    const int need_lo = hz[0] - 1, need_hi = hz_last + 1;
    if (need_hi - need_lo + 1 > kRing) {  // the host takes four slices only where they fit
      if (lane == 0) atomicExch(&p.counters[4], 1ull);
      return false;
    }
    if (need_lo > ring_hi || need_hi < ring_lo) {
      ring_lo = need_lo;
      ring_hi = need_lo - 1;
    }
    if (ring_lo < need_lo) ring_lo = need_lo;
    bool ok = true;
    while (ring_hi < need_hi && ok) {
      ++ring_hi;
      ok = load_slab<CAPS>(p, G, ring_hi, W, lane);
    }
    if (!ok) {
      if (lane == 0) atomicExch(&p.counters[4], 1ull);
      return false;
    }
    __syncwarp();
    for (int t = lane; t < kRing * SL; t += 32) {
      const int us = t / SL, k = t - SL * us, z = min(z0 + k, p.Mz - 1);
      W.zoff[us][k] = DS((double)(need_lo + us - p.ztab[z].x), p.zfv[z]);
    }
    Acc<SL> A;
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      A.sr[k].clear();
      A.si[k].clear();
      A.rm[k] = A.next[k] = FLT_MAX;
      A.id[k] = 0;
    }
    int nb = 0;
    // per slab of the step: the bins that overlap the depth window of the slices it serves
    auto window = [&](int u, float* t, bool* v, int& lo, int& hi) {
      const int slot = u & (kRing - 1);
      const float zo = __fmul_rn(G.a33s, (float)(u - hz[0]));
      // the reference's 27 cells in z: slab u serves slice k within one cell of its home cell
      float w_lo = 1e30f, w_hi = -1e30f;
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        t[k] = __fsub_rn(zv[k], zo);
        v[k] = has[k] && u - hz[k] >= -1 && u - hz[k] <= 1;
        if (v[k]) {
          w_lo = fminf(w_lo, t[k]);
          w_hi = fmaxf(w_hi, t[k]);
        }
      }
      lo = hi = 0;
      if (w_lo > w_hi) return;
      lo = W.bin[slot][max(0, min(kBins, (int)floorf((w_lo - r3) * inv_bin)))];
      hi = W.bin[slot][max(0, min(kBins, (int)ceilf((w_hi + r3) * inv_bin)))];
    };
    // one loop over slabs and rounds of 32 atoms, so that there is one copy of consume
    float t[SL];
    bool v[SL];
    int u = need_lo - 1, b = 0, hi = 0;
    for (;;) {
      while (b >= hi && u < need_hi) window(++u, t, v, b, hi);
      const bool more = b < hi;
      if (more) {
        // one atom per lane: kept if some column of the patch can accept it at some slice
        const int slot = u & (kRing - 1), j = b + lane;
        bool keep = false;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        float hm[SL];
        if (j < hi) {
          q = W.p[slot][j];
          float hmax = kOff;
#pragma unroll
          for (int k = 0; k < SL; ++k) {
            const float dz = q.z - t[k];
            hm[k] = v[k] ? cut2f - dz * dz : kOff;
            hmax = fmaxf(hmax, hm[k]);
          }
          const float dxr = fmaxf(0.f, fmaxf(G.xmin - q.x, q.x - G.xmax));
          const float dyr = fmaxf(0.f, fmaxf(G.ymin - q.y, q.y - G.ymax));
          keep = fmaf(dxr, dxr, dyr * dyr) <= hmax + 2.f * kGuard64;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int d = nb + __popc(m & lt);
          W.xy[d] = make_float2(q.x, q.y);
          W.ref[d] = make_int2(W.gi[slot][j], __float_as_int(q.w) | ((u - need_lo) << 16) | (j << 18));
#pragma unroll
          for (int k = 0; k < SL; ++k) W.hm[d][k] = hm[k];
        }
        nb += __popc(m);
        b += 32;
      }
      if (nb > (more ? kN - 33 : 0)) {
        consume<CAPS, SL, kDens>(p, W, nb, Xv, Yv, cut2f, T, s1024, ni2s2, A, act, n_acc, lane);
        n_tst += (unsigned long long)nb;
        nb = 0;
      }
      if (!more) break;
    }
    // density: where the FP32 minimum lies in rho's range, the exact distance of its atom; where the
    // FP32 distance cannot tell the nearest from the next, the exact minimum over all that it cannot
    double rho[SL];
    if constexpr (kDens) {
      bool want[SL], any = false, tie = false;
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        rho[k] = !p.use_density || A.rm[k] < rm_lo ? 1.0 : 0.0;
        want[k] = active && has[k] && p.use_density && A.rm[k] >= rm_lo && A.rm[k] <= fminf(rm_hi, 0.f);
        any = any || want[k];
        tie = tie || (want[k] && A.next[k] <= A.rm[k] + 2.f * kGuard64);
      }
      if (__any_sync(0xffffffffu, any)) {
        double best[SL];
#pragma unroll
        for (int k = 0; k < SL; ++k) {
          best[k] = DBL_MAX;
          if (want[k]) {
            const int us = A.id[k] & 3, slot = (need_lo + us) & (kRing - 1), j = A.id[k] >> 2;
            best[k] = exact_dd(p, W, W.gi[slot][j], __float_as_int(W.p[slot][j].w), us, k, lane);
          }
        }
        if (__any_sync(0xffffffffu, tie)) {
          for (int u = need_lo; u <= need_hi; ++u) {
            const int slot = u & (kRing - 1);
            int lo, hi;
            window(u, t, v, lo, hi);
            for (int j = lo; j < hi; ++j) {
              const float4 q = W.p[slot][j];
              const float dx = q.x - Xv, dy = q.y - Yv;
              const float h = fmaf(dx, dx, dy * dy);
#pragma unroll
              for (int k = 0; k < SL; ++k) {
                const float dz = q.z - t[k];
                if (want[k] && v[k] && h + dz * dz - cut2f <= A.rm[k] + 2.f * kGuard64) {
                  const double dd = exact_dd(p, W, W.gi[slot][j], __float_as_int(q.w), u - need_lo, k, lane);
                  if (dd <= p.cut2 && dd < best[k]) best[k] = dd;
                }
              }
            }
          }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < SL; ++k)
          if (want[k]) rho[k] = rho64(best[k], p.sigma);
        __syncwarp();
      }
    }
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      if (z0 + k >= z_hi) break;
      // with density, rho x and rho are stored; for the fixed-point integrator times its coefficients
      const bool fixed = p.fx_shift >= 0;
      double f = fixed ? p.fx_bg : 1.0;
      if constexpr (kDens) {
        f = DM(f, rho[k]);
        out_rho[((int64_t)(z0 + k) << 5) + lane] = __double_as_longlong(fixed ? DM(rho[k], p.fx_b0) : rho[k]);
      }
      out[((int64_t)(z0 + k) << 5) + lane] =
          sample(A.sr[k].lo, A.sr[k].hi, A.si[k].lo, A.si[k].hi, f, !kDens && fixed);
    }
  }
  if (p.want_stats) {
    unsigned long long acc_w = n_acc, tst_w = active ? (unsigned long long)SL * n_tst : 0u;
    for (int o = 16; o > 0; o >>= 1) {
      acc_w += __shfl_xor_sync(0xffffffffu, acc_w, o);
      tst_w += __shfl_xor_sync(0xffffffffu, tst_w, o);
    }
    if (lane == 0) {
      atomicAdd(&p.counters[2], tst_w);
      atomicAdd(&p.counters[3], acc_w);
    }
  }
  return true;
}

template <int CAPS, int SL, bool kDens, bool kMasked, int kMinBlocks>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks)
    k_field64(const ColumnJob* __restrict__ jobs, int n_jobs, FieldRange R, const long long* __restrict__ T) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpSmem<CAPS, SL>& W = reinterpret_cast<WarpSmem<CAPS, SL>*>(smem_raw)[warp];
  if ((int64_t)R.counters[0] > R.cap) return;  // the binning overflowed: the host retries
  int chunk = R.chunk, n_chunks = R.n_chunks, units = R.units();
  if constexpr (kMasked) {
    const int n = listed_patches(R), deep = jobs[0].p.Mz;
    chunk = warp_depth_chunk(n, deep, R.slots, kRule64);
    n_chunks = (deep + chunk - 1) / chunk;
    units = n * n_chunks;
  }
  for (;;) {
    int unit = 0;
    if (lane == 0) unit = (int)atomicAdd(R.work, 1u);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if (unit >= units) break;
    if (R.counters[4] != 0) break;  // a slab overflowed: the host recomputes with larger slabs
    int patch;
    const ColumnJob& J = field_patch(jobs, n_jobs, R.patch_lo + unit / n_chunks, patch);
    const int z_lo = unit % n_chunks * chunk, z_hi = min(J.p.Mz, z_lo + chunk);
    if (z_lo >= z_hi) continue;  // an image less deep than the batch's deepest
    const int64_t o = J.sample_base - R.origin + (int64_t)patch * J.p.Mz * 32;
    if constexpr (kMasked) patch = listed_patch(R, J.p, patch);
    if (!field_tile<CAPS, SL, kDens, kMasked>(J.p, W, patch, z_lo, z_hi, (longlong2*)R.samples + o, (long long*)R.rho64 + o, T,
                                               lane))
      break;
  }
}

// ------------------------------------------------------------------------------------------
// The column integrator
// ------------------------------------------------------------------------------------------

// A column's samples for column60: with density FP64, of which sparse columns need every bit, else units of
// 2^-60, exact to bg's own bits.
template <bool kDens>
struct FixedSamples {
  const longlong2* x;
  const long long* r;
  long long b0, a;
  struct Raw {
    longlong2 x;
    long long r;
  };
  __device__ __forceinline__ Raw load(int z) const {
    return Raw{x[(int64_t)z << 5], kDens ? r[(int64_t)z << 5] : b0};
  }
  __device__ __forceinline__ SFix coef(const Raw& s) const {
    if constexpr (kDens)
      return sfix(to60(__longlong_as_double(s.r)), to60(__longlong_as_double(s.x.x)),
                  to60(__longlong_as_double(s.x.y)), a);
    else
      return sfix(s.r, s.x.x, s.x.y, a);
  }
};

// A warp per patch and angle (warp w of the CTA takes angles w, w + warps, ...), one lane per
// column.  FP64 takes about 90 operations per double step, at 76 cycles each; in fixed point they are
// 156 multiply-adds of 4 cycles and as much again of additions and shifts.  The host takes
// fixed point where 2^-60 is no coarser than FP64 for these amplitudes (fixed_rule), and a warp with
// columns that turn out too weak for it (column60) repeats those in FP64.
template <bool kDens>
__global__ void __launch_bounds__(256) k_integrate64(const ColumnJob* __restrict__ jobs, int n_jobs, FieldRange R) {
  __shared__ double part[8][32];
  const int lane = threadIdx.x, warp = threadIdx.y, nw = blockDim.y;
  if (blockIdx.x == 0 && warp == 0 && lane == 0) *R.work = 0;  // for the next field kernel
  if ((int64_t)R.counters[0] > R.cap || R.counters[4] != 0) return;
  if (R.list && (int)blockIdx.x >= listed_patches(R)) return;
  int patch;
  const ColumnJob& J = field_patch(jobs, n_jobs, R.patch_lo + blockIdx.x, patch);
  const ColumnParams& p = J.p;
  const int64_t o = J.sample_base - R.origin + (int64_t)patch * p.Mz * 32 + lane;
  if (R.list) patch = listed_patch(R, J.p, patch);
  const int tiles_x = (p.ix1 - p.ix0 + 7) / 8;
  const int ix = p.ix0 + (patch % tiles_x) * 8 + (lane & 7), iy = p.iy0 + (patch / tiles_x) * 4 + (lane >> 3);
  const bool active = ix < p.ix1 && iy < p.iy1;
  bool wanted = active;
  if (p.tile_mask) wanted = active && p.tile_mask[(iy / p.mask_T) * p.mask_ntx + ix / p.mask_T] != 0;
  if (!__any_sync(0xffffffffu, wanted)) return;
  const double2* __restrict__ X = (const double2*)R.samples + o;
  const double* __restrict__ RH = R.rho64 + o;
  const double reach0 = fabs(p.b0) + fabs(p.bg);
  double total = 0.0;
  for (int k0 = 0; k0 < p.n_prec; k0 += nw) {
    const int k = k0 + warp;
    if (k < p.n_prec) {
      const double a = p.aa[k];
      const bool fixed = p.fx_shift >= 0;
      bool repeat = !fixed;
      if (fixed) {
        const FixedSamples<kDens> src{(const longlong2*)X, (const long long*)RH, to60(p.fx_b0), to60(DM(a, p.fx_a))};
        part[warp][lane] = column60(p.Mz, p.fx_shift, src, repeat);
        repeat = repeat && wanted;
      }
      if (__any_sync(0xffffffffu, repeat)) {
        // the stored samples are rho x and rho, or those times the fixed-point coefficients; of an image without
        // density in units of 2^-60, whatever the others of its batch have
        const double inv = fixed ? __ddiv_rn(1.0, p.fx_a) : 1.0;
        auto coef = [&](int z) {
          const double2 x = X[(int64_t)z << 5];
          const double r = kDens ? RH[(int64_t)z << 5] : 1.0;
          if (!fixed) return S64{kDens ? DM(p.b0, r) : p.b0, DM(p.bg, x.x), DM(p.bg, x.y)};
          if (kDens && p.use_density) return S64{DM(r, inv), DM(x.x, inv), DM(x.y, inv)};
          const double u = DM(inv, 0x1p-60);
          const long long xr = kDens ? to60(x.x) : __double_as_longlong(x.x),
                          xi = kDens ? to60(x.y) : __double_as_longlong(x.y);
          return S64{p.b0, DM(__ll2double_rn(xr), u), DM(__ll2double_rn(xi), u)};
        };
        const double ig = column64(p.Mz, p.dz, a, reach0 + fabs(a), coef);
        if (repeat) part[warp][lane] = ig;
      }
    }
    __syncthreads();
    if (warp == 0)
      for (int w = 0; w < min(nw, p.n_prec - k0); ++w) total = DA(total, part[w][lane]);
    __syncthreads();
  }
  if (warp == 0 && wanted) {
    if (p.finalize) {  // the precession average and the bright-field flip
      total = __ddiv_rn(total, p.fin_scale);
      if (p.fin_bright) total = DS(1.0, total);
    }
    p.img[ix + (int64_t)p.Mx * iy] = total;
  }
}

template <int CAPS, int SL, bool kDens, bool kMasked, int B>
cudaError_t launch(const ColumnJob* jobs, int n_jobs, FieldRange R, const long long* T, cudaStream_t st) {
  const size_t smem = sizeof(WarpSmem<CAPS, SL>) * kWarps;
  auto kernel = k_field64<CAPS, SL, kDens, kMasked, B>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int grid = sm_count() * B;
  split_depth(R, 1, kWarps * grid, kRule64);
  if (!R.list) grid = std::max(1, std::min(grid, (R.units() + kWarps - 1) / kWarps));
  ++launch_count();
  kernel<<<grid, kWarps * 32, smem, st>>>(jobs, n_jobs, R, T);
  return cudaGetLastError();
}

template <int SL, bool kDens, bool kMasked>
cudaError_t launch_tier(int tier, const ColumnJob* jobs, int n_jobs, const FieldRange& R, const long long* T,
                        cudaStream_t st) {
  if (tier >= 2) return launch<256, SL, kDens, kMasked, 1>(jobs, n_jobs, R, T, st);
  if (tier == 1) return launch<192, SL, kDens, kMasked, 1>(jobs, n_jobs, R, T, st);
  return launch<128, SL, kDens, kMasked, kField64Blocks>(jobs, n_jobs, R, T, st);
}

}  // namespace field64

int field64_patches(const ColumnParams& p) {
  const int Wd = p.ix1 - p.ix0, Hd = p.iy1 - p.iy0;
  return Wd <= 0 || Hd <= 0 ? 0 : ((Wd + 7) / 8) * ((Hd + 3) / 4);
}

// exp(-(j / 1024)^2 / 2) in units of 2^-58, j = 0 .. kGauss64Size - 1 (the library's exp: correctly
// rounded but for one value in a few thousand)
void gauss64_table(long long* t) {
  for (int j = 0; j < kGauss64Size; ++j)
    t[j] = std::llrint(std::ldexp(std::exp(-0.5 * ((double)j / 1024.0) * ((double)j / 1024.0)), 58));
}

cudaError_t launch_field64(const ColumnJob* d_jobs, int n_jobs, const FieldRange& R, int max_np, int slab_tier,
                           bool density, bool masked, bool four, const long long* d_gauss, cudaStream_t st) {
  using namespace field64;
  cudaError_t e = cudaSuccess;
  if (R.units() <= 0) return e;
#define STEM_F64(SL)                                                                                        \
  (masked ? (density ? launch_tier<SL, true, true>(slab_tier, d_jobs, n_jobs, R, d_gauss, st)               \
                     : launch_tier<SL, false, true>(slab_tier, d_jobs, n_jobs, R, d_gauss, st))             \
          : (density ? launch_tier<SL, true, false>(slab_tier, d_jobs, n_jobs, R, d_gauss, st)              \
                     : launch_tier<SL, false, false>(slab_tier, d_jobs, n_jobs, R, d_gauss, st)))
  e = four ? STEM_F64(4) : STEM_F64(2);
#undef STEM_F64
  if (e != cudaSuccess) return e;
  const dim3 block(32, std::min(8, max_np));
  ++launch_count();
  if (density)
    k_integrate64<true><<<R.patch_hi - R.patch_lo, block, 0, st>>>(d_jobs, n_jobs, R);
  else
    k_integrate64<false><<<R.patch_hi - R.patch_lo, block, 0, st>>>(d_jobs, n_jobs, R);
  return cudaGetLastError();
}

}  // namespace stem
