// K2+K3, FP32: the voxel field and its column integrator.
//
// The pixel loop of computeD2BI_img (Lib_DynamicalTwoBeamImaging.f90:1870-1900) with the
// neighbour search of Lib_LinkCell3D.f90:1515-1605 (k_field32) and the integrator of
// :2316-2480 (k_integrate32), for the FP32 path (k_column_fp32 in k_column.cu is the general
// form, for any cell size and slab occupancy).  The field samples pass through device memory
// (8 bytes a voxel, 12 with density): the field kernel then carries no integrator state, splits a
// column's depth over CTAs where an image has few columns, and runs once however many precession
// angles integrate over it.
//
// The field kernel: a CTA of four warps owns 16 x 8 pixel columns and a range of slices, each warp 32
// of the columns (8 x 4, 4 x 8 or 16 x 2: the tuning variants), four slices per step (two where some
// image's steps of four do not fit the ring).  Instruction issue bounds it (0.64 to 0.7 per cycle and
// sub-partition), then the shared-memory loads of the atoms and the FP32 pipe; so everything that does
// not depend on the column is done once for the four warps, and an atom's values are loaded for two columns:
// * The atoms of a link-cell slab (one z cell; a ring of four) within 3 sigma of the tile are
//   gathered into shared memory once per slab (a tile of one warp would gather 2.3 times as
//   many per column).
// * Per step, one thread per atom computes what depends on the atom and the depth alone, for the
//   atoms of the step's depth window (counted first, so that they lie densely): the largest in-plane r^2
//   each slice still accepts (hmax_k = (3 sigma)^2 - dz_k^2, or kOff where the reference's 27-cell
//   rule excludes the slab for that slice) and the Gaussian's depth factor times the phasor,
//   ex2(-dz_k^2) (cos, sin).
// * Each warp lists the atoms that some column of its patch accepts at some slice (distance to
//   the patch's sample rectangle against the largest hmax), ballot + popc, order kept.
// * A lane then takes two columns, and the two groups of 16 lanes take different listed atoms: the
//   in-plane distances (FP32x2), one ex2 per atom and column for all four slices (the Gaussian is
//   separable), and per slice the inclusive cutoff dxy^2 <= hmax_k and one FP32x2 multiply-add of the
//   weight into (cos, sin); the groups' sums are added at the end of the step.
// Measured on the 1.2M-atom image (566 x 566 x 240): 2.84 ms for the kernel before (a warp's own
// slabs, two slices per step, the integrator in the same kernel), 2.06 ms field + 0.15 ms integrator
// now; of a field of 2.12 ms 0.87 were the lists' sums (0.65 at the FP32 pipe's rate), 0.30 the depth terms, 0.29
// the gather, 0.26 the step's fixed cost, 0.16 the lists, 0.13 the exact recheck.  One column per lane
// ran 2.55 ms (the loads), four columns 2.22, six CTAs per SM instead of five 2.33, a producer warp per CTA
// 2.55, slabs per warp 2.35.
// Images of one patch shape are the same to the last bit whatever the slab capacity; the shapes
// distribute a list over the groups of lanes differently, so between shapes they agree to FP32 rounding.
// Lengths are scaled by s = sqrt(log2 e / 2 sigma^2), so a weight is ex2(-r'^2).
//
// Precision: FP32 throughout; the weight is the product of two ex2 values (a few ulp).  The FP32
// cutoff test may decide an atom within rounding of the cutoff differently from the reference;
// columns whose field sum is small enough for that to matter re-decide those atoms in the
// reference's FP64 arithmetic (exact_fix below).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "internal.h"
#include "slab_ring.cuh"
#include "two_beam32.h"

namespace stem {
namespace field32 {

using slab::Geo;
using slab::kRing;

constexpr float kOff = -1e30f;  // hmax of a slice the slab does not serve
constexpr int kTileX = 16, kTileY = 8;
constexpr int kCPL = 2;         // columns per lane
constexpr int kSegs = 32;       // cell runs looked up at a time, one per lane

// CAP: atoms per slab; WCAP: atoms in a step's depth window; NW: warps; SL: slices per step.
template <int CAP_, int WCAP_, int NW_, int SL_>
struct Smem {
  static constexpr int CAP = CAP_, WCAP = WCAP_, NW = NW_, SL = SL_;
  static constexpr int kRounds = (kRing * CAP + 32 * NW - 1) / (32 * NW);
  static_assert(kRounds <= 32 && kRounds * NW <= 64, "a thread's window flags and the warps' counts");
  float4 p[kRing * CAP];  // X', Y' (tile frame), z (own cell), kept atom
  float2 cs[kRing * CAP]; // (cos, sin) of the phase
  // the atoms of the step's depth window; entry WCAP accepts nothing (pads a list)
  float4 r[WCAP + 1];     // X', Y', the largest hmax with the margin of the patch test, kept atom
  typename std::conditional<SL == 4, float4, float2>::type h[WCAP + 1];  // hmax per slice
  float4 e0[WCAP + 1];    // ex2(-dz^2) (cos, sin) of slices 0 and 1
  float4 e1[SL == 4 ? WCAP + 1 : 1];  // of slices 2 and 3
  int4 seg[kSegs];        // the footprint's cell runs: first cell in the plane, cells, x shift, row
  int count[kRing];
  int cnt[2][NW];
  int wcnt[64];           // window atoms per round and warp
  int unit;
  unsigned short li[NW][WCAP + 4];  // byte offsets of the atoms listed for a warp's patch
};

template <int NW>
__device__ __forceinline__ void sync() {
  if constexpr (NW == 1) __syncwarp();
  else __syncthreads();
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ int warp_scan(int v, int lane) {  // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// The footprint's runs of consecutive cells (rows uy, runs in x, a run ends where x wraps): run
// s0 + lane of them.
struct Runs {
  int k_lo, n_run, n_seg;
};
__device__ __forceinline__ int4 run_of(const ColumnParams& p, const Geo& G, const Runs& R, int s) {
  const int k = R.k_lo + s % R.n_run, uy = G.uy_lo + s / R.n_run, shift = k * p.Ex;
  const int x0 = max(G.ux_lo, shift), x1 = min(G.ux_hi, shift + p.Ex - 1);
  return make_int4(p.Ex * slab::pos_mod(uy, p.Ey) + (x0 - shift), x1 - x0 + 1, shift, uy);
}

// Gather slab u (its cells in the tile's footprint, atoms within 3 sigma of the tile's sample
// rectangle) into its ring slot, in the order rows, runs, atoms; false (in every thread) when it
// holds more than CAP.  Every warp looks the runs up for itself (one per lane); the first 32 come
// from the table built once per unit.
template <typename W_>
__device__ __forceinline__ bool load_slab_cta(const ColumnParams& p, const Geo& G, const Runs& R, int u, W_& W) {
  constexpr int NW = W_::NW, CAP = W_::CAP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int cz = u;
  if (cz < 0 || cz >= p.Ez) cz = slab::pos_mod(u, p.Ez);
  const int slot = u & (kRing - 1);
  const int64_t plane = (int64_t)p.Ex * p.Ey * cz;
  int n = 0, par = 0;
  for (int s0 = 0; s0 < R.n_seg; s0 += kSegs) {
    const int ns = min(kSegs, R.n_seg - s0);
    int4 sg = make_int4(0, 0, 0, 0);
    int a_lo = 0, len = 0;
    if (lane < ns) {
      sg = s0 == 0 ? W.seg[lane] : run_of(p, G, R, s0 + lane);
      const int* c = p.cell_start + plane + sg.x;
      a_lo = c[0];
      len = c[sg.y] - a_lo;
    }
    const int incl = warp_scan(len, lane);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int first = incl - len;  // this lane's run covers the indices [first, incl)
    for (int b = 0; b < total; b += 32 * NW) {
      const int i = b + tid;
      int s = 0;
      for (int q = 1; q < ns; ++q) s += __shfl_sync(0xffffffffu, first, q) <= i;
      // (an empty run shares its successor's first index and is passed over)
      const int j = __shfl_sync(0xffffffffu, a_lo, s) + i - __shfl_sync(0xffffffffu, first, s);
      const int shift = __shfl_sync(0xffffffffu, sg.z, s), uy = __shfl_sync(0xffffffffu, sg.w, s);
      bool keep = false;
      float4 rec = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < total) keep = slab::slab_candidate<false>(p, G, j, shift, uy, rec);
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      int base = n, tot = __popc(m);
      if constexpr (NW > 1) {
        if (lane == 0) W.cnt[par][warp] = tot;
        sync<NW>();
        tot = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          const int c = W.cnt[par][w];
          if (w < warp) base += c;
          tot += c;
        }
      }
      if (n + tot > CAP) return false;
      if (keep) {
        const int d = slot * CAP + base + __popc(m & ((1u << lane) - 1));
        float sn, co;
        __sincosf(6.28318531f * rec.w, &sn, &co);  // the phase lies in [-1/2, 1/2) cycles
        W.p[d] = make_float4(rec.x, rec.y, rec.z, __int_as_float(j));
        W.cs[d] = make_float2(co, sn);
      }
      n += tot;
      par ^= 1;
    }
    if (s0 + kSegs < R.n_seg) sync<NW>();  // cnt[par] may still be read
  }
  if (tid == 0) W.count[slot] = n;
  sync<NW>();
  return true;
}

// The cutoff in the reference is an FP64 comparison, d.d <= (3 sigma)^2
// (Lib_LinkCell3D.f90:1594), and the phase field is discontinuous there: a voxel whose only
// neighbour lies at the cutoff has x = 0 on one side and a unit phasor on the other
// (S / max(1e-16, |S|), Lib_DynamicalTwoBeamImaging.f90:1877-1892).  The FP32 test may
// decide an atom within about 3e-5 (scaled r^2) of the cutoff differently.  That changes
// a voxel with many neighbours by a few 1e-6 in I at most, but a sparse one (a void's rim,
// or neighbours whose phases cancel) by up to 1e-2.  So after each step the columns whose
// field sum is small go through the warp's listed atoms again, re-decide in the reference's FP64
// arithmetic every atom the FP32 test placed within kGuard of the cutoff, and correct the
// sum for each decision that changes.  The pass repeats the step's FP32 operations on
// the same staged values, so it meets the same decisions; the FP64 distance uses the cell
// fractions the binning kept (2^-32 cells) and the reference's per-axis form
// d = a (f + (k - zi_frac)).
constexpr float kGuard = 1e-4f;  // scaled r^2; the FP32 test's error is below 3e-5
// |S|^2 below which a column re-decides its near-cutoff atoms.  A flipped atom weighs
// exp(-9/2) = 0.011 and moves x = S / |S| by at most 0.011 |e^(i phi) - x| / |S|; above
// |S| = 1/2, with the few-tenths-of-a-radian phase spread of neighbouring atoms, that
// changes I by a few 1e-5 at most.
constexpr float kSparse2 = 0.25f;

__device__ __forceinline__ int wrap_diff(int c, int h, int n) {  // c - h in -(n/2) .. n/2, periodic
  int d = c - h;
  if (d > n / 2) d -= n;
  else if (d < -(n / 2)) d += n;
  return d;
}

template <int SL>
struct Slices {
  int hz[SL];     // home z cell
  float zv[SL];   // scaled depth from the origin of home cell hz[0]
  bool has[SL];
};

// This lane's column, with what the exact distances need.
struct Column {
  float X, Y;
  int hx, hy;
  double fvx, fvy;
};

template <int SL>
struct Fix {
  float2 d[SL];  // corrections of the slices' sums
  int dn;        // change of the accepted count
};

template <typename W_>
__device__ __noinline__ Fix<W_::SL> exact_fix(const ColumnParams& p, const W_& W, int warp, int n, int z0, int need_lo,
                                              float a33s, float cut2, const Slices<W_::SL>& S, unsigned want,
                                              const Column& C) {
  constexpr int SL = W_::SL;
  Fix<SL> r;
#pragma unroll
  for (int k = 0; k < SL; ++k) r.d[k] = make_float2(0.f, 0.f);
  r.dn = 0;
  for (int i = 0; i < n; ++i) {
    const float4 e = W.r[W.li[warp][i] >> 4];
    const float dx = __fadd_rn(e.x, -C.X), dy = __fadd_rn(e.y, -C.Y);
    const float h = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
    float hm[SL];
    const auto hv = W.h[W.li[warp][i] >> 4];
    hm[0] = hv.x;
    hm[1] = hv.y;
    if constexpr (SL == 4) {
      hm[2] = hv.z;
      hm[3] = hv.w;
    }
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      if (!(want >> k & 1) || fabsf(h - hm[k]) > kGuard) continue;
      const int gi = __float_as_int(e.w);
      const int packed = __float_as_int(p.p32[gi].w);
      const int kx = wrap_diff(packed & 1023, C.hx, p.Ex), ky = wrap_diff((packed >> 10) & 1023, C.hy, p.Ey);
      const int kz = wrap_diff(packed >> 20, S.hz[k], p.Ez);
      const uint4 fr = p.fr32[gi];
      const double fx = (double)fr.x * 2.3283064365386963e-10, fy = (double)fr.y * 2.3283064365386963e-10,
                   fz = (double)fr.z * 2.3283064365386963e-10;
      const double d0 = __dmul_rn(p.a11, __dadd_rn(fx, __dsub_rn((double)kx, C.fvx)));
      const double d1 = __dmul_rn(p.a22, __dadd_rn(fy, __dsub_rn((double)ky, C.fvy)));
      const double d2 = __dmul_rn(p.a33, __dadd_rn(fz, __dsub_rn((double)kz, p.zfv[z0 + k])));
      const bool acc64 = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)) <= p.cut2;
      if (acc64 == (h <= hm[k])) continue;
      float sn, cs;
      __sincosf(6.28318531f * p.ph32[gi], &sn, &cs);
      const float w = ex2_approx(-h) * ex2_approx(hm[k] - cut2) * (acc64 ? 1.f : -1.f);  // dz^2 = cut2 - hmax
      r.d[k].x = fmaf(w, cs, r.d[k].x);
      r.d[k].y = fmaf(w, sn, r.d[k].y);
      r.dn += acc64 ? 1 : -1;
    }
  }
  return r;
}

__device__ __forceinline__ float rho_of(float r2min, float sig) {
  if (r2min < sig * sig) return 1.f;
  if (r2min > 4.f * sig * sig) return 0.f;
  const float xx = sqrtf(r2min) / sig - 1.f;
  return 1.f - xx * xx * xx * (10.f - 15.f * xx + 6.f * xx * xx);
}

// Column of lane `lane` of patch w (of four) in the 16 x 8 tile at (x0, y0).
template <int TX>
__device__ __forceinline__ void patch_column(int x0, int y0, int w, int lane, int& ix, int& iy) {
  const int wx = TX == 8 ? (w & 1) * 8 : TX == 4 ? w * 4 : 0;
  const int wy = TX == 8 ? (w >> 1) * 4 : TX == 4 ? 0 : w * 2;
  ix = x0 + wx + lane % TX;
  iy = y0 + wy + lane / TX;
}

// The slices [z_lo, z_hi) of one tile (NW = 4: its four patches; NW = 2: `patch` and the one below it; NW = 1:
// patch `patch` of it).
// Samples of patch w, slice z to out[((w * Mz + z) << 5) + lane].  False when a slab or a step's
// window overflows.
//
// The lanes' loop reads 14 floats per atom from shared memory, and a shared-memory read costs by
// the bytes it returns to the lanes, broadcast or not (measured: 0.47 16-byte reads per cycle and
// SM): with one column per lane these reads bound the kernel.  So a lane takes CPL columns (two or
// four of its patch, 32 / CPL lanes cover it) and the 32 / CPL-lane groups of a warp take different
// atoms; the groups' sums are added once per step, which leaves each lane with its own column.
template <int CPL, int TX, bool kDens, bool kStats, bool kMasked, typename W_>
__device__ __forceinline__ bool field_tile(const ColumnParams& p, W_& W, int patch, int z_lo, int z_hi,
                                           float2* __restrict__ out, float* __restrict__ out_rho) {
  constexpr int NW = W_::NW, SL = W_::SL, CAP = W_::CAP, WCAP = W_::WCAP;
  constexpr int LPG = 32 / CPL;  // lanes per group
  constexpr bool kSameX = LPG % TX == 0;  // a lane's columns share x
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = lane / LPG;
  const int tile = patch >> 2;
  auto patch_of = [&](int w) { return NW == 1 ? patch & 3 : NW == 2 ? (patch & 1) + 2 * w : w; };  // within the tile
  const int w4 = patch_of(warp);
  const int tiles_x = (p.ix1 - p.ix0 + kTileX - 1) / kTileX;
  const int x0 = p.ix0 + tile % tiles_x * kTileX, y0 = p.iy0 + tile / tiles_x * kTileY;
  int ix, iy;
  patch_column<TX>(x0, y0, w4, lane, ix, iy);
  const bool active = ix < p.ix1 && iy < p.iy1;
  // tile mask: a warp lists and sums when any of its columns is wanted (a patch may straddle
  // mask tiles); the integrator writes only the wanted ones
  bool wanted = active;
  if constexpr (kMasked) {
    if (p.tile_mask) wanted = active && p.tile_mask[(iy / p.mask_T) * p.mask_ntx + ix / p.mask_T] != 0;
  }
  const bool work = __any_sync(0xffffffffu, wanted);
  unsigned patches = 15;  // of the tile, with a wanted column
  if constexpr (NW == 1) {
    if (!work) return true;
  } else if constexpr (kMasked) {
    if (lane == 0) W.wcnt[warp] = work;
    sync<NW>();
    patches = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) patches |= W.wcnt[w] ? 1u << patch_of(w) : 0u;
    if (!patches) return true;
  }

  // the frame is the 16 x 8 tile's for any NW, so that the staged values do not depend on it, from
  // the cell of its middle: coordinates half as large round half as coarsely
  Geo G;
  G.ux_ref = p.xtab[min(x0 + kTileX / 2, p.ix1 - 1)].x;
  G.uy_ref = p.ytab[min(y0 + kTileY / 2, p.iy1 - 1)].x;
  G.scale = p.scale;
  G.a11s = p.a11s;
  G.a22s = p.a22s;
  G.a33s = p.a33s;
  const float cut2 = p.cut2s;
  G.pre2 = cut2 * 1.0002f + 1e-3f;
  auto col_x = [&](int2 t) { return __fmaf_rn(G.a11s, (float)(t.x - G.ux_ref), __int_as_float(t.y)); };
  auto col_y = [&](int2 t) { return __fmaf_rn(G.a22s, (float)(t.x - G.uy_ref), __int_as_float(t.y)); };
  // the CPL columns this lane sums: those of lanes lane % LPG + c LPG
  float nX[CPL], nY[CPL];
  unsigned act = 0;
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    int cx, cy;
    patch_column<TX>(x0, y0, w4, lane % LPG + c * LPG, cx, cy);
    nX[c] = -col_x(p.xtab[min(cx, p.ix1 - 1)]);
    nY[c] = -col_y(p.ytab[min(cy, p.iy1 - 1)]);
    if (cx < p.ix1 && cy < p.iy1) act |= 1u << c;
  }
  // this warp's sample rectangle (its columns on the image), as centre and half widths
  float pxc, pyc, pxh, pyh;
  Runs R;
  {
    int xa, ya, xb, yb;
    patch_column<TX>(x0, y0, w4, 0, xa, ya);
    patch_column<TX>(x0, y0, w4, 31, xb, yb);
    const float x_lo = col_x(p.xtab[min(xa, p.ix1 - 1)]), x_hi = col_x(p.xtab[min(xb, p.ix1 - 1)]);
    const float y_lo = col_y(p.ytab[min(ya, p.iy1 - 1)]), y_hi = col_y(p.ytab[min(yb, p.iy1 - 1)]);
    pxc = 0.5f * (x_lo + x_hi);
    pyc = 0.5f * (y_lo + y_hi);
    pxh = 0.5f * (x_hi - x_lo) + 2e-5f;  // the centre's rounding
    pyh = 0.5f * (y_hi - y_lo) + 2e-5f;
    // the gather's rectangle and cells: the tile's, or for one warp the patch's, or about the wanted patches
    int gx0 = x0, gx1 = min(x0 + kTileX, p.ix1) - 1, gy0 = y0, gy1 = min(y0 + kTileY, p.iy1) - 1;
    if (kMasked && NW > 1 && patches != 15) {
      int lx = 1 << 30, ly = 1 << 30, ux = 0, uy = 0;
#pragma unroll
      for (int w = 0; w < 4; ++w)
        if (patches >> w & 1) {
          int cx, cy;
          patch_column<TX>(x0, y0, w, 0, cx, cy);
          lx = min(lx, cx);
          ly = min(ly, cy);
          patch_column<TX>(x0, y0, w, 31, cx, cy);
          ux = max(ux, cx);
          uy = max(uy, cy);
        }
      gx0 = lx;
      gy0 = ly;
      gx1 = min(gx1, ux);
      gy1 = min(gy1, uy);
    }
    if constexpr (NW == 1) {
      gx0 = xa;
      gy0 = ya;
      gx1 = min(xb, p.ix1 - 1);
      gy1 = min(yb, p.iy1 - 1);
    }
    const int2 xl = p.xtab[gx0], xh = p.xtab[gx1], yl = p.ytab[gy0], yh = p.ytab[gy1];
    G.xmin = col_x(xl);
    G.xmax = col_x(xh);
    G.ymin = col_y(yl);
    G.ymax = col_y(yh);
    // the cells that reach within 3 sigma of the rectangle, at most one beyond its home cells (the
    // reference's 27-cell search)
    const float reach = sqrtf(G.pre2), ia = 1.f / G.a11s, ib = 1.f / G.a22s;
    G.ux_lo = max(xl.x - 1, G.ux_ref + (int)floorf((G.xmin - reach) * ia - 1e-4f));
    G.ux_hi = min(xh.x + 1, G.ux_ref + (int)floorf((G.xmax + reach) * ia + 1e-4f));
    G.uy_lo = max(yl.x - 1, G.uy_ref + (int)floorf((G.ymin - reach) * ib - 1e-4f));
    G.uy_hi = min(yh.x + 1, G.uy_ref + (int)floorf((G.ymax + reach) * ib + 1e-4f));
    R.k_lo = slab::floor_div(G.ux_lo, p.Ex);
    R.n_run = slab::floor_div(G.ux_hi, p.Ex) - R.k_lo + 1;
    R.n_seg = (G.uy_hi - G.uy_lo + 1) * R.n_run;
    if (tid < min(kSegs, R.n_seg)) W.seg[tid] = run_of(p, G, R, tid);  // the step's first barrier publishes it
  }
  const unsigned lt = (1u << lane) - 1;
  const float r3 = sqrtf(cut2) * 1.0001f + 1e-4f;  // z-window half width, rounded up
  out += (int64_t)(NW == 1 ? 0 : warp) * p.Mz * 32 + lane;
  out_rho += (int64_t)(NW == 1 ? 0 : warp) * p.Mz * 32 + lane;

  int ring_lo = 1 << 30, ring_hi = (1 << 30) - 1;  // empty
  unsigned n_acc = 0;
  unsigned long long n_tst = 0;
  for (int z0 = z_lo; z0 < z_hi; z0 += SL) {
    Slices<SL> S;
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      S.has[k] = z0 + k < p.Mz;
      const int2 e = p.ztab[S.has[k] ? z0 + k : z0];
      S.hz[k] = S.has[k] ? e.x : S.hz[0];
      S.zv[k] = S.has[k] ? __int_as_float(e.y) : 0.f;
    }
    // the table gives each pair's depths from its even slice's home cell
#pragma unroll
    for (int k = 2; k < SL; ++k)
      if (S.has[k]) S.zv[k] = __fadd_rn(S.zv[k], __fmul_rn(G.a33s, (float)(S.hz[k & ~1] - S.hz[0])));
    int hz_last = S.hz[0];
    float zv_last = S.zv[0];
#pragma unroll
    for (int k = 1; k < SL; ++k)
      if (S.has[k]) {
        hz_last = S.hz[k];
        zv_last = S.zv[k];
      }
    const int need_lo = S.hz[0] - 1, need_hi = hz_last + 1;
    bool ok = need_hi - need_lo + 1 <= kRing;  // the host takes four slices only where they fit
    if (need_lo > ring_hi || need_hi < ring_lo) {
      ring_lo = need_lo;
      ring_hi = need_lo - 1;
    }
    if (ring_lo < need_lo) ring_lo = need_lo;
    sync<NW>();  // every warp is done with the previous step's slabs and window
    while (ok && ring_hi < need_hi) {
      ++ring_hi;
      ok = load_slab_cta(p, G, R, ring_hi, W);
    }

    // the atoms of the slabs inside the step's depth window, in slab and gather order: flags and
    // counts first, then their depth terms, one atom per thread
    int n_win = 0;
    if (ok) {
      int pre[kRing + 1];  // first index of each slab in the step's index space
      pre[0] = 0;
#pragma unroll
      for (int s = 0; s < kRing; ++s) pre[s + 1] = pre[s] + (need_lo + s <= need_hi ? W.count[(need_lo + s) & (kRing - 1)] : 0);
      auto place = [&](int i, int& s) {  // slab number of index i, and its place in p
        s = (i >= pre[1]) + (i >= pre[2]) + (i >= pre[3]);
        const int first = s == 0 ? 0 : s == 1 ? pre[1] : s == 2 ? pre[2] : pre[3];
        return ((need_lo + s) & (kRing - 1)) * CAP + i - first;
      };
      const int total = pre[kRing], rounds = (total + 32 * NW - 1) / (32 * NW);
      unsigned flags = 0;
      for (int r = 0; r < rounds; ++r) {
        const int i = r * 32 * NW + tid;
        bool in = false;
        if (i < total) {
          int s;
          const int j = place(i, s);
          const float zr = __fadd_rn(W.p[j].z, __fmul_rn(G.a33s, (float)(s - 1)));
          in = zr >= S.zv[0] - r3 && zr <= zv_last + r3;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) flags |= 1u << r;
        if (lane == 0) W.wcnt[r * NW + warp] = __popc(m);
      }
      sync<NW>();
      const int nc = rounds * NW;
      const int c0 = lane < nc ? W.wcnt[lane] : 0;
      const int i0 = warp_scan(c0, lane);
      n_win = __shfl_sync(0xffffffffu, i0, 31);
      int c1 = 0, i1 = 0;
      if (W_::kRounds * NW > 32 && nc > 32) {
        c1 = 32 + lane < nc ? W.wcnt[32 + lane] : 0;
        i1 = n_win + warp_scan(c1, lane);
        n_win = __shfl_sync(0xffffffffu, i1, 31);
      }
      if (n_win > WCAP) ok = false;
      for (int r = 0; ok && r < rounds; ++r) {
        const int q = r * NW + warp;
        int base = __shfl_sync(0xffffffffu, i0 - c0, q & 31);
        if (W_::kRounds * NW > 32) {
          const int b1 = __shfl_sync(0xffffffffu, i1 - c1, q & 31);
          if (q >= 32) base = b1;
        }
        const bool in = flags >> r & 1;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (!in) continue;
        int s;
        const int j = place(r * 32 * NW + tid, s), d = base + __popc(m & lt);
        const float4 q4 = W.p[j];
        const float zo = __fmul_rn(G.a33s, (float)(s - 1));  // the slab's origin relative to hz[0]'s
        const float2 cs = W.cs[j];
        float hm[4] = {kOff, kOff, kOff, kOff}, hmax = kOff, w[4];
#pragma unroll
        for (int k = 0; k < SL; ++k) {
          const float dz = __fsub_rn(q4.z, __fsub_rn(S.zv[k], zo));
          // a slab serves a slice within the cutoff; with z cells shorter than 3 sigma the
          // reference searches only the 27 cells around each voxel's home cell, so it serves
          // a slice only within one cell of that slice's home z cell
          const int dc = need_lo + s - S.hz[k];
          hm[k] = S.has[k] && !(p.trunc_z && (dc < -1 || dc > 1)) ? __fmaf_rn(-dz, dz, cut2) : kOff;
          hmax = fmaxf(hmax, hm[k]);
          w[k] = ex2_approx(-dz * dz);
        }
        // margin: the lanes' own rounding of dxy^2 must not reach below the rectangle's
        W.r[d] = make_float4(q4.x, q4.y, fmaf(hmax, 1.0001f, 1e-4f), q4.w);
        if constexpr (SL == 4) W.h[d] = make_float4(hm[0], hm[1], hm[2], hm[3]);
        else W.h[d] = make_float2(hm[0], hm[1]);
        W.e0[d] = make_float4(w[0] * cs.x, w[0] * cs.y, w[1] * cs.x, w[1] * cs.y);
        if constexpr (SL == 4) W.e1[d] = make_float4(w[2] * cs.x, w[2] * cs.y, w[3] * cs.x, w[3] * cs.y);
      }
    }
    if (!ok) {
      if (tid == 0) atomicExch(&p.counters[4], 1ull);
      return false;  // the host recomputes with larger slabs, or the general kernel
    }
    sync<NW>();
    if (!work) continue;

    // the atoms that some column of the patch accepts at some slice
    unsigned short* L = W.li[warp];
    int n = 0;
    for (int i0 = 0; i0 < n_win; i0 += 32) {
      const int i = i0 + lane;
      bool keep = false;
      if (i < n_win) {
        const float4 q = W.r[i];
        const float dx = fmaxf(0.f, fabsf(q.x - pxc) - pxh), dy = fmaxf(0.f, fabsf(q.y - pyc) - pyh);
        keep = fmaf(dx, dx, dy * dy) <= q.z;
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) L[n + __popc(m & lt)] = (unsigned short)(i << 4);
      n += __popc(m);
    }
    if (lane < CPL) L[n + lane] = (unsigned short)(WCAP << 4);  // pads the list to whole rounds of the groups
    __syncwarp();

    float2 a[CPL][SL];
    float rm[CPL][SL];  // density: min of dxy^2 - hmax_k = r^2 - (3 sigma)^2
#pragma unroll
    for (int c = 0; c < CPL; ++c)
#pragma unroll
      for (int k = 0; k < SL; ++k) {
        a[c][k] = make_float2(0.f, 0.f);
        rm[c][k] = FLT_MAX;
      }
    const char* RB = reinterpret_cast<const char*>(W.r);
    const char* HB = reinterpret_cast<const char*>(W.h);
    const char* E0 = reinterpret_cast<const char*>(W.e0);
    const char* E1 = reinterpret_cast<const char*>(W.e1);
    // (unrolled by two, the loop's branch and index arithmetic cost two slices per step most: 4.8M atoms at one
    // sigma a slice 3.93 ms, 3.78 by four, 3.71 by eight; four slices 2.43, 2.39, 2.38)
#pragma unroll 8
    for (int i = 0; i < n; i += CPL) {
      const unsigned o = L[i + grp];
      const float2 q = *reinterpret_cast<const float2*>(RB + o);
      float4 hm = make_float4(kOff, kOff, kOff, kOff);
      if constexpr (SL == 4) {
        hm = *reinterpret_cast<const float4*>(HB + o);
      } else {
        const float2 h2 = *reinterpret_cast<const float2*>(HB + (o >> 1));
        hm.x = h2.x;
        hm.y = h2.y;
      }
      const float4 ea = *reinterpret_cast<const float4*>(E0 + o);
      float4 eb = make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (SL == 4) eb = *reinterpret_cast<const float4*>(E1 + o);
      float hh[CPL];
      if constexpr (CPL == 1) {
        const float dx = __fadd_rn(q.x, nX[0]), dy = __fadd_rn(q.y, nY[0]);
        hh[0] = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
      } else {
#pragma unroll
        for (int c = 0; c < CPL; c += 2) {  // two columns per FP32x2 operation, rounded as one column is
          const float2 dy = __fadd2_rn(make_float2(q.y, q.y), make_float2(nY[c], nY[c + 1]));
          float2 dx = make_float2(0.f, 0.f);
          if constexpr (kSameX) dx.x = dx.y = __fadd_rn(q.x, nX[0]);
          else dx = __fadd2_rn(make_float2(q.x, q.x), make_float2(nX[c], nX[c + 1]));
          const float2 h2 = __ffma2_rn(dx, dx, __fmul2_rn(dy, dy));
          hh[c] = h2.x;
          hh[c + 1] = h2.y;
        }
      }
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const float h = hh[c], w = ex2_approx(-h);
        const float2 ww = make_float2(w, w);
        if (h <= hm.x) a[c][0] = __ffma2_rn(ww, make_float2(ea.x, ea.y), a[c][0]);
        if (h <= hm.y) a[c][1] = __ffma2_rn(ww, make_float2(ea.z, ea.w), a[c][1]);
        if constexpr (SL == 4) {
          if (h <= hm.z) a[c][2] = __ffma2_rn(ww, make_float2(eb.x, eb.y), a[c][2]);
          if (h <= hm.w) a[c][3] = __ffma2_rn(ww, make_float2(eb.z, eb.w), a[c][3]);
        }
        if (kDens) {
          rm[c][0] = fminf(rm[c][0], h - hm.x);
          rm[c][1] = fminf(rm[c][1], h - hm.y);
          if constexpr (SL == 4) {
            rm[c][2] = fminf(rm[c][2], h - hm.z);
            rm[c][3] = fminf(rm[c][3], h - hm.w);
          }
        }
        if (kStats && (act >> c & 1)) {
          n_acc += (h <= hm.x) + (h <= hm.y);
          if constexpr (SL == 4) n_acc += (h <= hm.z) + (h <= hm.w);
        }
      }
    }
    if (kStats) n_tst += (unsigned long long)n;
    // the groups' sums: lane l is left with column l of the patch
#pragma unroll
    for (int half = CPL / 2; half >= 1; half /= 2) {
      const int o = half * LPG;         // partner: the group half away
      const bool up = (grp & half) != 0;  // keeps the upper half of the columns it still holds
#pragma unroll
      for (int c = 0; c < half; ++c)
#pragma unroll
        for (int k = 0; k < SL; ++k) {
          const float2 mine = up ? a[c + half][k] : a[c][k], other = up ? a[c][k] : a[c + half][k];
          a[c][k] = __fadd2_rn(mine, make_float2(__shfl_xor_sync(0xffffffffu, other.x, o),
                                                 __shfl_xor_sync(0xffffffffu, other.y, o)));
          if (kDens) {
            const float m = up ? rm[c + half][k] : rm[c][k], t = up ? rm[c][k] : rm[c + half][k];
            rm[c][k] = fminf(m, __shfl_xor_sync(0xffffffffu, t, o));
          }
        }
    }
    {
      // sparse or cancelling sums: re-decide the near-cutoff atoms exactly (see exact_fix)
      unsigned want = 0;
#pragma unroll
      for (int k = 0; k < SL; ++k)
        if (active && n > 0 && S.has[k] && fmaf(a[0][k].x, a[0][k].x, a[0][k].y * a[0][k].y) < kSparse2) want |= 1u << k;
      if (__any_sync(0xffffffffu, want != 0)) {
        if (want) {
          const int2 xt = p.xtab[ix], yt = p.ytab[iy];
          const Column C{col_x(xt), col_y(yt), xt.x, yt.x, p.xfv[ix], p.yfv[iy]};
          const Fix<SL> f = exact_fix(p, W, warp, n, z0, need_lo, G.a33s, cut2, S, want, C);
#pragma unroll
          for (int k = 0; k < SL; ++k) {
            a[0][k].x += f.d[k].x;
            a[0][k].y += f.d[k].y;
          }
          if (kStats) n_acc += (unsigned)f.dn;
        }
        __syncwarp();
      }
    }
#pragma unroll
    for (int k = 0; k < SL; ++k) {
      if (z0 + k >= z_hi) break;
      // x = S / max(1e-16, |S|); with density, rho x and rho are stored
      const float2 v = a[0][k];
      float inv = rsqrtf(fmaxf(fmaf(v.x, v.x, v.y * v.y), 1e-32f));
      if constexpr (kDens) {
        const float rho = p.use_density ? rho_of((cut2 + rm[0][k]) * p.r2_to_A2, (float)p.sigma) : 1.f;
        out_rho[(int64_t)(z0 + k) << 5] = rho;
        inv *= rho;
      }
      out[(int64_t)(z0 + k) << 5] = make_float2(v.x * inv, v.y * inv);
    }
  }
  if (kStats && work) {
    unsigned long long acc_w = n_acc, tst_w = active ? SL * n_tst : 0u;
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

// Persistent over the units (tile and range of slices) of every image of the range: each CTA
// takes the next one from a global counter.
template <typename W_, int CPL, int TX, bool kDens, bool kStats, bool kMasked, int kMinBlocks>
__global__ void __launch_bounds__(W_::NW * 32, kMinBlocks)
    k_field32(const ColumnJob* __restrict__ jobs, int n_jobs, FieldRange R) {
  constexpr int NW = W_::NW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  W_& W = *reinterpret_cast<W_*>(smem_raw);
  if ((int64_t)R.counters[0] > R.cap) return;  // the binning overflowed: the host retries
  if (threadIdx.x == 0) {
    W.r[W_::WCAP] = make_float4(0.f, 0.f, kOff, 0.f);
    if constexpr (W_::SL == 4) W.h[W_::WCAP] = make_float4(kOff, kOff, kOff, kOff);
    else W.h[W_::WCAP] = make_float2(kOff, kOff);
    W.e0[W_::WCAP] = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (W_::SL == 4) W.e1[W_::WCAP] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  int chunk = R.chunk, n_chunks = R.n_chunks, units = R.units() / NW;
  if constexpr (kMasked) {
    const int n = listed_patches(R), deep = jobs[0].p.Mz;
    chunk = warp_depth_chunk((n + NW - 1) / NW, deep, R.slots, kRule32);
    n_chunks = (deep + chunk - 1) / chunk;
    units = n / NW * n_chunks;
  }
  for (;;) {
    sync<NW>();
    // a slab overflowed: the host recomputes with larger slabs
    if (threadIdx.x == 0) W.unit = R.counters[4] != 0 ? units : (int)atomicAdd(R.work, 1u);
    sync<NW>();
    const int unit = W.unit;
    if (unit >= units) break;
    int patch;
    const ColumnJob& J = field_patch(jobs, n_jobs, R.patch_lo + unit / n_chunks * NW, patch);
    const int z_lo = unit % n_chunks * chunk, z_hi = min(J.p.Mz, z_lo + chunk);
    if (z_lo >= z_hi) continue;  // an image less deep than the batch's deepest
    const int64_t o = J.sample_base - R.origin + (int64_t)patch * J.p.Mz * 32;
    if constexpr (kMasked) patch = listed_patch(R, J.p, patch);
    if (!field_tile<CPL, TX, kDens, kStats, kMasked>(J.p, W, patch, z_lo, z_hi, (float2*)R.samples + o, R.rho32 + o))
      break;
  }
}

// ------------------------------------------------------------------------------------------
// The column integrator
// ------------------------------------------------------------------------------------------

// NH angle pairs of one column (T = float: one angle), |phi_g|^2 to out[0 ..].  The equations are
// linear, so the reference's renormalisation after every double step (:2466-2472) only scales
// phi: it is done every 8 steps and at the end (every step when a step could grow phi by more
// than a small factor), which drops a tenth of the operations.
template <typename T, int NH, bool kDens>
__device__ __forceinline__ void integrate(const ColumnParams& p, const float2* __restrict__ X,
                                          const float* __restrict__ RH, const T* a, int every, float* out) {
  T ph[NH][4];
#pragma unroll
  for (int k = 0; k < NH; ++k) {
    ph[k][0] = bc<T>(1.f);
    ph[k][1] = ph[k][2] = ph[k][3] = bc<T>(0.f);
  }
  const float b0 = (float)p.b0, bg = (float)p.bg, dz = (float)p.dz;
  auto sample = [&](int z) {
    const float2 x = X[(int64_t)z << 5];
    return Sample{kDens ? b0 * RH[(int64_t)z << 5] : b0, bg * x.x, bg * x.y};
  };
  Sample s0 = sample(0);
  int n = 0;
  // (1.2M atoms, one angle, 165 us with the steps' parts added one by one, 150 now; density, 128k atoms, 55 and 52,
  // 59 with eight steps unrolled)
  constexpr int kUnroll = kDens ? 2 : 8;
#pragma unroll kUnroll
  for (int z = 2; z <= p.Mz; z += 2) {  // the last sample of an even column is the first (:1898-1899)
    const Sample s1 = sample(z - 1), s2 = sample(z < p.Mz ? z : 0);
#pragma unroll
    for (int k = 0; k < NH; ++k) rk4<T>(s0, s1, s2, a[k], dz, ph[k]);
    s0 = s2;
    if (++n == every) {
      n = 0;
#pragma unroll
      for (int k = 0; k < NH; ++k) renormalise(ph[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < NH; ++k) {
    renormalise(ph[k]);
    const T ig = fma_(ph[k][2], ph[k][2], mul_(ph[k][3], ph[k][3]));
    if constexpr (std::is_same<T, float>::value) {
      out[0] = ig;
    } else {
      out[2 * k] = ig.x;
      out[2 * k + 1] = ig.y;
    }
  }
}

template <int TX>
__device__ __forceinline__ bool patch_pixel(const ColumnParams& p, int patch, int lane, int64_t& o) {
  const int tiles_x = (p.ix1 - p.ix0 + kTileX - 1) / kTileX, tile = patch >> 2;
  int ix, iy;
  patch_column<TX>(p.ix0 + tile % tiles_x * kTileX, p.iy0 + tile / tiles_x * kTileY, patch & 3, lane, ix, iy);
  o = ix + (int64_t)p.Mx * iy;
  if (ix >= p.ix1 || iy >= p.iy1) return false;
  return !p.tile_mask || p.tile_mask[(iy / p.mask_T) * p.mask_ntx + ix / p.mask_T] != 0;
}

__device__ __forceinline__ void write_pixel(const ColumnParams& p, int64_t o, double v) {
  if (p.finalize) {  // the precession average and the bright-field flip (k_epilogue's arithmetic)
    v = __ddiv_rn(v, p.fin_scale);
    if (p.fin_bright) v = __dsub_rn(1.0, v);
  }
  p.img[o] = v;
}

// Every image with one angle: a warp per patch, four patches per CTA.
template <int TX, bool kDens>
__global__ void __launch_bounds__(128) k_integrate32(const ColumnJob* __restrict__ jobs, int n_jobs, FieldRange R) {
  const int lane = threadIdx.x, g = R.patch_lo + blockIdx.x * 4 + threadIdx.y;
  if (g == R.patch_lo && lane == 0) *R.work = 0;  // for the next field kernel
  if ((int64_t)R.counters[0] > R.cap || R.counters[4] != 0 || g >= R.patch_hi) return;
  if (R.list && g - R.patch_lo >= listed_patches(R)) return;
  int patch;
  const ColumnJob& J = field_patch(jobs, n_jobs, g, patch);
  const int64_t o = J.sample_base - R.origin + (int64_t)patch * J.p.Mz * 32 + lane;
  if (R.list) patch = listed_patch(R, J.p, patch);
  int64_t px;
  const bool wanted = patch_pixel<TX>(J.p, patch, lane, px);
  if (!__any_sync(0xffffffffu, wanted)) return;
  const float a = J.p.aaf[0];
  float ig;
  integrate<float, 1, kDens>(J.p, (const float2*)R.samples + o, R.rho32 + o, &a, J.p.renorm32, &ig);
  if (wanted) write_pixel(J.p, px, (double)ig);
}

// Several angles: a CTA per patch; warp w takes the angles 2 NH w .. of every group of 16, the
// group's sum is formed in angle order, the groups' sums in FP64.
template <int TX, int NH, bool kDens>
__global__ void __launch_bounds__(128) k_integrate32_multi(const ColumnJob* __restrict__ jobs, int n_jobs,
                                                           FieldRange R) {
  __shared__ float part[16][32];
  const int lane = threadIdx.x, warp = threadIdx.y;
  if (blockIdx.x == 0 && warp == 0 && lane == 0) *R.work = 0;  // for the next field kernel
  if ((int64_t)R.counters[0] > R.cap || R.counters[4] != 0) return;
  int patch;
  const ColumnJob& J = field_patch(jobs, n_jobs, R.patch_lo + blockIdx.x, patch);
  const ColumnParams& p = J.p;
  int64_t px;
  const bool wanted = patch_pixel<TX>(p, patch, lane, px);
  if (!__any_sync(0xffffffffu, wanted)) return;
  const int64_t o = J.sample_base - R.origin + (int64_t)patch * p.Mz * 32 + lane;
  double total = 0.0;
  for (int k0 = 0; k0 < p.n_prec; k0 += 16) {
    const int np = min(16, p.n_prec - k0);
    for (int k = 2 * NH * warp; k < np; k += 2 * NH * blockDim.y) {
      float2 a[NH];  // the table is padded to an even count
      float ig[2 * NH];
#pragma unroll
      for (int i = 0; i < NH; ++i)
        a[i] = k + 2 * i < np ? make_float2(p.aaf[k0 + k + 2 * i], p.aaf[k0 + k + 2 * i + 1]) : make_float2(0.f, 0.f);
      integrate<float2, NH, kDens>(p, (const float2*)R.samples + o, R.rho32 + o, a, p.renorm32, ig);
#pragma unroll
      for (int i = 0; i < 2 * NH; ++i)
        if (k + i < np) part[k + i][lane] = ig[i];
    }
    __syncthreads();
    if (warp == 0) {
      float acc = 0.f;
      for (int k = 0; k < np; ++k) acc = __fadd_rn(acc, part[k][lane]);
      total += (double)acc;
    }
    __syncthreads();
  }
  if (warp == 0 && wanted) write_pixel(p, px, total);
}

template <int TX, bool kDens>
cudaError_t launch_integrate(const ColumnJob* jobs, int n_jobs, const FieldRange& R, int max_np, cudaStream_t st) {
  const int patches = R.patch_hi - R.patch_lo;
  ++launch_count();
  if (max_np <= 1)
    k_integrate32<TX, kDens><<<(patches + 3) / 4, dim3(32, 4), 0, st>>>(jobs, n_jobs, R);
  else if (max_np <= 8)
    k_integrate32_multi<TX, 1, kDens><<<patches, dim3(32, (max_np + 1) / 2), 0, st>>>(jobs, n_jobs, R);
  else
    k_integrate32_multi<TX, 2, kDens><<<patches, dim3(32, 4), 0, st>>>(jobs, n_jobs, R);
  return cudaGetLastError();
}

template <int CAP, int WCAP, int NW, int SL, int TX, bool kDens, bool kStats, bool kMasked, int B>
cudaError_t launch(const ColumnJob* jobs, int n_jobs, FieldRange R, int max_np, cudaStream_t st) {
  static_assert((sizeof(Smem<CAP, WCAP, NW, SL>) + 1024) * B <= 232448, "shared memory of B CTAs");
  using W = Smem<CAP, WCAP, NW, SL>;
  auto kernel = k_field32<W, kCPL, TX, kDens, kStats, kMasked, B>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W));
  if (e != cudaSuccess) return e;
  split_depth(R, NW, sm_count() * B, kRule32);
  const int grid = std::max(1, std::min(sm_count() * B, R.list ? R.patch_hi - R.patch_lo : R.units() / NW));
  ++launch_count();
  kernel<<<grid, NW * 32, sizeof(W), st>>>(jobs, n_jobs, R);
  e = cudaGetLastError();
  return e == cudaSuccess ? launch_integrate<TX, kDens>(jobs, n_jobs, R, max_np, st) : e;
}

// Tuning variants (tier 0): the patch shape and the slab capacity.  A masked launch takes its
// variant's patch shape, so that the masked columns equal the plain image's; tiers 1 and 2, the
// statistics and the two-slice instances use 8 x 4 patches.  Images of one patch shape are the same
// to the last bit (the shapes distribute an atom list over the groups of lanes differently).
template <int SL, bool kDens, bool kStats, bool kMasked>
cudaError_t dispatch(const ColumnJob* jobs, int n_jobs, const FieldRange& R, int max_np, int variant, int tier,
                     cudaStream_t st) {
  // Denser slabs, or coarser voxels: as much staging as three and as two CTAs per SM leave (four with two
  // slices per step, whose window entries are smaller), then one warp per patch, and at last a window that holds
  // all of its slabs.  With 352 / 704 atoms at two CTAs and then a warp per patch, 400k atoms of two interpenetrating
  // bcc cells at 1.2 A voxels took 1.98 ms (0.84 with slabs per warp before, 0.89 now), 0.6 A 2.71 (2.31, 2.34), 800k of
  // two fcc cells at 0.72 A 4.76 (2.20, 1.75), 400k fcc atoms at 0.9 A 0.83 (0.83, 0.69).
  if (tier >= 4) return launch<256, 1024, 1, SL, 8, kDens, kStats, kMasked, 2>(jobs, n_jobs, R, max_np, st);
  if (tier == 3) return launch<256, 512, 1, SL, 8, kDens, kStats, kMasked, SL == 2 ? 4 : 3>(jobs, n_jobs, R, max_np, st);
  if constexpr (kMasked)  // halves of tiles (field32_halves)
    if (tier == 0 && R.per_item == 2)
      return launch<SL == 2 ? 128 : 112, SL == 2 ? 240 : 208, 2, SL, 8, kDens, kStats, kMasked, 8>(jobs, n_jobs, R,
                                                                                                 max_np, st);
  if constexpr (SL == 4) {
    if (tier == 2) return launch<416, 960, 4, SL, 8, kDens, kStats, kMasked, 2>(jobs, n_jobs, R, max_np, st);
    if (tier == 1) return launch<288, 608, 4, SL, 8, kDens, kStats, kMasked, 3>(jobs, n_jobs, R, max_np, st);
  } else {
    if (tier == 2) return launch<512, 1024, 4, SL, 8, kDens, kStats, kMasked, 2>(jobs, n_jobs, R, max_np, st);
    if (tier == 1) return launch<320, 512, 4, SL, 8, kDens, kStats, kMasked, 4>(jobs, n_jobs, R, max_np, st);
    return launch<192, 384, 4, SL, 8, kDens, kStats, kMasked, 4>(jobs, n_jobs, R, max_np, st);
  }
  if constexpr (SL == 4 && !kStats) {
    switch (variant) {
      case 1: return launch<160, 288, 4, SL, 8, kDens, kStats, kMasked, kField32Blocks>(jobs, n_jobs, R, max_np, st);
      case 2: return launch<192, 384, 4, SL, 4, kDens, kStats, kMasked, 4>(jobs, n_jobs, R, max_np, st);
      case 3: return launch<160, 288, 4, SL, 4, kDens, kStats, kMasked, kField32Blocks>(jobs, n_jobs, R, max_np, st);
      case 4: return launch<192, 384, 4, SL, 16, kDens, kStats, kMasked, 4>(jobs, n_jobs, R, max_np, st);
      case 5: return launch<160, 288, 4, SL, 16, kDens, kStats, kMasked, kField32Blocks>(jobs, n_jobs, R, max_np, st);
      default: break;
    }
  }
  return launch<192, 384, 4, SL, 8, kDens, kStats, kMasked, 4>(jobs, n_jobs, R, max_np, st);
}

template <int SL, bool kDens>
cudaError_t dispatch2(const ColumnJob* jobs, int n_jobs, const FieldRange& R, int max_np, int variant, int tier,
                      bool stats, bool masked, cudaStream_t st) {
  if (stats) return dispatch<SL, kDens, true, false>(jobs, n_jobs, R, max_np, variant, tier, st);
  if (masked) return dispatch<SL, kDens, false, true>(jobs, n_jobs, R, max_np, variant, tier, st);
  return dispatch<SL, kDens, false, false>(jobs, n_jobs, R, max_np, variant, tier, st);
}

constexpr int kVariants = 6;
const char* const kNames[kVariants] = {"8x4 slab128", "8x4 slab96", "4x8 slab128", "4x8 slab96", "16x2 slab128",
                                       "16x2 slab96"};

}  // namespace field32

int field32_patches(const ColumnParams& p) {
  const int Wd = p.ix1 - p.ix0, Hd = p.iy1 - p.iy0;
  if (Wd <= 0 || Hd <= 0) return 0;
  return 4 * ((Wd + field32::kTileX - 1) / field32::kTileX) * ((Hd + field32::kTileY - 1) / field32::kTileY);
}

namespace {
__global__ void __launch_bounds__(256) k_wanted_tiles(const ColumnJob* __restrict__ job, int tiles, int across, int tx,
                                                      int ty, int* __restrict__ list,
                                                      unsigned long long* __restrict__ count) {
  const ColumnParams& p = job->p;
  const int i = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31;
  bool want = false;
  const int x0 = p.ix0 + i % across * tx, y0 = p.iy0 + i / across * ty;
  if (i < tiles && x0 < p.ix1) {
    const int x1 = min(x0 + tx, p.ix1) - 1, y1 = min(y0 + ty, p.iy1) - 1;
    for (int my = y0 / p.mask_T; my <= y1 / p.mask_T; ++my)
      for (int mx = x0 / p.mask_T; mx <= x1 / p.mask_T; ++mx) want = want || p.tile_mask[my * p.mask_ntx + mx] != 0;
  }
  const unsigned m = __ballot_sync(0xffffffffu, want);
  if (!m) return;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (want) list[base + __popc(m & ((1u << lane) - 1))] = i;
}
}  // namespace

cudaError_t launch_wanted_tiles(const ColumnJob* d_job, int tiles, int across, int tx, int ty, int* list,
                                unsigned long long* count, cudaStream_t st) {
  ++launch_count();
  k_wanted_tiles<<<(tiles + 255) / 256, 256, 0, st>>>(d_job, tiles, across, tx, ty, list, count);
  return cudaGetLastError();
}

// A mask whose tiles are an odd number of 8 pixels wide often wants one half of a 16 x 8 tile: two warps and the
// atoms about 8 x 8 pixels then (4.8M atoms, 480 slices, 7 % of the tiles of 8 pixels 4.44 ms, by whole tiles 5.73;
// all of them 49.3 and 44.0: above some 85 % whole tiles would be the better).
bool field32_halves(int mask_T, int variant, int slab_tier) {
  return mask_T % 16 != 0 && ring_variant_same(variant) && slab_tier == 0;
}

int ring_variant_count() { return field32::kVariants; }

int ring_variant_slab(int variant) { return variant == 1 || variant == 3 || variant == 5 ? 96 : 128; }

bool ring_variant_same(int variant) { return variant < 2; }  // the 8 x 4 patches

const char* ring_variant_name(int variant) {
  return variant >= 0 && variant < field32::kVariants ? field32::kNames[variant] : "invalid";
}

cudaError_t launch_field32(const ColumnJob* d_jobs, int n_jobs, const FieldRange& R, int max_np, bool density,
                           bool stats, bool masked, bool four, int variant, int slab_tier, cudaStream_t st) {
  if (masked && stats) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (R.units() <= 0) return e;
  using namespace field32;
  if (four)
    return density ? dispatch2<4, true>(d_jobs, n_jobs, R, max_np, variant, slab_tier, stats, masked, st)
                   : dispatch2<4, false>(d_jobs, n_jobs, R, max_np, variant, slab_tier, stats, masked, st);
  return density ? dispatch2<2, true>(d_jobs, n_jobs, R, max_np, variant, slab_tier, stats, masked, st)
                 : dispatch2<2, false>(d_jobs, n_jobs, R, max_np, variant, slab_tier, stats, masked, st);
}

}  // namespace stem
