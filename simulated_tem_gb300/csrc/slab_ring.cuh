// Staging of link-cell slabs for the column kernels: one warp gathers the atoms of a slab
// (one z cell of the link-cell grid) that lie within 3 sigma of its patch of pixel columns
// into warp-private shared memory, ordered by z bin, once per slab of its march in depth.
#pragma once
#include <cuda_runtime.h>

#include "internal.h"

namespace stem {
namespace slab {

constexpr int kRing = 4;    // resident slabs (unwrapped z cells u, slot u & 3)
constexpr int kBins = 32;   // z bins per slab for the window lookup (at most 32: one lane each)

// Lengths inside the kernel are scaled by s = sqrt(log2(e) / (2 sigma^2)), so that the
// Gaussian weight exp(-r^2 / (2 sigma^2)) is ex2(-r'^2) of the scaled distance r'.
struct Geo {
  int ux_lo, ux_hi, uy_lo, uy_hi, ux_ref, uy_ref;
  float xmin, xmax, ymin, ymax, pre2;
  float a11s, a22s, a33s, scale;
};

// The frame and footprint of a patch: its home cells' range with one cell around, and its columns'
// sample rectangle in scaled lengths from the patch's reference cell (the first home cell); Xv, Yv
// receive this lane's column.  Lanes off the image (not active) do not widen the footprint.
__device__ __forceinline__ void patch_frame(const ColumnParams& p, Geo& G, double sd, bool active, int hx, int hy,
                                            double fvx, double fvy, float& Xv, float& Yv) {
  G.scale = (float)sd;
  const int big = 1 << 29;
  const int mnx = __reduce_min_sync(0xffffffffu, active ? hx : big);
  const int mxx = __reduce_max_sync(0xffffffffu, active ? hx : -big);
  const int mny = __reduce_min_sync(0xffffffffu, active ? hy : big);
  const int mxy = __reduce_max_sync(0xffffffffu, active ? hy : -big);
  G.ux_lo = mnx - 1;
  G.ux_hi = mxx + 1;
  G.uy_lo = mny - 1;
  G.uy_hi = mxy + 1;
  G.ux_ref = mnx;
  G.uy_ref = mny;
  G.a11s = (float)(p.a11 * sd);
  G.a22s = (float)(p.a22 * sd);
  G.a33s = (float)(p.a33 * sd);
  Xv = (float)(p.a11 * (fvx + (double)(hx - G.ux_ref)) * sd);
  Yv = (float)(p.a22 * (fvy + (double)(hy - G.uy_ref)) * sd);
  const float fbig = 1e30f;
  float v = active ? Xv : fbig, w = active ? -Xv : fbig, y = active ? Yv : fbig, z = active ? -Yv : fbig;
  for (int o = 16; o > 0; o >>= 1) {
    v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    w = fminf(w, __shfl_xor_sync(0xffffffffu, w, o));
    y = fminf(y, __shfl_xor_sync(0xffffffffu, y, o));
    z = fminf(z, __shfl_xor_sync(0xffffffffu, z, o));
  }
  G.xmin = v;
  G.xmax = -w;
  G.ymin = y;
  G.ymax = -z;
}

__device__ __forceinline__ int pos_mod(int a, int n) {
  const int r = a % n;
  return r < 0 ? r + n : r;
}

__device__ __forceinline__ int floor_div(int a, int n) { return (a >= 0) ? a / n : -((-a + n - 1) / n); }

// One gathered candidate: atom j of a cell in row uy, x cells shifted by `shift` (an
// unwrapped run), in the warp's scaled frame; keep when within 3 sigma of the patch.
template <bool kCellCode>
__device__ __forceinline__ bool slab_candidate(const ColumnParams& p, const Geo& G, int j, int shift, int uy,
                                               float4& rec) {
  const float4 r = p.p32[j];
  const int packed = __float_as_int(r.w);
  const int cxu = (packed & 1023) + shift;
  const float X = __fmaf_rn(r.x, G.scale, __fmul_rn(G.a11s, (float)(cxu - G.ux_ref)));
  const float Y = __fmaf_rn(r.y, G.scale, __fmul_rn(G.a22s, (float)(uy - G.uy_ref)));
  const float dx = fmaxf(0.f, fmaxf(G.xmin - X, X - G.xmax));
  const float dy = fmaxf(0.f, fmaxf(G.ymin - Y, Y - G.ymax));
  const float w4 = kCellCode ? __int_as_float((cxu - G.ux_ref + 8) | ((uy - G.uy_ref + 8) << 8)) : p.ph32[j];
  rec = make_float4(X, Y, __fmul_rn(r.z, G.scale), w4);
  return dx * dx + dy * dy <= G.pre2;
}

// Appends the kept candidates of one 32-lane round (ballot + popc, order kept); false
// when the slab would exceed CAPS.
template <int CAPS>
__device__ __forceinline__ bool slab_append(float4* P, int* GI, int& n, bool keep, const float4& rec, int j,
                                            int lane) {
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  const int cnt = __popc(m);
  if (n + cnt > CAPS) return false;
  if (keep) {
    const int d = n + __popc(m & ((1u << lane) - 1));
    P[d] = rec;
    GI[d] = j;
  }
  n += cnt;
  return true;
}

// Gather slab u (its cells in the patch footprint, atoms within 3 sigma of the
// patch rectangle) into its ring slot and order it by z bin in place; false
// when it holds more than CAPS atoms.
// The fourth float of an entry holds the atom's unwrapped cell relative to the warp's
// reference cells, (ux - ux_ref + 8) | (uy - uy_ref + 8) << 8 (exact distances need it).  WS: any
// warp-memory layout with the slab arrays p, gi, bin and count.
//
// The footprint is rows uy of x runs (a run ends where x wraps): segments of consecutive
// atoms.  Up to 8 segments, the lanes look up all segment ranges at once,
// join them into one index space (the slot's bin array, free until the sort, holds the
// table) and gather two 32-lane rounds at a time; otherwise row by row, one round at a
// time.  Both routes visit the atoms in the same order (rows, runs, atoms), so the slab's contents
// and order do not depend on the route.
template <int CAPS, typename WS>
__device__ bool load_slab(const ColumnParams& p, const Geo& G, int u, WS& W, int lane) {
  const int cz = pos_mod(u, p.Ez);
  const int slot = u & (kRing - 1);
  float4* P = W.p[slot];
  int* GI = W.gi[slot];
  int n = 0;
  constexpr int kMaxSeg = 8;
  static_assert(4 * kMaxSeg + 1 <= kBins + 1, "the segment table lives in a slot's bin array");
  const int k_lo = floor_div(G.ux_lo, p.Ex), k_hi = floor_div(G.ux_hi, p.Ex);
  const int n_run = max(0, k_hi - k_lo + 1), n_seg = max(0, G.uy_hi - G.uy_lo + 1) * n_run;
  if (n_seg >= 1 && n_seg <= kMaxSeg) {
    int* seg = W.bin[slot];  // per segment: first index, first atom, x shift, row; then the total
    int len = 0, a_lo = 0, shift = 0, uy = 0;
    if (lane < n_seg) {
      const int k = k_lo + lane % n_run;
      uy = G.uy_lo + lane / n_run;
      shift = k * p.Ex;
      const int x0 = max(G.ux_lo, shift), x1 = min(G.ux_hi, shift + p.Ex - 1);
      const int64_t row_base = (int64_t)p.Ex * (pos_mod(uy, p.Ey) + (int64_t)p.Ey * cz);
      a_lo = p.cell_start[row_base + (x0 - shift)];
      len = p.cell_start[row_base + (x1 - shift) + 1] - a_lo;
    }
    int incl = len;
#pragma unroll
    for (int o = 1; o < kMaxSeg; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, kMaxSeg - 1);
    if (lane < n_seg) {
      seg[4 * lane] = incl - len;
      seg[4 * lane + 1] = a_lo;
      seg[4 * lane + 2] = shift;
      seg[4 * lane + 3] = uy;
    }
    if (lane == 0) seg[4 * n_seg] = total;
    __syncwarp();
    int sg = 0;  // this lane's segment (its indices only grow)
    auto locate = [&](int i, int& j, int& sh, int& y) {
      while (i >= seg[4 * (sg + 1)]) ++sg;
      j = seg[4 * sg + 1] + (i - seg[4 * sg]);
      sh = seg[4 * sg + 2];
      y = seg[4 * sg + 3];
    };
    constexpr int kRounds = 2;
    for (int b = 0; b < total; b += 32 * kRounds) {
      int j[kRounds];
      bool keep[kRounds];
      float4 rec[kRounds];
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const int i = b + 32 * r + lane;
        int sh = 0, y = 0;
        j[r] = 0;
        keep[r] = false;
        rec[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < total) {
          locate(i, j[r], sh, y);
          keep[r] = slab_candidate<true>(p, G, j[r], sh, y, rec[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
        if (b + 32 * r < total && !slab_append<CAPS>(P, GI, n, keep[r], rec[r], j[r], lane)) return false;
    }
  } else {
    for (int uy = G.uy_lo; uy <= G.uy_hi; ++uy) {
      const int64_t row_base = (int64_t)p.Ex * (pos_mod(uy, p.Ey) + (int64_t)p.Ey * cz);
      for (int k = k_lo; k <= k_hi; ++k) {
        const int shift = k * p.Ex;
        const int x0 = max(G.ux_lo, shift), x1 = min(G.ux_hi, shift + p.Ex - 1);
        const int a_lo = p.cell_start[row_base + (x0 - shift)];
        const int a_hi = p.cell_start[row_base + (x1 - shift) + 1];
        for (int b = a_lo; b < a_hi; b += 32) {
          const int j = b + lane;
          bool keep = false;
          float4 rec = make_float4(0.f, 0.f, 0.f, 0.f);
          if (j < a_hi) keep = slab_candidate<true>(p, G, j, shift, uy, rec);
          if (!slab_append<CAPS>(P, GI, n, keep, rec, j, lane)) return false;
        }
      }
    }
  }
  __syncwarp();
  // counting sort by z bin, in place: every lane first holds its atoms in registers;
  // within a bin the gather order is kept (deterministic)
  constexpr int kPer = CAPS / 32;
  const float inv_bin = kBins / G.a33s;
  int* hist = W.bin[slot];
  for (int b = lane; b <= kBins; b += 32) hist[b] = 0;
  __syncwarp();
  float4 e[kPer];
  int es[kPer];
  int eb[kPer], er[kPer];
  const unsigned lt = (1u << lane) - 1;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = lane + 32 * k;
    const bool valid = i < n;
    e[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    es[k] = 0;
    eb[k] = 0;
    er[k] = 0;
    const unsigned act = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      e[k] = P[i];
      es[k] = GI[i];
      eb[k] = min(kBins - 1, max(0, (int)floorf(e[k].z * inv_bin)));
      const unsigned m = __match_any_sync(act, eb[k]);
      er[k] = hist[eb[k]] + __popc(m & lt);
      __syncwarp(act);
      if ((m & lt) == 0) hist[eb[k]] += __popc(m);  // the group's first lane counts it
    }
    __syncwarp();
  }
  // exclusive scan of the 32 bin counts: bin starts, bin[kBins] = n
  {
    const int v = lane < kBins ? hist[lane] : 0;
    int incl = v;
    for (int o = 1; o < kBins; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncwarp();
    if (lane < kBins) hist[lane] = incl - v;
    if (lane == 0) hist[kBins] = n;
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    if (lane + 32 * k < n) {
      const int d = hist[eb[k]] + er[k];
      P[d] = e[k];
      GI[d] = es[k];
    }
  }
  __syncwarp();
  if (lane == 0) W.count[slot] = n;
  __syncwarp();
  return true;
}

}  // namespace slab
}  // namespace stem
