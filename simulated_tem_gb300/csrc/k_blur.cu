// K4: the separable Gaussian blur of d2bi's PNG output (src/d2bi.f90:1543-1624).
//
// x pass:  f_x(ix,iy) = sum_{jj=max(0,ix-Nk)}^{min(Nx-1,ix+Nk)} k(|jj-ix|) f(jj,iy),
//          w_stripe(ix) = 1 / sum of the same weights;
// y pass:  out(ix,iy) = [sum_jj k(|jj-iy|) f_x(ix,jj)] * w_stripe(ix) / (sum of those weights).
// The weights k are computed on the host exactly as the reference does; the
// sums run in ascending jj with separately rounded operations, so the result
// equals the reference's double arithmetic.
//
// FP64 arithmetic is what bounds it: one warp instruction per 19 cycles and SM.  The sum of the
// weights is the same for a whole column (row), so it is formed once per column and row, and the
// rounded products k f are formed by the integer units (rounded_product), which the FP64 unit's 76
// cycles per warp and scheduler leave idle: one FP64 instruction per tap is left of three.
// Both passes are one kernel: a warp sums 64 neighbouring pixels of a line from shared memory and
// writes them transposed, so that the second pass reads lines again.  The 8-byte stores of 32 lines
// meet in the L2 cache, which holds the intermediate image at the sizes d2bi produces.
// 1132 x 1131 pixels at t = 6.97 (71 taps): 1095 us with the sums of the weights and the products on
// the FP64 unit, 419 us now (whole call; the additions alone need 370).  300 x 200 at t = 3.3: 76 and
// 58 us, 70 x 61 at t = 6.9: 70 and 62 us, most of them the copy of the weights and the launches.
#include <cuda_runtime.h>

#include "internal.h"
#include "rounded_product.h"

namespace stem {
namespace {

constexpr int kOut = 64;     // pixels of a warp, two per lane
constexpr int kTaps = 96;    // taps per fill of the buffers: a blur of t <= 9.5 pixels takes one fill
constexpr int kBlurWarps = 4;

struct BlurLines {
  const double* in;
  double* out;             // transposed: pixel o of line l at o * lines + l
  int len, lines;
  const double* kern;
  int nk;
  double* w_out;           // first pass: 1 / sum per pixel of a line, then the sum per line of the second
  const double* w_line;    // second pass: the factor of each line, and
  const double* w_pix;     // the divisor of each pixel
};

// Sum of the weights that reach pixel o of a line, in ascending order.
__device__ __forceinline__ double weight_sum(const double* __restrict__ kern, int nk, int o, int len) {
  const int lo = max(0, o - nk), left = o - lo, right = min(len - 1 - o, nk);
  double ws = 0.0;
  for (int d = -left; d <= right; ++d) ws = __dadd_rn(ws, kern[abs(d)]);
  return ws;
}

template <bool kFirst>
__global__ void __launch_bounds__(32 * kBlurWarps) k_blur_lines(BlurLines a, int weight_blocks) {
  __shared__ uint4 s_f[kBlurWarps][kTaps + kOut];
  __shared__ uint4 s_k[kBlurWarps][kTaps];
  int64_t block = blockIdx.x;
  if constexpr (kFirst) {  // the first blocks: the weight sums of both passes
    if (block < weight_blocks) {
      const int64_t i = block * blockDim.x + threadIdx.x;
      if (i < a.len) a.w_out[i] = __ddiv_rn(1.0, weight_sum(a.kern, a.nk, (int)i, a.len));
      else if (i - a.len < a.lines) a.w_out[i] = weight_sum(a.kern, a.nk, (int)(i - a.len), a.lines);
      return;
    }
    block -= weight_blocks;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int segs = (a.len - 1) / kOut + 1;
  const int64_t unit = block * kBlurWarps + warp;
  // the warps of a block take neighbouring lines: their transposed stores share sectors
  const int64_t group = unit / ((int64_t)segs * kBlurWarps), rest = unit % ((int64_t)segs * kBlurWarps);
  const int64_t line = group * kBlurWarps + rest % kBlurWarps;
  if (line >= a.lines) return;
  const int base = (int)(rest / kBlurWarps) * kOut;
  const double* row = a.in + line * a.len;
  const int nk = a.nk;
  double acc0 = 0.0, acc1 = 0.0;
  uint4* bf = s_f[warp];
  uint4* bk = s_k[warp];
  const bool two = a.len - base > 32;
  // taps that lie outside the line for all of the warp's pixels add nothing
  const int64_t t_lo = max((int64_t)0, (int64_t)nk - base - (min(kOut, a.len - base) - 1)),
                t_hi = min((int64_t)2 * nk + 1, (int64_t)a.len - base + nk);
  for (int64_t t0 = t_lo; t0 < t_hi; t0 += kTaps) {
    const int n = (int)min((int64_t)kTaps, t_hi - t0);
    const int64_t j0 = base - nk + t0;  // the pixel of lane 0's first tap
    bool plain = true;
    __syncwarp();
    for (int i = lane; i < n + kOut - 1; i += 32) {
      const int64_t j = j0 + i;
      const uint64_t v = j >= 0 && j < a.len ? (uint64_t)__double_as_longlong(row[j]) : 0;
      bool ok;
      const RoundedFactor f = pixel_factor(v, ok);
      bf[i] = make_uint4(f.lo, f.hi, f.e, 0);
      plain &= ok;
    }
    for (int i = lane; i < n; i += 32) {
      const int64_t d = t0 + i - nk;
      bool ok;
      const RoundedFactor k = weight_factor((uint64_t)__double_as_longlong(a.kern[d < 0 ? -d : d]), ok);
      bk[i] = make_uint4(k.lo, k.hi, k.e, 0);
      plain &= ok;
    }
    plain = __all_sync(0xffffffffu, plain);
    if (plain) {
      // zero pixels, and those outside the line, are left out: a sum that began with +0 is never -0,
      // so adding a zero changes nothing
      const uint4* f0 = bf + lane;
      if (two) {
#pragma unroll 4
        for (int t = 0; t < n; ++t) {
          const uint4 k = bk[t], f = f0[t], g = f0[t + 32];
          const double p = __longlong_as_double((long long)rounded_product({f.x, f.y, f.z}, {k.x, k.y, k.z}));
          const double q = __longlong_as_double((long long)rounded_product({g.x, g.y, g.z}, {k.x, k.y, k.z}));
          if (f.y) acc0 = __dadd_rn(acc0, p);
          if (g.y) acc1 = __dadd_rn(acc1, q);
        }
      } else {
#pragma unroll 4
        for (int t = 0; t < n; ++t) {
          const uint4 k = bk[t], f = f0[t];
          const double p = __longlong_as_double((long long)rounded_product({f.x, f.y, f.z}, {k.x, k.y, k.z}));
          if (f.y) acc0 = __dadd_rn(acc0, p);
        }
      }
    } else {  // infinities, NaN, subnormal numbers, extreme magnitudes: the FP64 unit's products
      for (int t = 0; t < n; ++t) {
        const int64_t d = t0 + t - nk, j = j0 + t + lane;
        const double k = a.kern[d < 0 ? -d : d];
        if (j >= 0 && j < a.len) acc0 = __dadd_rn(acc0, __dmul_rn(k, row[j]));
        if (j + 32 >= 0 && j + 32 < a.len) acc1 = __dadd_rn(acc1, __dmul_rn(k, row[j + 32]));
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int o = base + lane + 32 * h;
    if (o >= a.len) break;
    double v = h ? acc1 : acc0;
    if constexpr (!kFirst) v = __ddiv_rn(__dmul_rn(v, a.w_line[line]), a.w_pix[o]);
    a.out[(int64_t)o * a.lines + line] = v;
  }
}

int64_t blur_blocks(int len, int lines) {
  const int64_t segs = (len - 1) / kOut + 1, groups = (lines - 1) / kBlurWarps + 1;
  return segs * groups;
}

}  // namespace

// d_tmp holds nx*ny + nx + ny doubles (the x-pass image transposed, w_stripe, the y pass's sums).
cudaError_t launch_blur(const double* d_in, double* d_tmp, double* d_out, int nx, int ny, const double* d_kernel,
                        int nk, cudaStream_t st) {
  const int64_t n = (int64_t)nx * ny;
  double* w = d_tmp + n;
  const int64_t wb = ((int64_t)nx + ny + 32 * kBlurWarps - 1) / (32 * kBlurWarps);
  const int64_t bx = blur_blocks(nx, ny) + wb, by = blur_blocks(ny, nx);
  if (bx > INT32_MAX || by > INT32_MAX) return cudaErrorInvalidValue;
  BlurLines a{d_in, d_tmp, nx, ny, d_kernel, nk, w, nullptr, nullptr};
  k_blur_lines<true><<<(unsigned)bx, 32 * kBlurWarps, 0, st>>>(a, (int)wb);
  BlurLines b{d_tmp, d_out, ny, nx, d_kernel, nk, nullptr, w, w + nx};
  k_blur_lines<false><<<(unsigned)by, 32 * kBlurWarps, 0, st>>>(b, 0);
  return cudaGetLastError();
}

}  // namespace stem
