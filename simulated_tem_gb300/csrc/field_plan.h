// The host's plan of a call's field: ranges of patches whose samples share one workspace.  Plain C++:
// the allocations and the split in depth are the caller's.
#pragma once

#include <math.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#ifdef __CUDACC__
#define FP_HD __host__ __device__
#else
#define FP_HD
#endif

namespace stem {

// Device memory that a context keeps for field samples.
struct SampleMemory {
  void* p = nullptr;
  size_t cap = 0;    // bytes
  int patience = 0;  // calls that make do with what is held before more is asked for again
};

// The bytes a call may lay its samples out in: `want`, at most `most` (an image's or batch's columns then
// run in several ranges), less on a full device, but at least `least`, one patch; 0: not even that.
// What is held and holds `least` is given up only for a larger buffer, and after a refusal the next
// kPatience calls do with it: a free, a failing allocation and a synchronisation of the device per call
// cost more than the further ranges.
constexpr int kPatience = 63;
template <typename Alloc, typename Release>
size_t sample_room(SampleMemory& m, size_t want, size_t least, size_t most, Alloc alloc, Release release) {
  if (most == 0) return 0;
  want = std::max(std::min(want, most), least);
  if (m.p && m.cap >= want) return want;
  if (m.p && m.cap >= least) {
    if (m.patience > 0) {
      --m.patience;
      return m.cap;
    }
    if (void* p = alloc(want)) {
      release(m.p);
      m.p = p;
      m.cap = want;
    } else {
      m.patience = kPatience;
    }
    return m.cap;
  }
  if (m.p) release(m.p);
  m = SampleMemory();
  for (size_t n = want;; n = std::max(n / 2, least)) {
    if (void* p = alloc(n)) {
      m.p = p;
      m.cap = n;
      m.patience = n < want ? kPatience : 0;
      return n;
    }
    if (n <= least) return 0;
  }
}

// The voxel field of a range of patches (warp tiles of 32 columns) of a batch, in a workspace of
// samples: patch by patch in job order, slice by slice, 32 lanes.  The work is handed out in units
// of one patch and `chunk` slices, so that few patches still fill the GPU.
struct FieldRange {
  void* samples = nullptr;  // the field x of a voxel (times rho with density): float2 or double2
  float* rho32 = nullptr;   // with density: rho
  double* rho64 = nullptr;
  int64_t origin = 0;       // index of the workspace's first sample in the batch's sample sequence
  int patch_lo = 0, patch_hi = 0;
  int deepest = 1;          // slices of the deepest image
  int n_chunks = 1;         // per patch: ceil(deepest / chunk)
  int chunk = 0;            // slices per unit, a multiple of 4 (split_depth)
  int job_lo = 0, n_jobs = 0;  // the range's jobs in the call's job table
  bool four = true;         // four slices per step (else two)
  int64_t rho_at = 0;       // where rho starts in the workspace, in values
  // of a tile-masked image, which is alone: the tiles that have a wanted column, in any order, and their number;
  // patches and samples are then counted along this list, and the split in depth follows the number
  const int* list = nullptr;
  const unsigned long long* n_list = nullptr;
  int per_item = 1;         // patches per listed tile (2: the left or right half of an FP32 tile)
  int slots = 1;            // units that the GPU works on at a time
  unsigned* work = nullptr;  // units handed out: zero before the field kernel, zeroed again by the integrator
  const unsigned long long* counters = nullptr;
  int64_t cap = 0;
  FP_HD int units() const { return (patch_hi - patch_lo) * n_chunks; }
};

// Splits the patches of a batch into ranges of at most `samples` samples, cut at multiples of
// `align` patches of an image.
template <typename Job>
void field_ranges(const Job* jobs, int n_jobs, int patches, int64_t samples, int align, int deepest,
                  std::vector<FieldRange>& out) {
  out.clear();
  int job = 0;
  for (int lo = 0; lo < patches;) {
    FieldRange R;
    R.patch_lo = lo;
    R.deepest = R.chunk = deepest;
    auto end_of = [&](int j) { return j + 1 < n_jobs ? jobs[j + 1].patch_base : patches; };
    while (end_of(job) <= lo) ++job;
    R.origin = jobs[job].sample_base + (int64_t)(lo - jobs[job].patch_base) * jobs[job].p.Mz * 32;
    int64_t left = samples;
    int hi = lo;
    for (int j = job; j < n_jobs; ++j) {
      const int64_t per = (int64_t)jobs[j].p.Mz * 32;
      const int begin = std::max(lo, jobs[j].patch_base), n = end_of(j) - begin;
      const int64_t fit = std::min<int64_t>(n, left / per / align * align);
      hi = begin + (int)fit;
      left -= fit * per;
      if (fit < n) break;
    }
    R.patch_hi = std::max(hi, lo + align);  // the workspace holds at least `align` of the deepest
    lo = R.patch_hi;
    out.push_back(R);
  }
}

// Slices per unit of work (a multiple of 4) of `tiles` tiles up to `deepest` slices deep, `slots` of
// which the GPU works on at a time (the CTAs of the instance that runs), when a unit costs `fixed` slices beside
// its own (the slabs it stages before its first step): of up to kPieces pieces the number with the shortest waves
// of units, the last one partly filled.  In the FP32 field a unit, a CTA each, that is left alone in its SM at the
// end runs faster, which leaves a tail of 0.7 waves: over 28 images and instances (45 to 2,556 tiles, 40 to 240 slices, one
// to five CTAs per SM) the pieces are within 1.5 % of the fastest in the mean, 5 % at worst; whole
// waves of five CTAs, whatever the instance, 10 and 43 % (648 tiles of 120 slices, four CTAs: 1.21 ms in one piece,
// 0.87 in five).  The FP64 field's units, a warp each, differ, and up to two waves of them wait for the
// longest, more even out: 128k atoms with density (1653 patches, 160 slices) 4766 us with 160 slices in 0.9 waves,
// 4512 with 40 in 3.6, 4352 with 20 in 7.2, 4530 with 8.
constexpr int kPieces = 64;
struct DepthRule {
  int fixed;
  float tail;
  bool two_whole;  // up to two waves are whole ones
};
constexpr DepthRule kRule32{4, 0.7f, false}, kRule64{1, 0.5f, true};
template <typename F>
FP_HD F depth_cost(int64_t tiles, int deepest, int slots, DepthRule rule, int pieces, int& chunk) {
  chunk = ((deepest + pieces - 1) / pieces + 3) & ~3;
  const F w = (F)(tiles * ((deepest + chunk - 1) / chunk)) / (F)slots;
  const F waves = rule.two_whole && w <= (F)2.0 ? (F)1.08 * ceil(w) : w + (F)rule.tail;
  return waves * (F)(chunk + rule.fixed);
}
// The range split for a kernel whose units are `align` patches and of which `slots` run at a time.
inline void split_depth(FieldRange& R, int align, int slots, DepthRule rule) {
  const int deepest = R.deepest;
  const int64_t tiles = std::max(1, (R.patch_hi - R.patch_lo) / align);
  R.slots = slots;
  int best = (deepest + 3) & ~3;
  double best_cost = -1;
  for (int pieces = 1; pieces <= (deepest + 3) / 4 && pieces <= kPieces; ++pieces) {
    int chunk;
    const double cost = depth_cost<double>(tiles, deepest, slots, rule, pieces, chunk);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = chunk;
    }
  }
  R.chunk = best;
  R.n_chunks = (deepest + best - 1) / best;
}

// The images of one group: those that march four slices per step, or two.
struct FieldGroup {
  int job_lo = 0, n_jobs = 0;
  int64_t patches = 0, samples = 0;
  int deepest = 1;
};

// The ranges of both groups.  `room(want, least)` gives the workspace's bytes, at least `least` and at most
// about `want`, or 0; it is asked once, for both groups, since a second answer may be a smaller buffer
// than the first one's ranges were laid out in.  False when there is no room.
template <typename Job, typename Room>
bool plan_ranges(const Job* jobs, const FieldGroup (&groups)[2], int align, size_t bytes_per_sample, Room room,
                 std::vector<FieldRange>& out) {
  out.clear();
  const size_t want = (size_t)std::max(groups[0].samples, groups[1].samples) * bytes_per_sample;
  size_t least = 0;
  for (const FieldGroup& g : groups)
    if (g.samples) least = std::max(least, (size_t)g.deepest * 32 * align * bytes_per_sample);
  if (least == 0) return true;
  const size_t got = room(want, least);
  if (got < least) return false;
  const int64_t n_room = (int64_t)(got / bytes_per_sample) & ~(int64_t)31;
  std::vector<FieldRange> part;
  for (int i = 0; i < 2; ++i) {
    const FieldGroup& g = groups[i];
    if (g.samples == 0) continue;
    field_ranges(jobs + g.job_lo, g.n_jobs, (int)g.patches, n_room, align, g.deepest, part);
    for (FieldRange& R : part) {
      R.job_lo = g.job_lo;
      R.n_jobs = g.n_jobs;
      R.four = i == 0;
      R.rho_at = 2 * n_room;
      out.push_back(R);
    }
  }
  return true;
}

}  // namespace stem
