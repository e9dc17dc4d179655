"""The plan of a call's field samples (field_plan.h): every range of patches lies in the buffer that is held
when the call runs, whatever the allocator gives, and the ranges cover all patches once."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "simulated_tem_gb300", "csrc")

RANGES = r"""
#include "field_plan.h"
#include <cstdio>
#include <random>
struct Params { int Mz; };
struct Job { Params p; int patch_base; int64_t sample_base; };
#define CHECK(c) do { if (!(c)) { std::printf("line %d: " #c "\n", __LINE__); return 1; } } while (0)
int main() {
  std::mt19937 rng(7);
  auto below = [&](int n) { return (int)(rng() % (unsigned)n); };
  for (int trial = 0; trial < 3000; ++trial) {
    const int align = trial % 2 ? 4 : 1;
    const size_t per = trial % 3 ? 8 : 24;
    std::vector<Job> jobs;
    stem::FieldGroup g[2];
    for (int i = 0; i < 2; ++i) {
      g[i].job_lo = (int)jobs.size();
      g[i].n_jobs = below(4);
      for (int j = 0; j < g[i].n_jobs; ++j) {
        const int mz = 1 + below(300), np = align * below(40);
        jobs.push_back({{mz}, (int)g[i].patches, g[i].samples});
        g[i].patches += np;
        g[i].samples += (int64_t)np * mz * 32;
        g[i].deepest = std::max(g[i].deepest, mz);
      }
    }
    // an allocator whose every answer is less than the one before
    size_t held = 0, scale = 1 + below(64);
    auto room = [&](size_t want, size_t least) {
      held = std::max(least, want / scale);
      scale *= 2;
      return held;
    };
    std::vector<stem::FieldRange> out;
    CHECK(stem::plan_ranges(jobs.data(), g, align, per, room, out));
    int next[2] = {0, 0};
    for (stem::FieldRange& R : out) {
      stem::split_depth(R, align, 1 + below(3000), trial % 5 ? stem::kRule32 : stem::kRule64);
      CHECK(R.chunk >= 4 && R.chunk % 4 == 0 && R.n_chunks * R.chunk >= R.deepest && (R.n_chunks - 1) * R.chunk < R.deepest);
      const int i = R.four ? 0 : 1;
      CHECK(R.patch_lo == next[i] && R.patch_hi > R.patch_lo && R.deepest == g[i].deepest);
      CHECK(R.job_lo == g[i].job_lo && R.n_jobs == g[i].n_jobs);
      next[i] = R.patch_hi;
      int64_t end = 0;  // samples of the range, from the workspace's start
      for (int j = g[i].job_lo; j < g[i].job_lo + g[i].n_jobs; ++j) {
        const int stop = j + 1 < g[i].job_lo + g[i].n_jobs ? jobs[j + 1].patch_base : (int)g[i].patches;
        const int lo = std::max(R.patch_lo, jobs[j].patch_base), hi = std::min(R.patch_hi, stop);
        if (lo >= hi) continue;
        const int64_t o = jobs[j].sample_base - R.origin;
        CHECK(o + (int64_t)(lo - jobs[j].patch_base) * jobs[j].p.Mz * 32 >= 0);
        end = std::max(end, o + (int64_t)(hi - jobs[j].patch_base) * jobs[j].p.Mz * 32);
      }
      CHECK(2 * end <= R.rho_at);                       // the field before rho,
      CHECK((size_t)(R.rho_at / 2) * per <= held);      // and all of it in what is held now
    }
    CHECK(next[0] == g[0].patches && next[1] == g[1].patches);
  }
  std::vector<stem::FieldRange> out;
  Job one{{10}, 0, 0};
  stem::FieldGroup g[2];
  g[0].n_jobs = 1;
  g[0].patches = 4;
  g[0].samples = 4 * 320;
  g[0].deepest = 10;
  CHECK(!stem::plan_ranges(&one, g, 4, 8, [](size_t, size_t) { return (size_t)0; }, out));
  std::puts("ok");
  return 0;
}
"""

ROOM = r"""
#include "field_plan.h"
#include <cstdio>
#include <cstdlib>
#include <map>
#define CHECK(c) do { if (!(c)) { std::printf("line %d: " #c "\n", __LINE__); return 1; } } while (0)
int main() {
  const size_t M = 1 << 20;
  size_t free_bytes = 100 * M, next = 64;
  std::map<void*, size_t> live;
  int calls = 0;
  auto alloc = [&](size_t n) -> void* {
    ++calls;
    if (n > free_bytes) return nullptr;
    free_bytes -= n;
    void* p = (void*)(next += 64);
    live[p] = n;
    return p;
  };
  auto release = [&](void* p) {
    ++calls;
    free_bytes += live.at(p);
    live.erase(p);
  };
  stem::SampleMemory m;
  auto room = [&](size_t want, size_t least, size_t most) {
    const size_t got = stem::sample_room(m, want, least, most, alloc, release);
    if (got && !(m.p && live.at(m.p) == m.cap && got <= m.cap)) std::abort();
    return got;
  };
  CHECK(room(10 * M, M, 64 * M) == 10 * M && room(4 * M, M, 64 * M) == 4 * M && calls == 1);
  CHECK(room(200 * M, M, 64 * M) == 64 * M && live.size() == 1);   // bounded, and the smaller one given back
  CHECK(room(200 * M, 70 * M, 64 * M) == 70 * M);                   // one patch takes more than the bound
  // a full device: half, then what is held call after call, and no allocator call in them
  release(m.p);
  m = stem::SampleMemory();
  free_bytes = 40 * M;
  CHECK(room(64 * M, M, 64 * M) == 32 * M);
  calls = 0;
  for (int i = 0; i < stem::kPatience; ++i) CHECK(room(64 * M, M, 64 * M) == 32 * M);
  CHECK(calls == 0);
  CHECK(room(64 * M, M, 64 * M) == 32 * M && calls == 1 && live.size() == 1);  // asked again, refused, kept
  free_bytes = 100 * M;
  for (int i = 0; i < stem::kPatience; ++i) CHECK(room(64 * M, M, 64 * M) == 32 * M);
  CHECK(room(64 * M, M, 64 * M) == 64 * M);                         // and again, with the memory there
  // down to one patch, and nothing
  release(m.p);
  m = stem::SampleMemory();
  free_bytes = 2040;
  CHECK(room(64 * M, 2000, 64 * M) == 2000);
  CHECK(room(64 * M, 5001, 64 * M) == 0 && live.empty() && !m.p && m.cap == 0);
  CHECK(room(64 * M, 1000, 0) == 0);
  std::puts("ok");
  return 0;
}
"""


def run(tmp_path, source):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-Wall", "-Wno-unknown-pragmas", "-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout


def test_ranges_lie_in_the_buffer_that_is_held(tmp_path):
    run(tmp_path, RANGES)


def test_the_memory_held_for_samples(tmp_path):
    run(tmp_path, ROOM)
