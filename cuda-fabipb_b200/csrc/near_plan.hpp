// near_plan.hpp -- how the symmetric near field cuts its work, and the scratch that it takes: host arithmetic on the
// parts' sizes alone.
//
// A task is a chunk of the larger part R of a near pair against all of the smaller part T.  It takes scratch slots
// (16 bytes in FP64, 8 in FP32): R's panels once for the pair, T's panels once for every chunk of R.
#pragma once
#include <algorithm>
#include <vector>

namespace fb {

constexpr double kNearScratch = 512.0 * 1024 * 1024;   // bytes
constexpr int kNearResidentWarps = 2368;               // 148 SMs with 16 warps

// Parts of a direct FP64 context: runs of 128 panels, at most 256 of them, so that the slots of every panel against
// every part stay within 4 KiB a panel (and below 2^31).  256 parts are 32,640 pairs, 14 for each resident warp.
// Against parts that keep the scratch within 512 MiB, which from 200,000 panels on are long and few: 204,800 panels
// 94.7 ms so and 91.7 with 256 parts, 401,408 393 and 352; 720,000 1,150 ms, 2,106 in ordered passes.
constexpr int kEqualParts = 256;
inline int equal_part_length(long long n) {
  const long long quantum = 64LL * kEqualParts;
  long long len = std::max(128LL, (n + quantum - 1) / quantum * 64);
  while ((double)n * ((n + len - 1) / len) > 2147483646.0) len += 64;
  return (int)len;
}
inline double equal_part_scratch(long long n) { return 16.0 * kEqualParts * n; }

struct NearPlan {
  bool tasks = false;    // false: every pair in the finishing kernel
  int chunk = 0;         // panels of R per task
  long long slots = 0;   // scratch of all tasks
  long long count = 0;   // tasks
};

// each_pair(f) calls f(a, b, on) once for every unordered pair of distinct near parts, on: the pair may be a task.
//
// The chunk: whole parts up to 256 panels; 64 when that leaves fewer padded 32 x 32 tiles than eight for each of the
// chip's resident warps (a task is one warp's serial work).  It is doubled until the slots are within the limit.  In
// an FMM context that is kNearScratch, or as much again as whole parts take if that is more (large leaves would
// otherwise take a copy of T per 256 panels of R: 2,100,000 panels in 56 leaves 6e9 slots instead of 2e8).  Never
// 2^31 slots, which the tasks count in int: the finishing kernel takes every pair then.
//
// A direct context (every part near every other) gives its limit in bytes.  Where that makes so few tasks that less
// than half of the resident warps are busy, the ordered passes, which evaluate each pair twice but fill the chip, are
// the faster ones.
template <typename EachPair>
NearPlan plan_near_tasks(const std::vector<int> &count, size_t slotBytes, double directLimit, EachPair each_pair) {
  int top = 1;
  for (int c : count) top = std::max(top, c);
  auto add = [&](NearPlan &p, int a, int b) {
    const int cr = std::max(count[a], count[b]), ct = std::min(count[a], count[b]);
    const int chunks = (cr + p.chunk - 1) / p.chunk;
    p.slots += cr + (long long)chunks * ct;
    p.count += chunks;
  };
  NearPlan small, large;   // both in the pass that finds which
  small.chunk = 64;
  large.chunk = 256;
  long long tiles = 0, whole = 0;
  each_pair([&](int a, int b, bool on) {
    tiles += (long long)((count[a] + 31) / 32) * ((count[b] + 31) / 32);
    if (!on) return;
    whole += count[a] + count[b];
    add(small, a, b);
    add(large, a, b);
  });
  const double limit = directLimit > 0.0 ? directLimit / slotBytes : std::max(kNearScratch / slotBytes, 2.0 * whole);
  NearPlan p = tiles < 8 * kNearResidentWarps ? small : large;
  auto fits = [&] { return (double)p.slots <= limit && p.slots < 2147483647LL; };
  while (!fits() && p.chunk < top) {
    p.chunk *= 2;
    p.slots = p.count = 0;
    each_pair([&](int a, int b, bool on) {
      if (on) add(p, a, b);
    });
  }
  p.tasks = p.count > 0 && fits();
  if (directLimit > 0.0 && p.chunk > 256 && 2 * p.count < kNearResidentWarps) p.tasks = false;
  return p;
}

}  // namespace fb
