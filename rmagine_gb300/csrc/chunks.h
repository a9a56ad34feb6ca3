// Pose chunks of the simulate host forms.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace rmg {

// The smallest rest that is worth a launch of its own, where `least` poses are
// the least of any other: 64 poses with a least of 49 take 256 us as 49 and 15 and
// 262 at once, 50 take 247 as 49 and 1 and 238 at once.
inline size_t least_rest(size_t least) { return least / 4; }

// Poses of a full chunk: at most `want` (what the staging memory is to hold), and
// ceil(n / 2) so that two chunks overlap, but no fewer than `least` and a small
// rest.
inline size_t chunk_poses(uint32_t n, size_t want, size_t least) {
  return std::min<size_t>(std::max<size_t>(1, want),
                          std::max<size_t>(((size_t)n + 1) / 2, std::min<size_t>(n, least + least_rest(least))));
}

// Full chunks of `chunk` poses, then the last two chunks' worth split in halving
// sizes (at least chunk / 8 and `least` poses), so that the work left after the
// final launch -- its copy, and forming its points -- is a small chunk's.  A last
// one of fewer than least_rest(least) poses goes with the chunk before it, or
// shares with it evenly where the two are more than `chunk`.  Returns the first
// pose of every chunk and n.
inline std::vector<uint32_t> chunk_schedule(uint32_t n, size_t chunk, size_t least) {
  std::vector<uint32_t> first{0};
  uint64_t p = 0;
  while (n - p > 2 * chunk) {
    p += chunk;
    first.push_back((uint32_t)p);
  }
  const uint64_t min_tail = std::max<uint64_t>(std::max<uint64_t>(1, least), chunk / 8);
  while (p < n) {
    const uint64_t rem = n - p;
    uint64_t take = rem <= min_tail ? rem : std::max<uint64_t>(min_tail, std::min<uint64_t>(chunk, (rem + 1) / 2));
    if (rem - take < least_rest(least)) take = rem <= chunk ? rem : (rem + 1) / 2;
    p += take;
    first.push_back((uint32_t)p);
  }
  return first;
}

}  // namespace rmg
