// hj_ranges.h -- memory bookkeeping (host only, no CUDA): the free ranges of a
// batch's particle pool, first fit (admission takes room for a bunch, retirement
// gives it back and merges it with its free neighbours), the sizes of cached
// blocks and the bounds of a caller's.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <utility>
#include <vector>

namespace hj_ranges {

// (start, length) of each free range: sorted, disjoint and never adjacent.
using Ranges = std::vector<std::pair<int64_t, int64_t>>;

// Room for n particles, rounded up to a multiple of 4 (at least 4, so every
// bunch starts on a 32-byte boundary), from the first free range that holds
// it.  Returns false, changing nothing, when none does.
inline bool take(Ranges& fr, int64_t n, int64_t* start, int64_t* cap) {
  const int64_t need = std::max<int64_t>((n + 3) / 4 * 4, 4);
  for (size_t i = 0; i < fr.size(); ++i) {
    auto& r = fr[i];
    if (r.second >= need) {
      *start = r.first;
      *cap = need;
      r.first += need;
      r.second -= need;
      if (r.second == 0) fr.erase(fr.begin() + i);
      return true;
    }
  }
  return false;
}

// Return [start, start + cap) to the free ranges.
inline void give(Ranges& fr, int64_t start, int64_t cap) {
  auto it = std::lower_bound(fr.begin(), fr.end(), std::make_pair(start, (int64_t)0));
  it = fr.insert(it, {start, cap});
  size_t i = it - fr.begin();
  if (i + 1 < fr.size() && fr[i].first + fr[i].second == fr[i + 1].first) {
    fr[i].second += fr[i + 1].second;
    fr.erase(fr.begin() + i + 1);
  }
  if (i > 0 && fr[i - 1].first + fr[i - 1].second == fr[i].first) {
    fr[i - 1].second += fr[i].second;
    fr.erase(fr.begin() + i);
  }
}

// Length of the largest free range.
inline int64_t largest(const Ranges& fr) {
  int64_t m = 0;
  for (const auto& r : fr) m = std::max(m, r.second);
  return m;
}

// Size of the block that serves b bytes: 2^k x {1, 1.25, 1.5, 1.75}, so that requests of
// similar sizes reuse each other's blocks, at least 4096.  A request beyond what the cache
// keeps (`kept` bytes) is not reused anyway and takes only its own pages: a turn log or a
// pool may need most of the device's memory.
inline size_t size_class(size_t b, size_t kept) {
  if (b <= 4096) return 4096;
  const int lg = b > kept ? 14 : 63 - __builtin_clzll((unsigned long long)b);
  const size_t step = size_t(1) << (lg - 2);
  return (b + step - 1) / step * step;
}

// Whether [p, p + bytes) lies in the allocation of `size` bytes at base.
inline bool covers(uint64_t base, uint64_t size, uint64_t p, uint64_t bytes) {
  return p >= base && p - base <= size && bytes <= size - (p - base);
}

}  // namespace hj_ranges
