// near_list.h -- sizes of the element sums' list of near pairs (8 bytes each).
//
// Which pairs are near is known only after the far kernel has run, so the list
// has a first size, and grows when an evaluation before counted more.  A list
// that its pairs do not fit is not used: every pair is tested again, which
// gives the same sums from no memory.  So the list has an upper limit (a share
// of the free memory, or the caller's), and stays as it is where the pairs would
// not fit below it: n x panels pairs can be any number of gigabytes.
#pragma once

#include <algorithm>
#include <cstddef>

// n particles, `panels` panels.  96 pairs a particle serve a wake around its
// bodies (67 a particle in the 2M-particle step).
inline size_t near_list_first(size_t n, size_t panels, size_t limit) {
  const size_t most = n * panels;
  const size_t want = std::max(std::max<size_t>((size_t)1 << 20, n * 96),
                               std::min<size_t>(most / 8, (size_t)1 << 26));
  return std::min(std::min(want, most), limit);
}

// after an evaluation that counted `seen` pairs on a list of `cap`
inline size_t near_list_next(size_t cap, unsigned long long seen, size_t limit) {
  if (seen <= cap || seen > limit) return cap;
  return (size_t)std::min<unsigned long long>(seen + seen / 4 + 1024, limit);
}
