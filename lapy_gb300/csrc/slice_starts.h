// Starts of a sliced matrix's slices (host logic only).
#pragma once
#include <cstdint>
#include <vector>

namespace lapy {

// starts[u] = sum of the sizes before u, starts[n] the total, which is
// returned: -1 (and nothing) when it does not fit into 32 bits.  One row of
// many entries pads the 31 beside it, so the sum can exceed 2^32 although the
// matrix has fewer than 2^31 entries.
inline int64_t slice_starts(const int32_t* size, int n, std::vector<int32_t>* starts) {
  int64_t sum = 0;
  for (int u = 0; u < n; ++u) sum += size[u];
  if (sum > INT32_MAX) return -1;
  starts->resize((size_t)n + 1);
  int32_t at = 0;
  for (int u = 0; u < n; ++u) {
    (*starts)[u] = at;
    at += size[u];
  }
  (*starts)[n] = at;
  return sum;
}

}  // namespace lapy
