// Host side of the cluster kernels' operator layout (see sg_cluster.cuh): rows renumbered by
// decreasing length, rows of at most 32 nonzeros interleaved by slices (padded to the slice's
// longest; a padding element is 0 in the gathered vector's last entry, one past the other
// operator's rows), longer rows row by row.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <numeric>
#include <vector>

namespace sg {

struct StartLen {
  int start, len;  // as the device's int2
};

// The numbering of one operator's rows.
struct RowOrder {
  int slice = 5;          // log2 of the rows of a slice
  std::vector<int> perm;  // position -> row
  std::vector<int> pos;   // row -> position
};

inline RowOrder order_rows(const int* ptr, int rows) {
  RowOrder o;
  long long in_long = 0;
  int longest = 0;
  for (int r = 0; r < rows; ++r) {
    const int len = ptr[r + 1] - ptr[r];
    if (len > 32) in_long += len;
    longest = std::max(longest, len);
  }
  // Mostly longer rows: eight to a slice, so that an operator of few rows (the 200 rows of a
  // facility-location LP, 40-160 nonzeros each) occupies every warp. (Not where the padding of
  // its shorter rows, three of four places, could pass 32-bit offsets.)
  o.slice = rows > 0 && 2 * in_long > ptr[rows] && ptr[rows] < (1 << 28) ? 3 : 5;
  // Stable counting sort by decreasing length.
  std::vector<int> at(static_cast<size_t>(longest) + 2, 0);
  for (int r = 0; r < rows; ++r) ++at[longest - (ptr[r + 1] - ptr[r]) + 1];
  std::partial_sum(at.begin(), at.end(), at.begin());
  o.perm.resize(rows);
  o.pos.resize(rows);
  for (int r = 0; r < rows; ++r) {
    const int p = at[longest - (ptr[r + 1] - ptr[r])]++;
    o.perm[p] = r;
    o.pos[r] = p;
  }
  return o;
}

// Starts and lengths by position and, per slice, the start and number of steps of its rows of at
// most 32 nonzeros (+ 256 when it has longer rows: RowShare::desc); returns the elements the
// operator's arrays take (padding of partly filled slices included).
inline long long place_rows(const int* ptr, const RowOrder& o, StartLen* sl, StartLen* desc) {
  const int rows = static_cast<int>(o.perm.size());
  const int slice_rows = 1 << o.slice;
  long long at = 0;
  for (int p = 0; p < rows; ++p) {
    const int len = ptr[o.perm[p] + 1] - ptr[o.perm[p]];
    sl[p].len = len;
    if (len > 32) {
      sl[p].start = static_cast<int>(at);
      at += len;
    }
  }
  for (int first = 0; first < rows; first += slice_rows) {
    const int last = std::min(rows, first + slice_rows);
    int width = 0;
    bool has_long = false;
    for (int p = first; p < last; ++p) {
      if (sl[p].len > 32) {
        has_long = true;
        continue;
      }
      width = std::max(width, sl[p].len);
      sl[p].start = static_cast<int>(at + (p - first));
    }
    desc[first >> o.slice] = {width > 0 ? static_cast<int>(at) : 0, width | (has_long ? 256 : 0)};
    at += static_cast<long long>(width) * 32;
  }
  return at;
}

inline int slices_of(const RowOrder& o) {
  return (static_cast<int>(o.perm.size()) + (1 << o.slice) - 1) >> o.slice;
}

// The place of nonzero k of the row at position p.
inline int place_of(const StartLen& sl, int k) {
  return sl.start + (sl.len <= 32 ? k << 5 : k);
}

}  // namespace sg
