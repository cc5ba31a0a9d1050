// Host side of the cluster kernels' operator layout (see sg_cluster.cuh): rows renumbered by
// decreasing length, rows of at most 32 nonzeros interleaved by slices, a lane or several to a row
// (padded to the slice's longest; a padding element is 0 in the gathered vector's last entry, one
// past the other operator's rows), longer rows row by row.
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
  int lanes = 1;          // lanes of a row of at most 32 nonzeros
  std::vector<int> perm;  // position -> row
  std::vector<int> pos;   // row -> position
};

inline RowOrder order_rows(const int* ptr, int rows, bool small = false) {
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
  // Small LPs (Batch::create): one CTA has more warps than the operator has slices of 32, and an
  // iteration is mostly the chain of a row's additions: 8 or 16 rows to a slice, 4 or 2 lanes a row.
  if (small) {
    if (rows <= 128) o.slice = rows <= 64 ? 3 : std::min(o.slice, 4);
    o.lanes = 32 >> o.slice;
  }
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
      width = std::max(width, (sl[p].len + o.lanes - 1) / o.lanes);
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

// The place of nonzero k of the row at position p (RowShare::place on the device).
inline int place_of(const StartLen& sl, int k, const RowOrder& o) {
  if (sl.len > 32) return sl.start + k;
  return sl.start + ((k / o.lanes) << 5) + ((k % o.lanes) << o.slice);
}

// The other layout, for an LP on one cluster of few rows a CTA (sg_chunk.cu). The rows, by
// decreasing length, are dealt out to the CTAs in turn; row l of CTA r has position
// r ceil(rows / size) + l (the CTA's entries of the gathered vector lie side by side: l size + r,
// tried first, sent every warp's 32 entries to one bank), and its nonzeros go to tasks, a warp's
// work each: 32 >> lanes rows of the CTA, 2^lanes lanes to a row, `steps` steps; nonzero k of a
// row is read at step k >> lanes by the row's lane k mod 2^lanes. Padding: value 0, index the other
// operator's positions.
struct Task {
  int place;  // first element, in the CTA's block
  int steps;
  int first;  // own row
  int rows;   // rows | lanes << 8
};

struct TaskLayout {
  int per = 0;                // positions of a CTA
  std::vector<int> perm, pos;  // position -> row (-1: none), row -> position
  std::vector<StartLen> row;  // per position: first element (of the whole layout), log2 lanes
  std::vector<Task> tasks;
  std::vector<int> task_off, elem_off;  // per CTA: first task and element
  std::vector<int> filled;  // and two numbers: rows with nonzeros, rows on several lanes
  int most_tasks = 0, most_elems = 0;
  int positions() const { return static_cast<int>(perm.size()); }
};

// limit: no row takes more steps (up to 32 lanes). 0: a row of at most 32 nonzeros by one lane,
// longer ones by 32 (the sums of FP32 keep their order).
inline TaskLayout make_tasks(const int* ptr, int rows, int size, int limit) {
  TaskLayout t;
  const RowOrder o = order_rows(ptr, rows);
  t.per = (rows + size - 1) / size;
  t.perm.assign(static_cast<size_t>(t.per) * size, -1);
  t.pos.resize(rows);
  t.row.assign(t.perm.size(), StartLen{0, 0});
  t.task_off.assign(1, 0);
  t.elem_off.assign(1, 0);
  auto lanes_of = [&](int len) {
    if (limit == 0) return len <= 32 ? 0 : 5;
    int lanes = 0;
    while (lanes < 5 && ((len - 1) >> lanes) >= limit) ++lanes;
    return lanes;
  };
  for (int rank = 0; rank < size; ++rank) {
    const int own = rows > rank ? (rows - rank - 1) / size + 1 : 0;
    const int first = rank * t.per;
    for (int l = 0; l < own; ++l) {
      const int r = o.perm[static_cast<size_t>(l) * size + rank];
      t.perm[first + l] = r;
      t.pos[r] = first + l;
    }
    auto length = [&](int l) { return ptr[t.perm[first + l] + 1] - ptr[t.perm[first + l]]; };
    int elems = 0, l = 0, count = 0, shared = 0;
    while (l < own && length(l) > 0) {
      const int lanes = lanes_of(length(l));
      Task k{elems, ((length(l) - 1) >> lanes) + 1, l, 0};
      int n = 0;
      for (; n < (32 >> lanes) && l < own && length(l) > 0 && lanes_of(length(l)) == lanes;
           ++n, ++l) {
        t.row[first + l] = StartLen{t.elem_off.back() + elems + (n << lanes), lanes};
      }
      k.rows = n | lanes << 8;
      if (lanes > 0) shared = l;
      t.tasks.push_back(k);
      ++count;
      elems += k.steps * 32;
    }
    t.filled.push_back(l);
    t.filled.push_back(shared);
    t.task_off.push_back(static_cast<int>(t.tasks.size()));
    t.elem_off.push_back(t.elem_off.back() + elems);
    t.most_tasks = std::max(t.most_tasks, count);
    t.most_elems = std::max(t.most_elems, elems);
  }
  return t;
}

}  // namespace sg
