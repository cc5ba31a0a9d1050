// The cluster kernels' operator layout (sg_cluster_layout.h), for random operators with and without
// several lanes a row: every nonzero has a place of its own inside the operator's elements, on a lane
// of its row and in a step that the row's slice walks, and the other places are as many as the
// padding.
#include <stdio.h>

#include <random>
#include <vector>

#include "sg_cluster_layout.h"

int main() {
  std::mt19937 rng(7);
  long long checked = 0;
  for (int round = 0; round < 600; ++round) {
    const int rows = round < 140 ? round : static_cast<int>(rng() % 700);
    const int most = 1 + static_cast<int>(rng() % 60);
    std::vector<int> ptr(rows + 1, 0);
    for (int r = 0; r < rows; ++r) ptr[r + 1] = ptr[r] + static_cast<int>(rng() % (most + 1));
    for (bool small : {false, true}) {
      const sg::RowOrder o = sg::order_rows(ptr.data(), rows, small);
      const int slices = sg::slices_of(o);
      std::vector<sg::StartLen> sl(rows + 1), desc(slices + 1);
      const long long elems = sg::place_rows(ptr.data(), o, sl.data(), desc.data());
      if (o.lanes != (small ? 32 >> o.slice : 1)) return printf("lanes\n"), 1;
      std::vector<char> used(elems, 0);
      for (int p = 0; p < rows; ++p) {
        const int r = o.perm[p];
        if (o.pos[r] != p || sl[p].len != ptr[r + 1] - ptr[r]) return printf("order\n"), 1;
        if (p > 0 && sl[p].len > sl[p - 1].len) return printf("not sorted\n"), 1;
        const sg::StartLen& d = desc[p >> o.slice];
        if (sl[p].len > 32 && !(d.len & 256)) return printf("long row unmarked\n"), 1;
        int last_step = -1, last_lane = -1;
        for (int k = 0; k < sl[p].len; ++k) {
          const int at = sg::place_of(sl[p], k, o);
          if (at < 0 || at >= elems || used[at]++) return printf("place\n"), 1;
          ++checked;
          if (sl[p].len > 32) continue;
          const int step = (at - d.start) / 32, lane = (at - d.start) % 32;
          if (at < d.start || step >= (d.len & 255)) return printf("outside the slice\n"), 1;
          if (lane % (1 << o.slice) != p % (1 << o.slice) || lane >> o.slice >= o.lanes) {
            return printf("lane\n"), 1;
          }
          if (step < last_step || (step == last_step && lane <= last_lane)) {
            return printf("order of steps\n"), 1;
          }
          last_step = step;
          last_lane = lane;
        }
      }
    }
  }
  printf("%lld nonzeros\n", checked);
  return 0;
}
