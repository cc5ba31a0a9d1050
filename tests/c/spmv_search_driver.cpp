// The device-pointer product's search of the row starts (lower_bound_ptr, put in by
// test_spmv_search.py) on the CPU, a host thread per lane of the warp, up to 2^31 - 1 rows: the
// starts are a sparse mapping, of which only the probed pages exist.
#include <stdio.h>
#include <sys/mman.h>

#include <algorithm>
#include <barrier>
#include <climits>
#include <thread>
#include <vector>

#define __device__
#define __forceinline__ inline

namespace {

struct Index {
  unsigned x;
};
thread_local Index threadIdx{0};
std::barrier<> lanes(32);
unsigned votes[2] = {0, 0};

unsigned ballot(bool p) {
  static thread_local int turn = 0;
  unsigned& v = votes[turn ^= 1];
  if (p) __atomic_fetch_or(&v, 1u << threadIdx.x, __ATOMIC_SEQ_CST);
  lanes.arrive_and_wait();
  const unsigned all = v;
  lanes.arrive_and_wait();
  if (threadIdx.x == 0) v = 0;
  return all;
}
#define __ballot_sync(mask, p) ballot(p)
#define __popc(v) __builtin_popcount(v)
using std::max;
using std::min;

// SEARCH

int search(const int* ptr, int m, long long key) {
  int found[32];
  std::vector<std::thread> warp;
  for (unsigned l = 0; l < 32; ++l) {
    warp.emplace_back([&, l] {
      threadIdx.x = l;
      found[l] = lower_bound_ptr(ptr, m, key);
    });
  }
  for (auto& t : warp) t.join();
  for (int l = 1; l < 32; ++l) {
    if (found[l] != found[0]) return -1;
  }
  return found[0];
}

}  // namespace

int main() {
  const size_t bytes = (static_cast<size_t>(INT_MAX) + 1) * sizeof(int);
  int* ptr = static_cast<int*>(mmap(nullptr, bytes, PROT_READ | PROT_WRITE,
                                    MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0));
  if (ptr == MAP_FAILED) return printf("no mapping\n"), 2;
  int bad = 0;
  for (int m : {1, 2, 31, 32, 33, 63, 1000, 1 << 20, (1 << 30) + 1, INT_MAX - 32, INT_MAX - 31,
                INT_MAX - 1, INT_MAX}) {
    // The last rows hold two nonzeros each, the others none.
    const int full = std::min(m, 1000);
    for (int k = 0; k <= full; ++k) ptr[m - full + k] = 2 * k;
    for (int k : {0, 1, full / 2, full - 1, full}) {
      for (int key : {2 * k - 1, 2 * k}) {
        if (key < 0) continue;
        const int want = key == 0 ? 0 : std::min(m, m - full + k);
        const int got = search(ptr, m, key);
        if (got != want) {
          ++bad;
          printf("%d rows, key %d: %d, not %d\n", m, key, got, want);
        }
      }
    }
    for (int k = 0; k <= full; ++k) ptr[m - full + k] = 0;
  }
  return bad != 0;
}
