// sg_cluster.cuh for cluster_failure_driver.cpp: barriers, reductions and stores between CTAs are
// the emulated cluster's, walks only wait, and waits fail where the driver says.
#pragma once

#include "emulated_device.h"

namespace sg {

constexpr int kThreads64 = 256, kThreads64Large = 512, kThreads32Few = 256, kThreads32Mid = 384, kThreads32 = 512;
constexpr int kMaxCluster = 16;
enum : int { kInDevice = 0, kVectorsShared = 1, kAllShared = 2, kModes = 3 };
enum : int { kOptimal = 0, kIterationLimit = 3, kTimeLimit = 4, kNumericalError = 5 };
inline unsigned long long globaltimer_ns() { return 0; }
inline thread_local unsigned char sg_smem[1 << 16];

struct ClusterShared {
  int fail = 0;
  unsigned stop = 0, next = 0;
  double red[1], peer[1];
};

// An address: the CTA above 24 bits, the place in its ClusterShared below.
inline unsigned cluster_rank() { return emu::rank; }
inline unsigned cluster_size() { return emu::size; }
inline void cluster_sync(unsigned) { emu::cluster.barrier(emu::rank); }
inline void cluster_init(ClusterShared& sh, unsigned size) {
  emu::cluster.shared[emu::rank] = &sh;
  cluster_sync(size);
}
inline unsigned shared_addr(const void* p) {
  return static_cast<unsigned>(static_cast<const char*>(p) -
                               static_cast<const char*>(emu::cluster.shared[emu::rank]));
}
inline unsigned map_rank(unsigned addr, unsigned rank) { return rank << 24 | addr; }
inline void st_cluster(unsigned addr, unsigned v) {
  if (!emu::cluster.touch(addr >> 24)) return;
  memcpy(static_cast<char*>(emu::cluster.shared[addr >> 24]) + (addr & 0xffffffu), &v, 4);
}
// CLUSTER_STOPPED

template <typename T, bool SHARED>
struct Array {
  T* a;
  Array(T* p) : a(p) {}
  T get(int i) const { return a[i]; }
  void set(int i, T v) const { a[i] = v; }
};
struct At {
  int ls, lane, l, p;
};
template <typename S>
S sh_copy(const S* p) {
  return *p;
}

template <typename V, int MODE>
struct alignas(16) Exchange {
  V* device;
  unsigned xs_at, ys_at, cmask_at, rmask_at;
  ClusterShared* sh;
  unsigned rank, size, tx[2];
  V* xs() const { return reinterpret_cast<V*>(sg_smem); }
  V* ys() const { return reinterpret_cast<V*>(sg_smem) + 64; }
  void put_x(const At&, V) const { store(); }
  void put_y(const At&, V) const { store(); }
  void store() const {
    for (unsigned r = 0; r < size; ++r) emu::cluster.touch(r);
  }
  bool wait(int) const {
    if (sh->fail != 0) emu::cluster.stray = true;  // none after one that gave up
    if (emu::waits++ >= emu::fail_at) {
      sh->fail = 1;
      emu::cluster.failed = true;
    }
    return sh->fail == 0;
  }
};
template <typename V, int MODE, int WHICH, bool OWN = false>
struct Sender {
  const Exchange<V, MODE>& ex;
  explicit Sender(const Exchange<V, MODE>& e) : ex(e) {}
  void put(const At&, V) const { ex.store(); }
};
enum : int { kWalkOne = 0, kWalkPairs = 1, kWalkLanes = 2 };
template <typename T, int WALK = kWalkOne>
struct alignas(16) RowShare {
  static constexpr bool kTasks = false;
  const int2 *sl, *desc;
  const int* idx;
  const T* val;
  int rows, slice;
  unsigned rank, size;
  int slices() const { return 1; }
  int own() const { return 1; }
  int place(const int2& row, int k) const { return row.x + k; }
};
// One own row, at position 0.
template <typename S, typename F>
void each_own(const S&, const F& f) {
  f(At{0, 0, 0, 0});
}
template <typename E, typename S>
void build_masks(E& ex, const S&, const S&) {
  cluster_sync(ex.size);
  cluster_sync(ex.size);
}
template <int K, unsigned MAXMASK = 0u>
void cluster_reduce(double (&v)[K], ClusterShared&, unsigned rank, unsigned size) {
  for (unsigned r = 0; r < size; ++r) emu::cluster.touch(r);
  emu::cluster.values[rank].assign(v, v + K);
  cluster_sync(size);
  for (int q = 0; q < K; ++q) {
    v[q] = 0.0;
    for (unsigned r = 0; r < size; ++r) {
      const double x = emu::cluster.values[r][q];
      v[q] = (MAXMASK >> q) & 1u ? fmax(v[q], x) : v[q] + x;
    }
  }
  cluster_sync(size);
}
inline void keep_branch(unsigned) {}
struct Ready {
  bool operator()() const { return true; }
};
template <typename A>
struct Zero {
  A operator()(const At&) const { return A(0); }
};
template <bool NC, bool MAXRED, typename S, typename P, typename I, typename F, typename R>
bool walk_rows(const S&, const P&, const I&, const F& f, const R& ready) {
  if (!ready()) return false;
  f(At{0, 0, 0, 0}, 1.0);
  return true;
}
template <typename S, typename P, typename I, typename F, typename R>
bool walk_step(const S& a, const P& p, const I& i, const F& f, const R& ready) {
  return walk_rows<true, false>(a, p, i, f, ready);
}

}  // namespace sg
