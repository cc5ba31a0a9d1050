// Stand-ins for the device behind cluster_failure_driver.cpp: one host thread is a CTA of one
// thread.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __noinline__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __restrict__

struct int2 {
  int x, y;
};
struct int4 {
  int x, y, z, w;
};
inline int2 make_int2(int x, int y) { return {x, y}; }
struct uint3 {
  unsigned x, y, z;
};
inline thread_local uint3 threadIdx{0, 0, 0}, blockIdx{0, 0, 0}, blockDim{32, 1, 1},
    gridDim{1, 1, 1};
using cudaStream_t = void*;
using cudaEvent_t = void*;
enum cudaError_t { cudaSuccess = 0 };
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
inline void __syncthreads() {}
inline bool __any_sync(unsigned, bool p) { return p; }
inline unsigned __activemask() { return 1u; }
inline unsigned __ballot_sync(unsigned, bool) { return 0u; }
template <typename T>
T __shfl_sync(unsigned, T v, int) {
  return v;
}
inline int __ffs(unsigned v) { return __builtin_ffs(static_cast<int>(v)); }
template <typename T>
T __ldg(const T* p) {
  return *p;
}
inline long long __double_as_longlong(double v) {
  long long b;
  memcpy(&b, &v, 8);
  return b;
}
inline int min(int a, int b) { return a < b ? a : b; }
inline std::mutex emu_atomics;
template <typename T, typename V>
T atomicAdd(T* p, V v) {
  std::lock_guard<std::mutex> l(emu_atomics);
  const T old = *p;
  *p += v;
  return old;
}
inline int atomicExch(int* p, int v) {
  std::lock_guard<std::mutex> l(emu_atomics);
  const int old = *p;
  *p = v;
  return old;
}

namespace emu {

struct Cluster {
  std::mutex mu;
  std::condition_variable cv;
  unsigned size = 1, arrived = 0, left = 0;
  long long phase = 0;
  std::vector<long long> passed;
  std::vector<char> ended;
  std::vector<void*> shared;
  std::vector<std::vector<double>> values;
  bool stray = false, failed = false;
  void reset(unsigned n) {
    size = n;
    arrived = left = 0;
    phase = 0;
    passed.assign(n, 0);
    ended.assign(n, 0);
    shared.assign(n, nullptr);
    values.assign(n, {});
    stray = failed = false;
  }
  void release() {
    if (arrived > 0 && arrived + left >= size) {
      arrived = 0;
      ++phase;
      cv.notify_all();
    }
  }
  void barrier(unsigned r) {  // a CTA that has ended counts as arrived
    std::unique_lock<std::mutex> l(mu);
    ++passed[r];
    const long long p = phase;
    ++arrived;
    release();
    cv.wait(l, [&] { return phase != p; });
  }
  void leave(unsigned r) {
    std::lock_guard<std::mutex> l(mu);
    ended[r] = 1;
    ++left;
    release();
  }
  bool sound() const {
    for (long long p : passed) {
      if (p != passed[0]) return false;
    }
    return !stray;
  }
  // A store into CTA r: false when that has ended.
  bool touch(unsigned r) {
    std::lock_guard<std::mutex> l(mu);
    if (ended[r]) stray = true;
    return !ended[r];
  }
};
inline Cluster cluster;
inline thread_local unsigned rank = 0, size = 1;
inline thread_local int waits = 0, fail_at = 0;
inline void enter(unsigned r, unsigned n, int at) {
  rank = r;
  size = n;
  waits = 0;
  fail_at = at;
  blockIdx.x = r;
  gridDim.x = n;
}

}  // namespace emu
