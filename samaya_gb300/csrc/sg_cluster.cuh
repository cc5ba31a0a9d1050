// One LP held by a thread-block cluster: the row walks, the vector exchange and the reductions of
// the kernels that run many iterations of one LP inside one launch (the batched solves and the
// unrolled layer).
//
// Layout of an operator (A by rows, or A' by rows: the LP's columns), made on the host
// (sg_cluster_layout.h): its rows are renumbered by decreasing length and taken in slices of 32
// (8 where most nonzeros sit in long rows). Rows of at most 32 nonzeros are stored slice by slice
// with their k-th nonzeros side by side (start + 32 k), so that a warp's loads are whole lines and
// the lanes of a slice end together; longer rows are stored row by row. (Small LPs, kWalkLanes: 8, 16
// or 32 rows to a slice, row r's nonzeros on lane r and every 2^slice-th after it in turn.) Slice s
// belongs to CTA
// s mod C of the cluster: sorted slices dealt out in turn balance the CTAs.
// Rows of random LPs hold 15 +- 4 nonzeros: unsorted, a warp's longest row keeps it half as long
// again, and the FP64 pipe (below) is busy for every lane that has nothing to add.
//
// The FP64 pipe bounds the FP64 kernels: a warp's FP64 instruction takes it for 19 clocks
// whatever lanes are active (1.68 lanes per clock and SM, latency 64 clocks, measured), so the
// epilogues fold the row's own term into the sum's start and compare on the integer pipe.
//
// Every CTA keeps its own copy of the two vectors that the products gather from (xs: one entry
// per column, ys: one per row) in shared memory, and the state of its own rows and columns. A
// row's update sends the new entry to the CTAs whose nonzeros read it, and to no others:
// st.async into their copy, completing on their mbarrier, so an exchange costs one remote
// store's latency and no cluster barrier. A barrier.cluster costs 720 clocks even for one CTA and
// its acquire drops the L1 contents, which hold the CTA's nonzeros from one iteration to the
// next (measured: re-reading 80 KB after it 2,700 clocks, after a block barrier 960).
//
// Why no entry is overwritten while it is still read: a CTA sends entries of xs after it has
// received every entry of ys that its columns read. Entry xs[j] in another CTA is read there by
// rows that have a nonzero in column j; each of them sends its own ys entry to column j's CTA,
// after its sum, so that CTA's wait covers all of them (and the same with xs and ys exchanged).
// A publication that does not alternate this way needs a cluster_sync before it.
//
// A wait is bounded, and it may give up in one CTA and not, or later, in another. A CTA whose wait
// gave up (ClusterShared::fail) waits no more and goes on through every cluster barrier of the
// kernel, and all CTAs leave a loop that holds such barriers together: by a reduction that carries
// the failure, or by cluster_stopped. (A look at `fail` in the wait itself took 1% of every solve.) One that left alone would arrive at its last
// barrier in the place of an earlier one and end, and the others would then store into the shared
// memory of a CTA that has ended.
//
// Every sum is taken in a fixed order, so a re-run is bit-identical.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sg_common.cuh"

namespace sg {

// Threads per CTA. FP64 kernels, bound by the FP64 pipe, take 256 of 128 registers, so that two CTAs
// share an SM and one's exchange overlaps the other's sums; 512 where the gathered vectors leave no
// room for a second CTA (Batch::plan_clusters). An FP32 solve has an SM to a CTA and is
// bound by the latency of its chains; how many threads share the registers follows the rows
// (Batch::plan_clusters): 256 of 255 registers, 384 of 168, 512 of 128.
constexpr int kThreads64 = 256;
constexpr int kThreads64Large = 512;
constexpr int kThreads32Few = 256;
constexpr int kThreads32Mid = 384;
constexpr int kThreads32 = 512;
constexpr int kMaxWarps = kThreads32 / 32;
constexpr int kMaxCluster = 16;
constexpr int kBatch = 4;  // nonzeros of a row loaded together (walk_rows spells out four)
// A wait for remote entries gives up after this many polls (each may suspend the thread for a
// while), far beyond any store's completion time.
constexpr int kClusterWaitTries = 1 << 22;

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned shared_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// The address of the same shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
  unsigned o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(addr), "r"(rank));
  return o;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
      "l"(__double_as_longlong(v)), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
      "r"(__float_as_uint(v)), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void st_async_if(unsigned on, unsigned addr, double v, unsigned bar) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n"
      " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n}" ::"r"(
          addr),
      "l"(__double_as_longlong(v)), "r"(bar), "r"(on)
      : "memory");
}
__device__ __forceinline__ void st_async_if(unsigned on, unsigned addr, float v, unsigned bar) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n"
      " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n}" ::"r"(
          addr),
      "r"(__float_as_uint(v)), "r"(bar), "r"(on)
      : "memory");
}

// Every thread of the cluster; orders shared and global accesses of all its CTAs.
__device__ __forceinline__ void cluster_sync(unsigned size) {
  if (size == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// Loads and stores at 32-bit shared addresses (a pointer into shared memory that is not known as
// one at compile time costs 64-bit arithmetic and a uniform-register move an access: 55,000 of
// 66,000 instructions an iteration of a 6,440-column FP32 LP were address arithmetic).
__device__ __forceinline__ float sh_load(unsigned a, float) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double sh_load(unsigned a, double) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ unsigned sh_load_u16(unsigned a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ unsigned sh_load_u32(unsigned a) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sh_store(unsigned a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void sh_store(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// A copy of a struct in shared memory, read anew where it stands: what a walk derives from it
// lives for that walk. (Held in registers across the iterations, the compiler keeps every walk's
// addresses there too, and spills: 25 million local loads in 63 iterations of 160 LPs.)
template <typename S>
__device__ __forceinline__ S sh_copy(const S* p) {
  static_assert(sizeof(S) % 16 == 0 && alignof(S) == 16, "whole 16-byte words");
  union U {
    S s;
    unsigned w[sizeof(S) / 4];
    __device__ U() {}
  } u;
  const unsigned a = shared_addr(p);
#pragma unroll
  for (unsigned k = 0; k < sizeof(S) / 16; ++k) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(u.w[4 * k]), "=r"(u.w[4 * k + 1]), "=r"(u.w[4 * k + 2]),
                   "=r"(u.w[4 * k + 3])
                 : "r"(a + 16 * k)
                 : "memory");
  }
  return u.s;
}

// An array in shared (SHARED) or device memory.
template <typename T, bool SHARED>
struct Array;
template <typename T>
struct Array<T, true> {
  unsigned a;
  __device__ __forceinline__ Array(T* p) : a(shared_addr(p)) {}
  __device__ __forceinline__ T get(int i) const {
    return sh_load(a + i * static_cast<int>(sizeof(T)), T());
  }
  __device__ __forceinline__ void set(int i, T v) const {
    sh_store(a + i * static_cast<int>(sizeof(T)), v);
  }
};
template <typename T>
struct Array<T, false> {
  T* a;
  __device__ __forceinline__ Array(T* p) : a(p) {}
  __device__ __forceinline__ T get(int i) const { return a[i]; }
  __device__ __forceinline__ void set(int i, T v) const { a[i] = v; }
};

// The part of a kernel's static shared memory that belongs to the cluster's exchange.
struct ClusterShared {
  unsigned long long bar[2];           // arrivals of xs [0] and ys [1] entries
  unsigned phase[2];                   // completed phases of each
  double red[24 * kMaxWarps];          // block reductions
  double peer[kMaxCluster * 24];       // the CTAs' totals of a cluster reduction
  unsigned count[2][kMaxCluster];      // entries this CTA sends to each other CTA
  unsigned incoming[2][kMaxCluster];   // entries each other CTA sends here
  unsigned distance[kMaxCluster];      // from a shared address here to the one in rank ^ q
  int fail;                            // a bounded wait gave up
  unsigned stop;                       // in some CTA of the cluster (cluster_stopped)
  int next;                            // work queue position
};

// Call once at kernel entry, before any exchange.
__device__ __forceinline__ void cluster_init(ClusterShared& sh, unsigned size) {
  if (threadIdx.x == 0) {
    for (int k = 0; k < 2; ++k) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_addr(&sh.bar[k]))
                   : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const unsigned here = shared_addr(&sh);
    for (unsigned q = 0; q < size; ++q) sh.distance[q] = map_rank(here, cluster_rank() ^ q) - here;
    sh.phase[0] = sh.phase[1] = 0;
    sh.fail = 0;
    sh.stop = 0u;
  }
  cluster_sync(size);
}

// A cluster barrier after which every CTA knows whether a wait gave up in any of them, before it.
// (Another cluster barrier lies between two of these, so that none is told of a later failure.)
__device__ __forceinline__ bool cluster_stopped(ClusterShared& sh, unsigned size) {
  if (threadIdx.x < size && sh.fail != 0) {
    st_cluster(map_rank(shared_addr(&sh.stop), threadIdx.x), 1u);
  }
  cluster_sync(size);
  return sh.stop != 0u;
}

// The kernels' dynamic shared memory. What lies there is kept as an offset into it: a 32-bit value,
// and the compiler sees shared addresses.
extern __shared__ __align__(16) unsigned char sg_smem[];

// What sits in a CTA's shared memory: nothing (then one CTA per cluster, and the gathered vectors
// in device memory), the gathered vectors and masks, or the state too.
enum : int { kInDevice = 0, kVectorsShared = 1, kAllShared = 2, kModes = 3 };

// An own row (or column) of the share: own slice, lane, ls 2^slice + lane, position.
struct At {
  int ls, lane, l, p;
};

// The gathered vectors of one LP and their exchange. V is the vectors' type. Entries are
// numbered by position (the operators' renumbered rows and columns).
template <typename V, int MODE>
struct alignas(16) Exchange {
  V* device;               // kInDevice: xs, then ys
  unsigned xs_at, ys_at;   // else their offsets (in entries from `device` in kInDevice)
  unsigned cmask_at, rmask_at;
  ClusterShared* sh;
  unsigned rank, size;
  unsigned tx[2];          // bytes arriving per publication of xs, ys

  // xs (n + 1) and ys (m + 1): this CTA's copies; the last entries, 0, are the padding's.
  __device__ __forceinline__ V* xs() const {
    if constexpr (MODE != kInDevice) return reinterpret_cast<V*>(sg_smem + xs_at);
    return device + xs_at;
  }
  __device__ __forceinline__ V* ys() const {
    if constexpr (MODE != kInDevice) return reinterpret_cast<V*>(sg_smem + ys_at);
    return device + ys_at;
  }
  // Own columns and rows: the CTAs that read the entry (bit q: rank ^ q).
  __device__ __forceinline__ unsigned short* cmask() const {
    return reinterpret_cast<unsigned short*>(sg_smem + cmask_at);
  }
  __device__ __forceinline__ unsigned short* rmask() const {
    return reinterpret_cast<unsigned short*>(sg_smem + rmask_at);
  }
  // Shared variables of the CTA rank ^ q lie at a fixed distance (ClusterShared::distance).
  __device__ __forceinline__ void send(unsigned mask, V* p, V v, int which) const {
    const unsigned a = shared_addr(p);
    const unsigned b = shared_addr(&sh->bar[which]);
    for (unsigned q = 1; q < size; ++q) {
      if ((mask >> q) & 1u) {
        const unsigned d = sh->distance[q];
        st_async(a + d, v, b + d);
      }
    }
  }
  // The new entry of an own column (own row), to every CTA that reads it.
  __device__ __forceinline__ void put_x(const At& at, V v) const {
    V* x = xs() + at.p;
    *x = v;
    if constexpr (MODE != kInDevice) {
      if (size > 1) send(cmask()[at.l], x, v, 0);
    }
  }
  __device__ __forceinline__ void put_y(const At& at, V v) const {
    V* y = ys() + at.p;
    *y = v;
    if constexpr (MODE != kInDevice) {
      if (size > 1) send(rmask()[at.l], y, v, 1);
    }
  }
  // After every thread of the CTA has put its entries: true when all entries read here have
  // arrived, false when the bounded wait gave up (uniform over the CTA; no wait follows that one, as
  // its phase may be open still). Two waits for the same vector have a barrier of the CTA between
  // them.
  __device__ __forceinline__ bool wait(int which) const {
    if (size == 1) {
      __syncthreads();
      return true;
    }
    const unsigned bar = shared_addr(&sh->bar[which]);
    const unsigned ph = sh->phase[which] & 1u;
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"(tx[which])
                   : "memory");
    }
    unsigned ok = 0;
    for (int k = 0; k < kClusterWaitTries && ok == 0; ++k) {
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}"
          : "=r"(ok)
          : "r"(bar), "r"(ph)
          : "memory");
    }
    if (ok == 0) sh->fail = 1;
    __syncthreads();
    if (threadIdx.x == 0) ++sh->phase[which];
    return sh->fail == 0;
  }
};

// put_x (WHICH 0) or put_y (1) of one walk, its addresses in registers. OWN: every lane goes
// through its own targets (the chunk kernel's clusters of up to 16; the batched kernels' of mostly
// 4 were 1-2% slower so).
template <typename V, int MODE, int WHICH, bool OWN = false>
struct Sender {
  Array<V, MODE != kInDevice> v;
  unsigned mask, bar, distance, size;
  __device__ __forceinline__ explicit Sender(const Exchange<V, MODE>& ex)
      : v(WHICH == 0 ? ex.xs() : ex.ys()),
        mask(shared_addr(WHICH == 0 ? ex.cmask() : ex.rmask())),
        bar(shared_addr(&ex.sh->bar[WHICH])),
        distance(shared_addr(&ex.sh->distance[0])),
        size(ex.size) {}
  __device__ __forceinline__ void put(const At& at, V value) const {
    v.set(at.p, value);
    if constexpr (MODE != kInDevice) {
      if (size > 1) {
        unsigned m = sh_load_u16(mask + 2 * at.l);
        if constexpr (OWN) {
          // Each lane its own targets, two at a time (every target in turn by the whole warp takes
          // 100 clocks each, 1,500 with 16 CTAs).
          const unsigned a = v.a + at.p * static_cast<int>(sizeof(V));
          while (m != 0u) {
            const unsigned q0 = 31 - __clz(m);
            m ^= 1u << q0;
            const unsigned q1 = 31 - __clz(m | 1u);
            const unsigned d0 = sh_load_u32(distance + 4 * q0);
            const unsigned d1 = sh_load_u32(distance + 4 * q1);
            st_async(a + d0, value, bar + d0);
            st_async_if(m, a + d1, value, bar + d1);
            m &= ~(1u << q1);
          }
        } else {
          for (unsigned q = 1; q < size; ++q) {
            if ((m >> q) & 1u) {
              const unsigned d = sh_load_u32(distance + 4 * q);
              st_async(v.a + at.p * static_cast<int>(sizeof(V)) + d, value, bar + d);
            }
          }
        }
      }
    }
  }
};

// How a share's slices are walked: one at a time, two (walk_pairs), or one whose rows take 32 >> slice
// lanes each.
enum : int { kWalkOne = 0, kWalkPairs = 1, kWalkLanes = 2 };

// A CTA's share of an operator by rows.
template <typename T, int WALK = kWalkOne>
struct alignas(16) RowShare {
  static constexpr bool kTasks = false;
  const int2* sl;  // per row (position): first nonzero, length
  // Per slice: the place of its rows' first nonzeros (lane 0's; rows of at most 32), their number
  // of steps, with kHasLong when the slice has longer rows.
  const int2* desc;
  const int* idx;
  const T* val;
  int rows;        // of the whole operator
  int slice;       // log2 of the rows of a slice
  unsigned rank, size;

  // Own slices; own rows, whole slices (the last may run past the operator's rows); the position
  // of own row l.
  __host__ __device__ __forceinline__ int slices() const {
    const int all = (rows + (1 << slice) - 1) >> slice;
    return all > static_cast<int>(rank)
               ? (all - static_cast<int>(rank) - 1) / static_cast<int>(size) + 1
               : 0;
  }
  // Own slice ls's entry of desc.
  __device__ __forceinline__ int2 steps(int ls) const {
    return __ldg(desc + (ls * static_cast<int>(size) + static_cast<int>(rank)));
  }
  __host__ __device__ __forceinline__ int own() const { return slices() << slice; }
  // Nonzero k of a row (its first, length): the place.
  __device__ __forceinline__ int place(const int2& row, int k) const {
    if (row.y > 32) return row.x + k;
    if constexpr (WALK == kWalkLanes) {
      return row.x + ((k >> (5 - slice)) << 5) + ((k & ((32 >> slice) - 1)) << slice);
    }
    return row.x + (k << 5);
  }
  __device__ __forceinline__ int position(int l) const {
    return ((((l >> slice) * static_cast<int>(size)) + static_cast<int>(rank)) << slice) +
           (l & ((1 << slice) - 1));
  }
};
constexpr int kHasLong = 256;  // as place_rows sets it

// f(at) for every own row of the share (thread tid takes own rows tid, tid + threads, ...).
template <typename T, int WALK, typename F>
__device__ __forceinline__ void each_own(const RowShare<T, WALK>& A, const F& f) {
  const int own = A.own();
  for (int l = threadIdx.x; l < own; l += blockDim.x) {
    const At at{l >> A.slice, l & ((1 << A.slice) - 1), l, A.position(l)};
    if (at.p < A.rows) f(at);
  }
}

// The bytes that arrive here per publication, from the entries that each CTA counted for each
// other (ClusterShared::count); ends with a cluster barrier.
template <typename V, int MODE>
__device__ __forceinline__ void settle_counts(Exchange<V, MODE>& ex) {
  ClusterShared& sh = *ex.sh;
  ex.tx[0] = ex.tx[1] = 0;
  __syncthreads();
  if (threadIdx.x < 2 * ex.size) {
    const unsigned which = threadIdx.x & 1u;
    const unsigned q = threadIdx.x >> 1;
    st_cluster(map_rank(shared_addr(&sh.incoming[which][q]), ex.rank ^ q), sh.count[which][q]);
  }
  cluster_sync(ex.size);
  for (unsigned q = 0; q < ex.size; ++q) {
    ex.tx[0] += sh.incoming[0][q] * static_cast<unsigned>(sizeof(V));
    ex.tx[1] += sh.incoming[1][q] * static_cast<unsigned>(sizeof(V));
  }
  // Nobody overwrites the counts of the next LP before all have read these.
  cluster_sync(ex.size);
}

// Fills the masks of the own rows and columns and the byte counts; ends with a cluster barrier.
template <typename V, int MODE, typename T, int WALK>
__device__ __forceinline__ void build_masks(Exchange<V, MODE>& ex, const RowShare<T, WALK>& K,
                                            const RowShare<T, WALK>& Kt) {
  ClusterShared& sh = *ex.sh;
  ex.tx[0] = ex.tx[1] = 0;
  if (ex.size == 1) {
    __syncthreads();
    return;
  }
  __syncthreads();
  if (threadIdx.x < 2 * kMaxCluster) (&sh.count[0][0])[threadIdx.x] = 0;
  __syncthreads();
  for (int which = 0; which < 2; ++which) {
    // Column j is read by the CTAs that own the rows of its nonzeros, row i by the CTAs that
    // own the columns of its nonzeros.
    const RowShare<T, WALK>& A = which == 0 ? Kt : K;
    const int other = which == 0 ? K.slice : Kt.slice;
    unsigned short* mask = which == 0 ? ex.cmask() : ex.rmask();
    each_own(A, [&](const At& at) {
      const int2 sl = __ldg(A.sl + at.p);
      unsigned m = 0;
      for (int k = 0; k < sl.y; ++k) {
        const int j = __ldg(A.idx + A.place(sl, k));
        m |= 1u << (((j >> other) & static_cast<int>(ex.size - 1)) ^ static_cast<int>(ex.rank));
      }
      m &= ~1u;
      mask[at.l] = static_cast<unsigned short>(m);
      while (m != 0u) {
        const unsigned q = __ffs(m) - 1;
        m &= m - 1u;
        atomicAdd(&sh.count[which][q], 1u);
      }
    });
  }
  settle_counts(ex);
}

// K sums (or maxima, bit q of MAXMASK) over the cluster, in a fixed order; every thread of every
// CTA receives the totals.
template <int K, unsigned MAXMASK = 0u>
__device__ __forceinline__ void cluster_reduce(double (&v)[K], ClusterShared& sh, unsigned rank,
                                               unsigned size) {
  static_assert(K <= 24, "peer slots");
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < K; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double t = __shfl_down_sync(0xffffffffu, v[q], o);
      v[q] = ((MAXMASK >> q) & 1u) ? fmax(v[q], t) : v[q] + t;
    }
  }
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < K; ++q) sh.red[q * kMaxWarps + warp] = v[q];
  }
  __syncthreads();
  if (threadIdx.x < K) {
    const bool mx = (MAXMASK >> threadIdx.x) & 1u;
    double t = sh.red[threadIdx.x * kMaxWarps];
    for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) {
      const double u = sh.red[threadIdx.x * kMaxWarps + w];
      t = mx ? fmax(t, u) : t + u;
    }
    if (size == 1) {
      sh.peer[threadIdx.x] = t;
    } else {
      const unsigned a = shared_addr(&sh.peer[rank * K + threadIdx.x]);
      for (unsigned q = 0; q < size; ++q) st_cluster(map_rank(a, q), t);
    }
  }
  cluster_sync(size);
#pragma unroll
  for (int q = 0; q < K; ++q) {
    double t = sh.peer[q];
    for (unsigned p = 1; p < size; ++p) {
      t = ((MAXMASK >> q) & 1u) ? fmax(t, sh.peer[p * K + q]) : t + sh.peer[p * K + q];
    }
    v[q] = t;
  }
  cluster_sync(size);
}

// NC: the matrix is not written by this kernel (loads through the read-only path).
template <bool NC, typename T>
__device__ __forceinline__ T ld_mat(const T* p) {
  if constexpr (NC) {
    return __ldg(p);
  } else {
    return *p;
  }
}

// In the body of a branch that all of `mask`'s lanes take together: keeps the body behind a jump.
// As predicated instructions its FP64 operations would take the pipe for 19 clocks each even with
// every lane off (measured on a walk of no rows: 8 of them, 1,400 clocks beside 15 busy warps).
__device__ __forceinline__ void keep_branch(unsigned mask) { __syncwarp(mask); }

// The parts of a slice's rows, on every 2^slice-th lane, added up (or their maximum).
template <bool MAXRED, typename ACC>
__device__ __forceinline__ ACC join_lanes(ACC s, int slice) {
  for (int o = 16; o >= 1 << slice; o >>= 1) {
    const ACC got = __shfl_xor_sync(0xffffffffu, s, o);
    s = MAXRED ? fmax(s, got) : s + got;
  }
  return s;
}

// s + the sum (or maximum) over the nonzeros of the slice's longer rows (lanes with a row, at
// position p; the others keep s), by the whole warp, four (FP64) or eight rows at a time so that
// their loads overlap: lane l takes nonzeros l, l + 32, ..., and the shuffle trees of the rows are
// folded into one (each step halves the sums a lane carries: 6 additions in place of 20, 9 in
// place of 40); every row's tree is the same as alone.
template <bool NC, bool MAXRED, typename T, int WALK, typename ACC, typename Prod>
__device__ __forceinline__ ACC long_rows(const RowShare<T, WALK> A, const Prod& prod, bool valid,
                                         int p, ACC s) {
  constexpr int kTogether = sizeof(ACC) == 8 ? 4 : 8;
  const int lane = threadIdx.x & 31;
  int2 sl = make_int2(0, 0);
  if (valid) sl = __ldg(A.sl + p);
  unsigned pending = __ballot_sync(0xffffffffu, sl.y > 32);
  while (pending != 0u) {
    int lb[kTogether], ll[kTogether];
    unsigned taken = 0;  // the lanes whose rows this round sums
    int most = 0;
#pragma unroll
    for (int u = 0; u < kTogether; ++u) {
      const int src = pending != 0u ? __ffs(pending) - 1 : 0;
      lb[u] = __shfl_sync(0xffffffffu, sl.x, src);
      ll[u] = __shfl_sync(0xffffffffu, sl.y, src);
      if (pending == 0u) ll[u] = 0;
      taken |= pending & (0u - pending);
      pending &= pending - 1u;
      most = max(most, ll[u]);
    }
    ACC t[kTogether];
#pragma unroll
    for (int u = 0; u < kTogether; ++u) t[u] = ACC(0);
    for (int first = 0; first < most; first += 32) {
      const int k = first + lane;
      T la[kTogether];
      int lj[kTogether];
#pragma unroll
      for (int u = 0; u < kTogether; ++u) {
        la[u] = T(0);
        lj[u] = 0;
        if (k < ll[u]) {
          la[u] = ld_mat<NC>(A.val + lb[u] + k);
          lj[u] = __ldg(A.idx + lb[u] + k);
        }
      }
#pragma unroll
      for (int u = 0; u < kTogether; ++u) {
        if (first < ll[u]) {
          if constexpr (sizeof(ACC) == 8) keep_branch(0xffffffffu);
          const ACC q = prod(la[u], lj[u]);
          const ACC n = MAXRED ? fmax(t[u], q) : t[u] + q;
          t[u] = k < ll[u] ? n : t[u];
        }
      }
    }
    // Folded tree: the upper half of the lanes goes on with the upper half of the rows; when one
    // row is left, plain steps finish it. Row u ends in lanes u 32/kTogether and on.
    int o = 16;
#pragma unroll
    for (int h = kTogether / 2; h > 0; h >>= 1, o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int u = 0; u < h; ++u) {
        const ACC give = up ? t[u] : t[u + h];
        const ACC keep = up ? t[u + h] : t[u];
        const ACC got = __shfl_xor_sync(0xffffffffu, give, o);
        t[u] = MAXRED ? fmax(keep, got) : keep + got;
      }
    }
#pragma unroll
    for (; o > 0; o >>= 1) {
      const ACC got = __shfl_xor_sync(0xffffffffu, t[0], o);
      t[0] = MAXRED ? fmax(t[0], got) : t[0] + got;
    }
    const int u = __popc(taken & ((1u << lane) - 1u));
    const ACC mine = __shfl_sync(0xffffffffu, t[0], (u * (32 / kTogether)) & 31);
    if ((taken >> lane) & 1u) s = MAXRED ? fmax(s, mine) : s + mine;
  }
  return s;
}

// f(at, s) for every own row of the share, s = init(at) + the sum of prod(val, idx) over the row's
// nonzeros (or the maximum, with init 0). A row of at most 32 nonzeros is summed by its thread in
// index order, as many steps as its slice's longest (a shorter row's padding adds 0 times the
// gathered vector's last entry, 0), with kWalkLanes by its lanes and a tree over them; longer rows
// by long_rows. Then every row's (first) lane runs f, so that the updates of a slice run side by
// side. ready() waits for the gathered vector after
// the first loads are on their way (every thread calls it once; false ends the walk).
//
// walk_one: a slice at a time, four steps' nonzeros loaded while the four before are summed (of the
// same slice or the warp's slice before).
template <bool NC, bool MAXRED, typename T, int WALK, typename Prod, typename Init, typename F,
          typename Ready>
__device__ __forceinline__ bool walk_one(const RowShare<T, WALK> A, const Prod& prod,
                                         const Init& init, const F& f, const Ready& ready) {
  using ACC = decltype(prod(T(), 0));
  constexpr int B = kBatch;
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  const bool lane_in = lane < (1 << A.slice);
  const int own = A.slices();
  T a[B];
  int j[B];
  // Nonzeros k .. k + B - 1 of a slice's rows.
  auto fetch = [&](int2 d, int k) {
    const T* val = A.val + (d.x + lane + (k << 5));
    const int* idx = A.idx + (d.x + lane + (k << 5));
    const int left = (d.y & 255) - k;
#pragma unroll
    for (int u = 0; u < B; ++u) {
      if (u < left) {
        a[u] = ld_mat<NC>(val + (u << 5));
        j[u] = __ldg(idx + (u << 5));
      }
    }
  };
  int ls = threadIdx.x >> 5;
  int2 d = ls < own ? A.steps(ls) : make_int2(0, 0);
  fetch(d, 0);
  if (!ready()) return false;
  while (ls < own) {
    const int next = ls + warps;
    const At at{ls, lane, (ls << A.slice) + lane,
                ((ls * static_cast<int>(A.size) + static_cast<int>(A.rank)) << A.slice) + lane};
    const bool valid = lane_in && at.p < A.rows;
    const int2 dn = next < own ? A.steps(next) : make_int2(0, 0);
    ACC s = ACC(0);
    if (valid) s = init(at);
    const int width = d.y & 255;
    for (int k = 0;; k += B) {
      T ca[B];
      int cj[B];
      const bool more = k + B < width;
#pragma unroll
      for (int u = 0; u < B; ++u) {
        ca[u] = a[u];
        cj[u] = j[u];
      }
      fetch(more ? d : dn, more ? k + B : 0);
      const int left = width - k;
      auto step = [&](int u) {
        const ACC q = prod(ca[u], cj[u]);
        s = MAXRED ? fmax(s, q) : s + q;
      };
      // Behind jumps (keep_branch): exactly the steps that are left.
      if (left >= 4) {
        keep_branch(0xffffffffu);
        step(0);
        step(1);
        step(2);
        step(3);
      } else if (left >= 2) {
        keep_branch(0xffffffffu);
        step(0);
        step(1);
        if (left == 3) {
          keep_branch(0xffffffffu);
          step(2);
        }
      } else if (left == 1) {
        keep_branch(0xffffffffu);
        step(0);
      }
      if (!more) break;
    }
    if constexpr (WALK == kWalkLanes) s = join_lanes<MAXRED>(s, A.slice);
    if (d.y >= kHasLong) s = long_rows<NC, MAXRED>(A, prod, valid, at.p, s);
    if (valid) f(at, s);
    d = dn;
    ls = next;
  }
  return true;
}

// walk_pairs: two slices at a time, so that 16 loads a thread are on their way.
template <bool NC, bool MAXRED, typename T, typename Prod, typename Init, typename F,
          typename Ready>
__device__ __forceinline__ bool walk_pairs(const RowShare<T, kWalkPairs> A, const Prod& prod,
                                           const Init& init, const F& f, const Ready& ready) {
  using ACC = decltype(prod(T(), 0));
  constexpr int B = kBatch;
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  const bool lane_in = lane < (1 << A.slice);
  const int own = A.slices();
  bool called = false;
  for (int ls = threadIdx.x >> 5; ls < own || !called; ls += 2 * warps) {
    int2 d[2];
    ACC s[2];
    At at[2];
    bool valid[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int q = ls + h * warps;
      d[h] = q < own ? A.steps(q) : make_int2(0, 0);
      at[h] = At{q, lane, (q << A.slice) + lane,
                 ((q * static_cast<int>(A.size) + static_cast<int>(A.rank)) << A.slice) + lane};
      valid[h] = lane_in && q < own && at[h].p < A.rows;
      s[h] = ACC(0);
    }
    const int width = max(d[0].y & 255, d[1].y & 255);
    for (int k = 0; k == 0 || k < width; k += B) {
      T a[2][B];
      int j[2][B];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const T* val = A.val + (d[h].x + lane + (k << 5));
        const int* idx = A.idx + (d[h].x + lane + (k << 5));
        const int left = (d[h].y & 255) - k;
#pragma unroll
        for (int u = 0; u < B; ++u) {
          if (u < left) {
            a[h][u] = ld_mat<NC>(val + (u << 5));
            j[h][u] = __ldg(idx + (u << 5));
          }
        }
      }
      if (!called) {
        if (!ready()) return false;
        called = true;
      }
      if (k == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (valid[h]) s[h] = init(at[h]);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int left = (d[h].y & 255) - k;
#pragma unroll
        for (int u = 0; u < B; ++u) {
          if (u < left) {
            const ACC q = prod(a[h][u], j[h][u]);
            s[h] = MAXRED ? fmax(s[h], q) : s[h] + q;
          }
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (d[h].y >= kHasLong) s[h] = long_rows<NC, MAXRED>(A, prod, valid[h], at[h].p, s[h]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (valid[h]) f(at[h], s[h]);
    }
  }
  return true;
}

template <bool NC, bool MAXRED, typename T, int WALK, typename Prod, typename Init, typename F,
          typename Ready>
__device__ __forceinline__ bool walk_rows(const RowShare<T, WALK>& A, const Prod& prod,
                                          const Init& init, const F& f, const Ready& ready) {
  if constexpr (WALK == kWalkPairs) {
    return walk_pairs<NC, MAXRED>(A, prod, init, f, ready);
  } else {
    return walk_one<NC, MAXRED>(A, prod, init, f, ready);
  }
}

// The walk of a step (NC, sums): a share of tasks has its own (sg_chunk.cu).
template <typename Share, typename Prod, typename Init, typename F, typename Ready>
__device__ __forceinline__ bool walk_step(const Share& A, const Prod& prod, const Init& init,
                                          const F& f, const Ready& ready) {
  if constexpr (Share::kTasks) {
    return A.walk(prod, init, f, ready);
  } else {
    return walk_rows<true, false>(A, prod, init, f, ready);
  }
}

// ready of a walk whose gathered vector is in place.
struct Ready {
  __device__ __forceinline__ bool operator()() const { return true; }
};

// init of a plain sum.
template <typename ACC>
struct Zero {
  __device__ __forceinline__ ACC operator()(const At&) const { return ACC(0); }
};

}  // namespace sg
