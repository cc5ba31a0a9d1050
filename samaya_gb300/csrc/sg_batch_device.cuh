// Device pieces shared by the batched kernels: a matrix's share of one CTA, the shared-memory
// layout, projections and launches (see sg_cluster.cuh and sg_batch.cuh).
#pragma once

#include <math.h>
#include <stdint.h>

#include "sg_batch.cuh"
#include "sg_cluster.cuh"

namespace sg {

namespace {

__device__ __forceinline__ double lam_of(double g, double lo, double up) {
  const bool hl = lo > -INFINITY;
  const bool hu = up < INFINITY;
  return hl && hu ? g : hl ? fmax(g, 0.0) : hu ? fmin(g, 0.0) : 0.0;
}

// fmin(fmax(v, lo), hi). In FP64 the comparisons run on the integer pipe, on the doubles' bits
// mapped to a signed order (-0 below +0; a NaN becomes lo, as fmax makes it): the FP64 pipe, two
// operations a clock per SM, bounds these kernels.
__device__ __forceinline__ float clamp_to(float v, float lo, float hi) {
  return fminf(fmaxf(v, lo), hi);
}
__device__ __forceinline__ double clamp_to(double v, double lo, double hi) {
  const long long bv = __double_as_longlong(v);
  const long long bl = __double_as_longlong(lo);
  const long long bh = __double_as_longlong(hi);
  const long long kl = bl ^ ((bl >> 63) & 0x7fffffffffffffffLL);
  const long long kh = bh ^ ((bh >> 63) & 0x7fffffffffffffffLL);
  const bool nan = (bv & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
  const long long kv = bv ^ ((bv >> 63) & 0x7fffffffffffffffLL);
  const bool low = nan || kv < kl;
  const double r = low ? lo : v;
  return (low ? kl : kv) > kh ? hi : r;
}

template <typename T>
struct GatherT {
  const T* x;
  __device__ __forceinline__ T operator()(T a, int j) const { return a * x[j]; }
};
template <typename T>
struct GatherD {
  const T* x;
  __device__ __forceinline__ double operator()(T a, int j) const {
    return static_cast<double>(a) * static_cast<double>(x[j]);
  }
};

// The products of a walk over the gathered vector x.
template <typename T, int MODE>
struct Gather {
  Array<T, MODE != kInDevice> x;
  __device__ __forceinline__ T operator()(T a, int j) const { return a * x.get(j); }
};

// A matrix's share of one CTA.
template <typename T, typename Share = RowShare<T>>
struct MatShare {
  int m, n;
  long long kz, tz;        // first element of A's and A''s arrays
  const int *kperm, *tperm;  // position -> row, column
  Share K, Kt;             // own rows of A and of A'
  int nr, nc;              // own rows and columns, whole slices
};

template <typename T, typename Share = RowShare<T>>
__device__ __forceinline__ MatShare<T, Share> mat_share(const BatchView& b, int g, const T* kval,
                                                        const T* tval, unsigned rank,
                                                        unsigned size) {
  MatShare<T, Share> s;
  s.m = b.mat_m[g];
  s.n = b.mat_n[g];
  s.kz = b.mat_k_off[g];
  s.tz = b.mat_t_off[g];
  s.kperm = b.k_perm + b.mat_row_off[g];
  s.tperm = b.t_perm + b.mat_col_off[g];
  s.K = Share{b.k_sl + b.mat_row_off[g], b.k_desc + b.mat_kd_off[g], b.k_idx + s.kz,
              kval + s.kz, s.m, b.mat_slice[2 * g], rank, size};
  s.Kt = Share{b.t_sl + b.mat_col_off[g], b.t_desc + b.mat_td_off[g], b.t_idx + s.tz,
               tval + s.tz, s.n, b.mat_slice[2 * g + 1], rank, size};
  s.nr = s.K.own();
  s.nc = s.Kt.own();
  return s;
}

// Shared memory, in order: the gathered vectors, the masks (clusters of several CTAs), the state.
// The vectors sit at the same place in every CTA of a cluster.
template <typename V, int MODE, typename T, typename Share>
__device__ __forceinline__ Exchange<V, MODE> make_exchange(const MatShare<T, Share>& s,
                                                           ClusterShared& sh, V* spill,
                                                           unsigned rank, unsigned size) {
  Exchange<V, MODE> ex;
  ex.sh = &sh;
  ex.rank = rank;
  ex.size = size;
  ex.device = spill;
  if constexpr (MODE != kInDevice) {
    ex.xs_at = 0u;
    ex.ys_at = (s.n + 1) * static_cast<unsigned>(sizeof(V));
    ex.cmask_at = ex.ys_at + (s.m + 1) * static_cast<unsigned>(sizeof(V));
    ex.rmask_at = ex.cmask_at + s.nc * 2;
  } else {
    ex.xs_at = 0u;
    ex.ys_at = s.n + 1;
    ex.cmask_at = ex.rmask_at = 0u;
  }
  if (threadIdx.x == 0) ex.xs()[s.n] = ex.ys()[s.m] = V(0);
  build_masks(ex, s.K, s.Kt);
  return ex;
}

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

// The configuration of a launch of `clusters` clusters of `size` CTAs.
struct ClusterLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  template <typename... Params>
  cudaError_t set(void (*kernel)(Params...), int size, int clusters, int threads, size_t smem,
                  cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kClusterSmemMax));
    if (e == cudaSuccess && size > 8) {
      e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                               cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    cfg.gridDim = dim3(clusters * size);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return e;
  }
};

template <typename... Params, typename... Args>
cudaError_t launch_clusters(void (*kernel)(Params...), int size, int clusters, int threads,
                            size_t smem, cudaStream_t s, Args... args) {
  ClusterLaunch l;
  const cudaError_t e = l.set(kernel, size, clusters, threads, smem, s);
  return e != cudaSuccess ? e : cudaLaunchKernelEx(&l.cfg, kernel, args...);
}

// Whether the device can hold a cluster of this kernel at all. A process that owns a slice of the
// GPU may have no GPC with that many SMs to itself. A kernel and size found to fit with the most
// shared memory fit with any: the device is asked once for them (30 to 60 us; a solve_pdlp call on
// a facility-location LP of 40 x 150 takes 2,030).
template <typename... Params>
bool clusters_fit(void (*kernel)(Params...), int size, int threads, size_t smem) {
  if (size > cluster_limit()) return false;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return false;
  const void* address = reinterpret_cast<const void*>(kernel);
  if (known_to_fit(address, device, size, threads, false)) return true;
  auto asked = [&](size_t bytes) {
    ClusterLaunch l;
    int clusters = 0;
    if (l.set(kernel, size, 1, threads, bytes, nullptr) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &l.cfg) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return clusters > 0;
  };
  if (asked(kClusterSmemMax)) return known_to_fit(address, device, size, threads, true);
  return asked(smem);
}

}  // namespace

}  // namespace sg
