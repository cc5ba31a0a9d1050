// The PDHG steps of one LP on a cluster, with the state they keep (see sg_cluster.cuh).
#pragma once

#include "sg_batch_device.cuh"

namespace sg {

namespace {

// The state of the own columns and rows that every iteration reads, one array after another
// (array k of own entry l, position p): the point, the sum since the restart (FP32: the running
// average; Halpern: the anchor) and the scaled problem; the rows' extrapolated point (negated),
// dual and its sum.
enum : int {
  kPoint = 0, kSum = 1, kCost = 2, kLower = 3, kUpper = 4, kBar = 5, kDual = 6, kDualSum = 7
};
constexpr int kColArrays = 5, kRowArrays = 8;  // solve_state_bytes

// Slice by slice, 32 entries of each array (a constant distance between a row's values): in shared
// memory the CTA's own slices, in device memory all slices.
template <typename T, int MODE>
struct alignas(16) SolveState {
  T* device;                   // not kAllShared: the columns' arrays
  long long rows_device;       // and how far on the rows' are
  unsigned cols_at, rows_at;   // kAllShared: offsets
  unsigned rank, size;
  __device__ __forceinline__ T* col_base() const {
    if constexpr (MODE == kAllShared) return reinterpret_cast<T*>(sg_smem + cols_at);
    return device;
  }
  __device__ __forceinline__ T* row_base() const {
    if constexpr (MODE == kAllShared) return reinterpret_cast<T*>(sg_smem + rows_at);
    return device + rows_device;
  }
  __device__ __forceinline__ T& col(int k, const At& at) const {
    if constexpr (MODE == kAllShared) {
      return reinterpret_cast<T*>(sg_smem + cols_at)[(at.ls * kColArrays + k) * 32 + at.lane];
    } else {
      return device[(static_cast<long long>(at.ls * size + rank) * kColArrays + k) * 32 + at.lane];
    }
  }
  __device__ __forceinline__ T& row(int k, const At& at) const {
    if constexpr (MODE == kAllShared) {
      return reinterpret_cast<T*>(sg_smem + rows_at)[(at.ls * kRowArrays + k) * 32 + at.lane];
    } else {
      return device[rows_device +
                    (static_cast<long long>(at.ls * size + rank) * kRowArrays + k) * 32 + at.lane];
    }
  }
};

// One operator's state arrays (the columns' or the rows') in a walk: entry k of the own row `at`.
template <typename T, int MODE, int ARRAYS>
struct StepState {
  Array<T, MODE == kAllShared> base;
  unsigned rank, size;
  struct Entry {
    Array<T, MODE == kAllShared> e;
    __device__ __forceinline__ T get(int k) const { return e.get(32 * k); }
    __device__ __forceinline__ void set(int k, T v) const { e.set(32 * k, v); }
  };
  __device__ __forceinline__ Entry at(const At& a) const {
    Entry r{base};
    if constexpr (MODE == kAllShared) {
      r.e.a += (a.ls * (ARRAYS * 32) + a.lane) * static_cast<int>(sizeof(T));
    } else {
      r.e.a += static_cast<long long>(a.ls * static_cast<int>(size) + static_cast<int>(rank)) *
                   (ARRAYS * 32) + a.lane;
    }
    return r;
  }
};

// Device storage of an instance beside the state: the second point (the restart point, or
// Halpern's T(z)), the columns' saved extrapolated point, by position.
template <typename T>
struct Second {
  T* st;  // x (n), r (m), y (m), saved (n)
  int n, m;
  __device__ __forceinline__ T& x(int p) const { return st[p]; }
  __device__ __forceinline__ T& r(int p) const { return st[n + p]; }
  __device__ __forceinline__ T& y(int p) const { return st[n + m + p]; }
  __device__ __forceinline__ T& saved(int p) const { return st[n + 2 * m + p]; }
};

// The average of `count` points whose sum is s (FP64; FP32 keeps the average itself).
__device__ __forceinline__ double average(double s, double inv_count) { return s * inv_count; }
__device__ __forceinline__ float average(float s, double) { return s; }

template <typename T, int MODE>
__device__ __forceinline__ StepState<T, MODE, kColArrays> col_state(const SolveState<T, MODE>& S) {
  return {S.col_base(), S.rank, S.size};
}
template <typename T, int MODE>
__device__ __forceinline__ StepState<T, MODE, kRowArrays> row_state(const SolveState<T, MODE>& S) {
  return {S.row_base(), S.rank, S.size};
}

// What the walks need of an instance, in shared memory (sh_copy).
template <typename T, int MODE, typename Share = RowShare<T>, typename State = SolveState<T, MODE>>
struct StepContext {
  MatShare<T, Share> M;
  Exchange<T, MODE> ex;
  State S;
  Second<T> Z;
  T weight[64], rest[64];  // run_steps
};

// One PDHG iteration (FP64: sums since the restart in place of running averages, one addition
// less each, and the row's own term as the sum's start). xs has been put, not waited for; so it
// is afterwards.
template <typename T, int MODE, typename Share, typename State>
__device__ __forceinline__ bool classic_step(const StepContext<T, MODE, Share, State>* ctx, T tau, T sig,
                                             T ta, T tb) {
  constexpr bool kF64 = sizeof(T) == 8;
  {
    const auto K = sh_copy(&ctx->M.K);
    const auto ex = sh_copy(&ctx->ex);
    const auto R = row_state(sh_copy(&ctx->S));
    const Sender<T, MODE, 1, Share::kTasks> y_out(ex);
    const bool ok = walk_step(
        K, Gather<T, MODE>{ex.xs()},
        [&](const At& at) { return kF64 ? R.at(at).get(kBar) : T(0); },
        [&](const At& at, T s) {
          const auto e = R.at(at);
          const T res = kF64 ? s : s + e.get(kBar);
          const T yn = e.get(kDual) + sig * res;
          e.set(kDual, yn);
          y_out.put(at, yn);
          const T lo = e.get(kLower);
          const T up = e.get(kUpper);
          const T r = e.get(kPoint);
          if constexpr (kF64) {
            e.set(kDualSum, e.get(kDualSum) + yn);
            // An equality row's logical is its bound from the first step on: a warp of such
            // rows skips the logicals.
            const bool steady = same_bits(lo, up) && same_bits(r, lo);
            const unsigned here = __activemask();
            if (__any_sync(here, !steady)) {
              keep_branch(here);
              const T rn = clamp_to(r - tau * (e.get(kCost) - yn), lo, up);
              e.set(kPoint, rn);
              e.set(kBar, fma(-2.0, rn, r));
              e.set(kSum, e.get(kSum) + rn);
            } else {
              e.set(kBar, -lo);
            }
          } else {
            const T rn = clamp_to(r - tau * (e.get(kCost) - yn), lo, up);
            e.set(kPoint, rn);
            e.set(kBar, -(rn + (rn - r)));
            e.set(kDualSum, tb * e.get(kDualSum) + ta * yn);
            e.set(kSum, tb * e.get(kSum) + ta * rn);
          }
        },
        [&]() { return ex.wait(0); });
    if (!ok) return false;
  }
  const auto Kt = sh_copy(&ctx->M.Kt);
  const auto ex = sh_copy(&ctx->ex);
  const auto C = col_state(sh_copy(&ctx->S));
  const Sender<T, MODE, 0, Share::kTasks> x_out(ex);
  return walk_step(
      Kt, Gather<T, MODE>{ex.ys()},
      [&](const At& at) { return kF64 ? C.at(at).get(kCost) : T(0); },
      [&](const At& at, T s) {
        const auto e = C.at(at);
        const T x = e.get(kPoint);
        const T g = kF64 ? s : e.get(kCost) + s;
        const T v = clamp_to(x - tau * g, e.get(kLower), e.get(kUpper));
        e.set(kPoint, v);
        x_out.put(at, kF64 ? fma(T(2), v, -x) : v + (v - x));
        e.set(kSum, kF64 ? e.get(kSum) + v : tb * e.get(kSum) + ta * v);
      },
      [&]() { return ex.wait(1); });
}

// One reflected Halpern iteration z+ = N + w (z0 - N), N = 2 T(z) - z, w = 1 / (k + 2) (k:
// iterations since the restart), T the PDHG map in primal-first order, as the single-LP engine's
// halpern_primal / halpern_dual kernels compute it; the anchor is in the sums' place, and T(z)
// (the point the evaluation, the restarts and the answer use) is written when it is `measured`.
// ys has been put, not waited for; so it is afterwards.
template <typename T, int MODE, typename Share, typename State>
__device__ __forceinline__ bool halpern_step(const StepContext<T, MODE, Share, State>* ctx, T tau, T sig, T w,
                                             bool measured) {
  constexpr bool kF64 = sizeof(T) == 8;
  const Second<T>& Z = ctx->Z;
  {
    const auto Kt = sh_copy(&ctx->M.Kt);
    const auto ex = sh_copy(&ctx->ex);
    const auto C = col_state(sh_copy(&ctx->S));
    const Sender<T, MODE, 0, Share::kTasks> x_out(ex);
    const bool ok = walk_step(
        Kt, Gather<T, MODE>{ex.ys()},
        [&](const At& at) { return kF64 ? C.at(at).get(kCost) : T(0); },
        [&](const At& at, T s) {
          const auto e = C.at(at);
          const T x = e.get(kPoint);
          const T g = kF64 ? s : e.get(kCost) + s;
          const T xh = clamp_to(x - tau * g, e.get(kLower), e.get(kUpper));
          const T refl = kF64 ? fma(T(2), xh, -x) : xh + (xh - x);
          x_out.put(at, refl);
          e.set(kPoint, refl + w * (e.get(kSum) - refl));
          if (measured) Z.x(at.p) = xh;
        },
        [&]() { return ex.wait(1); });
    if (!ok) return false;
  }
  const auto K = sh_copy(&ctx->M.K);
  const auto ex = sh_copy(&ctx->ex);
  const auto R = row_state(sh_copy(&ctx->S));
  const Sender<T, MODE, 1, Share::kTasks> y_out(ex);
  return walk_step(
      K, Gather<T, MODE>{ex.xs()}, Zero<T>(),
      [&](const At& at, T s) {
        const auto e = R.at(at);
        const T y = e.get(kDual);
        const T r = e.get(kPoint);
        const T rh = clamp_to(r - tau * (e.get(kCost) - y), e.get(kLower), e.get(kUpper));
        const T rrefl = kF64 ? fma(T(2), rh, -r) : rh + (rh - r);
        const T yh = y + sig * (s - rrefl);
        const T yrefl = kF64 ? fma(T(2), yh, -y) : yh + (yh - y);
        const T yn = yrefl + w * (e.get(kDualSum) - yrefl);
        e.set(kDual, yn);
        y_out.put(at, yn);
        e.set(kPoint, rrefl + w * (e.get(kSum) - rrefl));
        if (measured) {
          Z.y(at.p) = yh;
          Z.r(at.p) = rh;
        }
      },
      [&]() { return ex.wait(0); });
}

// `count` iterations, the last of them measured, before_last() just before it; xs (Halpern: ys)
// put, not waited for, before and after. ctx->weight and rest hold the steps' weights. (Inlined:
// in a called function every global load takes two more instructions for its descriptor.)
template <bool HALPERN, typename T, int MODE, typename Share, typename State, typename BeforeLast>
__device__ __forceinline__ bool run_steps(const StepContext<T, MODE, Share, State>* ctx,
                                          int count, T tau, T sig,
                                          const BeforeLast& before_last) {
  bool ok = true;
  for (int i = 0; i < count && ok; ++i) {
    if (i == count - 1) before_last();
    if constexpr (HALPERN) {
      ok = halpern_step(ctx, tau, sig, ctx->weight[i], i == count - 1);
    } else {
      ok = classic_step(ctx, tau, sig, ctx->weight[i], ctx->rest[i]);
    }
  }
  return ok;
}

}  // namespace

}  // namespace sg
