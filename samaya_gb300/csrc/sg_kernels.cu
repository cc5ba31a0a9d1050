// Kernels of the GB300 PDLP engine: the two fused PDHG step kernels, the evaluation kernels, the
// single-CTA decision kernels, restarts, infeasibility/unboundedness detection and the
// device-side setup (Ruiz, power iteration, norms).
//
// Reference algorithm: src/lp/pdlp.cpp (CPU loop and decisions) and src/gpu/pdhg_core.cu (its
// GPU arithmetic). Here every decision of the loop runs on the device, so a chunk of
// kCheckFrequency iterations plus its evaluation replays from one CUDA graph.
#include <math.h>

#include <type_traits>

#include "sg_kernels.cuh"
#include "sg_tile.cuh"

namespace sg {

namespace {

template <typename T>
__device__ __forceinline__ T clampv(T v, T lo, T hi) {
  return fmin(fmax(v, lo), hi);
}

// Doubles compared through their bit patterns mapped to a signed integer order, on the integer
// pipe (GB300's FP64 pipe is small): the same as fmin(fmax(v, lo), hi) for numbers (with
// -0 ordered below +0).
__device__ __forceinline__ long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

template <>
__device__ __forceinline__ double clampv<double>(double v, double lo, double hi) {
  const double r = order_key(v) < order_key(lo) ? lo : v;
  return order_key(r) > order_key(hi) ? hi : r;
}

// The extrapolated point 2 v+ - v (one fused operation in FP64).
template <typename T>
__device__ __forceinline__ T extrapolate(T vn, T v) {
  return vn + (vn - v);
}

template <>
__device__ __forceinline__ double extrapolate<double>(double vn, double v) {
  return fma(2.0, vn, -v);
}

// lambda of the reduced cost g for a variable with bounds [lo, up] (pdlp.cpp:455-465).
__device__ __forceinline__ double bound_part(double g, double lo, double up) {
  const bool hl = lo > -INFINITY;
  const bool hu = up < INFINITY;
  return hl && hu ? g : hl ? fmax(g, 0.0) : hu ? fmin(g, 0.0) : 0.0;
}

// Plain loads: a step launch's CTAs are there while the launch before them still writes x
// (wait_for_previous), which the read-only path does not allow.
template <typename T, typename ACC>
struct Gather1 {
  const T* x;
  __device__ __forceinline__ ACC operator()(int, T a, int j) const {
    return static_cast<ACC>(a) * static_cast<ACC>(x[j]);
  }
};

template <typename T>
struct Gather2 {
  const T* x0;
  const T* x1;
  __device__ __forceinline__ double operator()(int v, T a, int j) const {
    return static_cast<double>(a) * static_cast<double>(ldg((v == 0 ? x0 : x1) + j));
  }
};

// ------------------------------------------------------------------------------------------
// Step kernels. One PDHG iteration (pdlp.cpp:574-641; pdhg_core.cu:23-50) is two launches:
//   dual   (rows of K):  y+ = y + sigma (K xbar - rbar - q); r+ = proj(r - tau (c_r - y+));
//                        rbar' = r+ + (r+ - r); averages of y and r
//   primal (rows of K'): x+ = proj(x - tau (c_x + K' y+)); xbar' = x+ + (x+ - x); average of x
// The extrapolation of the reference's first kernel is produced by the previous step's
// epilogue (xbar'), so the SpMV gathers one vector.

template <typename T, typename ACC>
struct DualEpi {
  const T* y;
  T* y_new;
  const T* vr;   // r (n offset applied)
  T* vr_new;
  T* vbar_r;
  const T* c;
  const T* l;
  const T* u;
  const T* q;
  T* yerg;
  T* verg_r;
  ACC sigma, tau, alpha, beta;
  struct Pre {
    ACC rbar, q, y, r, c, l, u, yerg, rerg;
  };
  __device__ __forceinline__ Pre load(int i) const {
    Pre p;
    p.rbar = static_cast<ACC>(vbar_r[i]);
    p.q = q != nullptr ? static_cast<ACC>(q[i]) : ACC(0);
    p.y = static_cast<ACC>(y[i]);
    p.r = static_cast<ACC>(vr[i]);
    p.c = static_cast<ACC>(c[i]);
    p.l = static_cast<ACC>(l[i]);
    p.u = static_cast<ACC>(u[i]);
    p.yerg = static_cast<ACC>(yerg[i]);
    p.rerg = static_cast<ACC>(verg_r[i]);
    return p;
  }
  __device__ __forceinline__ void row(int i, const ACC (&s)[1], const Pre& p) {
    ACC res = s[0] - p.rbar;
    if (q != nullptr) res -= p.q;
    const ACC yn = p.y + sigma * res;
    y_new[i] = static_cast<T>(yn);
    ACC rn = p.r - tau * (p.c - yn);
    rn = clampv<ACC>(rn, p.l, p.u);
    vr_new[i] = static_cast<T>(rn);
    vbar_r[i] = static_cast<T>(extrapolate<ACC>(rn, p.r));
    yerg[i] = static_cast<T>(beta * p.yerg + alpha * yn);
    verg_r[i] = static_cast<T>(beta * p.rerg + alpha * rn);
  }
  __device__ __forceinline__ void row(int i, const ACC (&s)[1]) { row(i, s, load(i)); }
  __device__ __forceinline__ void long_row(int, int i, const ACC (&s)[1]) { row(i, s); }
};

// The bounds of column j: the shared pair when every column has it (no loads), else the
// vectors.
template <typename T, typename ACC>
struct ColBounds {
  const T* l;
  const T* u;
  int uniform;
  ACC lo, hi;
  __device__ __forceinline__ void load(int j, ACC& pl, ACC& pu) const {
    if (uniform) {
      pl = lo;
      pu = hi;
    } else {
      pl = static_cast<ACC>(l[j]);
      pu = static_cast<ACC>(u[j]);
    }
  }
};

template <typename T, typename ACC>
__device__ __forceinline__ ColBounds<T, ACC> col_bounds(const IterView<T>& it) {
  return ColBounds<T, ACC>{it.lower, it.upper, it.xb_uniform, static_cast<ACC>(it.xb_lo),
                           static_cast<ACC>(it.xb_hi)};
}

template <typename T, typename ACC>
struct PrimalEpi {
  const T* x;
  T* x_new;
  T* xbar;
  const T* c;
  ColBounds<T, ACC> b;
  T* xerg;
  ACC tau, alpha, beta;
  struct Pre {
    ACC x, c, l, u, xerg;
  };
  __device__ __forceinline__ Pre load(int j) const {
    Pre p;
    p.x = static_cast<ACC>(x[j]);
    p.c = static_cast<ACC>(c[j]);
    b.load(j, p.l, p.u);
    p.xerg = static_cast<ACC>(xerg[j]);
    return p;
  }
  // The column's new values, written to x_new, xbar and xerg.
  static constexpr int kIn = 3, kOut = 3;
  __device__ __forceinline__ void update(const Pre& p, ACC s, ACC (&o)[kOut]) const {
    ACC xn = p.x - tau * (p.c + s);
    xn = clampv<ACC>(xn, p.l, p.u);
    o[0] = xn;
    o[1] = extrapolate<ACC>(xn, p.x);
    o[2] = beta * p.xerg + alpha * xn;
  }
  __device__ __forceinline__ void row(int j, const ACC (&s)[1], const Pre& p) {
    ACC o[kOut];
    update(p, s[0], o);
    x_new[j] = static_cast<T>(o[0]);
    xbar[j] = static_cast<T>(o[1]);
    xerg[j] = static_cast<T>(o[2]);
  }
  // The vectors that Pre reads beside the bounds, and those that update fills.
  __device__ __forceinline__ const T* in(int k) const { return k == 0 ? x : k == 1 ? c : xerg; }
  __device__ __forceinline__ T* out(int k) const { return k == 0 ? x_new : k == 1 ? xbar : xerg; }
  __device__ __forceinline__ static Pre pre(const ACC (&v)[kIn], ACC l, ACC u) {
    return Pre{v[0], v[1], l, u, v[2]};
  }
  __device__ __forceinline__ void row(int j, const ACC (&s)[1]) { row(j, s, load(j)); }
  __device__ __forceinline__ void long_row(int, int j, const ACC (&s)[1]) { row(j, s); }
};

template <typename T>
using Acc = T;  // FP64 storage accumulates in FP64, FP32 storage in FP32.

// Step launches behind another step launch of the chunk start before it has ended
// (programmatic dependent launch): a step's CTAs let the next launch's in as soon as they run
// themselves, and these read the control block (which no step writes) and take the step's
// scalars while the last CTAs before them finish; wait_for_previous() returns when that launch
// has ended and its writes are visible. Every CTA waits, also one with nothing to do: the launch
// after it relies on the one before it having ended. (A power-law LP of 400,000 x 800,000, 192
// iterations: 17.9 ms without, 17.2 with; the transportation LPs 1%. Fetching the first tile's
// nonzeros into L2 before the wait gave nothing.)
__device__ __forceinline__ void let_next_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A primal step over an operator of exactly two nonzeros a column (the columns of a transportation
// or network-flow LP): a thread takes kWide<T> consecutive columns, 16 bytes of every vector, so
// that all its loads are 16 bytes wide and on their way together. Bound by memory (36 bytes a
// column in FP32, shared bounds not counted; 2 million columns 14.5 us by run_tiles, a column a
// thread and 256 after another, 10.3 so).
template <typename T>
constexpr int kWide = 16 / static_cast<int>(sizeof(T));

template <typename T>
__device__ __forceinline__ void load_wide(const T* p, T (&v)[kWide<T>]) {
  *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
}
template <typename T>
__device__ __forceinline__ void store_wide(T* p, const T (&v)[kWide<T>]) {
  *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(v);
}

template <typename T, typename Epi>
__device__ __forceinline__ void two_nonzero_columns(const OpView<T>& Kt, const T* y, Epi& epi) {
  using ACC = Acc<T>;
  constexpr int W = kWide<T>;
  const int n = Kt.rows;
  const int j0 = (blockIdx.x * kBlock + threadIdx.x) * W;
  if (j0 + W > n) {
    for (int j = j0; j < n; ++j) {
      ACC s[1] = {ACC(0)};
      for (int q = 2 * j; q < 2 * j + 2; ++q) s[0] += ldg(Kt.val + q) * y[ldg(Kt.idx + q)];
      epi.row(j, s);
    }
    return;
  }
  alignas(16) int idx[2 * W];
  alignas(16) T val[2][W];
  alignas(16) T in[Epi::kIn][W];
  alignas(16) T lo[W], up[W];
#pragma unroll
  for (int k = 0; k < W / 2; ++k) {
    *reinterpret_cast<int4*>(idx + 4 * k) =
        __ldg(reinterpret_cast<const int4*>(Kt.idx + 2 * static_cast<size_t>(j0)) + k);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    *reinterpret_cast<float4*>(val[k]) =
        __ldg(reinterpret_cast<const float4*>(Kt.val + 2 * static_cast<size_t>(j0)) + k);
  }
#pragma unroll
  for (int k = 0; k < Epi::kIn; ++k) load_wide(epi.in(k) + j0, in[k]);
  if (!epi.b.uniform) {
    load_wide(epi.b.l + j0, lo);
    load_wide(epi.b.u + j0, up);
  }
  alignas(16) T out[Epi::kOut][W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    ACC s = ACC(0);
#pragma unroll
    for (int q = 2 * w; q < 2 * w + 2; ++q) s += val[q / W][q % W] * y[idx[q]];
    ACC v[Epi::kIn], o[Epi::kOut];
#pragma unroll
    for (int k = 0; k < Epi::kIn; ++k) v[k] = in[k][w];
    epi.update(Epi::pre(v, epi.b.uniform ? epi.b.lo : lo[w], epi.b.uniform ? epi.b.hi : up[w]), s,
               o);
#pragma unroll
    for (int k = 0; k < Epi::kOut; ++k) out[k][w] = static_cast<T>(o[k]);
  }
#pragma unroll
  for (int k = 0; k < Epi::kOut; ++k) {
    T* p = epi.out(k);
    if (p != nullptr) store_wide(p + j0, out[k]);
  }
}

// The scalars of one step launch. FP64 kernels compute them once per CTA (thread 0) and share
// them: an FP64 division in every thread of thousands of CTAs kept GB300's small FP64 pipe
// busy. FP32 kernels compute the average weight in FP32 per thread.
template <typename ACC>
struct StepScalars {
  ACC sigma, tau, alpha, beta;
};

template <typename ACC>
__device__ __forceinline__ StepScalars<ACC> step_scalars(const Ctl* __restrict__ ctl,
                                                         long long k) {
  if constexpr (std::is_same<ACC, double>::value) {
    __shared__ StepScalars<double> sh;
    if (threadIdx.x == 0) {
      const double alpha = 1.0 / static_cast<double>(k + 1);
      sh.sigma = ctl->sigma;
      sh.tau = ctl->tau;
      sh.alpha = alpha;
      sh.beta = 1.0 - alpha;
    }
    __syncthreads();
    return sh;
  } else {
    // FP32: lane 0 of each warp converts and divides, the warp shuffles the results (the
    // shared-memory broadcast above put a dependent load and a barrier in front of every CTA's
    // first load: slower; per thread, the FP64 -> FP32 and 64-bit integer conversions ran on
    // the FP64 pipe in every thread). Every lane is active at kernel entry.
    StepScalars<ACC> s{};
    if ((threadIdx.x & 31) == 0) {
      s.sigma = static_cast<ACC>(ctl->sigma);
      s.tau = static_cast<ACC>(ctl->tau);
      s.alpha = ACC(1) / static_cast<ACC>(k + 1);
      s.beta = ACC(1) - s.alpha;
    }
    s.sigma = __shfl_sync(0xffffffffu, s.sigma, 0);
    s.tau = __shfl_sync(0xffffffffu, s.tau, 0);
    s.alpha = __shfl_sync(0xffffffffu, s.alpha, 0);
    s.beta = __shfl_sync(0xffffffffu, s.beta, 0);
    return s;
  }
}

// Two variants of each step kernel (TileSet::variant, one per operator, picked by the tile
// tuner or the built-in rule):
//   0: many CTAs per SM resident (operators of short rows, where occupancy hides the latency),
//      as many as fit without spills: the primal step 6 (40 registers) in FP32 and 5 (48) in
//      FP64; the dual step, whose epilogue preloads eight or nine row values, 5 in FP32 and 4
//      (64) in FP64 (a few bytes spill; at 3 per SM, spill-free, the power-law LP's FP64 dual
//      step took 108 us instead of 92);
//   1: 128 registers, the warp-per-row and segment loops unrolled twice as deep (operators of
//      long rows, whose few CTAs need more loads in flight each; at 3 CTAs per SM, 80
//      registers, no faster on the transportation LP);
//   3 (primal steps only): operators of two nonzeros a column (two_nonzero_columns);
//   2 (dual steps only): variant 0 plus the kind-3 row groups and the staged kind-1 segments
//      of a tile set that has them.
// (Measured and not kept: a third variant loading a short row's first three pairs of
// nonzeros together at 4 CTAs per SM; no faster on the transportation or power-law LPs.)
template <typename T>
constexpr int step_min_blocks(int variant, bool dual) {
  if (variant == 1) return 2;
  if (variant == 2) return sizeof(T) == 8 ? 3 : 4;
  if (variant == 3) return 4;
  if (sizeof(T) == 8) return dual ? 4 : 5;
  return dual ? 5 : 6;
}

template <typename T, int VAR>
__global__ void __launch_bounds__(kBlock, step_min_blocks<T>(VAR, true)) dual_step_kernel(
    const Ctl* __restrict__ ctl, OpView<T> K, IterView<T> it, int j) {
  let_next_start();
  const long long t = ctl->t + j;
  const bool idle = ctl->done || t >= ctl->max_iter;
  using ACC = Acc<T>;
  const int p = static_cast<int>(t & 1);
  const long long k = ctl->k + j;
  const StepScalars<ACC> sc = step_scalars<ACC>(ctl, k);
  DualEpi<T, ACC> epi;
  const int n = it.n;
  epi.y = it.y(p);
  epi.y_new = it.y(p ^ 1);
  epi.vr = it.v(p) + n;
  epi.vr_new = it.v(p ^ 1) + n;
  epi.vbar_r = it.Vbar + n;
  epi.c = it.cost + n;
  epi.l = it.lower + n;
  epi.u = it.upper + n;
  epi.q = it.rhs;
  epi.yerg = it.Yerg;
  epi.verg_r = it.Verg + n;
  epi.sigma = sc.sigma;
  epi.tau = sc.tau;
  epi.alpha = sc.alpha;
  epi.beta = sc.beta;
  wait_for_previous();
  if (idle) return;
  Gather1<T, ACC> g{it.Vbar};
  run_tiles<T, ACC, 1, Gather1<T, ACC>, DualEpi<T, ACC>, false, VAR == 1, VAR == 2>(
      K.ts, K.ptr, K.idx, K.val, g, epi);
}

template <typename T, int VAR>
__global__ void __launch_bounds__(kBlock, step_min_blocks<T>(VAR, false)) primal_step_kernel(
    const Ctl* __restrict__ ctl, OpView<T> Kt, IterView<T> it, int j) {
  let_next_start();
  const long long t = ctl->t + j;
  const bool idle = ctl->done || t >= ctl->max_iter;
  using ACC = Acc<T>;
  const int p = static_cast<int>(t & 1);
  const long long k = ctl->k + j;
  const StepScalars<ACC> sc = step_scalars<ACC>(ctl, k);
  PrimalEpi<T, ACC> epi;
  epi.x = it.v(p);
  epi.x_new = it.v(p ^ 1);
  epi.xbar = it.Vbar;
  epi.c = it.cost;
  epi.b = col_bounds<T, ACC>(it);
  epi.xerg = it.Verg;
  epi.tau = sc.tau;
  epi.alpha = sc.alpha;
  epi.beta = sc.beta;
  wait_for_previous();
  if (idle) return;
  if constexpr (VAR == 3) {
    two_nonzero_columns<T>(Kt, it.y(p ^ 1), epi);
  } else {
    Gather1<T, ACC> g{it.y(p ^ 1)};
    run_tiles<T, ACC, 1, Gather1<T, ACC>, PrimalEpi<T, ACC>, false, VAR == 1>(
        Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi);
  }
}

// ------------------------------------------------------------------------------------------
// Reflected Halpern PDHG (the engine's SG_ALGORITHM_HALPERN; no reference counterpart). With
// T the PDHG map z = (v, y) -> (v^, y^) (primal first: v^ = proj(v - tau (c - K'y)),
// y^ = y + sigma (K (2 v^ - v) - q)) and z0 the point of the last restart, one iteration is
//   z+ = lambda (2 T(z) - z) + (1 - lambda) z0,  lambda = (k + 1) / (k + 2)
// (Halpern's iteration on the reflected map 2T - I, nonexpansive, so z -> a fixed point of T).
// The primal launch runs first: x^ and the reflected 2 x^ - x (written to Vbar, the dual
// launch's SpMV input) and x+ from y; then the dual launch: the logicals' r^ from the old y,
// y^, and r+, y+. T(z) lands in Verg / Yerg, the evaluation's second iterate and the answer.

// z+ = N + w (z0 - N) with N = 2 z^ - z the reflected point and w = 1 - lambda = 1 / (k + 2).
template <typename ACC>
__device__ __forceinline__ ACC halpern_mix(ACC reflected, ACC z0, ACC w) {
  return reflected + w * (z0 - reflected);
}

template <>
__device__ __forceinline__ double halpern_mix<double>(double reflected, double z0, double w) {
  return fma(w, z0 - reflected, reflected);
}

// T(z) is read only by the evaluation after a chunk's last step (and by the restart, the
// precision switch and the answer, all after an evaluation), so only that step writes it: the
// chunk's last launch, or the step that reaches max_iter. Saves one vector write per
// iteration (8 MB of the 104 MB an FP32 primal step of the transportation LP moves).
__device__ __forceinline__ bool halpern_writes_hat(const Ctl* ctl, long long t, int j) {
  return j == kCheckFrequency - 1 || t + 1 >= ctl->max_iter;
}

template <typename T, typename ACC>
struct HalpernPrimalEpi {
  const T* x;
  T* x_new;
  T* xbar;   // 2 x^ - x, the dual launch's SpMV input
  T* xhat;   // x^ (T(z)'s primal part), written only when `hat`
  const T* x0;
  const T* c;
  ColBounds<T, ACC> b;
  ACC tau, w;
  bool hat;
  struct Pre {
    ACC x, c, l, u, x0;
  };
  __device__ __forceinline__ Pre load(int j) const {
    Pre p;
    p.x = static_cast<ACC>(x[j]);
    p.c = static_cast<ACC>(c[j]);
    b.load(j, p.l, p.u);
    p.x0 = static_cast<ACC>(x0[j]);
    return p;
  }
  // The column's new values, written to x_new, xbar and (when `hat`) xhat.
  static constexpr int kIn = 3, kOut = 3;
  __device__ __forceinline__ void update(const Pre& p, ACC s, ACC (&o)[kOut]) const {
    const ACC xh = clampv<ACC>(p.x - tau * (p.c + s), p.l, p.u);
    const ACC refl = extrapolate<ACC>(xh, p.x);
    o[0] = halpern_mix<ACC>(refl, p.x0, w);
    o[1] = refl;
    o[2] = xh;
  }
  __device__ __forceinline__ void row(int j, const ACC (&s)[1], const Pre& p) {
    ACC o[kOut];
    update(p, s[0], o);
    if (hat) xhat[j] = static_cast<T>(o[2]);
    xbar[j] = static_cast<T>(o[1]);
    x_new[j] = static_cast<T>(o[0]);
  }
  __device__ __forceinline__ const T* in(int k) const { return k == 0 ? x : k == 1 ? c : x0; }
  __device__ __forceinline__ T* out(int k) const {
    return k == 0 ? x_new : k == 1 ? xbar : hat ? xhat : nullptr;
  }
  __device__ __forceinline__ static Pre pre(const ACC (&v)[kIn], ACC l, ACC u) {
    return Pre{v[0], v[1], l, u, v[2]};
  }
  __device__ __forceinline__ void row(int j, const ACC (&s)[1]) { row(j, s, load(j)); }
  __device__ __forceinline__ void long_row(int, int j, const ACC (&s)[1]) { row(j, s); }
};

template <typename T, typename ACC>
struct HalpernDualEpi {
  const T* y;
  T* y_new;
  T* yhat;
  const T* y0;
  const T* vr;   // r (n offset applied)
  T* vr_new;
  T* vr_hat;
  const T* r0;
  const T* c;
  const T* l;
  const T* u;
  const T* q;
  ACC sigma, tau, w;
  bool hat;  // write T(z) (y^, r^)
  struct Pre {
    ACC y, r, c, l, u, q, y0, r0;
  };
  __device__ __forceinline__ Pre load(int i) const {
    Pre p;
    p.y = static_cast<ACC>(y[i]);
    p.r = static_cast<ACC>(vr[i]);
    p.c = static_cast<ACC>(c[i]);
    p.l = static_cast<ACC>(l[i]);
    p.u = static_cast<ACC>(u[i]);
    p.q = q != nullptr ? static_cast<ACC>(q[i]) : ACC(0);
    p.y0 = static_cast<ACC>(y0[i]);
    p.r0 = static_cast<ACC>(r0[i]);
    return p;
  }
  __device__ __forceinline__ void row(int i, const ACC (&s)[1], const Pre& p) {
    // The logical's primal step uses the old dual (primal first), then the dual step sees the
    // row's reflected logical: K (2 v^ - v) = A (2 x^ - x) - (2 r^ - r).
    const ACC rh = clampv<ACC>(p.r - tau * (p.c - p.y), p.l, p.u);
    const ACC rrefl = extrapolate<ACC>(rh, p.r);
    ACC res = s[0] - rrefl;
    if (q != nullptr) res -= p.q;
    const ACC yh = p.y + sigma * res;
    if (hat) {
      yhat[i] = static_cast<T>(yh);
      vr_hat[i] = static_cast<T>(rh);
    }
    y_new[i] = static_cast<T>(halpern_mix<ACC>(extrapolate<ACC>(yh, p.y), p.y0, w));
    vr_new[i] = static_cast<T>(halpern_mix<ACC>(rrefl, p.r0, w));
  }
  __device__ __forceinline__ void row(int i, const ACC (&s)[1]) { row(i, s, load(i)); }
  __device__ __forceinline__ void long_row(int, int i, const ACC (&s)[1]) { row(i, s); }
};

template <typename T, int VAR>
__global__ void __launch_bounds__(kBlock, step_min_blocks<T>(VAR, false)) halpern_primal_kernel(
    const Ctl* __restrict__ ctl, OpView<T> Kt, IterView<T> it, int j) {
  let_next_start();
  const long long t = ctl->t + j;
  const bool idle = ctl->done || t >= ctl->max_iter;
  using ACC = Acc<T>;
  const int p = static_cast<int>(t & 1);
  // alpha = 1 / (k' + 1) with k' = k + 1: the Halpern weight 1 / (k + 2).
  const StepScalars<ACC> sc = step_scalars<ACC>(ctl, ctl->k + j + 1);
  HalpernPrimalEpi<T, ACC> epi;
  epi.x = it.v(p);
  epi.x_new = it.v(p ^ 1);
  epi.xbar = it.Vbar;
  epi.xhat = it.Verg;
  epi.x0 = it.Vrst;
  epi.c = it.cost;
  epi.b = col_bounds<T, ACC>(it);
  epi.tau = sc.tau;
  epi.w = sc.alpha;
  epi.hat = halpern_writes_hat(ctl, t, j);
  wait_for_previous();
  if (idle) return;
  if constexpr (VAR == 3) {
    two_nonzero_columns<T>(Kt, it.y(p), epi);
  } else {
    Gather1<T, ACC> g{it.y(p)};
    run_tiles<T, ACC, 1, Gather1<T, ACC>, HalpernPrimalEpi<T, ACC>, false, VAR == 1>(
        Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi);
  }
}

template <typename T, int VAR>
__global__ void __launch_bounds__(kBlock, step_min_blocks<T>(VAR, true)) halpern_dual_kernel(
    const Ctl* __restrict__ ctl, OpView<T> K, IterView<T> it, int j) {
  let_next_start();
  const long long t = ctl->t + j;
  const bool idle = ctl->done || t >= ctl->max_iter;
  using ACC = Acc<T>;
  const int p = static_cast<int>(t & 1);
  const StepScalars<ACC> sc = step_scalars<ACC>(ctl, ctl->k + j + 1);
  HalpernDualEpi<T, ACC> epi;
  const int n = it.n;
  epi.y = it.y(p);
  epi.y_new = it.y(p ^ 1);
  epi.yhat = it.Yerg;
  epi.y0 = it.Yrst;
  epi.vr = it.v(p) + n;
  epi.vr_new = it.v(p ^ 1) + n;
  epi.vr_hat = it.Verg + n;
  epi.r0 = it.Vrst + n;
  epi.c = it.cost + n;
  epi.l = it.lower + n;
  epi.u = it.upper + n;
  epi.q = it.rhs;
  epi.sigma = sc.sigma;
  epi.tau = sc.tau;
  epi.w = sc.alpha;
  epi.hat = halpern_writes_hat(ctl, t, j);
  wait_for_previous();
  if (idle) return;
  Gather1<T, ACC> g{it.Vbar};
  run_tiles<T, ACC, 1, Gather1<T, ACC>, HalpernDualEpi<T, ACC>, false, VAR == 1, VAR == 2>(
      K.ts, K.ptr, K.idx, K.val, g, epi);
}

// ------------------------------------------------------------------------------------------
// Evaluation (pdhg_core.cu:102-144 / pdlp.cpp:411-488): the seven sums of the current and the
// average iterate in the space before equilibration, plus the restart distances, from one
// pass over each operator (both iterates share the matrix read). W0 = 1 measures the second
// slot alone (the Halpern solves decide on T(z) only; the current iterate's sums stay 0).

template <typename T, int W0 = 0>
struct EvalRowEpi {
  // rows of K: logicals r and duals y
  const T* vr[2];
  const T* y[2];
  const T* vr_rst;
  const T* y_rst;
  EvalView ev;
  int n;
  double acc[kEvalSums];
  double* long_terms;
  __device__ __forceinline__ void terms(int i, const double (&s)[2 - W0],
                                        double (&a)[kEvalSums]) {
    const double rs = ev.rs[i];
    const double irs = ev.inv_rs[i];
    const double c = ev.cost[n + i];
    const double lo = ev.lower[n + i];
    const double up = ev.upper[n + i];
    const double q = ev.rhs != nullptr ? ev.rhs[i] : 0.0;
#pragma unroll
    for (int w = W0; w < 2; ++w) {
      const double vrv = static_cast<double>(vr[w][i]);
      const double yv = static_cast<double>(y[w][i]);
      const double value = vrv * irs;
      const double yo = yv * rs;
      const double g = c - yo;
      const double e = s[w - W0] * irs - value - q;
      a[w * 7 + 0] += e * e;
      a[w * 7 + 5] += value * value;
      a[w * 7 + 6] += yo * yo;
      a[w * 7 + 2] += c * value;
      const double lam = bound_part(g, lo, up);
      a[w * 7 + 1] += (g - lam) * (g - lam);
      if (lam > 0.0) a[w * 7 + 3] += lam * lo;
      if (lam < 0.0) a[w * 7 + 3] += lam * up;
      // With a right-hand side ([A -I] v = q) the dual objective carries -y'q.
      if (q != 0.0) a[w * 7 + 3] -= yo * q;
      const double dv = vrv - static_cast<double>(vr_rst[i]);
      const double dy = yv - static_cast<double>(y_rst[i]);
      a[14 + 2 * w] += dv * dv;
      a[15 + 2 * w] += dy * dy;
    }
  }
  __device__ __forceinline__ void row(int i, const double (&s)[2 - W0]) { terms(i, s, acc); }
  __device__ __forceinline__ void long_row(int lrow, int i, const double (&s)[2 - W0]) {
    double a[kEvalSums];
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) a[q] = 0.0;
    terms(i, s, a);
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) long_terms[lrow * kMaxSums + q] = a[q];
  }
};

template <typename T, int W0 = 0>
struct EvalColEpi {
  // rows of K': structurals x
  const T* x[2];
  const T* x_rst;
  EvalView ev;
  int m;
  double acc[kEvalSums];
  double* long_terms;
  __device__ __forceinline__ void terms(int j, const double (&s)[2 - W0],
                                        double (&a)[kEvalSums]) {
    const double cs = ev.cs[j];
    const double ics = ev.inv_cs[j];
    const double c = ev.cost[j];
    const double lo = ev.lower[j];
    const double up = ev.upper[j];
#pragma unroll
    for (int w = W0; w < 2; ++w) {
      const double xv = static_cast<double>(x[w][j]);
      const double value = xv * cs;
      const double g = c + (m > 0 ? s[w - W0] * ics : 0.0);
      a[w * 7 + 4] += value * value;
      a[w * 7 + 2] += c * value;
      const double lam = bound_part(g, lo, up);
      a[w * 7 + 1] += (g - lam) * (g - lam);
      if (lam > 0.0) a[w * 7 + 3] += lam * lo;
      if (lam < 0.0) a[w * 7 + 3] += lam * up;
      const double dv = xv - static_cast<double>(x_rst[j]);
      a[14 + 2 * w] += dv * dv;
    }
  }
  __device__ __forceinline__ void row(int j, const double (&s)[2 - W0]) { terms(j, s, acc); }
  __device__ __forceinline__ void long_row(int lrow, int j, const double (&s)[2 - W0]) {
    double a[kEvalSums];
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) a[q] = 0.0;
    terms(j, s, a);
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) long_terms[lrow * kMaxSums + q] = a[q];
  }
};

// Stores the grid totals (the split rows' terms are added by grid_reduce).
struct EvalFin {
  Ctl* c;
  __device__ __forceinline__ void operator()(const double (&tot)[kEvalSums]) const {
    for (int q = 0; q < kEvalSums; ++q) {
      c->eval_r[q] = tot[q];
      c->eval_c[q] = 0.0;
    }
  }
};

__device__ __forceinline__ int eval_parity(const Ctl* ctl, int fixed_parity) {
  if (fixed_parity >= 0) return fixed_parity;
  long long steps = ctl->max_iter - ctl->t;
  if (steps > kCheckFrequency) steps = kCheckFrequency;
  return static_cast<int>((ctl->t + steps) & 1);
}

// One launch over both operators: the first grid_t CTAs take the columns (rows of K'), the rest the
// rows, and one reduction adds them up into eval_r (eval_c 0). (A launch each took 18 and 14 us on
// a 200 x 500 LP, most of it in the two reductions.)
template <typename T, int W0>
__global__ void __launch_bounds__(kBlock) eval_kernel(Ctl* ctl, OpView<T> K, OpView<T> Kt,
                                                      IterView<T> it, EvalView ev, RedView red,
                                                      int grid_t, int fixed_parity) {
  if (fixed_parity < 0 && ctl->done) return;
  const int cur = eval_parity(ctl, fixed_parity);
  double acc[kEvalSums];
  const int b = blockIdx.x;
  if (b < grid_t) {
    EvalColEpi<T, W0> epi;
    epi.x[0] = it.v(cur);
    epi.x[1] = it.Verg;
    epi.x_rst = it.Vrst;
    epi.ev = ev;
    epi.m = it.m;
    epi.long_terms = red.long_terms + static_cast<size_t>(K.ts.nlong) * kMaxSums;
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) epi.acc[q] = 0.0;
    if constexpr (W0 == 0) {
      Gather2<T> g{it.y(cur), it.Yerg};
      run_tiles<T, double, 2>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi, b, grid_t);
    } else {
      Gather1<T, double> g{it.Yerg};
      run_tiles<T, double, 1>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi, b, grid_t);
    }
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) acc[q] = epi.acc[q];
  } else {
    EvalRowEpi<T, W0> epi;
    const int n = it.n;
    epi.vr[0] = it.v(cur) + n;
    epi.vr[1] = it.Verg + n;
    epi.y[0] = it.y(cur);
    epi.y[1] = it.Yerg;
    epi.vr_rst = it.Vrst + n;
    epi.y_rst = it.Yrst;
    epi.ev = ev;
    epi.n = n;
    epi.long_terms = red.long_terms;
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) epi.acc[q] = 0.0;
    if constexpr (W0 == 0) {
      Gather2<T> g{it.v(cur), it.Verg};
      run_tiles<T, double, 2>(K.ts, K.ptr, K.idx, K.val, g, epi, b - grid_t,
                              gridDim.x - grid_t);
    } else {
      Gather1<T, double> g{it.Verg};
      run_tiles<T, double, 1>(K.ts, K.ptr, K.idx, K.val, g, epi, b - grid_t,
                              gridDim.x - grid_t);
    }
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) acc[q] = epi.acc[q];
  }
  grid_reduce<kEvalSums>(acc, red.partial, red.counter, smem_red(), EvalFin{ctl},
                         red.long_terms, K.ts.nlong + Kt.ts.nlong);
}

// The same sums for an FP32 operator, which is always an inner problem already in its own
// equilibrated space (unit scales) with its own FP32 cost, bounds and right-hand side: FP32
// products, row sums and terms (GB300's FP64 rate is a small fraction of its FP32 rate, and FP64
// terms made these kernels arithmetic-bound), FP64 grid totals. Precision ~1e-6 relative is
// ample for the inner tolerance; the refined point is assessed by the FP64 evaluation above.

__device__ __forceinline__ float bound_part32(float g, float lo, float up) {
  const bool hl = lo > -INFINITY;
  const bool hu = up < INFINITY;
  return hl && hu ? g : hl ? fmaxf(g, 0.0f) : hu ? fminf(g, 0.0f) : 0.0f;
}

struct Gather2f {
  const float* x0;
  const float* x1;
  __device__ __forceinline__ float operator()(int v, float a, int j) const {
    return a * ldg((v == 0 ? x0 : x1) + j);
  }
};

template <int W0 = 0>
struct EvalRowEpi32 {
  const float* vr[2];
  const float* y[2];
  const float* vr_rst;
  const float* y_rst;
  const float* c;  // row parts (n offset applied)
  const float* l;
  const float* u;
  const float* q;
  float acc[kEvalSums];
  double* long_terms;
  __device__ __forceinline__ void terms(int i, const float (&s)[2 - W0], float (&a)[kEvalSums]) {
    const float c_i = c[i];
    const float lo = l[i];
    const float up = u[i];
    const float q_i = q != nullptr ? q[i] : 0.0f;
#pragma unroll
    for (int w = W0; w < 2; ++w) {
      const float value = vr[w][i];
      const float yv = y[w][i];
      const float g = c_i - yv;
      const float e = s[w - W0] - value - q_i;
      a[w * 7 + 0] += e * e;
      a[w * 7 + 5] += value * value;
      a[w * 7 + 6] += yv * yv;
      a[w * 7 + 2] += c_i * value;
      const float lam = bound_part32(g, lo, up);
      a[w * 7 + 1] += (g - lam) * (g - lam);
      if (lam > 0.0f) a[w * 7 + 3] += lam * lo;
      if (lam < 0.0f) a[w * 7 + 3] += lam * up;
      a[w * 7 + 3] -= yv * q_i;
      const float dv = value - vr_rst[i];
      const float dy = yv - y_rst[i];
      a[14 + 2 * w] += dv * dv;
      a[15 + 2 * w] += dy * dy;
    }
  }
  __device__ __forceinline__ void row(int i, const float (&s)[2 - W0]) { terms(i, s, acc); }
  __device__ __forceinline__ void long_row(int lrow, int i, const float (&s)[2 - W0]) {
    float a[kEvalSums];
#pragma unroll
    for (int q2 = 0; q2 < kEvalSums; ++q2) a[q2] = 0.0f;
    terms(i, s, a);
#pragma unroll
    for (int q2 = 0; q2 < kEvalSums; ++q2) long_terms[lrow * kMaxSums + q2] = a[q2];
  }
};

template <int W0 = 0>
struct EvalColEpi32 {
  const float* x[2];
  const float* x_rst;
  const float* c;
  const float* l;
  const float* u;
  int m;
  float acc[kEvalSums];
  double* long_terms;
  __device__ __forceinline__ void terms(int j, const float (&s)[2 - W0], float (&a)[kEvalSums]) {
    const float c_j = c[j];
    const float lo = l[j];
    const float up = u[j];
#pragma unroll
    for (int w = W0; w < 2; ++w) {
      const float value = x[w][j];
      const float g = c_j + (m > 0 ? s[w - W0] : 0.0f);
      a[w * 7 + 4] += value * value;
      a[w * 7 + 2] += c_j * value;
      const float lam = bound_part32(g, lo, up);
      a[w * 7 + 1] += (g - lam) * (g - lam);
      if (lam > 0.0f) a[w * 7 + 3] += lam * lo;
      if (lam < 0.0f) a[w * 7 + 3] += lam * up;
      const float dv = value - x_rst[j];
      a[14 + 2 * w] += dv * dv;
    }
  }
  __device__ __forceinline__ void row(int j, const float (&s)[2 - W0]) { terms(j, s, acc); }
  __device__ __forceinline__ void long_row(int lrow, int j, const float (&s)[2 - W0]) {
    float a[kEvalSums];
#pragma unroll
    for (int q2 = 0; q2 < kEvalSums; ++q2) a[q2] = 0.0f;
    terms(j, s, a);
#pragma unroll
    for (int q2 = 0; q2 < kEvalSums; ++q2) long_terms[lrow * kMaxSums + q2] = a[q2];
  }
};

template <int W0>
__global__ void __launch_bounds__(kBlock) eval32_kernel(Ctl* ctl, OpView<float> K,
                                                        OpView<float> Kt, IterView<float> it,
                                                        RedView red, int grid_t,
                                                        int fixed_parity) {
  if (fixed_parity < 0 && ctl->done) return;
  const int cur = eval_parity(ctl, fixed_parity);
  double acc[kEvalSums];
  const int b = blockIdx.x;
  if (b < grid_t) {
    EvalColEpi32<W0> epi;
    epi.x[0] = it.v(cur);
    epi.x[1] = it.Verg;
    epi.x_rst = it.Vrst;
    epi.c = it.cost;
    epi.l = it.lower;
    epi.u = it.upper;
    epi.m = it.m;
    epi.long_terms = red.long_terms + static_cast<size_t>(K.ts.nlong) * kMaxSums;
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) epi.acc[q] = 0.0f;
    if constexpr (W0 == 0) {
      Gather2f g{it.y(cur), it.Yerg};
      run_tiles<float, float, 2>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi, b, grid_t);
    } else {
      Gather1<float, float> g{it.Yerg};
      run_tiles<float, float, 1>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi, b, grid_t);
    }
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) acc[q] = epi.acc[q];
  } else {
    const int n = it.n;
    EvalRowEpi32<W0> epi;
    epi.vr[0] = it.v(cur) + n;
    epi.vr[1] = it.Verg + n;
    epi.y[0] = it.y(cur);
    epi.y[1] = it.Yerg;
    epi.vr_rst = it.Vrst + n;
    epi.y_rst = it.Yrst;
    epi.c = it.cost + n;
    epi.l = it.lower + n;
    epi.u = it.upper + n;
    epi.q = it.rhs;
    epi.long_terms = red.long_terms;
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) epi.acc[q] = 0.0f;
    if constexpr (W0 == 0) {
      Gather2f g{it.v(cur), it.Verg};
      run_tiles<float, float, 2>(K.ts, K.ptr, K.idx, K.val, g, epi, b - grid_t,
                                 gridDim.x - grid_t);
    } else {
      Gather1<float, float> g{it.Verg};
      run_tiles<float, float, 1>(K.ts, K.ptr, K.idx, K.val, g, epi, b - grid_t,
                                 gridDim.x - grid_t);
    }
#pragma unroll
    for (int q = 0; q < kEvalSums; ++q) acc[q] = epi.acc[q];
  }
  grid_reduce<kEvalSums>(acc, red.partial, red.counter, smem_red(), EvalFin{ctl},
                         red.long_terms, K.ts.nlong + Kt.ts.nlong);
}

// ------------------------------------------------------------------------------------------
// Decisions (pdlp.cpp:493-541, 674-713, 1069-1131), one thread.

struct Meas {
  double rp, rd, rg, pobj, dobj;
};

__device__ Meas finish_sums(const Ctl* c, const double* s) {
  // s = (primal_sq, dual_sq, primal_obj, dual_obj, x_sq, r_sq, y_sq)
  Meas r;
  const double primal_res = sqrt(s[0]);
  const double dual_res = sqrt(s[1]);
  const double gap = s[2] - s[3];
  const double primal_scale = 1.0 + c->a_norm_max_col * sqrt(s[4]) + sqrt(s[5]) + c->q_norm;
  const double dual_scale = 1.0 + c->at_norm_max_row * sqrt(s[6]) + c->c_norm;
  const double gap_scale = 1.0 + fabs(s[2]) + fabs(s[3]);
  r.rp = c->m > 0 ? primal_res / primal_scale : 0.0;
  r.rd = c->m > 0 ? dual_res / dual_scale : 0.0;
  r.rg = gap / gap_scale;
  r.pobj = s[2];
  r.dobj = s[3];
  return r;
}

__device__ __forceinline__ double kkt_weighted(double omega, const Meas& e) {
  return sqrt(omega * omega * e.rp * e.rp + e.rd * e.rd / (omega * omega) + e.rg * e.rg);
}

__device__ __forceinline__ bool converged(const Meas& e, double tol) {
  return e.rp < tol && e.rd < tol && fabs(e.rg) < tol;
}

__device__ void set_answer(Ctl* c, int status, const Meas& e, long long iterations, int avg) {
  c->status = status;
  c->res[0] = e.rp;
  c->res[1] = e.rd;
  c->res[2] = e.rg;
  c->pobj = e.pobj;
  c->dobj = e.dobj;
  c->iterations = iterations;
  c->result_average = avg;
  c->done = 1;
}

// Termination test after the evaluation (cur, avg: its measures); schedules the detection checks.
__device__ __forceinline__ void decide_termination(Ctl* c, const Meas& cur, const Meas& avg) {
  long long steps = c->max_iter - c->t;
  if (steps > kCheckFrequency) steps = kCheckFrequency;
  const long long t_new = c->t + steps;
  c->evaluations += 1;
  if (!c->halpern && converged(cur, c->tol)) {
    set_answer(c, kOptimal, cur, t_new, 0);
    c->t = t_new;
    return;
  }
  if (converged(avg, c->tol)) {
    set_answer(c, kOptimal, avg, t_new, 1);
    c->t = t_new;
    return;
  }
  if (c->stall_limit > 0) {
    const double ec = fmax(fmax(cur.rp, cur.rd), fabs(cur.rg));
    const double ea = fmax(fmax(avg.rp, avg.rd), fabs(avg.rg));
    const bool use_avg = c->halpern || ea < ec;
    const double e = use_avg ? ea : ec;
    if (e < 0.8 * c->stall_best) {
      c->stall_best = e;
      c->stall_evals = 0;
    } else if (++c->stall_evals >= (e < c->stall_floor ? c->stall_limit : 8 * c->stall_limit)) {
      set_answer(c, kIterationLimit, use_avg ? avg : cur, t_new, use_avg ? 1 : 0);
      c->t = t_new;
      return;
    }
  }
  c->detect_pending = !c->no_detect && detection_due(t_new) && c->m > 0 ? 1 : 0;
  for (int q = 0; q < 8; ++q) c->det_flags[q] = 0;
}

// Detection verdict, then PDLP's adaptive restart and primal-weight update; advances the
// iteration counters and applies the iteration and time limits.
__device__ __forceinline__ void decide_restart(Ctl* c, const Meas& cur, const Meas& avg,
                                               double kkt_cur, double kkt_avg) {
  long long steps = c->max_iter - c->t;
  if (steps > kCheckFrequency) steps = kCheckFrequency;
  const long long t_new = c->t + steps;
  const long long iter = t_new - 1;
  if (c->detect_pending) {
    if (c->det_flags[0]) {
      set_answer(c, kInfeasible, cur, t_new, 0);
      c->t = t_new;
      return;
    }
    if (c->det_flags[1]) {
      set_answer(c, kUnbounded, cur, t_new, 0);
      c->t = t_new;
      return;
    }
  }
  const long long k_new = c->k + steps;
  const double omega = c->omega;
  const bool to_average = c->halpern || kkt_avg < kkt_cur;
  const double cand = to_average ? kkt_avg : kkt_cur;
  if (!(c->kkt_at_restart < INFINITY)) c->kkt_at_restart = cand;
  const bool restart = cand <= 0.2 * c->kkt_at_restart ||
                       (cand <= 0.8 * c->kkt_at_restart && cand > c->kkt_previous) ||
                       static_cast<double>(k_new) >= c->art_frac * static_cast<double>(iter + 1);
  c->kkt_previous = cand;
  c->last_kkt = cand;
  if (restart) {
    const double dx = sqrt(c->eval_c[to_average ? 16 : 14] + c->eval_r[to_average ? 16 : 14]);
    const double dy = sqrt(c->eval_r[to_average ? 17 : 15]);
    if (dx > 1e-10 && dy > 1e-10) {
      const double w = exp(0.5 * log(dy / dx) + 0.5 * log(omega));
      c->omega = w;
      c->tau = c->eta / w;
      c->sigma = c->eta * w;
    }
    c->restart_pending = 1;
    c->restart_to_avg = to_average ? 1 : 0;
    c->k = 0;
    c->kkt_at_restart = cand;
    c->kkt_previous = INFINITY;
    c->restarts += 1;
  } else {
    c->k = k_new;
  }
  c->t = t_new;
  // Halpern: the answer is T(z) (within the bounds), not the Halpern iterate.
  const int ans = c->halpern ? 1 : 0;
  if (c->t >= c->max_iter) {
    set_answer(c, kIterationLimit, ans ? avg : cur, c->max_iter, ans);
    return;
  }
  if (c->deadline_ns != 0ull && globaltimer_ns() > c->deadline_ns) {
    set_answer(c, kTimeLimit, ans ? avg : cur, c->t, ans);
  }
}

// The decisions by one warp: the termination test (FIRST), the restart (LAST), or both when no
// detection is due between them. Bound by latency: on the control block in device memory, every
// read behind a write to it, the two kernels took 20 us (under a profiler's cold caches); here it
// is copied to shared memory, and two lanes measure the two iterates side by side.
template <bool FIRST, bool LAST>
__global__ void decide_kernel(Ctl* ctl) {
  __shared__ __align__(16) unsigned long long copy[(sizeof(Ctl) + 7) / 8];
  static_assert(sizeof(Ctl) % 8 == 0, "copied by 8 bytes");
  constexpr int kWords = sizeof(Ctl) / 8;
  const int lane = threadIdx.x;
  unsigned long long* from = reinterpret_cast<unsigned long long*>(ctl);
  for (int k = lane; k < kWords; k += 32) copy[k] = from[k];
  __syncwarp();
  Ctl* c = reinterpret_cast<Ctl*>(copy);
  if (FIRST) {
    if (lane == 0) {
      c->restart_pending = 0;
      c->detect_pending = 0;
    }
    __syncwarp();
  }
  const bool done = c->done != 0;
  if (!done && lane < 2) {
    // Lane 0 the current iterate, lane 1 the average.
    Meas e;
    if (FIRST) {
      double s[7];
      for (int q = 0; q < 7; ++q) s[q] = c->eval_c[7 * lane + q] + c->eval_r[7 * lane + q];
      e = finish_sums(c, s);
      const double w[5] = {e.rp, e.rd, e.rg, e.pobj, e.dobj};
      for (int q = 0; q < 5; ++q) c->meas[lane][q] = w[q];
    } else {
      e = Meas{c->meas[lane][0], c->meas[lane][1], c->meas[lane][2], c->meas[lane][3],
               c->meas[lane][4]};
    }
    const double kkt = LAST ? kkt_weighted(c->omega, e) : 0.0;
    const double kkt_avg = __shfl_sync(3u, kkt, 1);
    __syncwarp(3u);
    if (lane == 0) {
      const Meas avg{c->meas[1][0], c->meas[1][1], c->meas[1][2], c->meas[1][3], c->meas[1][4]};
      if (FIRST) decide_termination(c, e, avg);
      if (LAST && !c->done) decide_restart(c, e, avg, kkt, kkt_avg);
    }
  }
  __syncwarp();
  for (int k = lane; k < kWords; k += 32) from[k] = copy[k];
}

// Restart at the candidate (pdhg_core.cu:362-380 + advance()): it becomes the current point
// (both ping-pong buffers), the extrapolated point (no momentum) and the restart point.
template <typename T>
__global__ void restart_kernel(const Ctl* __restrict__ ctl, IterView<T> it) {
  if (!ctl->restart_pending) return;
  const int cur = static_cast<int>(ctl->t & 1);
  const bool avg = ctl->restart_to_avg != 0;
  const int nt = it.n + it.m;
  const T* vc = avg ? it.Verg : it.v(cur);
  const T* yc = avg ? it.Yerg : it.y(cur);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
    const T val = vc[k];
    it.Vrst[k] = val;
    it.V[0][k] = val;
    it.V[1][k] = val;
    it.Vbar[k] = val;
    if (k < it.m) {
      const T yv = yc[k];
      it.Yrst[k] = yv;
      it.Y[0][k] = yv;
      it.Y[1][k] = yv;
    }
  }
}

__global__ void set_deadline_kernel(Ctl* c, unsigned long long budget_ns) {
  if (threadIdx.x == 0 && blockIdx.x == 0) c->deadline_ns = globaltimer_ns() + budget_ns;
}

// The answer in the LpProblem's space (pdlp.cpp:1167-1189): x = v cs, r = v / rs, y = y rs.
template <typename T>
__global__ void extract_kernel(const Ctl* __restrict__ ctl, IterView<T> it, EvalView ev,
                               double* x_out, double* y_out, double* dual_ray) {
  const int cur = static_cast<int>(ctl->t & 1);
  const bool avg = ctl->result_average != 0;
  const T* v = avg ? it.Verg : it.v(cur);
  const T* y = avg ? it.Yerg : it.y(cur);
  const int n = it.n;
  const int nt = n + it.m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
    if (k < n) {
      x_out[k] = static_cast<double>(v[k]) * ev.cs[k];
    } else {
      x_out[k] = static_cast<double>(v[k]) / ev.rs[k - n];
    }
    if (k < it.m) {
      y_out[k] = static_cast<double>(y[k]) * ev.rs[k];
      if (dual_ray != nullptr) dual_ray[k] = static_cast<double>(it.Yerg[k]);
    }
  }
}

// ------------------------------------------------------------------------------------------
// Infeasibility and unboundedness detection (pdlp.cpp:715-1043), on the device: Farkas
// certificate from the average dual, improving ray from the difference of consecutive
// iterates. Gated by Ctl::detect_pending; scalars land in Ctl::det / det_flags.

template <typename T>
__global__ void __launch_bounds__(kBlock) det_farkas_rows_kernel(Ctl* c, IterView<T> it,
                                                                 EvalView ev, RedView red) {
  if (c->done || !c->detect_pending) return;
  __shared__ double scratch[kMaxSums * (kBlock / 32)];
  double a[2] = {0.0, 0.0};  // max |yf|, sum |yf|
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < it.m; i += gridDim.x * blockDim.x) {
    const double yf = fabs(static_cast<double>(it.Yerg[i]) * ev.rs[i]);
    a[0] = fmax(a[0], yf);
    a[1] += yf;
  }
  grid_reduce<2, 1u>(a, red.partial, red.counter, scratch, [c](const double (&t)[2]) {
    c->det[0] = t[0];
    c->det[1] = t[1];
  });
}

// A'yf by columns: aty_j = (K' yerg)_j / cs_j, stored, and sum |aty_j|.
template <typename T>
struct FarkasColEpi {
  double* aty;
  const double* cs;
  double acc[1];
  __device__ __forceinline__ void row(int j, const double (&s)[1]) {
    const double a = s[0] / cs[j];
    aty[j] = a;
    acc[0] += fabs(a);
  }
  __device__ __forceinline__ void long_row(int lrow, int j, const double (&s)[1]) {
    const double a = s[0] / cs[j];
    aty[j] = a;
    long_abs[lrow * kMaxSums] = fabs(a);
  }
  double* long_abs;
};

template <typename T>
__global__ void __launch_bounds__(kBlock) det_farkas_cols_kernel(Ctl* c, OpView<T> Kt,
                                                                 IterView<T> it, EvalView ev,
                                                                 RedView red, double* aty) {
  if (c->done || !c->detect_pending) return;
  FarkasColEpi<T> epi;
  epi.aty = aty;
  epi.cs = ev.cs;
  epi.acc[0] = 0.0;
  epi.long_abs = red.long_terms;
  struct G {
    const T* y;
    __device__ __forceinline__ double operator()(int, T a, int i) const {
      return static_cast<double>(a) * static_cast<double>(ldg(y + i));
    }
  } g{it.Yerg};
  run_tiles<T, double, 1>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, g, epi);
  grid_reduce<1>(epi.acc, red.partial, red.counter, smem_red(), [c](const double (&t)[1]) {
    // w_scale: columns first, then the logicals' |yf| (pdlp.cpp:761-767).
    c->det[1] = t[0] + c->det[1];
  }, red.long_terms, Kt.ts.nlong);
}

template <typename T>
__global__ void __launch_bounds__(kBlock) det_farkas_bounds_kernel(Ctl* c, IterView<T> it,
                                                                   EvalView ev, RedView red,
                                                                   const double* aty) {
  if (c->done || !c->detect_pending) return;
  __shared__ double scratch[kMaxSums * (kBlock / 32)];
  const double y_max = c->det[0];
  const double tol = 1e-9 * c->det[1];
  const int n = it.n;
  const int nt = n + it.m;
  // min_f finite part, max_f finite part, min_f has -inf, max_f has +inf, scale
  double a[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
    const double raw = k < n ? aty[k] : -(static_cast<double>(it.Yerg[k - n]) * ev.rs[k - n]);
    const double lo = ev.lower[k];
    const double up = ev.upper[k];
    const double coef = fabs(raw) <= tol ? 0.0 : raw;
    if (coef > 0) {
      if (lo > -INFINITY) a[0] += coef * lo; else a[2] = 1.0;
      if (up < INFINITY) a[1] += coef * up; else a[3] = 1.0;
    } else if (coef < 0) {
      if (up < INFINITY) a[0] += coef * up; else a[2] = 1.0;
      if (lo > -INFINITY) a[1] += coef * lo; else a[3] = 1.0;
    }
    const double w = k < n ? raw / y_max : -raw / y_max;
    if (fabs(w) > 1e-9) {
      if (lo > -INFINITY) a[4] = fmax(a[4], fabs(w * lo));
      if (up < INFINITY) a[4] = fmax(a[4], fabs(w * up));
    }
  }
  grid_reduce<5, 0x1Cu>(a, red.partial, red.counter, scratch, [c](const double (&t)[5]) {
    const double min_f = t[2] > 0.0 ? -INFINITY : t[0];
    const double max_f = t[3] > 0.0 ? INFINITY : t[1];
    double scale = t[4];
    if (!isfinite(scale)) scale = 0.0;
    const double margin = 1e-8 * (1.0 + scale);
    c->det[2] = min_f;
    c->det[3] = max_f;
    c->det[4] = scale;
    const bool found = c->det[0] > 1e-6 && ((isfinite(min_f) && min_f > margin) ||
                                            (isfinite(max_f) && max_f < -margin));
    c->det_flags[0] = found ? 1 : 0;
  });
}

// Ray candidate d = v_new - v: v_max = max |d|.
template <typename T>
__global__ void __launch_bounds__(kBlock) det_ray_max_kernel(Ctl* c, IterView<T> it, RedView red) {
  if (c->done || !c->detect_pending || c->det_flags[0]) return;
  __shared__ double scratch[kMaxSums * (kBlock / 32)];
  const int cur = static_cast<int>(((c->t + (c->max_iter - c->t < kCheckFrequency
                                                  ? c->max_iter - c->t
                                                  : kCheckFrequency))) & 1);
  const T* vn = it.v(cur);
  const T* vo = it.v(cur ^ 1);
  const int nt = it.n + it.m;
  double a[1] = {0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
    a[0] = fmax(a[0], fabs(static_cast<double>(vn[k]) - static_cast<double>(vo[k])));
  }
  grid_reduce<1, 1u>(a, red.partial, red.counter, scratch,
                     [c](const double (&t)[1]) { c->det[5] = t[0]; });
}

// Columns of the ray: cost_dir (structural part), bound checks and the polished ray x
// (pdlp.cpp:887-964). ray_x (n) in the LpProblem's space.
template <typename T>
__global__ void __launch_bounds__(kBlock) det_ray_cols_kernel(Ctl* c, IterView<T> it, EvalView ev,
                                                              RedView red, double* ray_x) {
  if (c->done || !c->detect_pending || c->det_flags[0]) return;
  __shared__ double scratch[kMaxSums * (kBlock / 32)];
  const int cur = static_cast<int>(((c->t + (c->max_iter - c->t < kCheckFrequency
                                                  ? c->max_iter - c->t
                                                  : kCheckFrequency))) & 1);
  const T* vn = it.v(cur);
  const T* vo = it.v(cur ^ 1);
  const double v_max = c->det[5];
  double a[2] = {0.0, 0.0};  // cost_dir (cols), bound failure
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < it.n; j += gridDim.x * blockDim.x) {
    const double d = (static_cast<double>(vn[j]) - static_cast<double>(vo[j])) / v_max;
    double xj = d * ev.cs[j];
    a[0] += ev.cost[j] * xj;
    const double lo = ev.lower[j];
    const double up = ev.upper[j];
    const bool lb = lo > -INFINITY / 2;
    const bool ub = up < INFINITY / 2;
    const bool fixed = lb && ub && (up - lo <= 1e-10 * (1.0 + fabs(lo)));
    if (lb && ub) {
      if (fabs(xj) > (fixed ? 1e-3 : 1e-4)) a[1] = 1.0;
      xj = 0.0;
    } else if (lb) {
      if (xj < -1e-4) a[1] = 1.0;
      xj = fmax(xj, 0.0);
    } else if (ub) {
      if (xj > 1e-4) a[1] = 1.0;
      xj = fmin(xj, 0.0);
    }
    ray_x[j] = xj;
  }
  grid_reduce<2, 2u>(a, red.partial, red.counter, scratch, [c](const double (&t)[2]) {
    c->det[7] = t[0];
    c->det_flags[4] = t[1] > 0.0 ? 0 : 1;
  });
}

// Rows of the ray: primal feasibility of the raw direction and cost_dir of the logicals
// (NV 0: K d_x), and the row bounds of the polished ray (NV 1: K (ray_x / cs)).
template <typename T>
struct RayRowEpi {
  const T* vn;
  const T* vo;
  double inv_vmax;
  EvalView ev;
  int n;
  double acc[3];  // primal_feas^2, cost_dir (rows), row failure
  double* long_terms;
  __device__ __forceinline__ void terms(int i, const double (&s)[2], double (&a)[3]) {
    const double rs = ev.rs[i];
    const double dr = (static_cast<double>(vn[n + i]) - static_cast<double>(vo[n + i])) * inv_vmax;
    const double res = s[0] / rs - dr / rs;
    a[0] += res * res;
    a[1] += ev.cost[n + i] * (dr / rs);
    const double av = s[1] / rs;
    const double lo = ev.lower[n + i];
    const double up = ev.upper[n + i];
    const bool lb = lo > -INFINITY / 2;
    const bool ub = up < INFINITY / 2;
    const bool fixed = lb && ub && (up - lo <= 1e-10 * (1.0 + fabs(lo)));
    if (lb && ub) {
      if (fabs(av) > (fixed ? 1e-3 : 1e-4)) a[2] = 1.0;
    } else if (lb) {
      if (av < -1e-4) a[2] = 1.0;
    } else if (ub) {
      if (av > 1e-4) a[2] = 1.0;
    }
  }
  __device__ __forceinline__ void row(int i, const double (&s)[2]) { terms(i, s, acc); }
  __device__ __forceinline__ void long_row(int lrow, int i, const double (&s)[2]) {
    double a[3] = {0.0, 0.0, 0.0};
    terms(i, s, a);
    for (int q = 0; q < 3; ++q) long_terms[lrow * kMaxSums + q] = a[q];
  }
};

template <typename T>
__global__ void __launch_bounds__(kBlock) det_ray_rows_kernel(Ctl* c, OpView<T> K, IterView<T> it,
                                                              EvalView ev, RedView red,
                                                              const double* ray_x) {
  if (c->done || !c->detect_pending || c->det_flags[0]) return;
  const int cur = static_cast<int>(((c->t + (c->max_iter - c->t < kCheckFrequency
                                                  ? c->max_iter - c->t
                                                  : kCheckFrequency))) & 1);
  RayRowEpi<T> epi;
  epi.vn = it.v(cur);
  epi.vo = it.v(cur ^ 1);
  epi.inv_vmax = 1.0;
  const double v_max = c->det[5];
  epi.ev = ev;
  epi.n = it.n;
  epi.acc[0] = epi.acc[1] = epi.acc[2] = 0.0;
  epi.long_terms = red.long_terms;
  struct G {
    const T* vn;
    const T* vo;
    const double* ray_x;
    const double* cs;
    double v_max;
    __device__ __forceinline__ double operator()(int v, T a, int j) const {
      if (v == 0) {
        const double d = (static_cast<double>(vn[j]) - static_cast<double>(vo[j])) / v_max;
        return static_cast<double>(a) * d;
      }
      return static_cast<double>(a) * (ray_x[j] / cs[j]);
    }
  } g{epi.vn, epi.vo, ray_x, ev.cs, v_max};
  epi.inv_vmax = 1.0 / v_max;
  run_tiles<T, double, 2>(K.ts, K.ptr, K.idx, K.val, g, epi);
  grid_reduce<3, 4u>(epi.acc, red.partial, red.counter, smem_red(),
                     [c](const double (&t)[3]) {
    const double cd = t[1];
    const double fail = t[2];
    const double primal_feas = sqrt(t[0]);
    const double cost_dir = c->det[7] + cd;
    c->det[6] = primal_feas;
    c->det[7] = cost_dir;
    const bool ok = c->det_flags[4] != 0 && !(fail > 0.0);
    c->det_flags[1] = (c->det[5] > 1e-6 && primal_feas < 1e-6 && cost_dir < -1e-8 && ok) ? 1 : 0;
  }, red.long_terms, K.ts.nlong);
}

// ------------------------------------------------------------------------------------------
// Setup on the device (pdlp.cpp:36-187, 289-299, 377-394, 490-492), FP64.

struct MaxNormEpi {
  double most;
  __device__ __forceinline__ void row(int, const double (&s)[1]) { most = fmax(most, sqrt(s[0])); }
  __device__ __forceinline__ void long_row(int, int, const double (&s)[1]) {
    most = fmax(most, sqrt(s[0]));
  }
};

struct SqProd {
  __device__ __forceinline__ double operator()(int, double a, int) const { return a * a; }
};

// The largest column norm (rows of K', the first grid_t CTAs) and the largest row norm.
__global__ void __launch_bounds__(kBlock) max_norm_kernel(Ctl* c, OpView<double> K,
                                                          OpView<double> Kt, RedView red,
                                                          int grid_t) {
  MaxNormEpi epi{0.0};
  const int b = blockIdx.x;
  const bool cols = b < grid_t;
  if (cols) {
    run_tiles<double, double, 1>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, SqProd{}, epi, b, grid_t);
  } else {
    run_tiles<double, double, 1>(K.ts, K.ptr, K.idx, K.val, SqProd{}, epi, b - grid_t,
                                 gridDim.x - grid_t);
  }
  double most[2] = {cols ? epi.most : 0.0, cols ? 0.0 : epi.most};
  grid_reduce<2, 3u>(most, red.partial, red.counter, smem_red(), [c](const double (&t)[2]) {
    c->a_norm_max_col = t[0];
    c->at_norm_max_row = t[1];
  });
}

__global__ void __launch_bounds__(kBlock) sum_sq_kernel(const double* x, int len, RedView red,
                                                        double* out_sqrt) {
  __shared__ double scratch[kMaxSums * (kBlock / 32)];
  double a[1] = {0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < len; k += gridDim.x * blockDim.x) {
    a[0] += x[k] * x[k];
  }
  grid_reduce<1>(a, red.partial, red.counter, scratch,
                 [out_sqrt](const double (&t)[1]) { *out_sqrt = sqrt(t[0]); });
}

// Ruiz norms of D_r A D_c: product (a * scale[col])^2, row norm = rowscale * sqrt(sum).
struct RuizProd {
  const double* other;
  __device__ __forceinline__ double operator()(int, double a, int j) const {
    const double v = a * other[j];
    return v * v;
  }
};

// A scaling pass: every column (rows of K', the first grid_t CTAs) and every row (rows of K)
// takes its statistic with the old scales and writes its new scale to the other buffer, so a
// pass is one launch and needs no scratch vectors. (As three launches, K' and K statistics and
// an update, 22 passes' worth took 1.7 ms of a 1,000 x 2,000 transportation LP's solve: the
// update's square root and quotient alone 64 us of FP64 pipe a pass.)
struct ScalePair {
  const double* cs;
  const double* rs;
  double* cs_new;
  double* rs_new;
};

// The reference's pass (pdlp.cpp:109-187): scale / norm within [1e-8, 1e8], the norm sqrt(sum)
// times the scale; `changed` when a scale moved by more than a tenth.
struct RuizEpi {
  const double* own;
  double* out;
  double changed[1];
  double* long_terms;
  __device__ __forceinline__ double update(int r, double sum) const {
    const double old = own[r];
    const double nv = sqrt(sum) * old;
    const double s = nv > 0 ? fmax(1e-8, fmin(1e8, old / nv)) : old;
    out[r] = s;
    return fabs(s - old) / fmax(fabs(old), 1.0) > 0.1 ? 1.0 : 0.0;
  }
  __device__ __forceinline__ void row(int r, const double (&s)[1]) {
    changed[0] = fmax(changed[0], update(r, s[0]));
  }
  __device__ __forceinline__ void long_row(int lrow, int r, const double (&s)[1]) {
    long_terms[lrow * kMaxSums] = update(r, s[0]);
  }
};

__global__ void __launch_bounds__(kBlock) ruiz_pass_kernel(Ctl* c, OpView<double> K,
                                                           OpView<double> Kt, ScalePair sc,
                                                           RedView red, int grid_t) {
  if (c->ruiz_done) {
    // No pass since has moved a scale: both buffers take the current ones.
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < Kt.rows + K.rows;
         k += gridDim.x * blockDim.x) {
      if (k < Kt.rows) {
        sc.cs_new[k] = sc.cs[k];
      } else {
        sc.rs_new[k - Kt.rows] = sc.rs[k - Kt.rows];
      }
    }
    return;
  }
  RuizEpi epi{nullptr, nullptr, {0.0}, nullptr};
  const int b = blockIdx.x;
  if (b < grid_t) {
    epi.own = sc.cs;
    epi.out = sc.cs_new;
    epi.long_terms = red.long_terms + static_cast<size_t>(K.ts.nlong) * kMaxSums;
    run_tiles<double, double, 1>(Kt.ts, Kt.ptr, Kt.idx, Kt.val, RuizProd{sc.rs}, epi, b, grid_t);
  } else {
    epi.own = sc.rs;
    epi.out = sc.rs_new;
    epi.long_terms = red.long_terms;
    run_tiles<double, double, 1>(K.ts, K.ptr, K.idx, K.val, RuizProd{sc.cs}, epi, b - grid_t,
                                 gridDim.x - grid_t);
  }
  grid_reduce<1, 1u>(epi.changed, red.partial, red.counter, smem_red(),
                     [c](const double (&t)[1]) { c->ruiz_done = t[0] > 0.0 ? 0 : 1; },
                     red.long_terms, K.ts.nlong + Kt.ts.nlong);
}

// A_eq = D_r A D_c on both operators: K entries (a rs_i) cs_j, K' entries (a cs_j) rs_i, the
// association of apply_equilibration for A and A' (pdlp.cpp:204, 265-266). A warp takes 256
// consecutive nonzeros: two of its lanes find the first's and the last's row in the row starts,
// each nonzero's own row lies between (a search over all rows for every nonzero took 118 us for
// the 4 million of a 1,000 x 2,000 transportation LP).
__device__ __forceinline__ int row_between(const int* ptr, int lo, int hi, int k) {
  while (hi - lo > 1) {  // ptr[lo] <= k < ptr[hi]
    const int mid = (lo + hi) >> 1;
    if (__ldg(ptr + mid) <= k) lo = mid; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void scale_nonzeros(const OpView<double>& A, const double* given,
                                               const double* own, const double* other, int k0,
                                               int k1) {
  const int lane = threadIdx.x & 31;
  const int edge = lane == 0 ? k0 : k1 - 1;
  int found = 0;
  if (lane < 2) found = row_between(A.ptr, 0, A.rows, edge);
  const int r0 = __shfl_sync(0xffffffffu, found, 0);
  const int r1 = __shfl_sync(0xffffffffu, found, 1) + 1;
  for (int k = k0 + lane; k < k1; k += 32) {
    const int r = row_between(A.ptr, r0, r1, k);
    A.val[k] = given[k] * __ldg(own + r) * __ldg(other + A.idx[k]);
  }
}

__global__ void __launch_bounds__(kBlock) apply_scaling_kernel(
    OpView<double> K, OpView<double> Kt, const double* k_given, const double* t_given,
    const double* __restrict__ rs, const double* __restrict__ cs, int nnz) {
  constexpr int kPerWarp = 256;
  const int parts = (nnz + kPerWarp - 1) / kPerWarp;
  const int warps = gridDim.x * (kBlock / 32);
  for (int w = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); w < 2 * parts; w += warps) {
    const bool rows = w < parts;
    const int k0 = (rows ? w : w - parts) * kPerWarp;
    const int k1 = min(k0 + kPerWarp, nnz);
    if (rows) {
      scale_nonzeros(K, k_given, rs, cs, k0, k1);
    } else {
      scale_nonzeros(Kt, t_given, cs, rs, k0, k1);
    }
  }
}

// A column's bound over its scale. 0 and infinity, the usual bounds, stay: a warp of such skips
// the quotient (150 us for 2 million columns with two quotients each, on the FP64 pipe).
__device__ __forceinline__ double bound_over(double b, double scale) {
  const long long mag = __double_as_longlong(b) & 0x7fffffffffffffffLL;
  const bool stays = mag == 0 || mag == 0x7ff0000000000000LL;
  const unsigned here = __activemask();
  if (__any_sync(here, !stays)) {
    __syncwarp(here);  // a branch, not predicated instructions
    if (!stays) b = b / scale;
  }
  return b;
}

// The equilibrated cost and bounds, the evaluation's copies of the given ones, and the scales'
// reciprocals.
__global__ void scale_vectors_kernel(int n, int m, const double* cs, const double* rs,
                                     const double* cost, const double* lower, const double* upper,
                                     double* cost_eq, double* lower_eq, double* upper_eq,
                                     double* cost_ev, double* lower_ev, double* upper_ev,
                                     double* inv_cs, double* inv_rs) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n + m; k += gridDim.x * blockDim.x) {
    const double c0 = cost[k], lo = lower[k], up = upper[k];
    cost_ev[k] = c0;
    lower_ev[k] = lo;
    upper_ev[k] = up;
    if (k < n) {
      const double c = cs[k];
      inv_cs[k] = 1.0 / c;
      cost_eq[k] = c0 * c;
      lower_eq[k] = bound_over(lo, c);
      upper_eq[k] = bound_over(up, c);
    } else {
      const double r = rs[k - n];
      inv_rs[k - n] = 1.0 / r;
      cost_eq[k] = c0 * r;
      lower_eq[k] = lo * r;
      upper_eq[k] = up * r;
    }
  }
}

// Power iteration (pdlp.cpp:36-103) on A_eq: v = A' u, u = A v, sigma = |u| / |v|. In place of
// u / |u| the A' product takes u times a power of two that brings |u| into [1, 2): sigma does
// not see the length, the scaling is exact, and the quotients' launch between two products goes
// (21 of 63, 19 us each for 400,000 rows).
struct StoreSqEpi {
  double* out;
  double scale;  // a power of two
  double acc[1];
  double* long_terms;
  __device__ __forceinline__ void row(int r, const double (&s)[1]) {
    const double v = s[0] * scale;
    out[r] = v;
    acc[0] += v * v;
  }
  __device__ __forceinline__ void long_row(int lrow, int r, const double (&s)[1]) {
    const double v = s[0] * scale;
    out[r] = v;
    long_terms[lrow * kMaxSums] = v * v;
  }
};

__global__ void __launch_bounds__(kBlock) power_spmv_kernel(Ctl* c, OpView<double> A,
                                                            const double* x, double* y,
                                                            RedView red, int which) {
  if (c->power_done) return;
  StoreSqEpi epi;
  epi.out = y;
  epi.scale = which == 0 ? inverse_power(c->power_unorm) : 1.0;
  epi.acc[0] = 0.0;
  epi.long_terms = red.long_terms;
  run_tiles<double, double, 1>(A.ts, A.ptr, A.idx, A.val, Gather1<double, double>{x}, epi);
  grid_reduce<1>(epi.acc, red.partial, red.counter, smem_red(),
                 [c, which](const double (&t)[1]) {
    const double nrm = sqrt(t[0]);
    if (which == 0) {
      c->power_vnorm = nrm;
      if (nrm == 0.0) c->power_done = 1;
    } else {
      c->power_unorm = nrm;
      if (nrm == 0.0) {
        c->power_done = 1;
      } else {
        c->power_sigma = nrm / c->power_vnorm;
      }
    }
  }, red.long_terms, A.ts.nlong);
}

__global__ void power_finish_kernel(Ctl* c) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double L = 1.0;
  if (c->m > 0 && !c->power_done) {
    const double la = c->power_sigma * 1.01;
    L = sqrt(la * la + 1.0);
  } else if (c->m > 0 && c->power_done && c->power_sigma > 0.0) {
    // A zero vector after some iterations: the reference returns 1 (pdlp.cpp:74, 92).
    L = 1.0;
  }
  c->op_norm = L;
  c->eta = 0.99 / L;
  c->omega = 1.0;
  c->tau = c->eta;
  c->sigma = c->eta;
}

__global__ void init_state_kernel(Ctl* c) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  c->t = 0;
  c->k = 0;
  c->kkt_at_restart = INFINITY;
  c->kkt_previous = INFINITY;
  c->status = kRunning;
  c->done = 0;
  c->result_average = 0;
  c->restart_pending = 0;
  c->detect_pending = 0;
  c->iterations = 0;
  c->restarts = 0;
  c->evaluations = 0;
  c->res[0] = c->res[1] = c->res[2] = 0.0;
}

template <typename Src, typename Dst>
__global__ void convert_kernel(const Src* src, Dst* dst, long long count) {
  for (long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<long long>(gridDim.x) * blockDim.x) {
    dst[k] = static_cast<Dst>(src[k]);
  }
}

struct StoreEpi {
  double* out;
  __device__ __forceinline__ void row(int r, const double (&s)[1]) { out[r] = s[0]; }
  __device__ __forceinline__ void long_row(int, int r, const double (&s)[1]) { out[r] = s[0]; }
};

__global__ void __launch_bounds__(kBlock) spmv_kernel(OpView<double> A, const double* x,
                                                      double* y) {
  StoreEpi epi{y};
  run_tiles<double, double, 1>(A.ts, A.ptr, A.idx, A.val, Gather1<double, double>{x}, epi);
}

// ------------------------------------------------------------------------------------------
// Enhanced preconditioning (the engine's own, not the reference's): Ruiz equilibration in the
// infinity norm (10 passes: every row and column divided by the square root of its largest
// scaled magnitude) followed by Pock-Chambolle scaling with alpha = 1 (divide by the square
// root of the scaled absolute row / column sums), both updating rows and columns from the same
// matrix. Statistics by the tile kernel: products |a| * scale[other], max (Ruiz) or sum (PC).

struct AbsProd {
  const double* other;
  __device__ __forceinline__ double operator()(int, double a, int j) const {
    return fabs(a) * other[j];
  }
};

// scale / sqrt(statistic times scale) where that is positive. (Not scale * rsqrt(): its last bit is
// off the same way in every column of a transportation LP, whose duals of 256 iterations then were
// 2.4e-14 off in place of 2e-15.)
struct RescaleEpi {
  const double* own;
  double* out;
  __device__ __forceinline__ void row(int r, const double (&s)[1]) {
    const double old = own[r];
    const double stat = s[0] * old;
    out[r] = stat > 0.0 ? old / sqrt(stat) : old;
  }
  __device__ __forceinline__ void long_row(int, int r, const double (&s)[1]) { row(r, s); }
};

template <bool MAXRED>
__global__ void __launch_bounds__(kBlock) abs_pass_kernel(OpView<double> K, OpView<double> Kt,
                                                          ScalePair sc, int grid_t) {
  const int b = blockIdx.x;
  if (b < grid_t) {
    RescaleEpi epi{sc.cs, sc.cs_new};
    run_tiles<double, double, 1, AbsProd, RescaleEpi, MAXRED>(
        Kt.ts, Kt.ptr, Kt.idx, Kt.val, AbsProd{sc.rs}, epi, b, grid_t);
  } else {
    RescaleEpi epi{sc.rs, sc.rs_new};
    run_tiles<double, double, 1, AbsProd, RescaleEpi, MAXRED>(
        K.ts, K.ptr, K.idx, K.val, AbsProd{sc.cs}, epi, b - grid_t, gridDim.x - grid_t);
  }
}

// Initial primal weight |c| / |b| of the equilibrated problem (b: each row's largest finite
// bound magnitude), 1 when either is ~0.
__global__ void __launch_bounds__(kBlock) primal_weight_init_kernel(Ctl* c, int n, int m,
                                                                    const double* cost_eq,
                                                                    const double* lower_eq,
                                                                    const double* upper_eq,
                                                                    RedView red) {
  __shared__ double scratch[kMaxSums * (kBlock / 32)];
  double a[2] = {0.0, 0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n + m; k += gridDim.x * blockDim.x) {
    if (k < n) {
      a[0] += cost_eq[k] * cost_eq[k];
    } else {
      const double lo = lower_eq[k];
      const double up = upper_eq[k];
      const double b = fmax(isfinite(lo) ? fabs(lo) : 0.0, isfinite(up) ? fabs(up) : 0.0);
      a[1] += b * b;
    }
  }
  grid_reduce<2>(a, red.partial, red.counter, scratch, [c](const double (&t)[2]) {
    const double cn = sqrt(t[0]);
    const double bn = sqrt(t[1]);
    const double w = (cn > 1e-10 && bn > 1e-10) ? cn / bn : 1.0;
    c->omega = w;
    c->tau = c->eta / w;
    c->sigma = c->eta * w;
  });
}

int vec_grid(long long len) {
  long long g = (len + kBlock - 1) / kBlock;
  if (g < 1) g = 1;
  if (g > 4096) g = 4096;
  return static_cast<int>(g);
}

}  // namespace

size_t tile_smem_bytes(const TileSet& ts, int nv, size_t acc_bytes) {
  return tile_smem_size(nv, acc_bytes, ts.cap_nnz, ts.cap_rows);
}

namespace {

// The dual step launches: the kind-3 staging or the staged segments' chunk buffers when the
// tile set has them (both in the variant-2 kernels).
template <typename T>
bool dual_variant2(const TileSet& ts) {
  return ts.groups > 0 || ts.staged;
}
template <typename T>
size_t dual_smem_bytes(const TileSet& ts) {
  if (!dual_variant2<T>(ts)) return tile_smem_bytes(ts, 1, sizeof(T));
  const size_t g = group_smem_size<T, Acc<T>>();
  const size_t c = staged_smem_size<T>();
  return g > c ? g : c;
}

}  // namespace

void configure_kernels() {
  // Opt in to large dynamic shared memory; the launch sizes themselves follow each operator's
  // tile capacity, so occupancy is set by the actual size.
  const int big = 200 * 1024;
  cudaFuncSetAttribute(det_ray_rows_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(det_ray_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(dual_step_kernel<double, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(primal_step_kernel<double, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(dual_step_kernel<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(primal_step_kernel<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(dual_step_kernel<double, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(dual_step_kernel<double, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(primal_step_kernel<double, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(dual_step_kernel<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(dual_step_kernel<float, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(primal_step_kernel<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_dual_kernel<double, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_primal_kernel<double, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_dual_kernel<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_primal_kernel<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_dual_kernel<double, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_dual_kernel<double, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_primal_kernel<double, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_dual_kernel<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_dual_kernel<float, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(halpern_primal_kernel<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(det_farkas_cols_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(det_farkas_cols_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(max_norm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(ruiz_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(power_spmv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(spmv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(abs_pass_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(abs_pass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
}

namespace {

// A step launch; `behind`: the launch before it on the stream is a step of the same chunk.
template <typename T>
void launch_step(void (*kernel)(const Ctl*, OpView<T>, IterView<T>, int), const Ctl* ctl,
                 const OpView<T>& A, const IterView<T>& it, int j, int grid, size_t smem,
                 bool behind, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = behind ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, ctl, A, it, j);
}

}  // namespace

template <typename T>
void launch_dual_step(const Ctl* ctl, const OpView<T>& K, const IterView<T>& it, int j, int grid,
                      cudaStream_t s, bool behind) {
  if (K.ts.ntiles == 0) return;
  launch_step<T>(dual_variant2<T>(K.ts)  ? dual_step_kernel<T, 2>
                 : K.ts.variant == 1     ? dual_step_kernel<T, 1>
                                         : dual_step_kernel<T, 0>,
                 ctl, K, it, j, grid, dual_smem_bytes<T>(K.ts), behind, s);
}

// The launch of a primal step: columns of two nonzeros, or tiles. In FP64 two_nonzero_columns takes
// 80,000 columns and more, when every SM has a CTA of 512: fewer keep more of the FP64 pipes busy in
// tiles (transportation LPs, 320 iterations, ms, by columns against tiles: 100 x 200 3.89 and 3.62,
// 150 x 400 5.53 and 5.22, 200 x 500 6.10 and 6.20, 301 x 703 5.10 and 5.52, 500 x 1,000 7.46 and
// 8.08). In FP32 all (50 x 130 3.70 and 3.81, 60 x 200 3.30 and 3.29, 100 x 200 3.10 and 3.20, 500 x
// 1,000 5.32 and 5.55).
template <typename T>
int primal_variant(const OpView<T>& Kt) {
  const bool wide = Kt.ts.uniform_len == 2 && (sizeof(T) == 4 || Kt.rows >= 80000);
  return wide ? 3 : Kt.ts.variant == 1 ? 1 : 0;
}
template <typename T>
int primal_grid(const OpView<T>& Kt, int grid) {
  constexpr int kColumns = kBlock * kWide<T>;
  return primal_variant(Kt) == 3 ? (Kt.rows + kColumns - 1) / kColumns : grid;
}

template <typename T>
void launch_primal_step(const Ctl* ctl, const OpView<T>& Kt, const IterView<T>& it, int j,
                        int grid, cudaStream_t s, bool behind) {
  if (Kt.ts.ntiles == 0) return;
  const int v = primal_variant(Kt);
  launch_step<T>(v == 3   ? primal_step_kernel<T, 3>
                 : v == 1 ? primal_step_kernel<T, 1>
                          : primal_step_kernel<T, 0>,
                 ctl, Kt, it, j, primal_grid(Kt, grid), tile_smem_bytes(Kt.ts, 1, sizeof(T)),
                 behind, s);
}

template <typename T>
void launch_halpern_primal(const Ctl* ctl, const OpView<T>& Kt, const IterView<T>& it, int j,
                           int grid, cudaStream_t s, bool behind) {
  if (Kt.ts.ntiles == 0) return;
  const int v = primal_variant(Kt);
  launch_step<T>(v == 3   ? halpern_primal_kernel<T, 3>
                 : v == 1 ? halpern_primal_kernel<T, 1>
                          : halpern_primal_kernel<T, 0>,
                 ctl, Kt, it, j, primal_grid(Kt, grid), tile_smem_bytes(Kt.ts, 1, sizeof(T)),
                 behind, s);
}

template <typename T>
void launch_halpern_dual(const Ctl* ctl, const OpView<T>& K, const IterView<T>& it, int j,
                         int grid, cudaStream_t s, bool behind) {
  if (K.ts.ntiles == 0) return;
  launch_step<T>(dual_variant2<T>(K.ts)  ? halpern_dual_kernel<T, 2>
                 : K.ts.variant == 1     ? halpern_dual_kernel<T, 1>
                                         : halpern_dual_kernel<T, 0>,
                 ctl, K, it, j, grid, dual_smem_bytes<T>(K.ts), behind, s);
}

template <typename T>
void launch_eval(Ctl* ctl, const OpView<T>& K, const OpView<T>& Kt, const IterView<T>& it,
                 const EvalView& ev, const RedView& red, int grid_k, int grid_t,
                 int fixed_parity, cudaStream_t s, bool second_only) {
  const size_t sm = tile_smem_bytes(K.ts, 2, 8);
  const int grid = grid_t + grid_k;
  if constexpr (std::is_same<T, float>::value) {
    // FP32 operators carry their own (equilibrated) data: `ev` is not used.
    (void)ev;
    if (second_only) {
      eval32_kernel<1><<<grid, kBlock, sm, s>>>(ctl, K, Kt, it, red, grid_t, fixed_parity);
    } else {
      eval32_kernel<0><<<grid, kBlock, sm, s>>>(ctl, K, Kt, it, red, grid_t, fixed_parity);
    }
  } else {
    if (second_only) {
      eval_kernel<T, 1><<<grid, kBlock, sm, s>>>(ctl, K, Kt, it, ev, red, grid_t, fixed_parity);
    } else {
      eval_kernel<T, 0><<<grid, kBlock, sm, s>>>(ctl, K, Kt, it, ev, red, grid_t, fixed_parity);
    }
  }
}

void launch_decide(Ctl* ctl, cudaStream_t s) { decide_kernel<true, true><<<1, 32, 0, s>>>(ctl); }
void launch_decide_a(Ctl* ctl, cudaStream_t s) { decide_kernel<true, false><<<1, 32, 0, s>>>(ctl); }
void launch_decide_b(Ctl* ctl, cudaStream_t s) { decide_kernel<false, true><<<1, 32, 0, s>>>(ctl); }

template <typename T>
void launch_restart(const Ctl* ctl, const IterView<T>& it, cudaStream_t s) {
  restart_kernel<T><<<vec_grid(it.n + it.m), kBlock, 0, s>>>(ctl, it);
}

template <typename T>
void launch_detect(Ctl* ctl, const OpView<T>& K, const OpView<T>& Kt, const IterView<T>& it,
                   const EvalView& ev, const RedView& red, double* scratch_n, double* scratch_nt,
                   int grid_k, int grid_t, cudaStream_t s) {
  (void)scratch_nt;
  const int gm = vec_grid(it.m) < 1024 ? vec_grid(it.m) : 1024;
  const int gn = vec_grid(it.n) < 1024 ? vec_grid(it.n) : 1024;
  const int gnt = vec_grid(it.n + it.m) < 1024 ? vec_grid(it.n + it.m) : 1024;
  det_farkas_rows_kernel<T><<<gm, kBlock, 0, s>>>(ctl, it, ev, red);
  det_farkas_cols_kernel<T><<<grid_t, kBlock, tile_smem_bytes(Kt.ts, 1, 8), s>>>(ctl, Kt, it, ev,
                                                                                red, scratch_n);
  det_farkas_bounds_kernel<T><<<gnt, kBlock, 0, s>>>(ctl, it, ev, red, scratch_n);
  det_ray_max_kernel<T><<<gnt, kBlock, 0, s>>>(ctl, it, red);
  det_ray_cols_kernel<T><<<gn, kBlock, 0, s>>>(ctl, it, ev, red, scratch_n);
  det_ray_rows_kernel<T><<<grid_k, kBlock, tile_smem_bytes(K.ts, 2, 8), s>>>(ctl, K, it, ev, red,
                                                                             scratch_n);
}

template <typename T>
void launch_extract(const Ctl* ctl, const IterView<T>& it, const EvalView& ev, double* x_out,
                    double* y_out, double* dual_ray, double* primal_ray_src, cudaStream_t s) {
  (void)primal_ray_src;
  extract_kernel<T><<<vec_grid(it.n + it.m), kBlock, 0, s>>>(ctl, it, ev, x_out, y_out, dual_ray);
}

void launch_setup_norms(Ctl* ctl, const OpView<double>& K, const OpView<double>& Kt,
                        const double* cost, const RedView& red, int grid_k, int grid_t,
                        cudaStream_t s) {
  if (K.rows > 0) {
    max_norm_kernel<<<grid_t + grid_k, kBlock, tile_smem_bytes(K.ts, 1, 8), s>>>(ctl, K, Kt, red,
                                                                                 grid_t);
  }
  const int nt = K.rows + Kt.rows;
  sum_sq_kernel<<<vec_grid(nt) < 1024 ? vec_grid(nt) : 1024, kBlock, 0, s>>>(cost, nt, red,
                                                                          &ctl->c_norm);
}

__global__ void reciprocal_kernel(const double* a, double* out, int count) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    out[k] = 1.0 / a[k];
  }
}

// Gather neighbours: rows i and i + 1, each of more than 32 nonzeros, whose k-th nonzeros lie
// 1 to 4 columns apart at 7 of 8 sampled positions k (the rows of a 2-D variable array x[k][j]
// summed over k: the candidates of the kind-3 row groups).
__global__ void row_neighbours_kernel(int m, const int* __restrict__ ptr,
                                      const int* __restrict__ idx, unsigned char* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    unsigned char a = 0;
    if (i + 1 < m) {
      const int b0 = ptr[i];
      const int b1 = ptr[i + 1];
      const int len = min(b1 - b0, ptr[i + 2] - b1);
      if (len > 32) {
        int hits = 0;
        for (int q = 0; q < 8; ++q) {
          const int k = static_cast<int>(static_cast<long long>(q) * len / 8);
          const int d = idx[b1 + k] - idx[b0 + k];
          hits += d != 0 && d >= -4 && d <= 4;
        }
        a = hits >= 7;
      }
    }
    out[i] = a;
  }
}

void launch_row_neighbours(int m, const int* ptr, const int* idx, unsigned char* out,
                           cudaStream_t s) {
  if (m <= 0) return;
  row_neighbours_kernel<<<vec_grid(m) < 1024 ? vec_grid(m) : 1024, kBlock, 0, s>>>(m, ptr, idx,
                                                                                  out);
}

void launch_reciprocals(const double* a, double* out, int count, cudaStream_t s) {
  if (count <= 0) return;
  reciprocal_kernel<<<vec_grid(count) < 1024 ? vec_grid(count) : 1024, kBlock, 0, s>>>(a, out,
                                                                                     count);
}

void launch_ruiz(Ctl* ctl, const OpView<double>& K, const OpView<double>& Kt, double* rs,
                 double* cs, double* rn, double* cn, const RedView& red, int grid_k, int grid_t,
                 cudaStream_t s) {
  const size_t sm = tile_smem_bytes(K.ts, 1, 8);
  for (int pass = 0; pass < 10; ++pass) {
    const ScalePair sc = pass % 2 == 0 ? ScalePair{cs, rs, cn, rn} : ScalePair{cn, rn, cs, rs};
    ruiz_pass_kernel<<<grid_t + grid_k, kBlock, sm, s>>>(ctl, K, Kt, sc, red, grid_t);
  }
}

void launch_enhanced_scaling(const OpView<double>& K, const OpView<double>& Kt, double* rs,
                             double* cs, double* rn, double* cn, int grid_k, int grid_t,
                             cudaStream_t s) {
  const size_t sm = tile_smem_bytes(K.ts, 1, 8);
  for (int pass = 0; pass < 11; ++pass) {
    const ScalePair sc = pass % 2 == 1 ? ScalePair{cs, rs, cn, rn} : ScalePair{cn, rn, cs, rs};
    if (pass < 10) {
      abs_pass_kernel<true><<<grid_t + grid_k, kBlock, sm, s>>>(K, Kt, sc, grid_t);
    } else {
      abs_pass_kernel<false><<<grid_t + grid_k, kBlock, sm, s>>>(K, Kt, sc, grid_t);
    }
  }
}

void launch_primal_weight_init(Ctl* ctl, int n, int m, const double* cost_eq,
                               const double* lower_eq, const double* upper_eq,
                               const RedView& red, cudaStream_t s) {
  const int g = vec_grid(n + m) < 1024 ? vec_grid(n + m) : 1024;
  primal_weight_init_kernel<<<g, kBlock, 0, s>>>(ctl, n, m, cost_eq, lower_eq, upper_eq, red);
}

void launch_apply_scaling(const OpView<double>& K, const OpView<double>& Kt,
                          const double* k_given, const double* t_given, const double* rs,
                          const double* cs, long long nnz, cudaStream_t s) {
  if (nnz == 0) return;
  apply_scaling_kernel<<<vec_grid(nnz / 4), kBlock, 0, s>>>(K, Kt, k_given, t_given, rs, cs,
                                                            static_cast<int>(nnz));
}

void launch_scale_vectors(int n, int m, const double* cs, const double* rs, const double* cost,
                          const double* lower, const double* upper, double* cost_eq,
                          double* lower_eq, double* upper_eq, double* cost_ev,
                          double* lower_ev, double* upper_ev, double* inv_cs, double* inv_rs,
                          cudaStream_t s) {
  scale_vectors_kernel<<<vec_grid(n + m), kBlock, 0, s>>>(
      n, m, cs, rs, cost, lower, upper, cost_eq, lower_eq, upper_eq, cost_ev, lower_ev, upper_ev,
      inv_cs, inv_rs);
}

// The start of a solve's setup: the control block, and both scale buffers at 1.
__global__ void setup_begin_kernel(Ctl* ctl, Ctl value, int n, int m, double* cs, double* cn,
                                   double* rs, double* rn) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *ctl = value;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n + m; k += gridDim.x * blockDim.x) {
    if (k < n) {
      cs[k] = cn[k] = 1.0;
    } else {
      rs[k - n] = rn[k - n] = 1.0;
    }
  }
}

void launch_setup_begin(Ctl* ctl, const Ctl& value, int n, int m, double* cs, double* cn,
                        double* rs, double* rn, cudaStream_t s) {
  setup_begin_kernel<<<vec_grid(n + m), kBlock, 0, s>>>(ctl, value, n, m, cs, cn, rs, rn);
}

void launch_power_finish(Ctl* ctl, cudaStream_t s) { power_finish_kernel<<<1, 32, 0, s>>>(ctl); }

void launch_power_iteration(Ctl* ctl, const OpView<double>& K, const OpView<double>& Kt,
                            double* u, double* v, const RedView& red, int iters, int grid_k,
                            int grid_t, cudaStream_t s) {
  const int m = K.rows;
  if (m > 0) {
    const int gm = vec_grid(m) < 1024 ? vec_grid(m) : 1024;
    sum_sq_kernel<<<gm, kBlock, 0, s>>>(u, m, red, &ctl->power_unorm);
    for (int it = 0; it < iters; ++it) {
      if (Kt.ts.ntiles > 0) {
        power_spmv_kernel<<<grid_t, kBlock, tile_smem_bytes(Kt.ts, 1, 8), s>>>(ctl, Kt, u, v, red, 0);
      }
      if (K.ts.ntiles > 0) {
        power_spmv_kernel<<<grid_k, kBlock, tile_smem_bytes(K.ts, 1, 8), s>>>(ctl, K, v, u, red, 1);
      }
    }
  }
  launch_power_finish(ctl, s);
}

void launch_init_state(Ctl* ctl, cudaStream_t s) { init_state_kernel<<<1, 32, 0, s>>>(ctl); }

__global__ void step_ctl_kernel(Ctl* c, double tau, double sigma, long long t, long long k,
                                long long max_iter) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  c->tau = tau;
  c->sigma = sigma;
  c->t = t;
  c->k = k;
  c->done = 0;
  c->max_iter = max_iter;
}

void launch_step_ctl(Ctl* ctl, double tau, double sigma, long long t, long long k,
                     long long max_iter, cudaStream_t s) {
  step_ctl_kernel<<<1, 32, 0, s>>>(ctl, tau, sigma, t, k, max_iter);
}

void launch_set_deadline(Ctl* ctl, double seconds, cudaStream_t s) {
  const double ns = seconds * 1e9;
  const unsigned long long budget = ns > 1.8e19 ? 18000000000000000000ull
                                                : static_cast<unsigned long long>(ns);
  set_deadline_kernel<<<1, 32, 0, s>>>(ctl, budget);
}

template <typename Src, typename Dst>
void launch_convert(const Src* src, Dst* dst, long long count, cudaStream_t s) {
  if (count <= 0) return;
  convert_kernel<Src, Dst><<<vec_grid(count), kBlock, 0, s>>>(src, dst, count);
}

void launch_spmv(const OpView<double>& A, const double* x, double* y, int grid, cudaStream_t s) {
  if (A.ts.ntiles == 0) return;
  spmv_kernel<<<grid, kBlock, tile_smem_bytes(A.ts, 1, 8), s>>>(A, x, y);
}

// Explicit instantiations.
template void launch_dual_step<double>(const Ctl*, const OpView<double>&, const IterView<double>&,
                                       int, int, cudaStream_t, bool);
template void launch_dual_step<float>(const Ctl*, const OpView<float>&, const IterView<float>&, int,
                                      int, cudaStream_t, bool);
template void launch_primal_step<double>(const Ctl*, const OpView<double>&,
                                         const IterView<double>&, int, int, cudaStream_t, bool);
template void launch_primal_step<float>(const Ctl*, const OpView<float>&, const IterView<float>&,
                                        int, int, cudaStream_t, bool);
template void launch_halpern_primal<double>(const Ctl*, const OpView<double>&,
                                            const IterView<double>&, int, int, cudaStream_t, bool);
template void launch_halpern_primal<float>(const Ctl*, const OpView<float>&,
                                           const IterView<float>&, int, int, cudaStream_t, bool);
template void launch_halpern_dual<double>(const Ctl*, const OpView<double>&,
                                          const IterView<double>&, int, int, cudaStream_t, bool);
template void launch_halpern_dual<float>(const Ctl*, const OpView<float>&,
                                         const IterView<float>&, int, int, cudaStream_t, bool);
template void launch_eval<double>(Ctl*, const OpView<double>&, const OpView<double>&,
                                  const IterView<double>&, const EvalView&, const RedView&, int,
                                  int, int, cudaStream_t, bool);
template void launch_eval<float>(Ctl*, const OpView<float>&, const OpView<float>&,
                                 const IterView<float>&, const EvalView&, const RedView&, int, int,
                                 int, cudaStream_t, bool);
template void launch_restart<double>(const Ctl*, const IterView<double>&, cudaStream_t);
template void launch_restart<float>(const Ctl*, const IterView<float>&, cudaStream_t);
template void launch_detect<double>(Ctl*, const OpView<double>&, const OpView<double>&,
                                    const IterView<double>&, const EvalView&, const RedView&,
                                    double*, double*, int, int, cudaStream_t);
template void launch_detect<float>(Ctl*, const OpView<float>&, const OpView<float>&,
                                   const IterView<float>&, const EvalView&, const RedView&, double*,
                                   double*, int, int, cudaStream_t);
template void launch_extract<double>(const Ctl*, const IterView<double>&, const EvalView&, double*,
                                     double*, double*, double*, cudaStream_t);
template void launch_extract<float>(const Ctl*, const IterView<float>&, const EvalView&, double*,
                                    double*, double*, double*, cudaStream_t);
template void launch_convert<double, float>(const double*, float*, long long, cudaStream_t);
template void launch_convert<float, double>(const float*, double*, long long, cudaStream_t);

}  // namespace sg
