// The up to kCheckFrequency iterations between two evaluations of a small LP, in one launch of
// one thread-block cluster.
//
// Launched step by step, an iteration of a small LP is two kernels of five dependent L2 round
// trips each and two launches, 9-17 us whatever its size; here the iterates and the matrix stay in
// the cluster's shared memory, and a half step ends in an exchange: 3.3 us for a random LP of 200 x
// 500 (FP64, bound by latency: loads, chains of FP64 operations, exchanges), 7.1 for one of 3,500 x
// 7,000 (bound by the FP64 pipes of 16 SMs). With the batched solves' walks, a row on a lane and
// the nonzeros in L1, these took 4.4 and 7.9. Engine::plan_chunk says where this kernel is taken.
#include "sg_chunk.cuh"
#include "sg_cluster_steps.cuh"

namespace sg {

namespace {

// A CTA's share of an operator in tasks, its elements and tasks in shared memory.
template <typename T>
struct alignas(16) TaskShare {
  using Value = T;
  static constexpr bool kTasks = true;
  int own;                            // rows
  int first;                          // position of the first
  unsigned rank, size;
  unsigned val_at, idx_at, task_at;   // shared addresses
  unsigned sums_at;
  int tasks, pad;
  int shared_rows, filled;            // the first rows take several lanes; the last have no nonzeros

  __device__ __forceinline__ int4 task(int t) const {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(task_at + 16 * t)
                 : "memory");
    return v;
  }

  // f(at, init(at) + sum) for every own row. Where a row has a lane to itself, the lane runs f; the
  // sums of rows on several lanes, a shuffle tree's, go to shared memory, and a thread per row runs
  // f after them. (With a lane per row everywhere, as walk_one has it, an LP of 200 x 500 left 12
  // of 16 warps idle, and one warp's 20 nonzeros took 3,500 of an iteration's 7,800 clocks.)
  // MAXRED: the maximum of the products, none negative (FP64: their bits compare as integers).
  template <bool MAXRED = false, typename Prod, typename Init, typename F, typename Ready>
  __device__ __forceinline__ bool walk(const Prod& prod, const Init& init, const F& f,
                                       const Ready& ready) const {
    auto join = [](T p, T q) {
      if constexpr (MAXRED) {
        return __double_as_longlong(p) > __double_as_longlong(q) ? p : q;
      } else {
        return p + q;
      }
    };
    // B steps' elements loaded while the B before are summed (of the same task or the warp's task
    // before).
    constexpr int B = sizeof(T) == 8 ? 4 : 8;
    const int lane = threadIdx.x & 31;
    T a[B];
    unsigned j[B];
    auto fetch = [&](const int4& d, int k) {
      const unsigned val = val_at + (d.x + lane + 32 * k) * static_cast<int>(sizeof(T));
      const unsigned idx = idx_at + (d.x + lane + 32 * k) * 2;
      const int left = d.y - k;
#pragma unroll
      for (int u = 0; u < B; ++u) {
        if (u < left) {
          a[u] = sh_load(val + 32 * u * static_cast<int>(sizeof(T)), T());
          j[u] = sh_load_u16(idx + 64 * u);
        }
      }
    };
    int t = threadIdx.x >> 5;
    int4 d = t < tasks ? task(t) : make_int4(0, 0, 0, 0);
    fetch(d, 0);
    if (!ready()) return false;
    while (t < tasks) {
      t += kChunkThreads / 32;
      const int4 dn = t < tasks ? task(t) : make_int4(0, 0, 0, 0);
      T s = T(0);
      for (int k = 0;; k += B) {
        T ca[B];
        unsigned cj[B];
        const bool more = k + B < d.y;
#pragma unroll
        for (int u = 0; u < B; ++u) {
          ca[u] = a[u];
          cj[u] = j[u];
        }
        fetch(more ? d : dn, more ? k + B : 0);
        const int left = d.y - k;
        if (left >= B) {
          if constexpr (sizeof(T) == 8) keep_branch(0xffffffffu);
#pragma unroll
          for (int u = 0; u < B; ++u) s = join(s, prod(ca[u], static_cast<int>(cj[u])));
        } else {
#pragma unroll
          for (int u = 0; u < B - 1; ++u) {
            if (u < left) {
              if constexpr (sizeof(T) == 8) keep_branch(0xffffffffu);
              s = join(s, prod(ca[u], static_cast<int>(cj[u])));
            }
          }
        }
        if (!more) break;
      }
      const int lanes = d.w >> 8;
      if (lanes == 0) {
        if (lane < (d.w & 255)) {
          const int l = d.z + lane;
          const At at{l, 0, l, first + l};
          f(at, join(init(at), s));
        }
      } else {
        for (int o = (1 << lanes) >> 1; o > 0; o >>= 1) {
          s = join(s, __shfl_xor_sync(0xffffffffu, s, o));
        }
        const int r = lane >> lanes;
        if ((lane & ((1 << lanes) - 1)) == 0 && r < (d.w & 255)) {
          sh_store(sums_at + (d.z + r) * static_cast<int>(sizeof(T)), s);
        }
      }
      d = dn;
    }
    const int rest = shared_rows + own - filled;
    if (rest == 0) return true;
    __syncthreads();
    for (int k = threadIdx.x; k < rest; k += kChunkThreads) {
      const bool sum = k < shared_rows;
      const int l = sum ? k : k - shared_rows + filled;
      const At at{l, 0, l, first + l};
      T s = init(at);
      if (sum) s = join(s, sh_load(sums_at + l * static_cast<int>(sizeof(T)), T()));
      f(at, s);
    }
    return true;
  }
};

// f(at) for every own row.
template <typename T, typename F>
__device__ __forceinline__ void each_own(const TaskShare<T>& A, const F& f) {
  for (int l = threadIdx.x; l < A.own; l += blockDim.x) f(At{l, 0, l, A.first + l});
}

// The state in shared memory, array after array (SolveState's, without slices).
template <typename T>
struct alignas(16) FlatState {
  unsigned cols_at, rows_at;      // shared addresses
  unsigned cols_bytes, rows_bytes;  // of an array
  struct Entry {
    unsigned a, array;
    __device__ __forceinline__ T get(int k) const { return sh_load(a + k * array, T()); }
    __device__ __forceinline__ void set(int k, T v) const { sh_store(a + k * array, v); }
  };
  struct Arrays {
    unsigned base, array;
    __device__ __forceinline__ Entry at(const At& p) const {
      return Entry{base + p.l * static_cast<unsigned>(sizeof(T)), array};
    }
  };
  __device__ __forceinline__ Entry col(const At& at) const {
    return Arrays{cols_at, cols_bytes}.at(at);
  }
  __device__ __forceinline__ Entry row(const At& at) const {
    return Arrays{rows_at, rows_bytes}.at(at);
  }
};
template <typename T>
__device__ __forceinline__ typename FlatState<T>::Arrays col_state(const FlatState<T>& S) {
  return {S.cols_at, S.cols_bytes};
}
template <typename T>
__device__ __forceinline__ typename FlatState<T>::Arrays row_state(const FlatState<T>& S) {
  return {S.rows_at, S.rows_bytes};
}

template <typename T>
__device__ __forceinline__ TaskShare<T> task_share(const ChunkOp<T>& op, int rows, unsigned rank,
                                                   unsigned size, unsigned sums_at) {
  const unsigned base = shared_addr(sg_smem);
  TaskShare<T> s;
  s.own = rows > static_cast<int>(rank)
              ? (rows - static_cast<int>(rank) - 1) / static_cast<int>(size) + 1
              : 0;
  s.first = static_cast<int>(rank) * op.per;
  s.rank = rank;
  s.size = size;
  s.val_at = base + op.val_at;
  s.idx_at = base + op.idx_at;
  s.task_at = base + op.task_at;
  s.sums_at = base + sums_at;
  s.tasks = op.task_off[rank + 1] - op.task_off[rank];
  s.filled = op.filled[2 * rank];
  s.shared_rows = op.filled[2 * rank + 1];
  return s;
}

// The CTA's block of an operator to shared memory.
template <typename T>
__device__ __forceinline__ void load_block(const ChunkOp<T>& op, unsigned rank) {
  T* val = reinterpret_cast<T*>(sg_smem + op.val_at);
  unsigned short* idx = reinterpret_cast<unsigned short*>(sg_smem + op.idx_at);
  int4* task = reinterpret_cast<int4*>(sg_smem + op.task_at);
  const int e0 = op.elem_off[rank];
  const int elems = op.elem_off[rank + 1] - e0;
  for (int k = threadIdx.x; k < elems; k += kChunkThreads) {
    val[k] = op.val[e0 + k];
    idx[k] = op.idx[e0 + k];
  }
  const int t0 = op.task_off[rank];
  const int tasks = op.task_off[rank + 1] - t0;
  for (int k = threadIdx.x; k < tasks; k += kChunkThreads) task[k] = op.task[t0 + k];
}

// Masks of the own columns (which 0) or rows (1): the CTAs that own the other operator's rows of
// their nonzeros (`per` positions each).
template <typename T>
__device__ __forceinline__ void task_masks(const TaskShare<T>& A, int per, unsigned short* mask,
                                           ClusterShared& sh, int which) {
  const int lane = threadIdx.x & 31;
  for (int t = threadIdx.x >> 5; t < A.tasks; t += kChunkThreads / 32) {
    const int4 d = A.task(t);
    const int lanes = d.w >> 8;
    unsigned m = 0;
    for (int k = 0; k < d.y; ++k) {
      const int j = static_cast<int>(sh_load_u16(A.idx_at + (d.x + lane + 32 * k) * 2));
      const unsigned owner = static_cast<unsigned>(j / per);  // size: padding
      if (owner < A.size) m |= 1u << (owner ^ A.rank);
    }
    for (int o = (1 << lanes) >> 1; o > 0; o >>= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
    const int r = lane >> lanes;
    if ((lane & ((1 << lanes) - 1)) == 0 && r < (d.w & 255)) {
      m &= ~1u;
      mask[d.z + r] = static_cast<unsigned short>(m);
      while (m != 0u) {
        const unsigned q = __ffs(m) - 1;
        m &= m - 1u;
        atomicAdd(&sh.count[which][q], 1u);
      }
    }
  }
}

// The LP's share of this CTA in shared memory, its masks and counts; ends with a cluster barrier.
template <typename T>
__device__ __forceinline__ void begin_cluster(const ChunkView<T>& c, ClusterShared& sh,
                                              unsigned rank, unsigned size,
                                              MatShare<T, TaskShare<T>>* m,
                                              Exchange<T, kAllShared>* e) {
  load_block(c.K, rank);
  load_block(c.Kt, rank);
  MatShare<T, TaskShare<T>>& M = *m;
  M.m = c.m;
  M.n = c.n;
  M.kz = M.tz = 0;
  M.kperm = c.K.perm;
  M.tperm = c.Kt.perm;
  M.K = task_share(c.K, c.m, rank, size, c.sums_at);
  M.Kt = task_share(c.Kt, c.n, rank, size, c.sums_at);
  M.nr = M.K.own;
  M.nc = M.Kt.own;
  Exchange<T, kAllShared>& ex = *e;
  ex.sh = &sh;
  ex.rank = rank;
  ex.size = size;
  ex.device = nullptr;
  ex.xs_at = 0u;
  ex.ys_at = (c.np + 1) * static_cast<unsigned>(sizeof(T));
  ex.cmask_at = ex.ys_at + (c.mp + 1) * static_cast<unsigned>(sizeof(T));
  ex.rmask_at = ex.cmask_at + M.nc * 2;
  if (threadIdx.x == 0) ex.xs()[c.np] = ex.ys()[c.mp] = T(0);
  for (int k = threadIdx.x; k < M.nc + M.nr; k += kChunkThreads) ex.cmask()[k] = 0;
  if (threadIdx.x < 2 * kMaxCluster) (&sh.count[0][0])[threadIdx.x] = 0;
  __syncthreads();
  task_masks(M.Kt, c.K.per, ex.cmask(), sh, 0);
  task_masks(M.K, c.Kt.per, ex.rmask(), sh, 1);
  settle_counts(ex);
}

template <typename T>
__device__ __forceinline__ FlatState<T> flat_state(const ChunkView<T>& c,
                                                   const MatShare<T, TaskShare<T>>& M) {
  const unsigned base = shared_addr(sg_smem);
  return FlatState<T>{base + c.cols_at, base + c.rows_at,
                      M.nc * static_cast<unsigned>(sizeof(T)),
                      M.nr * static_cast<unsigned>(sizeof(T))};
}

// The scaling passes of the setup (sg_kernels.cu: ruiz_pass_kernel, abs_pass_kernel) from the given
// values: the scales are the gathered vectors, xs the columns', ys the rows'. Both statistics are
// taken with the old scales; a cluster barrier, then every new scale is sent. Bound by latency;
// 10 or 11 launches took 0.1 ms of a small LP's solve, one takes 0.03.
template <bool RUIZ>
__global__ void __launch_bounds__(kChunkThreads, 1)
    chunk_scale_kernel(ChunkView<double> c, double* cs, double* rs) {
  __shared__ ClusterShared sh;
  const unsigned rank = cluster_rank();
  const unsigned size = cluster_size();
  cluster_init(sh, size);
  MatShare<double, TaskShare<double>> M;
  Exchange<double, kAllShared> ex;
  begin_cluster(c, sh, rank, size, &M, &ex);
  const FlatState<double> S = flat_state(c, M);
  const Sender<double, kAllShared, 0, true> x_out(ex);
  const Sender<double, kAllShared, 1, true> y_out(ex);
  const Array<double, true> x(ex.xs()), y(ex.ys());
  const Zero<double> zero;
  for (int p = threadIdx.x; p < c.np; p += kChunkThreads) x.set(p, 1.0);
  for (int p = threadIdx.x; p < c.mp; p += kChunkThreads) y.set(p, 1.0);
  cluster_sync(size);
  auto cols = [&](const At& at, double s) { S.col(at).set(0, s); };
  auto rows = [&](const At& at, double s) { S.row(at).set(0, s); };
  bool ok = true;
  constexpr int kPasses = RUIZ ? 10 : 11;
  for (int pass = 0; pass < kPasses; ++pass) {
    double moved[1] = {0.0};
    if constexpr (RUIZ) {
      auto by_y = [&](double a, int j) { return (a * y.get(j)) * (a * y.get(j)); };
      auto by_x = [&](double a, int j) { return (a * x.get(j)) * (a * x.get(j)); };
      M.Kt.walk(by_y, zero, cols, Ready());
      __syncthreads();
      M.K.walk(by_x, zero, rows, Ready());
    } else {
      auto by_y = [&](double a, int j) { return fabs(a) * y.get(j); };
      auto by_x = [&](double a, int j) { return fabs(a) * x.get(j); };
      if (pass < 10) {
        M.Kt.walk<true>(by_y, zero, cols, Ready());
        __syncthreads();
        M.K.walk<true>(by_x, zero, rows, Ready());
      } else {
        M.Kt.walk(by_y, zero, cols, Ready());
        __syncthreads();
        M.K.walk(by_x, zero, rows, Ready());
      }
    }
    cluster_sync(size);
    auto next = [&](double old, double stat) {
      if constexpr (RUIZ) {
        const double nv = sqrt(stat) * old;
        const double s = nv > 0 ? fmax(1e-8, fmin(1e8, old / nv)) : old;
        if (fabs(s - old) / fmax(fabs(old), 1.0) > 0.1) moved[0] = 1.0;
        return s;
      } else {
        const double by = stat * old;
        return by > 0.0 ? old / sqrt(by) : old;
      }
    };
    each_own(M.Kt, [&](const At& at) { x_out.put(at, next(x.get(at.p), S.col(at).get(0))); });
    each_own(M.K, [&](const At& at) { y_out.put(at, next(y.get(at.p), S.row(at).get(0))); });
    ok = ok && ex.wait(0) && ex.wait(1);
    if constexpr (RUIZ) {
      double all[2] = {moved[0], ok ? 0.0 : 1.0};
      cluster_reduce<2, 3u>(all, sh, rank, size);
      ok = all[1] == 0.0;
      if (all[0] == 0.0 || !ok) break;
    }
  }
  each_own(M.Kt, [&](const At& at) { cs[M.tperm[at.p]] = x.get(at.p); });
  each_own(M.K, [&](const At& at) { rs[M.kperm[at.p]] = y.get(at.p); });
  if (threadIdx.x == 0 && !ok) atomicExch(c.wait_error, 1);
  cluster_sync(size);
}

// The power iteration of the setup (pdlp.cpp:36-103; power_spmv_kernel's products): 20 times
// v = A' u, u = A v, and |u| / |v| of the last. The lengths are taken in the first iteration, whose
// u is brought into [1, 2) and whose growth the later ones undo by a power of two (exact), and in
// the last. 40 launches took 0.3 ms of a 200 x 500 LP's solve, one takes 0.08.
__global__ void __launch_bounds__(kChunkThreads, 1)
    chunk_power_kernel(Ctl* ctl, ChunkView<double> c, const double* u0, int iterations) {
  __shared__ ClusterShared sh;
  const unsigned rank = cluster_rank();
  const unsigned size = cluster_size();
  cluster_init(sh, size);
  MatShare<double, TaskShare<double>> M;
  Exchange<double, kAllShared> ex;
  begin_cluster(c, sh, rank, size, &M, &ex);
  const FlatState<double> S = flat_state(c, M);
  const Sender<double, kAllShared, 0, true> x_out(ex);
  const Sender<double, kAllShared, 1, true> y_out(ex);
  const Gather<double, kAllShared> from_x{ex.xs()}, from_y{ex.ys()};
  const Zero<double> zero;
  each_own(M.K, [&](const At& at) { y_out.put(at, u0[M.kperm[at.p]]); });
  double sigma = 0.0, growth = 1.0;
  bool ok = true, vanished = false;
  // (A CTA whose wait gave up stays to the reduction of the last iteration, where all know.)
  for (int k = 0; k < iterations && !vanished; ++k) {
    const bool lengths = k == 0 || k == iterations - 1;
    double v2[1] = {0.0}, u2[1] = {0.0};
    ok = ok && M.Kt.walk(from_y, zero,
                         [&](const At& at, double s) {
                           x_out.put(at, s);
                           if (lengths) v2[0] += s * s;
                         },
                         [&] { return ex.wait(1); });
    ok = ok && M.K.walk(from_x, zero,
                        [&](const At& at, double s) {
                          if (lengths) {
                            u2[0] += s * s;
                            S.row(at).set(0, s);
                          } else {
                            y_out.put(at, s * growth);
                          }
                        },
                        [&] { return ex.wait(0); });
    if (lengths) {
      double all[3] = {v2[0], u2[0], ok ? 0.0 : 1.0};
      cluster_reduce<3>(all, sh, rank, size);
      ok = all[2] == 0.0;
      if (!ok) break;
      const double vn = sqrt(all[0]), un = sqrt(all[1]);
      vanished = vn == 0.0 || un == 0.0;
      if (!vanished) {
        sigma = un / vn;
        growth = inverse_power(sigma * sigma);
        const double start = inverse_power(un);
        if (k < iterations - 1) {
          each_own(M.K, [&](const At& at) { y_out.put(at, S.row(at).get(0) * start); });
        }
      }
    }
  }
  if (threadIdx.x == 0) {
    if (!ok) atomicExch(c.wait_error, 1);
    if (rank == 0) {
      ctl->power_sigma = sigma;
      ctl->power_done = vanished ? 1 : 0;
    }
  }
  cluster_sync(size);
}

template <typename T, bool HALPERN>
__global__ void __launch_bounds__(kChunkThreads, 1)
    chunk_kernel(Ctl* ctl, ChunkView<T> c, IterView<T> it) {
  constexpr int MODE = kAllShared;
  constexpr bool kF64 = sizeof(T) == 8;
  __shared__ ClusterShared sh;
  __shared__ StepContext<T, MODE, TaskShare<T>, FlatState<T>> ctx;
  if (ctl->done) return;
  const long long t = ctl->t;
  const long long k0 = ctl->k;
  const long long left = ctl->max_iter - t;
  const int steps = static_cast<int>(left < kCheckFrequency ? left : kCheckFrequency);
  if (steps <= 0) return;
  const unsigned rank = cluster_rank();
  const unsigned size = cluster_size();
  cluster_init(sh, size);
  const int n = c.n;
  MatShare<T, TaskShare<T>> M;
  Exchange<T, MODE> ex;
  begin_cluster(c, sh, rank, size, &M, &ex);
  const Second<T> Z{c.second, c.np, c.mp};
  const FlatState<T> S = flat_state(c, M);
  if (threadIdx.x == 0) {
    ctx.M = M;
    ctx.ex = ex;
    ctx.S = S;
    ctx.Z = Z;
  }
  // The steps' weights as the step kernels take them (sg_kernels.cu).
  if (threadIdx.x < steps) {
    const long long k = k0 + threadIdx.x + (HALPERN ? 2 : 1);
    const T w = T(1) / static_cast<T>(k);
    ctx.weight[threadIdx.x] = w;
    ctx.rest[threadIdx.x] = T(1) - w;
  }
  // The state; FP64 averages as sums.
  const int cur = static_cast<int>(t & 1);
  const T* v = it.v(cur);
  const T* y = it.y(cur);
  const T count = static_cast<T>(k0);
  auto sum_of = [&](T average) { return !kF64 ? average : k0 == 0 ? T(0) : average * count; };
  each_own(M.Kt, [&](const At& at) {
    const int j = M.tperm[at.p];
    S.col(at).set(kPoint, v[j]);
    S.col(at).set(kSum, HALPERN ? it.Vrst[j] : sum_of(it.Verg[j]));
    S.col(at).set(kCost, it.cost[j]);
    S.col(at).set(kLower, it.xb_uniform ? it.xb_lo : it.lower[j]);
    S.col(at).set(kUpper, it.xb_uniform ? it.xb_hi : it.upper[j]);
    if (!HALPERN) ex.put_x(at, it.Vbar[j]);
  });
  each_own(M.K, [&](const At& at) {
    const int i = M.kperm[at.p];
    const int q = n + i;
    S.row(at).set(kPoint, v[q]);
    S.row(at).set(kCost, it.cost[q]);
    S.row(at).set(kLower, it.lower[q]);
    S.row(at).set(kUpper, it.upper[q]);
    S.row(at).set(kDual, y[i]);
    if (HALPERN) {
      S.row(at).set(kSum, it.Vrst[q]);
      S.row(at).set(kDualSum, it.Yrst[i]);
      ex.put_y(at, y[i]);
    } else {
      S.row(at).set(kSum, sum_of(it.Verg[q]));
      S.row(at).set(kDualSum, sum_of(it.Yerg[i]));
      S.row(at).set(kBar, -it.Vbar[q]);
    }
  });
  __syncthreads();
  bool ok = run_steps<HALPERN, T, MODE, TaskShare<T>, FlatState<T>>(
      &ctx, steps, static_cast<T>(ctl->tau), static_cast<T>(ctl->sigma), [&] {
        // The other buffers hold the iterate before the last.
        const int other = static_cast<int>((t + steps + 1) & 1);
        __syncthreads();
        each_own(ctx.M.Kt, [&](const At& at) {
          it.v(other)[ctx.M.tperm[at.p]] = ctx.S.col(at).get(kPoint);
        });
        each_own(ctx.M.K, [&](const At& at) {
          const int i = ctx.M.kperm[at.p];
          it.v(other)[ctx.M.n + i] = ctx.S.row(at).get(kPoint);
          it.y(other)[i] = ctx.S.row(at).get(kDual);
        });
      });
  ok = ok && ex.wait(HALPERN ? 1 : 0);
  if (ok) {
    const int now = static_cast<int>((t + steps) & 1);
    const T inv = T(1) / static_cast<T>(k0 + steps);
    auto average_of = [&](T sum) { return kF64 ? sum * inv : sum; };
    each_own(M.Kt, [&](const At& at) {
      const int j = M.tperm[at.p];
      it.v(now)[j] = S.col(at).get(kPoint);
      it.Vbar[j] = ex.xs()[at.p];
      it.Verg[j] = HALPERN ? Z.x(at.p) : average_of(S.col(at).get(kSum));
    });
    each_own(M.K, [&](const At& at) {
      const int i = M.kperm[at.p];
      const int q = n + i;
      it.v(now)[q] = S.row(at).get(kPoint);
      it.y(now)[i] = S.row(at).get(kDual);
      if (HALPERN) {
        it.Verg[q] = Z.r(at.p);
        it.Yerg[i] = Z.y(at.p);
      } else {
        const T lo = S.row(at).get(kLower);
        it.Vbar[q] = -S.row(at).get(kBar);
        it.Yerg[i] = average_of(S.row(at).get(kDualSum));
        // An FP64 step leaves the sums of equality rows, whose logicals are their bound from
        // the first step on, to this.
        it.Verg[q] = kF64 && lo == S.row(at).get(kUpper)
                         ? average_of(sum_of(it.Verg[q]) + static_cast<T>(steps) * lo)
                         : average_of(S.row(at).get(kSum));
      }
    });
  } else if (threadIdx.x == 0) {
    atomicExch(c.wait_error, 1);
    ctl->status = kNumericalError;
    ctl->done = 1;
  }
  cluster_sync(size);  // no CTA leaves while another may still send to it
}

// A warp per row of A and of A': its nonzeros' new column numbers or values.
template <typename T, bool INDICES>
__global__ void chunk_fill_kernel(ChunkView<T> c, OpView<T> K, OpView<T> Kt) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < c.m + c.n; w += warps) {
    const bool rows = w < c.m;
    const int r = rows ? w : w - c.m;
    const OpView<T>& A = rows ? K : Kt;
    const ChunkOp<T>& C = rows ? c.K : c.Kt;
    const int* other = rows ? c.Kt.pos : c.K.pos;
    const int b = A.ptr[r];
    const int len = A.ptr[r + 1] - b;
    const int2 place = C.row[C.pos[r]];
    for (int k = lane; k < len; k += 32) {
      const int at = place.x + ((k >> place.y) << 5) + (k & ((1 << place.y) - 1));
      if constexpr (INDICES) {
        C.idx[at] = static_cast<unsigned short>(other[A.idx[b + k]]);
      } else {
        C.val[at] = A.val[b + k];
      }
    }
  }
}

int fill_grid(int rows) {
  const int blocks = (rows + 7) / 8;
  return blocks < 1 ? 1 : blocks < 1216 ? blocks : 1216;
}

}  // namespace

template <typename T>
bool place_chunk(ChunkView<T>* v, const TaskLayout& k, const TaskLayout& t) {
  const size_t nc = t.per;
  const size_t nr = k.per;
  v->np = t.positions();
  v->mp = k.positions();
  v->K.per = k.per;
  v->Kt.per = t.per;
  if (v->np > 65535 || v->mp > 65535) return false;  // 16-bit column numbers
  // The gathered vectors and the masks come first (chunk_kernel).
  size_t at = (static_cast<size_t>(v->np) + v->mp + 2) * sizeof(T) + 2 * (nc + nr);
  auto take = [&](size_t bytes) {
    at = (at + 15) & ~static_cast<size_t>(15);
    const unsigned here = static_cast<unsigned>(at);
    at += bytes;
    return here;
  };
  v->cols_at = take(kColArrays * nc * sizeof(T));
  v->rows_at = take(kRowArrays * nr * sizeof(T));
  v->sums_at = take((nc > nr ? nc : nr) * sizeof(T));
  v->K.val_at = take(k.most_elems * sizeof(T));
  v->Kt.val_at = take(t.most_elems * sizeof(T));
  v->K.idx_at = take(k.most_elems * sizeof(unsigned short));
  v->Kt.idx_at = take(t.most_elems * sizeof(unsigned short));
  v->K.task_at = take(k.most_tasks * sizeof(Task));
  v->Kt.task_at = take(t.most_tasks * sizeof(Task));
  v->smem = at;
  return at <= kClusterSmemMax;
}

// (The scaling and power kernels take the same launch and less static shared memory.)
template <typename T>
bool chunk_fits(const ChunkView<T>& c, bool halpern) {
  return halpern ? clusters_fit(chunk_kernel<T, true>, c.size, kChunkThreads, c.smem)
                 : clusters_fit(chunk_kernel<T, false>, c.size, kChunkThreads, c.smem);
}

template <typename T>
void launch_chunk_indices(const ChunkView<T>& c, const OpView<T>& K, const OpView<T>& Kt,
                          cudaStream_t s) {
  chunk_fill_kernel<T, true><<<fill_grid(c.m + c.n), 256, 0, s>>>(c, K, Kt);
}

template <typename T>
void launch_chunk_values(const ChunkView<T>& c, const OpView<T>& K, const OpView<T>& Kt,
                         cudaStream_t s) {
  chunk_fill_kernel<T, false><<<fill_grid(c.m + c.n), 256, 0, s>>>(c, K, Kt);
}

template <typename T>
cudaError_t launch_chunk(Ctl* ctl, const ChunkView<T>& c, const IterView<T>& it, bool halpern,
                         cudaStream_t s) {
  auto go = [&](auto kernel) {
    return launch_clusters(kernel, c.size, 1, kChunkThreads, c.smem, s, ctl, c, it);
  };
  return halpern ? go(chunk_kernel<T, true>) : go(chunk_kernel<T, false>);
}

cudaError_t launch_chunk_power(Ctl* ctl, const ChunkView<double>& c, const double* u0,
                               int iterations, cudaStream_t s) {
  return launch_clusters(chunk_power_kernel, c.size, 1, kChunkThreads, c.smem, s, ctl, c, u0,
                         iterations);
}

cudaError_t launch_chunk_scale(const ChunkView<double>& c, const double* k_given,
                               const double* t_given, bool ruiz, double* cs, double* rs,
                               cudaStream_t s) {
  ChunkView<double> g = c;
  g.K.val = const_cast<double*>(k_given);
  g.Kt.val = const_cast<double*>(t_given);
  return launch_clusters(ruiz ? chunk_scale_kernel<true> : chunk_scale_kernel<false>, c.size, 1,
                         kChunkThreads, c.smem, s, g, cs, rs);
}

template bool place_chunk<double>(ChunkView<double>*, const TaskLayout&, const TaskLayout&);
template bool place_chunk<float>(ChunkView<float>*, const TaskLayout&, const TaskLayout&);
template bool chunk_fits<double>(const ChunkView<double>&, bool);
template bool chunk_fits<float>(const ChunkView<float>&, bool);
template void launch_chunk_indices<double>(const ChunkView<double>&, const OpView<double>&,
                                           const OpView<double>&, cudaStream_t);
template void launch_chunk_indices<float>(const ChunkView<float>&, const OpView<float>&,
                                          const OpView<float>&, cudaStream_t);
template void launch_chunk_values<double>(const ChunkView<double>&, const OpView<double>&,
                                          const OpView<double>&, cudaStream_t);
template void launch_chunk_values<float>(const ChunkView<float>&, const OpView<float>&,
                                         const OpView<float>&, cudaStream_t);
template cudaError_t launch_chunk<double>(Ctl*, const ChunkView<double>&, const IterView<double>&,
                                          bool, cudaStream_t);
template cudaError_t launch_chunk<float>(Ctl*, const ChunkView<float>&, const IterView<float>&,
                                         bool, cudaStream_t);

}  // namespace sg
