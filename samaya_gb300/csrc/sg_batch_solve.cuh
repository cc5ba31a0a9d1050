// The batched solve: persistent clusters that run whole PDLP solves (see sg_batch.cu).
//
// FP64 steps are bound by the FP64 pipe (busy 47-53% of the time) and by the walks' load latency
// before a cluster's exchange; FP32 ones by the instructions around each nonzero (addresses,
// bounds of the row). One CTA per LP (a block barrier a half step, unsorted rows, the nonzeros
// of a row side by side, averages and evaluation sums in separate passes) took 25.4 ms for 256
// iterations of 160 random LPs of 100-2,500 rows in FP64, clusters of four 13.4 ms; 512
// Halpern iterations of 256 facility-location nodes (40 x 160) with FP32 storage 53.6 ms,
// now, still a CTA per LP, 21.4 ms.
#pragma once

#include "sg_cluster_steps.cuh"

namespace sg {

// ------------------------------------------------------------------------------------------
// Solve: persistent clusters, one instance at a time.

namespace {

struct Meas {
  double rp, rd, rg, pobj, dobj;
};

__device__ __forceinline__ Meas finish7(const double* s, double amc, double amr, double cnorm,
                                        int m) {
  Meas r;
  const double ps = 1.0 + amc * sqrt(s[4]) + sqrt(s[5]);
  const double ds = 1.0 + amr * sqrt(s[6]) + cnorm;
  const double gs = 1.0 + fabs(s[2]) + fabs(s[3]);
  r.rp = m > 0 ? sqrt(s[0]) / ps : 0.0;
  r.rd = m > 0 ? sqrt(s[1]) / ds : 0.0;
  r.rg = (s[2] - s[3]) / gs;
  r.pobj = s[2];
  r.dobj = s[3];
  return r;
}

__device__ __forceinline__ double kkt_w(double w, const Meas& e) {
  return sqrt(w * w * e.rp * e.rp + e.rd * e.rd / (w * w) + e.rg * e.rg);
}

// The given problem and the scales of an instance, by position.
struct Given {
  const int *kperm, *tperm;
  const double *cost, *lower, *upper;  // (columns, rows) in the caller's order
  const double *cs, *rs, *ics, *irs;
  int n;
};

// What the evaluation needs beside the steps' context; evaluate_point is a call of its own, so
// that its registers are not the step's.
template <typename T, int MODE, typename Share>
struct EvalContext : StepContext<T, MODE, Share> {
  Given G;
};

// One iterate's sums (7 evaluation sums in the original space, pdlp.cpp:411-488, and the restart
// distances of v and y) into e: which 0 the current point, 1 the average, 2 Halpern's T(z). The
// evaluated vectors take the place of xs and ys.
template <typename T, int MODE, typename Share>
__device__ __noinline__ bool evaluate_point(const EvalContext<T, MODE, Share>* ctx, int which,
                                            double inv_k, double (&e)[9]) {
  constexpr bool kF64 = sizeof(T) == 8;
  const MatShare<T, Share>& M = ctx->M;
  const Exchange<T, MODE>& ex = ctx->ex;
  const SolveState<T, MODE>& S = ctx->S;
  const Second<T>& Z = ctx->Z;
  const Given& G = ctx->G;
  auto vx = [&](const At& at) -> T {
    return which == 0 ? S.col(kPoint, at)
           : which == 1 ? static_cast<T>(average(S.col(kSum, at), inv_k)) : Z.x(at.p);
  };
  auto vy = [&](const At& at) -> T {
    return which == 0 ? S.row(kDual, at)
           : which == 1 ? static_cast<T>(average(S.row(kDualSum, at), inv_k)) : Z.y(at.p);
  };
  auto vr = [&](const At& at) -> T {
    if (which == 2) return Z.r(at.p);
    if (which == 0) return S.row(kPoint, at);
    if (kF64 && S.row(kLower, at) == S.row(kUpper, at)) return S.row(kLower, at);
    return static_cast<T>(average(S.row(kSum, at), inv_k));
  };
  const bool halpern = which == 2;
#pragma unroll
  for (int q = 0; q < 9; ++q) e[q] = 0.0;
  each_own(M.Kt, [&](const At& at) { ex.put_x(at, vx(at)); });
  each_own(M.K, [&](const At& at) { ex.put_y(at, vy(at)); });
  if (!ex.wait(0) || !ex.wait(1)) return false;
  const int m = M.m;
  walk_rows<true, false>(M.K, GatherD<T>{ex.xs()}, Zero<double>(), [&](const At& at, double s) {
    const int k = G.n + G.kperm[at.p];
    const double irs = G.irs[at.p];
    const double rv = static_cast<double>(vr(at));
    const double yv = static_cast<double>(vy(at));
    const double value = rv * irs;
    const double yo = yv * G.rs[at.p];
    const double c = G.cost[k];
    const double g = c - yo;
    const double ep = s * irs - value;
    const double lo = G.lower[k];
    const double up = G.upper[k];
    e[0] += ep * ep;
    e[5] += value * value;
    e[6] += yo * yo;
    e[2] += c * value;
    const double lam = lam_of(g, lo, up);
    e[1] += (g - lam) * (g - lam);
    if (lam > 0.0) e[3] += lam * lo;
    if (lam < 0.0) e[3] += lam * up;
    const double dv = rv - static_cast<double>(halpern ? S.row(kSum, at) : Z.r(at.p));
    const double dy = yv - static_cast<double>(halpern ? S.row(kDualSum, at) : Z.y(at.p));
    e[7] += dv * dv;
    e[8] += dy * dy;
  }, Ready());
  walk_rows<true, false>(M.Kt, GatherD<T>{ex.ys()}, Zero<double>(), [&](const At& at, double s) {
    const int k = G.tperm[at.p];
    const double xv = static_cast<double>(vx(at));
    const double value = xv * G.cs[at.p];
    const double c = G.cost[k];
    const double g = c + (m > 0 ? s * G.ics[at.p] : 0.0);
    const double lo = G.lower[k];
    const double up = G.upper[k];
    e[4] += value * value;
    e[2] += c * value;
    const double lam = lam_of(g, lo, up);
    e[1] += (g - lam) * (g - lam);
    if (lam > 0.0) e[3] += lam * lo;
    if (lam < 0.0) e[3] += lam * up;
    const double dv = xv - static_cast<double>(halpern ? S.col(kSum, at) : Z.x(at.p));
    e[7] += dv * dv;
  }, Ready());
  return true;
}

// Runs one instance (a wait that gave up is in sh.fail). Storage, products and step sums in T
// (GB300's FP64 pipe is small), the evaluation in FP64.
template <typename T, int MODE, bool halpern, typename Share>
__device__ void solve_instance(const BatchView& b, int inst, ClusterShared& sh,
                               EvalContext<T, MODE, Share>* ctx, unsigned rank,
                               unsigned size) {
  constexpr bool kF64 = sizeof(T) == 8;
  const int g = b.inst_mat[inst];
  const T* kval = reinterpret_cast<const T*>(kF64 ? static_cast<const void*>(b.k_val)
                                                  : static_cast<const void*>(b.k_val32));
  const T* tval = reinterpret_cast<const T*>(kF64 ? static_cast<const void*>(b.t_val)
                                                  : static_cast<const void*>(b.t_val32));
  MatShare<T, Share> M = mat_share<T, Share>(b, g, kval, tval, rank, size);
  const int m = M.m;
  const int n = M.n;
  const long long nt = static_cast<long long>(n) + m;
  const long long vo = b.vec_off[inst];
  const Given G{M.kperm, M.tperm, b.cost + vo, b.lower + vo, b.upper + vo,
                b.cs + b.mat_col_off[g], b.rs + b.mat_row_off[g], b.ics + b.mat_col_off[g],
                b.irs + b.mat_row_off[g], n};
  const MatInfo mi = b.info[g];
  // Device storage (instance_elements): the gathered vectors where they do not fit, the second
  // points, the state where it does not fit.
  T* st = reinterpret_cast<T*>(b.state) + b.state_off[inst];
  const Second<T> Z{st + nt + 2, n, m};
  Exchange<T, MODE> ex = make_exchange<T, MODE>(M, sh, st, rank, size);
  SolveState<T, MODE> S;
  S.device = st + 3 * nt + 2;
  S.rows_device = (share_rows(n, M.Kt.slice, 1) >> M.Kt.slice) * 32 * kColArrays;
  S.cols_at = static_cast<unsigned>(cluster_vector_bytes(n, m, M.Kt.slice, M.K.slice,
                                                         static_cast<int>(size), sizeof(T)));
  S.rows_at = S.cols_at + M.Kt.slices() * static_cast<unsigned>(32 * kColArrays * sizeof(T));
  S.rank = rank;
  S.size = size;
  if (threadIdx.x == 0) {
    ctx->M = M;
    ctx->ex = ex;
    ctx->S = S;
    ctx->Z = Z;
    ctx->G = G;
  }
  // Scaled problem, zero iterates, ||c||.
  double nrm[3] = {0.0, 0.0, 0.0};
  each_own(M.Kt, [&](const At& at) {
    const int k = G.tperm[at.p];
    const double sc = G.cs[at.p];
    const double c0 = G.cost[k];
    const double c = c0 * sc;
    S.col(kCost, at) = static_cast<T>(c);
    S.col(kLower, at) = static_cast<T>(G.lower[k] / sc);
    S.col(kUpper, at) = static_cast<T>(G.upper[k] / sc);
    S.col(kPoint, at) = S.col(kSum, at) = Z.x(at.p) = T(0);
    nrm[0] += c0 * c0;
    nrm[1] += c * c;
  });
  each_own(M.K, [&](const At& at) {
    const int k = n + G.kperm[at.p];
    const double r = G.rs[at.p];
    const double c0 = G.cost[k];
    const double lo = G.lower[k] * r;
    const double up = G.upper[k] * r;
    S.row(kCost, at) = static_cast<T>(c0 * r);
    S.row(kLower, at) = static_cast<T>(lo);
    S.row(kUpper, at) = static_cast<T>(up);
    S.row(kPoint, at) = S.row(kSum, at) = S.row(kBar, at) = T(0);
    S.row(kDual, at) = S.row(kDualSum, at) = Z.r(at.p) = Z.y(at.p) = T(0);
    nrm[0] += c0 * c0;
    const double bb = fmax(isfinite(lo) ? fabs(lo) : 0.0, isfinite(up) ? fabs(up) : 0.0);
    nrm[2] += bb * bb;
  });
  cluster_reduce<3>(nrm, sh, rank, size);
  const double c_norm = sqrt(nrm[0]);
  double omega = 1.0;
  if (b.algorithm >= 1) {
    const double cn = sqrt(nrm[1]), bn = sqrt(nrm[2]);
    omega = (cn > 1e-10 && bn > 1e-10) ? cn / bn : 1.0;
  }
  const double eta = mi.eta;
  double tau = eta / omega, sigma = eta * omega;
  long long max_iter = b.max_iter;
  if (max_iter <= 0) {
    max_iter = 10000LL * nt / 10;
    if (max_iter < 10000LL) max_iter = 10000LL;
    if (max_iter > 1000000LL) max_iter = 1000000LL;
  }
  double kar = INFINITY, kprev = INFINITY;
  long long t = 0, k_since = 0, restarts = 0;
  int status = kIterationLimit;
  int result_avg = 0;
  double inv_k = 1.0;  // 1 / iterations since the restart, at an evaluation
  Meas final_meas{0, 0, 0, 0, 0};
  bool ok = true;
  // The gathered vector the first step reads.
  if (halpern) {
    each_own(M.K, [&](const At& at) { ex.put_y(at, T(0)); });
  } else {
    each_own(M.Kt, [&](const At& at) { ex.put_x(at, T(0)); });
  }
  while (t < max_iter) {
    // The iterations up to the next evaluation.
    long long steps = 64 - t % 64;
    if (steps > max_iter - t) steps = max_iter - t;
    // The steps' weights, a thread each (a double division by every thread of every step would
    // take the FP64 pipe for 4,000 clocks a step).
    __syncthreads();
    if (threadIdx.x < steps) {
      const double k = static_cast<double>(k_since + static_cast<int>(threadIdx.x));
      ctx->weight[threadIdx.x] = static_cast<T>(1.0 / (k + (halpern ? 2.0 : 1.0)));
      ctx->rest[threadIdx.x] = static_cast<T>(1.0 - 1.0 / (k + 1.0));
    }
    __syncthreads();
    ok = run_steps<halpern, T, MODE, Share, SolveState<T, MODE>>(
        ctx, static_cast<int>(steps), static_cast<T>(tau), static_cast<T>(sigma), [] {});
    t += steps;
    k_since += steps;
    ok = ok && ex.wait(halpern ? 1 : 0);
    // Evaluation of the current and the average iterate; Halpern: only T(z) (the Halpern iterate
    // itself can leave the bounds).
    if (!halpern) {
      each_own(M.Kt, [&](const At& at) { Z.saved(at.p) = ex.xs()[at.p]; });
      inv_k = 1.0 / static_cast<double>(k_since);
    }
    // a: the current iterate's 7 sums, the average's 7, the distances (v, y) of each, and
    // whether the time limit has passed (1, asked by one thread, so that all agree) and CTAs' waits
    // gave up (2 each).
    double a[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) a[q] = 0.0;
    for (int w = halpern ? 1 : 0; w < 2; ++w) {
      cluster_sync(size);  // every CTA has read xs and ys, their last entries in place
      double e[9] = {};
      ok = ok && evaluate_point<T, MODE, Share>(ctx, halpern ? 2 : w, inv_k, e);
      if (w == 0) {
#pragma unroll
        for (int q = 0; q < 7; ++q) a[q] = e[q];
        a[14] = e[7];
        a[15] = e[8];
      } else {
#pragma unroll
        for (int q = 0; q < 7; ++q) a[7 + q] = e[q];
        a[16] = e[7];
        a[17] = e[8];
      }
    }
    if (rank == 0 && threadIdx.x == 0) {
      const unsigned long long deadline = *b.deadline;
      if (deadline != 0ull && globaltimer_ns() > deadline) a[18] = 1.0;
    }
    if (threadIdx.x == 0 && !ok) a[18] += 2.0;
    cluster_reduce<19>(a, sh, rank, size);
    if (a[18] >= 2.0) {
      ok = false;
      break;
    }
    const Meas mc = finish7(a, mi.a_norm_max_col, mi.at_norm_max_row, c_norm, m);
    const Meas ma = finish7(a + 7, mi.a_norm_max_col, mi.at_norm_max_row, c_norm, m);
    const double tol = b.tol;
    if (!halpern && mc.rp < tol && mc.rd < tol && fabs(mc.rg) < tol) {
      status = kOptimal;
      final_meas = mc;
      break;
    }
    if (ma.rp < tol && ma.rd < tol && fabs(ma.rg) < tol) {
      status = kOptimal;
      result_avg = 1;
      final_meas = ma;
      break;
    }
    final_meas = halpern ? ma : mc;
    // Restart (pdlp.cpp:1069-1131); the Halpern iteration restarts to T(z).
    const double kc = kkt_w(omega, mc), ka = kkt_w(omega, ma);
    const bool to_avg = halpern || ka < kc;
    const double cand = halpern ? ka : fmin(kc, ka);
    if (!(kar < INFINITY)) kar = cand;
    const bool restart = cand <= 0.2 * kar || (cand <= 0.8 * kar && cand > kprev) ||
                         static_cast<double>(k_since) >= b.art_frac * static_cast<double>(t);
    kprev = cand;
    if (restart) {
      const double dx = sqrt(to_avg ? a[16] : a[14]);
      const double dy = sqrt(to_avg ? a[17] : a[15]);
      if (dx > 1e-10 && dy > 1e-10) {
        omega = exp(0.5 * log(dy / dx) + 0.5 * log(omega));
        tau = eta / omega;
        sigma = eta * omega;
      }
      // The candidate becomes the point, the extrapolated point and the anchor; a sum starts
      // again from nothing (an FP32 average is replaced by the first step's weight 1).
      each_own(M.Kt, [&](const At& at) {
        const T v = halpern  ? Z.x(at.p)
                    : to_avg ? static_cast<T>(average(S.col(kSum, at), inv_k))
                             : S.col(kPoint, at);
        S.col(kPoint, at) = v;
        if (halpern) {
          S.col(kSum, at) = v;
        } else {
          Z.x(at.p) = v;
          Z.saved(at.p) = v;
          if (kF64) S.col(kSum, at) = T(0);
        }
      });
      each_own(M.K, [&](const At& at) {
        T v, y;
        if (halpern) {
          v = Z.r(at.p);
          y = Z.y(at.p);
        } else if (to_avg) {
          v = kF64 && S.row(kLower, at) == S.row(kUpper, at)
                  ? S.row(kLower, at)
                  : static_cast<T>(average(S.row(kSum, at), inv_k));
          y = static_cast<T>(average(S.row(kDualSum, at), inv_k));
        } else {
          v = S.row(kPoint, at);
          y = S.row(kDual, at);
        }
        S.row(kPoint, at) = v;
        S.row(kDual, at) = y;
        if (halpern) {
          S.row(kSum, at) = v;
          S.row(kDualSum, at) = y;
        } else {
          S.row(kBar, at) = -v;
          Z.r(at.p) = v;
          Z.y(at.p) = y;
          if (kF64) S.row(kSum, at) = S.row(kDualSum, at) = T(0);
        }
      });
      k_since = 0;
      kar = cand;
      kprev = INFINITY;
      ++restarts;
    }
    if (a[18] != 0.0) {
      status = kTimeLimit;
      break;
    }
    // The gathered vector the next iteration reads first.
    if (halpern) {
      each_own(M.K, [&](const At& at) { ex.put_y(at, S.row(kDual, at)); });
    } else {
      each_own(M.Kt, [&](const At& at) { ex.put_x(at, Z.saved(at.p)); });
    }
  }
  // Entries put after the last evaluation are taken in before anyone goes on.
  if (ok && status == kIterationLimit) ok = ex.wait(halpern ? 1 : 0);
  __syncthreads();
  // Answer in the LpProblem's space (Halpern: T(z), within the bounds).
  double* xo = b.x_out + vo;
  double* yo = b.y_out + b.row_off[inst];
  each_own(M.Kt, [&](const At& at) {
    const T v = halpern      ? Z.x(at.p)
                : result_avg ? static_cast<T>(average(S.col(kSum, at), inv_k))
                             : S.col(kPoint, at);
    xo[G.tperm[at.p]] = static_cast<double>(v) * G.cs[at.p];
  });
  each_own(M.K, [&](const At& at) {
    T v, y;
    if (halpern) {
      v = Z.r(at.p);
      y = Z.y(at.p);
    } else if (result_avg) {
      v = kF64 && S.row(kLower, at) == S.row(kUpper, at)
              ? S.row(kLower, at)
              : static_cast<T>(average(S.row(kSum, at), inv_k));
      y = static_cast<T>(average(S.row(kDualSum, at), inv_k));
    } else {
      v = S.row(kPoint, at);
      y = S.row(kDual, at);
    }
    xo[n + G.kperm[at.p]] = static_cast<double>(v) / G.rs[at.p];
    yo[G.kperm[at.p]] = static_cast<double>(y) * G.rs[at.p];
  });
  if (rank == 0 && threadIdx.x == 0) {
    InstResult& r = b.results[inst];
    r.status = ok ? status : kNumericalError;
    r.iterations = status == kIterationLimit ? max_iter : t;
    r.rel_primal = final_meas.rp;
    r.rel_dual = final_meas.rd;
    r.rel_gap = final_meas.rg;
    r.primal_obj = final_meas.pobj;
    r.dual_obj = final_meas.dobj;
    r.restarts = restarts;
  }
  if (!ok && threadIdx.x == 0) atomicExch(b.wait_error, 1);
}

// The next position of the work queue, the same for every thread of the cluster; past its end when
// a wait gave up in one of the CTAs.
__device__ __forceinline__ int next_instance(unsigned* queue, ClusterShared& sh, unsigned rank,
                                             unsigned size) {
  // The last instance is done, its position read by all.
  const bool stopped = cluster_stopped(sh, size);
  if (rank == 0 && threadIdx.x == 0) {
    const unsigned q = stopped ? 0x7fffffffu : atomicAdd(queue, 1u);
    for (unsigned p = 0; p < size; ++p) st_cluster(map_rank(shared_addr(&sh.next), p), q);
  }
  cluster_sync(size);
  return sh.next;
}

}  // namespace

template <typename T, int MODE, bool HALPERN, int THREADS, int WALK = kWalkOne>
__global__ void __launch_bounds__(THREADS, sizeof(T) == 8 && THREADS == kThreads64 ? 2 : 1)
    batch_solve_kernel(BatchView b, InstanceList list) {
  using Share = RowShare<T, WALK>;
  __shared__ ClusterShared sh;
  __shared__ EvalContext<T, MODE, Share> ctx;
  const unsigned rank = cluster_rank();
  const unsigned size = cluster_size();
  cluster_init(sh, size);
  for (;;) {
    const int q = next_instance(b.queue + MODE, sh, rank, size);
    if (q >= list.count) break;
    solve_instance<T, MODE, HALPERN, Share>(b, list.inst[q], sh, &ctx, rank, size);
  }
  cluster_sync(size);
}

// go() with the kernel of a mode and number of threads (Batch::plan_clusters). FP32 with 512 threads
// walks two slices at a time: 128 registers and one slice's loads on their way are too few.
template <typename T, typename Go>
auto with_solve_kernel(int algorithm, int mode, const ClusterPlan& p, const Go& go) {
  const bool h = algorithm == 2;
  const int threads = p.threads[mode];
  if (p.small) {
    constexpr int kFew = sizeof(T) == 4 ? kThreads32Few : kThreads64;
    return h ? go(batch_solve_kernel<T, kAllShared, true, kFew, kWalkLanes>)
             : go(batch_solve_kernel<T, kAllShared, false, kFew, kWalkLanes>);
  }
  if constexpr (sizeof(T) == 4) {
    if (mode == kAllShared && threads == kThreads32Few) {
      return h ? go(batch_solve_kernel<T, kAllShared, true, kThreads32Few>)
               : go(batch_solve_kernel<T, kAllShared, false, kThreads32Few>);
    }
    if (mode == kAllShared && threads == kThreads32Mid) {
      return h ? go(batch_solve_kernel<T, kAllShared, true, kThreads32Mid>)
               : go(batch_solve_kernel<T, kAllShared, false, kThreads32Mid>);
    }
    if (mode == kAllShared) {
      return go(batch_solve_kernel<T, kAllShared, true, kThreads32, kWalkPairs>);
    }
  } else if (mode == kAllShared) {
    return h ? go(batch_solve_kernel<T, kAllShared, true, kThreads64>)
             : go(batch_solve_kernel<T, kAllShared, false, kThreads64>);
  }
  constexpr int kMost = sizeof(T) == 4 ? kThreads32 : kThreads64Large;
  constexpr int kWalk = sizeof(T) == 4 ? kWalkPairs : kWalkOne;
  if constexpr (sizeof(T) == 8) {
    if (mode == kVectorsShared && threads == kThreads64) {
      return h ? go(batch_solve_kernel<T, kVectorsShared, true, kThreads64>)
               : go(batch_solve_kernel<T, kVectorsShared, false, kThreads64>);
    }
  }
  if (mode == kVectorsShared) {
    return h ? go(batch_solve_kernel<T, kVectorsShared, true, kMost, kWalk>)
             : go(batch_solve_kernel<T, kVectorsShared, false, kMost, kWalk>);
  }
  return h ? go(batch_solve_kernel<T, kInDevice, true, kMost, kWalk>)
           : go(batch_solve_kernel<T, kInDevice, false, kMost, kWalk>);
}

template <typename T>
cudaError_t launch_solve(const BatchView& b, const ClusterPlan& p, int mode, cudaStream_t s) {
  const InstanceList list = p.group[mode];
  const int clusters = list.count < p.clusters ? list.count : p.clusters;
  return with_solve_kernel<T>(b.algorithm, mode, p, [&](auto kernel) {
    return launch_clusters(kernel, p.size, clusters, p.threads[mode], p.smem[mode], s, b, list);
  });
}

template <typename T>
bool solve_fits(const ClusterPlan& p, int algorithm) {
  for (int mode = 0; mode < kModes; ++mode) {
    if (p.group[mode].count > 0 && !with_solve_kernel<T>(algorithm, mode, p, [&](auto kernel) {
          return clusters_fit(kernel, p.size, p.threads[mode], p.smem[mode]);
        })) {
      return false;
    }
  }
  return true;
}

}  // namespace sg
