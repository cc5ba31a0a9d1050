#include "sg_batch_device.cuh"

namespace sg {

// ------------------------------------------------------------------------------------------
// Unrolled PDHG and its adjoint (the differentiable layer). Per instance (one cluster), K
// iterations of the fixed-step PDHG — tau = sigma = eta, primal weight 1, no restarts and no
// averaging — from zero on the equilibrated problem (the reference's step, pdlp.cpp:574-641):
//   y+ = y + sigma (A x_bar - r_bar);  v+ = P(v - tau (c + [A -I]' y+));  v_bar+ = 2 v+ - v
// with v = (x, r) and P the projection on [l, u]. The state (v, v_bar, y) is saved every
// `every` iterations. The adjoint recomputes each segment forward from its checkpoint, keeping
// for every projection which bound it met, then runs the transposed recurrences backwards:
//   V = v_hat + 2 b_hat;  z_hat = [l < z < u] V;  l_hat += [z <= l] V;  u_hat += [z >= u] V
//   v_hat' = z_hat - b_hat;  g_hat = -tau z_hat;  c_hat += g_hat
//   y_hat' = y_hat + [A -I] g_hat;  b_hat' = [A -I]' (sigma y_hat')
// (the costs, bounds and iterates map to the LpProblem's space by the column and row scales).
// The elementwise part of a backward step runs in the epilogues of the step before it, so a
// backward step is two walks and two exchanges, as a forward step is.
//
// Bound by the FP64 pipe and, with four CTAs to an LP, by the exchanges: 64 LPs of 500 x 1,200,
// 256 iterations forward and backward: 11.0 ms with a CTA per LP and block barriers, 7.1 with
// clusters of two, 6.2 with four.

namespace {

// A double's bits mapped to a signed order, -0 equal to +0.
__device__ __forceinline__ long long order_of(double x) {
  const long long b = __double_as_longlong(x);
  return (b << 1) == 0 ? 0 : b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// 1: z <= lo (out = lo), 2: z >= up (out = up), 0: between (or NaN). On the integer pipe.
__device__ __forceinline__ unsigned char project(double z, double lo, double up, double* out) {
  const long long kz = order_of(z);
  const bool nan = (__double_as_longlong(z) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
  if (!nan && kz <= order_of(lo)) {
    *out = lo;
    return 1;
  }
  if (!nan && kz >= order_of(up)) {
    *out = up;
    return 2;
  }
  *out = z;
  return 0;
}

// The state of one instance's own columns and rows, arrays one after another as in SolveState:
// the point and the scaled problem, the rows' extrapolated point (negated) and dual; the
// adjoint's v_hat, b_hat, the gradients, and the rows' g_hat and y_hat.
enum : int { kUPoint = 0, kUCost = 1, kULower = 2, kUUpper = 3, kUBar = 4, kUDual = 5 };
// Adjoint arrays, after the forward's: columns from kUCols, rows from kURows.
enum : int { kAV = 0, kAB = 1, kAGc = 2, kAGl = 3, kAGu = 4, kAG = 5, kAY = 6 };
constexpr int kUCols = 4, kURows = 6;  // arrays of the forward (unroll_state_bytes: 4 and 6)
constexpr int kACols = 5, kARows = 7;  // and of the adjoint beside them

// Slice by slice, as SolveState.
template <int MODE>
struct alignas(16) UnrollState {
  double* device;              // not kAllShared: the columns' arrays
  long long rows_device;       // and how far on the rows' are
  unsigned cols_at, rows_at;   // kAllShared: offsets
  int col_arrays, row_arrays;
  unsigned rank, size, pad[2];
  // Entry of an own column or row: its arrays lie 32 entries apart.
  struct Entry {
    Array<double, MODE == kAllShared> e;
    __device__ __forceinline__ double get(int k) const { return e.get(32 * k); }
    __device__ __forceinline__ void set(int k, double v) const { e.set(32 * k, v); }
  };
  __device__ __forceinline__ Entry col_entry(const At& at) const { return Entry{&col(0, at)}; }
  __device__ __forceinline__ Entry row_entry(const At& at) const { return Entry{&row(0, at)}; }
  __device__ __forceinline__ double& col(int k, const At& at) const {
    if constexpr (MODE == kAllShared) {
      return reinterpret_cast<double*>(sg_smem + cols_at)[(at.ls * col_arrays + k) * 32 + at.lane];
    } else {
      return device[(static_cast<long long>(at.ls * size + rank) * col_arrays + k) * 32 + at.lane];
    }
  }
  __device__ __forceinline__ double& row(int k, const At& at) const {
    if constexpr (MODE == kAllShared) {
      return reinterpret_cast<double*>(sg_smem + rows_at)[(at.ls * row_arrays + k) * 32 + at.lane];
    } else {
      return device[rows_device +
                    (static_cast<long long>(at.ls * size + rank) * row_arrays + k) * 32 + at.lane];
    }
  }
  __device__ __forceinline__ double& acol(int k, const At& at) const { return col(kUCols + k, at); }
  __device__ __forceinline__ double& arow(int k, const At& at) const { return row(kURows + k, at); }
};

template <int MODE, int WALK>
struct Unroll {
  MatShare<double, RowShare<double, WALK>> M;
  Exchange<double, MODE> ex;
  UnrollState<MODE> S;
  const double *cs, *rs;
  double eta;
  long long vo, nt;
};

template <int MODE, int WALK>
__device__ __forceinline__ Unroll<MODE, WALK> unroll_begin(const BatchView& b, const UnrollView& u,
                                                     int inst, bool adjoint, ClusterShared& sh,
                                                     unsigned rank,
                                                     unsigned size) {
  using Share = RowShare<double, WALK>;
  Unroll<MODE, WALK> p;
  const int g = b.inst_mat[inst];
  p.M = mat_share<double, Share>(b, g, b.k_val, b.t_val, rank, size);
  MatShare<double, Share>& M = p.M;
  p.nt = static_cast<long long>(M.n) + M.m;
  p.cs = b.cs + b.mat_col_off[g];
  p.rs = b.rs + b.mat_row_off[g];
  p.eta = b.info[g].eta;
  p.vo = b.vec_off[inst];
  double* st = reinterpret_cast<double*>(b.state) + b.state_off[inst];
  p.ex = make_exchange<double, MODE>(M, sh, st, rank, size);
  UnrollState<MODE>& S = p.S;
  S.col_arrays = adjoint ? kUCols + kACols : kUCols;
  S.row_arrays = adjoint ? kURows + kARows : kURows;
  S.device = st + 3 * p.nt + 2;
  S.rows_device = (share_rows(M.n, M.Kt.slice, 1) >> M.Kt.slice) * 32 * S.col_arrays;
  S.cols_at = static_cast<unsigned>(cluster_vector_bytes(
      M.n, M.m, M.Kt.slice, M.K.slice, static_cast<int>(size), sizeof(double)));
  S.rows_at = S.cols_at + M.Kt.slices() * static_cast<unsigned>(32 * S.col_arrays * sizeof(double));
  S.rank = rank;
  S.size = size;
  // The equilibrated cost and bounds.
  const double* c0 = b.cost + p.vo;
  const double* l0 = b.lower + p.vo;
  const double* u0 = b.upper + p.vo;
  each_own(M.Kt, [&](const At& at) {
    const int k = M.tperm[at.p];
    const double sc = p.cs[at.p];
    S.col(kUCost, at) = c0[k] * sc;
    S.col(kULower, at) = l0[k] / sc;
    S.col(kUUpper, at) = u0[k] / sc;
  });
  each_own(M.K, [&](const At& at) {
    const int k = M.n + M.kperm[at.p];
    const double sc = p.rs[at.p];
    S.row(kUCost, at) = c0[k] * sc;
    S.row(kULower, at) = l0[k] * sc;
    S.row(kUUpper, at) = u0[k] * sc;
  });
  return p;
}

// One fixed-step iteration; `mask` (n + m bytes by position, null: not kept) records the
// projections. An equality row's logical is its bound from the first step on: a warp of such rows
// skips the logicals unless the mask is kept (which side its z lies on depends on the dual). xs
// has been put, not waited for; so it is afterwards.
template <int MODE, int WALK>
__device__ __forceinline__ bool unroll_step(const Unroll<MODE, WALK>* p, double tau, double sigma,
                                            unsigned char* mask) {
  {
    const auto K = sh_copy(&p->M.K);
    const auto ex = sh_copy(&p->ex);
    const auto S = sh_copy(&p->S);
    const int n = p->M.n;
    const Sender<double, MODE, 1> y_out(ex);
    const bool ok = walk_rows<true, false>(
        K, Gather<double, MODE>{ex.xs()},
        [&](const At& at) { return S.row_entry(at).get(kUBar); },
        [&](const At& at, double sum) {
          const auto e = S.row_entry(at);
          const double yn = e.get(kUDual) + sigma * sum;
          e.set(kUDual, yn);
          y_out.put(at, yn);
          const double r = e.get(kUPoint);
          const double lo = e.get(kULower);
          const double up = e.get(kUUpper);
          const bool steady = mask == nullptr && same_bits(lo, up) && same_bits(r, lo);
          const unsigned here = __activemask();
          if (__any_sync(here, !steady)) {
            keep_branch(here);
            double rn;
            const unsigned char c = project(r - tau * (e.get(kUCost) - yn), lo, up, &rn);
            if (mask != nullptr) mask[n + at.p] = c;
            e.set(kUPoint, rn);
            e.set(kUBar, fma(-2.0, rn, r));
          } else {
            e.set(kUBar, -lo);
          }
        },
        [&]() { return ex.wait(0); });
    if (!ok) return false;
  }
  const auto Kt = sh_copy(&p->M.Kt);
  const auto ex = sh_copy(&p->ex);
  const auto S = sh_copy(&p->S);
  const Sender<double, MODE, 0> x_out(ex);
  return walk_rows<true, false>(
      Kt, Gather<double, MODE>{ex.ys()},
      [&](const At& at) { return S.col_entry(at).get(kUCost); },
      [&](const At& at, double sum) {
        const auto e = S.col_entry(at);
        const double x = e.get(kUPoint);
        double xn;
        const unsigned char c = project(x - tau * sum, e.get(kULower), e.get(kUUpper), &xn);
        if (mask != nullptr) mask[at.p] = c;
        e.set(kUPoint, xn);
        x_out.put(at, fma(2.0, xn, -x));
      },
      [&]() { return ex.wait(1); });
}

// The backward step's elementwise part for one entry (its adjoint arrays from `from` on): returns
// g_hat.
template <typename Entry>
__device__ __forceinline__ double adjoint_entry(const Entry& e, int from, double bh,
                                                unsigned char code, double tau) {
  const double V = fma(2.0, bh, e.get(from + kAV));
  double gh = 0.0;
  if (code == 0) {
    gh = -tau * V;
    e.set(from + kAV, V - bh);
    e.set(from + kAGc, e.get(from + kAGc) + gh);
  } else {
    const int k = from + (code == 1 ? kAGl : kAGu);
    e.set(k, e.get(k) + V);
    e.set(from + kAV, -bh);
  }
  return gh;
}

template <int MODE, int WALK>
__device__ bool unroll_forward(const BatchView& b, const UnrollView& u, int inst,
                               ClusterShared& sh, Unroll<MODE, WALK>* ctx, unsigned rank,
                               unsigned size) {
  const Unroll<MODE, WALK> p = unroll_begin<MODE, WALK>(b, u, inst, false, sh, rank, size);
  if (threadIdx.x == 0) *ctx = p;
  const UnrollState<MODE>& S = p.S;
  const auto& M = p.M;
  const long long nt = p.nt;
  each_own(M.Kt, [&](const At& at) { S.col(kUPoint, at) = 0.0; });
  each_own(M.K, [&](const At& at) {
    S.row(kUPoint, at) = S.row(kUBar, at) = S.row(kUDual, at) = 0.0;
  });
  each_own(M.Kt, [&](const At& at) { p.ex.put_x(at, 0.0); });
  __syncthreads();
  double* ck = u.ck + u.ck_off[inst];
  const long long stride = 2 * nt + M.m;
  bool ok = true;
  for (int it = 0; it < u.iterations && ok; ++it) {
    if (it % u.every == 0) {
      __syncthreads();  // the step before is done
      double* c = ck + static_cast<long long>(it / u.every) * stride;
      each_own(M.Kt, [&](const At& at) {
        c[at.p] = S.col(kUPoint, at);
        c[nt + at.p] = p.ex.xs()[at.p];
      });
      each_own(M.K, [&](const At& at) {
        c[M.n + at.p] = S.row(kUPoint, at);
        c[nt + M.n + at.p] = S.row(kUBar, at);
        c[2 * nt + at.p] = S.row(kUDual, at);
      });
      __syncthreads();  // read above by other threads than update them
    }
    ok = unroll_step(ctx, p.eta, p.eta, nullptr);
  }
  if (ok) ok = p.ex.wait(0);
  __syncthreads();
  double* vo = u.v_out + p.vo;
  each_own(M.Kt, [&](const At& at) { vo[M.tperm[at.p]] = S.col(kUPoint, at) * p.cs[at.p]; });
  each_own(M.K, [&](const At& at) { vo[M.n + M.kperm[at.p]] = S.row(kUPoint, at) / p.rs[at.p]; });
  return !cluster_stopped(sh, size);
}

template <int MODE, int WALK>
__device__ bool unroll_adjoint(const BatchView& b, const UnrollView& u, int inst,
                               ClusterShared& sh, Unroll<MODE, WALK>* ctx, unsigned rank,
                               unsigned size) {
  const Unroll<MODE, WALK> p = unroll_begin<MODE, WALK>(b, u, inst, true, sh, rank, size);
  if (threadIdx.x == 0) *ctx = p;
  const UnrollState<MODE>& S = p.S;
  const auto& M = p.M;
  const long long nt = p.nt;
  const double tau = p.eta, sigma = p.eta;
  const double* gv = u.grad_v + p.vo;
  // Adjoint of v_K in the equilibrated space: x = x_eq cs, r = r_eq / rs.
  each_own(M.Kt, [&](const At& at) {
    S.acol(kAV, at) = gv[M.tperm[at.p]] * p.cs[at.p];
    S.acol(kAB, at) = S.acol(kAGc, at) = S.acol(kAGl, at) = S.acol(kAGu, at) = 0.0;
  });
  each_own(M.K, [&](const At& at) {
    S.arow(kAV, at) = gv[M.n + M.kperm[at.p]] / p.rs[at.p];
    S.arow(kAB, at) = S.arow(kAGc, at) = S.arow(kAGl, at) = S.arow(kAGu, at) = 0.0;
    S.arow(kAY, at) = 0.0;
  });
  const double* ck = u.ck + u.ck_off[inst];
  unsigned char* mask = u.mask + u.mask_off[inst];
  const long long stride = 2 * nt + M.m;
  bool ok = true;
  for (int seg = u.nck - 1; seg >= 0; --seg) {
    const int k0 = seg * u.every;
    const int len = min(u.every, u.iterations - k0);
    const double* c = ck + static_cast<long long>(seg) * stride;
    // xs and ys of the segment before are read by all.
    if (cluster_stopped(sh, size)) break;
    each_own(M.Kt, [&](const At& at) {
      S.col(kUPoint, at) = c[at.p];
      p.ex.put_x(at, c[nt + at.p]);
    });
    each_own(M.K, [&](const At& at) {
      S.row(kUPoint, at) = c[M.n + at.p];
      S.row(kUBar, at) = c[nt + M.n + at.p];
      S.row(kUDual, at) = c[2 * nt + at.p];
    });
    for (int t = 0; t < len && ok; ++t) {
      ok = unroll_step(ctx, tau, sigma, mask + static_cast<long long>(t) * nt);
    }
    ok = ok && p.ex.wait(0);
    cluster_sync(size);  // the last x_bar is in place everywhere: xs may be sent again
    auto col = [&](const At& at, double bh, const unsigned char* mk, const UnrollState<MODE>& S,
                   const Sender<double, MODE, 0>& x_out) {
      x_out.put(at, adjoint_entry(S.col_entry(at), kUCols, bh, mk[at.p], tau));
    };
    auto row = [&](const At& at, double bh, const unsigned char* mk, const UnrollState<MODE>& S) {
      const auto e = S.row_entry(at);
      e.set(kURows + kAG, adjoint_entry(e, kURows, bh, mk[M.n + at.p], tau));
    };
    if (ok) {
      const unsigned char* mk = mask + static_cast<long long>(len - 1) * nt;
      const Sender<double, MODE, 0> x_out(p.ex);
      each_own(M.Kt, [&](const At& at) { col(at, S.acol(kAB, at), mk, S, x_out); });
      each_own(M.K, [&](const At& at) { row(at, S.arow(kAB, at), mk, S); });
    }
    for (int t = len - 1; t >= 0 && ok; --t) {
      const unsigned char* before = t > 0 ? mask + static_cast<long long>(t - 1) * nt : nullptr;
      {
        const auto K = sh_copy(&ctx->M.K);
        const auto ex = sh_copy(&ctx->ex);
        const auto S = sh_copy(&ctx->S);
        const Sender<double, MODE, 1> y_out(ex);
        ok = walk_rows<true, false>(
            K, Gather<double, MODE>{ex.xs()},
            [&](const At& at) { return -S.row_entry(at).get(kURows + kAG); },
            [&](const At& at, double sum) {
              const auto e = S.row_entry(at);
              const double yt = e.get(kURows + kAY) + sum;
              e.set(kURows + kAY, yt);
              const double sy = sigma * yt;
              y_out.put(at, sy);
              if (before != nullptr) {
                row(at, -sy, before, S);
              } else {
                e.set(kURows + kAB, -sy);
              }
            },
            [&]() { return ex.wait(0); });
      }
      if (!ok) break;
      // The last step of a segment sends no xs; the next segment starts with a barrier.
      const auto Kt = sh_copy(&ctx->M.Kt);
      const auto ex = sh_copy(&ctx->ex);
      const auto S = sh_copy(&ctx->S);
      const Sender<double, MODE, 0> x_out(ex);
      ok = walk_rows<true, false>(
          Kt, Gather<double, MODE>{ex.ys()}, Zero<double>(),
          [&](const At& at, double sum) {
            if (before != nullptr) {
              col(at, sum, before, S, x_out);
            } else {
              S.col_entry(at).set(kUCols + kAB, sum);
            }
          },
          [&]() { return ex.wait(1); });
    }
  }
  __syncthreads();
  // Gradients in the LpProblem's space: c_eq = c s, l_eq = l / cs (columns), l rs (rows).
  double* gc = u.grad_cost + p.vo;
  double* gl = u.grad_lower + p.vo;
  double* gu = u.grad_upper + p.vo;
  each_own(M.Kt, [&](const At& at) {
    const int k = M.tperm[at.p];
    const double sc = p.cs[at.p];
    gc[k] = S.acol(kAGc, at) * sc;
    gl[k] = S.acol(kAGl, at) / sc;
    gu[k] = S.acol(kAGu, at) / sc;
  });
  each_own(M.K, [&](const At& at) {
    const int k = M.n + M.kperm[at.p];
    const double sc = p.rs[at.p];
    gc[k] = S.arow(kAGc, at) * sc;
    gl[k] = S.arow(kAGl, at) * sc;
    gu[k] = S.arow(kAGu, at) * sc;
  });
  return !cluster_stopped(sh, size);
}

}  // namespace

template <bool ADJOINT, int MODE, int PER_SM = 2, int WALK = kWalkOne, int THREADS = kThreads64>
__global__ void __launch_bounds__(THREADS, PER_SM) unroll_kernel(BatchView b, UnrollView u,
                                                                    InstanceList list) {
  __shared__ ClusterShared sh;
  __shared__ Unroll<MODE, WALK> ctx;
  const unsigned rank = cluster_rank();
  const unsigned size = cluster_size();
  cluster_init(sh, size);
  bool ok = true;
  for (int q = blockIdx.x / size; q < list.count && ok; q += gridDim.x / size) {
    if constexpr (ADJOINT) {
      ok = unroll_adjoint<MODE, WALK>(b, u, list.inst[q], sh, &ctx, rank, size);
    } else {
      ok = unroll_forward<MODE, WALK>(b, u, list.inst[q], sh, &ctx, rank, size);
    }
  }
  if (!ok && threadIdx.x == 0) atomicExch(b.wait_error, 1);
  cluster_sync(size);
}

namespace {

// go() with the kernel of a mode; `alone`: the adjoint's variant with an SM to a CTA.
template <typename Go>
auto with_unroll_kernel(int adjoint, int mode, bool alone, const ClusterPlan& p, const Go& go) {
  if (p.small && adjoint && alone) return go(unroll_kernel<true, kAllShared, 1, kWalkLanes>);
  if (p.small) {
    return adjoint ? go(unroll_kernel<true, kAllShared, 2, kWalkLanes>)
                   : go(unroll_kernel<false, kAllShared, 2, kWalkLanes>);
  }
  if (mode == kAllShared && adjoint && alone) return go(unroll_kernel<true, kAllShared, 1>);
  if (mode == kAllShared) {
    return adjoint ? go(unroll_kernel<true, kAllShared>) : go(unroll_kernel<false, kAllShared>);
  }
  if (mode == kVectorsShared && p.threads[mode] == kThreads64) {
    return adjoint ? go(unroll_kernel<true, kVectorsShared>)
                   : go(unroll_kernel<false, kVectorsShared>);
  }
  constexpr int kMost = kThreads64Large;
  if (mode == kVectorsShared) {
    return adjoint ? go(unroll_kernel<true, kVectorsShared, 1, kWalkOne, kMost>)
                   : go(unroll_kernel<false, kVectorsShared, 1, kWalkOne, kMost>);
  }
  return adjoint ? go(unroll_kernel<true, kInDevice, 1, kWalkOne, kMost>)
                 : go(unroll_kernel<false, kInDevice, 1, kWalkOne, kMost>);
}

}  // namespace

bool unroll_fits(const ClusterPlan& p, int adjoint) {
  for (int mode = 0; mode < kModes; ++mode) {
    for (bool alone : {false, true}) {
      if (p.group[mode].count > 0 &&
          !with_unroll_kernel(adjoint, mode, alone, p, [&](auto kernel) {
            return clusters_fit(kernel, p.size, p.threads[mode], p.smem[mode]);
          })) {
        return false;
      }
    }
  }
  return true;
}

cudaError_t launch_unroll(const BatchView& b, const UnrollView& u, const ClusterPlan& p,
                          int adjoint, const GroupStreams& gs, cudaStream_t s) {
  return for_groups(p, gs, s, cudaSuccess, [&](int mode, cudaStream_t gst) {
    const InstanceList list = p.group[mode];
    const int clusters = list.count < p.clusters ? list.count : p.clusters;
    // The adjoint's values take 215 registers; with 128, two CTAs to an SM, some are read anew. While
    // every CTA finds an SM of its own the variant of 215 runs (the adjoint of 200 iterations: 1 LP of
    // 300 x 660 2.08 ms, 2.31 without; 64 of 150 x 330 2.07 and 2.33). Clusters of 4 and more leave SMs
    // of a GPC over: 16 clusters of 8 no longer ran side by side (2.63 ms with two CTAs to an SM, 3.87
    // without).
    const int side_by_side = p.size <= 2   ? p.sms / p.size
                             : p.size == 4 ? p.sms / p.size * 3 / 4
                                           : p.sms / p.size / 2;
    const bool alone = clusters <= side_by_side;
    return with_unroll_kernel(adjoint, mode, alone, p, [&](auto kernel) {
      return launch_clusters(kernel, p.size, clusters, p.threads[mode], p.smem[mode], gst, b, u, list);
    });
  });
}

}  // namespace sg
