// Batched PDLP: many LPs in one persistent launch (the engine's own; the reference solves one
// LP at a time). Instances are stored as a segmented concatenated CSR: matrices (each by rows,
// A, and by columns, A') concatenated with offsets, several instances may share one matrix
// (branch-and-bound node relaxations: one A, many bound vectors), and every instance has its
// own cost and bounds.
//
// Two kernels:
//   batch_setup_kernel   one thread-block cluster per matrix: the residual-scale norms of A,
//                        Ruiz (or the enhanced preconditioning), A_eq, and ||[A_eq -I]|| by
//                        power iteration — shared by every instance of that matrix;
//   batch_solve_kernel   (sg_batch_solve.cuh) persistent clusters pull instances from a work
//                        queue (largest first) and run the whole PDLP of one instance inside the
//                        cluster: the fused steps, the evaluation every 64 iterations, the
//                        termination test, the restarts and the primal-weight update of the
//                        single-LP engine (the reference's rules, pdlp.cpp:493-541, 674-713,
//                        1069-1131), per instance.
// The walks over rows and columns and the exchange between a cluster's CTAs are in
// sg_cluster.cuh; the cluster size follows the batch (Batch::make_plan).
#include "sg_batch_device.cuh"

namespace sg {

// ------------------------------------------------------------------------------------------
// Setup: one cluster per matrix. FP64: bound by the FP64 pipe (about 100 operations per nonzero
// in all) when the matrices fill the chip, by the exchanges when a single matrix is set up.
namespace {

template <int MODE, int WALK>
__device__ void setup_matrix(const BatchView& b, int g, ClusterShared& sh,
                             unsigned rank, unsigned size) {
  using Share = RowShare<double, WALK>;
  MatShare<double, Share> M =
      mat_share<double, Share>(b, g, b.k_val0, b.t_val0, rank, size);
  const int m = M.m;
  const int n = M.n;
  // By position: scales, their reciprocals, scratch.
  double* cs = b.cs + b.mat_col_off[g];
  double* rs = b.rs + b.mat_row_off[g];
  double* ics = b.ics + b.mat_col_off[g];
  double* irs = b.irs + b.mat_row_off[g];
  double* cn = ics;
  double* rn = irs;
  Exchange<double, MODE> ex = make_exchange<double, MODE>(
      M, sh, b.spill + b.mat_col_off[g] + b.mat_row_off[g] + 2 * g, rank, size);
  const Share& K0 = M.K;
  const Share& T0 = M.Kt;
  const Zero<double> zero_init;
  // Relative-residual scales of the original matrix (pdlp.cpp:377-394).
  double norms[2] = {0.0, 0.0};
  if (m > 0) {
    struct Sq {
      __device__ double operator()(double a, int) const { return a * a; }
    } sq;
    walk_rows<true, false>(T0, sq, zero_init,
                           [&](const At&, double s) { norms[0] = fmax(norms[0], sqrt(s)); }, Ready());
    walk_rows<true, false>(K0, sq, zero_init,
                           [&](const At&, double s) { norms[1] = fmax(norms[1], sqrt(s)); }, Ready());
    cluster_reduce<2, 3u>(norms, sh, rank, size);
  }
  // Preconditioning: the scales are the gathered vectors (xs the columns', ys the rows').
  double* xs = ex.xs();
  double* ys = ex.ys();
  for (int j = threadIdx.x; j < n; j += blockDim.x) xs[j] = 1.0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) ys[i] = 1.0;
  cluster_sync(size);
  bool ok = true;  // (no loop ends on it: they hold cluster barriers)
  if (m > 0 && n > 0) {
    // Both statistics are taken with the old scales, then every own scale is updated and sent.
    if (b.algorithm >= 1) {
      struct Abs {
        const double* o;
        __device__ double operator()(double a, int j) const { return fabs(a) * o[j]; }
      };
      for (int pass = 0; pass < 11; ++pass) {
        auto fc = [&](const At& at, double s) { cn[at.p] = s * xs[at.p]; };
        auto fr = [&](const At& at, double s) { rn[at.p] = s * ys[at.p]; };
        if (pass < 10) {
          walk_rows<true, true>(T0, Abs{ys}, zero_init, fc, Ready());
          walk_rows<true, true>(K0, Abs{xs}, zero_init, fr, Ready());
        } else {
          walk_rows<true, false>(T0, Abs{ys}, zero_init, fc, Ready());
          walk_rows<true, false>(K0, Abs{xs}, zero_init, fr, Ready());
        }
        cluster_sync(size);
        each_own(T0, [&](const At& at) {
          const double old = xs[at.p];
          ex.put_x(at, cn[at.p] > 0.0 ? old / sqrt(cn[at.p]) : old);
        });
        each_own(K0, [&](const At& at) {
          const double old = ys[at.p];
          ex.put_y(at, rn[at.p] > 0.0 ? old / sqrt(rn[at.p]) : old);
        });
        ok = ok && ex.wait(0) && ex.wait(1);
      }
    } else {
      // The reference's L2 Ruiz (pdlp.cpp:109-187).
      struct Sq2 {
        const double* o;
        __device__ double operator()(double a, int j) const {
          const double v = a * o[j];
          return v * v;
        }
      };
      for (int pass = 0; pass < 10; ++pass) {
        walk_rows<true, false>(T0, Sq2{ys}, zero_init,
                               [&](const At& at, double s) { cn[at.p] = sqrt(s) * xs[at.p]; }, Ready());
        walk_rows<true, false>(K0, Sq2{xs}, zero_init,
                               [&](const At& at, double s) { rn[at.p] = sqrt(s) * ys[at.p]; }, Ready());
        cluster_sync(size);
        double changed[1] = {0.0};
        auto rescaled = [&](double old, double nv) {
          if (!(nv > 0)) return old;
          const double s = fmax(1e-8, fmin(1e8, old / nv));
          if (fabs(s - old) / fmax(fabs(old), 1.0) > 0.1) changed[0] = 1.0;
          return s;
        };
        each_own(T0, [&](const At& at) { ex.put_x(at, rescaled(xs[at.p], cn[at.p])); });
        each_own(K0, [&](const At& at) { ex.put_y(at, rescaled(ys[at.p], rn[at.p])); });
        ok = ok && ex.wait(0) && ex.wait(1);
        cluster_reduce<1, 1u>(changed, sh, rank, size);
        if (changed[0] == 0.0) break;
      }
    }
  }
  // A_eq: K entries (a rs_i) cs_j, K' entries (a cs_j) rs_i; the scales by position.
  double* kv = b.k_val + M.kz;
  double* tv = b.t_val + M.tz;
  {
    auto scale_rows = [&](const Share& A, const double* own, const double* other,
                          double* out, float* out32, double* scale) {
      const int lane = threadIdx.x & 31;
      const int stride = 1 << A.slice;
      for (int ls = threadIdx.x >> 5;; ls += blockDim.x >> 5) {
        const int first = (ls * static_cast<int>(size) + static_cast<int>(rank)) << A.slice;
        if (first >= A.rows) break;
        const int p = first + lane;
        const bool valid = lane < stride && p < A.rows;
        int2 sl = make_int2(0, 0);
        double own_scale = 0.0;
        if (valid) {
          sl = __ldg(A.sl + p);
          own_scale = own[p];
          scale[p] = own_scale;
        }
        auto put = [&](int q, double sc) {
          const double v = __ldg(A.val + q) * sc * other[__ldg(A.idx + q)];
          out[q] = v;
          if (out32 != nullptr) out32[q] = static_cast<float>(v);
        };
        if (sl.y <= 32) {
          for (int k = 0; k < sl.y; ++k) put(A.place(sl, k), own_scale);
        }
        unsigned pending = __ballot_sync(0xffffffffu, sl.y > 32);
        while (pending != 0u) {
          const int src = __ffs(pending) - 1;
          pending &= pending - 1u;
          const int at = __shfl_sync(0xffffffffu, sl.x, src);
          const int len = __shfl_sync(0xffffffffu, sl.y, src);
          const double sc = __shfl_sync(0xffffffffu, own_scale, src);
          for (int k = lane; k < len; k += 32) put(at + k, sc);
        }
      }
    };
    scale_rows(K0, ys, xs, kv, b.fp32 ? b.k_val32 + M.kz : nullptr, rs);
    scale_rows(T0, xs, ys, tv, b.fp32 ? b.t_val32 + M.tz : nullptr, cs);
  }
  cluster_sync(size);
  // Power iteration (pdlp.cpp:36-103): ys holds u, xs holds v = A_eq' u.
  double L = 1.0;
  if (m > 0) {
    Share K = K0;
    K.val = kv;
    Share T = T0;
    T.val = tv;
    double ss[1] = {0.0};
    each_own(K, [&](const At& at) {
      const double u = b.power_start[M.kperm[at.p]];
      ss[0] += u * u;
    });
    cluster_reduce<1>(ss, sh, rank, size);
    double un = sqrt(ss[0]);
    each_own(K, [&](const At& at) { ex.put_y(at, b.power_start[M.kperm[at.p]] / un); });
    ok = ok && ex.wait(1);
    double sigma = 0.0;
    bool zero = false;
    for (int it = 0; it < 20; ++it) {
      double acc[1] = {0.0};
      walk_rows<false, false>(T, GatherT<double>{ys}, zero_init, [&](const At& at, double s) {
        ex.put_x(at, s);
        acc[0] += s * s;
      }, Ready());
      ok = ok && ex.wait(0);
      cluster_reduce<1>(acc, sh, rank, size);
      const double vn = sqrt(acc[0]);
      if (vn == 0.0) {
        zero = true;
        break;
      }
      // u = A_eq v, kept unscaled in rn until its norm is known.
      acc[0] = 0.0;
      walk_rows<false, false>(K, GatherT<double>{xs}, zero_init, [&](const At& at, double s) {
        rn[at.p] = s;
        acc[0] += s * s;
      }, Ready());
      cluster_reduce<1>(acc, sh, rank, size);
      un = sqrt(acc[0]);
      if (un == 0.0) {
        zero = true;
        break;
      }
      sigma = un / vn;
      const double inv = 1.0 / un;
      each_own(K, [&](const At& at) { ex.put_y(at, rn[at.p] * inv); });
      ok = ok && ex.wait(1);
    }
    if (!zero) {
      const double la = sigma * 1.01;
      L = sqrt(la * la + 1.0);
    }
  }
  __syncthreads();
  each_own(T0, [&](const At& at) { ics[at.p] = 1.0 / cs[at.p]; });
  each_own(K0, [&](const At& at) { irs[at.p] = 1.0 / rs[at.p]; });
  if (threadIdx.x == 0 && !ok) atomicExch(b.wait_error, 1);
  if (rank == 0 && threadIdx.x == 0) {
    MatInfo* info = b.info + g;
    info->eta = 0.99 / L;
    info->a_norm_max_col = norms[0];
    info->at_norm_max_row = norms[1];
  }
}

}  // namespace

template <int WALK, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kThreads64 ? 2 : 1)
    batch_setup_kernel(BatchView b, unsigned smem_bytes) {
  __shared__ ClusterShared sh;
  const unsigned rank = cluster_rank();
  const unsigned size = cluster_size();
  cluster_init(sh, size);
  const int g = blockIdx.x / size;
  if (cluster_vector_bytes(b.mat_n[g], b.mat_m[g], b.mat_slice[2 * g + 1], b.mat_slice[2 * g],
                           static_cast<int>(size), sizeof(double)) <= smem_bytes) {
    setup_matrix<kVectorsShared, WALK>(b, g, sh, rank, size);
  } else if constexpr (WALK == kWalkOne) {
    setup_matrix<kInDevice, WALK>(b, g, sh, rank, size);
  }
  cluster_sync(size);  // no CTA leaves while another may still send to it
}

__global__ void batch_deadline_kernel(unsigned long long* word, unsigned long long budget_ns) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  *word = budget_ns == 0ull ? 0ull : globaltimer_ns() + budget_ns;
}

// The groups run side by side: a later group's clusters start as the earlier one's end.
cudaError_t launch_batch(const BatchView& b, const ClusterPlan& setup, const ClusterPlan& solve,
                         unsigned long long budget_ns, const GroupStreams& gs, cudaStream_t s) {
  batch_deadline_kernel<<<1, 32, 0, s>>>(const_cast<unsigned long long*>(b.deadline), budget_ns);
  cudaMemsetAsync(b.queue, 0, kModes * sizeof(unsigned), s);
  cudaError_t e = launch_batch_setup(b, setup, s);
  return for_groups(solve, gs, s, e, [&](int mode, cudaStream_t gst) {
    return b.fp32 ? launch_solve32(b, solve, mode, gst) : launch_solve64(b, solve, mode, gst);
  });
}

namespace {

auto setup_kernel(const ClusterPlan& p) {
  return p.small                       ? batch_setup_kernel<kWalkLanes, kThreads64>
         : p.threads[0] == kThreads64 ? batch_setup_kernel<kWalkOne, kThreads64>
                                       : batch_setup_kernel<kWalkOne, kThreads64Large>;
}

}  // namespace

bool setup_fits(const ClusterPlan& p) {
  return clusters_fit(setup_kernel(p), p.size, p.threads[0], p.smem[0]);
}

cudaError_t launch_batch_setup(const BatchView& b, const ClusterPlan& setup, cudaStream_t s) {
  return launch_clusters(setup_kernel(setup), setup.size, b.nmat, setup.threads[0], setup.smem[0], s,
                         b, static_cast<unsigned>(setup.smem[0]));
}

}  // namespace sg
