// The up to kCheckFrequency iterations between two evaluations of a small LP, in one launch of
// one thread-block cluster.
//
// Launched step by step, an iteration of a small LP is two kernels of five dependent L2 round
// trips each and two launches, 12-17 us whatever its size; here the iterates stay in the cluster's
// shared memory, the nonzeros in its L1 caches, and a half step ends in an exchange: 5.4 us for a
// random LP of 200 x 500 (FP64, bound by the exchanges and the loads' latency), 10.6 for one of
// 5,000 x 10,000 (bound by the FP64 pipes of 16 SMs). Engine::plan_chunk says where it is taken.
#include "sg_chunk.cuh"
#include "sg_cluster_steps.cuh"

namespace sg {

namespace {

constexpr int kChunkThreads = 512;

template <typename T, bool HALPERN>
__global__ void __launch_bounds__(kChunkThreads, 1)
    chunk_kernel(Ctl* ctl, ChunkView<T> c, IterView<T> it) {
  constexpr int MODE = kAllShared;
  constexpr bool kF64 = sizeof(T) == 8;
  __shared__ ClusterShared sh;
  __shared__ StepContext<T, MODE> ctx;
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
  MatShare<T> M;
  M.m = c.m;
  M.n = n;
  M.kz = M.tz = 0;
  M.kperm = c.K.perm;
  M.tperm = c.Kt.perm;
  M.K = RowShare<T>{c.K.sl, c.K.desc, c.K.idx, c.K.val, c.m, c.K.slice, rank, size};
  M.Kt = RowShare<T>{c.Kt.sl, c.Kt.desc, c.Kt.idx, c.Kt.val, n, c.Kt.slice, rank, size};
  M.nr = M.K.own();
  M.nc = M.Kt.own();
  const Second<T> Z{c.second, n, c.m};
  const Exchange<T, MODE> ex = make_exchange<T, MODE>(M, sh, nullptr, rank, size);
  SolveState<T, MODE> S;
  S.device = nullptr;
  S.rows_device = 0;
  S.cols_at = static_cast<unsigned>(cluster_vector_bytes(n, c.m, c.Kt.slice, c.K.slice,
                                                         static_cast<int>(size), sizeof(T)));
  S.rows_at = S.cols_at + M.Kt.slices() * static_cast<unsigned>(32 * kColArrays * sizeof(T));
  S.rank = rank;
  S.size = size;
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
    S.col(kPoint, at) = v[j];
    S.col(kSum, at) = HALPERN ? it.Vrst[j] : sum_of(it.Verg[j]);
    S.col(kCost, at) = it.cost[j];
    S.col(kLower, at) = it.xb_uniform ? it.xb_lo : it.lower[j];
    S.col(kUpper, at) = it.xb_uniform ? it.xb_hi : it.upper[j];
    if (!HALPERN) ex.put_x(at, it.Vbar[j]);
  });
  each_own(M.K, [&](const At& at) {
    const int i = M.kperm[at.p];
    const int q = n + i;
    S.row(kPoint, at) = v[q];
    S.row(kCost, at) = it.cost[q];
    S.row(kLower, at) = it.lower[q];
    S.row(kUpper, at) = it.upper[q];
    S.row(kDual, at) = y[i];
    if (HALPERN) {
      S.row(kSum, at) = it.Vrst[q];
      S.row(kDualSum, at) = it.Yrst[i];
      ex.put_y(at, y[i]);
    } else {
      S.row(kSum, at) = sum_of(it.Verg[q]);
      S.row(kDualSum, at) = sum_of(it.Yerg[i]);
      S.row(kBar, at) = -it.Vbar[q];
    }
  });
  __syncthreads();
  bool ok = run_steps<T, MODE, HALPERN>(
      &ctx, steps, static_cast<T>(ctl->tau), static_cast<T>(ctl->sigma), [&] {
        // The other buffers hold the iterate before the last.
        const int other = static_cast<int>((t + steps + 1) & 1);
        __syncthreads();
        each_own(ctx.M.Kt, [&](const At& at) {
          it.v(other)[ctx.M.tperm[at.p]] = ctx.S.col(kPoint, at);
        });
        each_own(ctx.M.K, [&](const At& at) {
          const int i = ctx.M.kperm[at.p];
          it.v(other)[ctx.M.n + i] = ctx.S.row(kPoint, at);
          it.y(other)[i] = ctx.S.row(kDual, at);
        });
      });
  ok = ok && ex.wait(HALPERN ? 1 : 0);
  if (ok) {
    const int now = static_cast<int>((t + steps) & 1);
    const T inv = T(1) / static_cast<T>(k0 + steps);
    auto average_of = [&](T sum) { return kF64 ? sum * inv : sum; };
    each_own(M.Kt, [&](const At& at) {
      const int j = M.tperm[at.p];
      it.v(now)[j] = S.col(kPoint, at);
      it.Vbar[j] = ex.xs()[at.p];
      it.Verg[j] = HALPERN ? Z.x(at.p) : average_of(S.col(kSum, at));
    });
    each_own(M.K, [&](const At& at) {
      const int i = M.kperm[at.p];
      const int q = n + i;
      it.v(now)[q] = S.row(kPoint, at);
      it.y(now)[i] = S.row(kDual, at);
      if (HALPERN) {
        it.Verg[q] = Z.r(at.p);
        it.Yerg[i] = Z.y(at.p);
      } else {
        const T lo = S.row(kLower, at);
        it.Vbar[q] = -S.row(kBar, at);
        it.Yerg[i] = average_of(S.row(kDualSum, at));
        // An FP64 step leaves the sums of equality rows, whose logicals are their bound from
        // the first step on, to this.
        it.Verg[q] = kF64 && lo == S.row(kUpper, at)
                         ? average_of(sum_of(it.Verg[q]) + static_cast<T>(steps) * lo)
                         : average_of(S.row(kSum, at));
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
    const ClusterOp<T>& C = rows ? c.K : c.Kt;
    const int* other = rows ? c.Kt.pos : c.K.pos;
    const int b = A.ptr[r];
    const int2 sl = C.sl[C.pos[r]];
    for (int k = lane; k < sl.y; k += 32) {
      const int at = nonzero_at(sl.x, sl.y, k);
      if constexpr (INDICES) {
        C.idx[at] = other[A.idx[b + k]];
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

size_t chunk_smem_bytes(int n, int m, int tslice, int kslice, int size, size_t elem) {
  return cluster_vector_bytes(n, m, tslice, kslice, size, elem) +
         solve_state_bytes(share_rows(n, tslice, size) >> tslice,
                           share_rows(m, kslice, size) >> kslice, elem);
}

bool chunk_fits(size_t smem) { return smem <= kClusterSmemMax; }

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

template void launch_chunk_indices<double>(const ChunkView<double>&, const OpView<double>&,
                                           const OpView<double>&, cudaStream_t);
template void launch_chunk_values<double>(const ChunkView<double>&, const OpView<double>&,
                                          const OpView<double>&, cudaStream_t);
template void launch_chunk_values<float>(const ChunkView<float>&, const OpView<float>&,
                                         const OpView<float>&, cudaStream_t);
template cudaError_t launch_chunk<double>(Ctl*, const ChunkView<double>&, const IterView<double>&,
                                          bool, cudaStream_t);
template cudaError_t launch_chunk<float>(Ctl*, const ChunkView<float>&, const IterView<float>&,
                                         bool, cudaStream_t);

}  // namespace sg
