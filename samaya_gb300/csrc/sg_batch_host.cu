// Host side of the batched PDLP engine (see sg_batch.cu).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <functional>
#include <limits>
#include <mutex>
#include <numeric>
#include <queue>
#include <random>
#include <set>
#include <tuple>
#include <utility>

#include "../../include/sg_pdlp.h"
#include "sg_batch.cuh"
#include "sg_cluster_layout.h"

namespace sg {

bool known_to_fit(const void* kernel, int device, int size, int threads, bool add) {
  static std::mutex mu;
  static std::set<std::tuple<const void*, int, int, int>> known;  // kernels x devices x sizes
  std::lock_guard<std::mutex> lock(mu);
  const std::tuple<const void*, int, int, int> key{kernel, device, size, threads};
  if (add) known.insert(key);
  return known.count(key) != 0;
}

template <typename T>
int Batch::alloc(T** p, size_t count) {
  *p = nullptr;
  const cudaError_t e =
      cudaMalloc(reinterpret_cast<void**>(p), std::max<size_t>(count, 1) * sizeof(T));
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported here, not by the next call
    return e == cudaErrorMemoryAllocation ? SG_ERR_OUT_OF_MEMORY : SG_ERR_CUDA;
  }
  allocs_.push_back(*p);
  return SG_OK;
}

Batch::~Batch() {
  if (stream_) cudaStreamSynchronize(stream_);
  for (void* p : allocs_) cudaFree(p);
  for (void* p : {static_cast<void*>(u_.ck), static_cast<void*>(u_.mask),
                  const_cast<void*>(static_cast<const void*>(u_.ck_off)),
                  const_cast<void*>(static_cast<const void*>(u_.mask_off))}) {
    if (p) cudaFree(p);
  }
  if (wait_host_) cudaFreeHost(wait_host_);
  if (groups_.fork) cudaEventDestroy(groups_.fork);
  for (int mode = 0; mode < kModes; ++mode) {
    if (groups_.join[mode]) cudaEventDestroy(groups_.join[mode]);
    if (groups_.stream[mode]) cudaStreamDestroy(groups_.stream[mode]);
  }
  if (stream_) cudaStreamDestroy(stream_);
}

#define SG_B_TRY(call)                                     \
  do {                                                     \
    const int rc_ = (call);                                \
    if (rc_ != SG_OK) {                                    \
      if (err) *err = std::string("batch: ") + #call;     \
      delete b;                                            \
      return rc_;                                          \
    }                                                      \
  } while (0)

#define SG_B_CUDA(call)                                                              \
  do {                                                                               \
    const cudaError_t e_ = (call);                                                   \
    if (e_ != cudaSuccess) {                                                         \
      if (err) *err = std::string(#call) + ": " + cudaGetErrorString(e_);           \
      delete b;                                                                      \
      return e_ == cudaErrorMemoryAllocation ? SG_ERR_OUT_OF_MEMORY : SG_ERR_CUDA; \
    }                                                                                \
  } while (0)

int Batch::create(Batch** out, int nmat, const int* mat_m, const int* mat_n,
                  const int64_t* mat_colptr, const int32_t* mat_rowidx, const double* mat_val,
                  int count, const int* inst_mat, const double* cost, const double* lower,
                  const double* upper, double tol, long long max_iter, double time_limit,
                  int precision, int algorithm, std::string* err) {
  *out = nullptr;
  if (nmat <= 0 || count <= 0 || mat_m == nullptr || mat_n == nullptr || mat_colptr == nullptr ||
      inst_mat == nullptr || cost == nullptr || lower == nullptr || upper == nullptr) {
    if (err) *err = "invalid argument";
    return SG_ERR_INVALID_ARGUMENT;
  }
  // Host layout of the matrices.
  std::vector<long long> nnz_off(nmat + 1, 0), col_off(nmat + 1, 0), row_off(nmat + 1, 0),
      cp_off(nmat + 1, 0);
  for (int g = 0; g < nmat; ++g) {
    if (mat_m[g] < 0 || mat_n[g] < 0) {
      if (err) *err = "negative dimension";
      return SG_ERR_INVALID_ARGUMENT;
    }
    cp_off[g + 1] = cp_off[g] + mat_n[g] + 1;
    const int64_t* cp = mat_colptr + cp_off[g];
    const long long nnz = cp[mat_n[g]];
    if (cp[0] != 0 || nnz < 0 || nnz >= std::numeric_limits<int>::max()) {
      if (err) *err = "bad column starts";
      return SG_ERR_INVALID_ARGUMENT;
    }
    for (int j = 0; j < mat_n[g]; ++j) {
      if (cp[j + 1] < cp[j]) {
        if (err) *err = "column starts decrease";
        return SG_ERR_INVALID_ARGUMENT;
      }
    }
    nnz_off[g + 1] = nnz_off[g] + nnz;
    col_off[g + 1] = col_off[g] + mat_n[g];
    row_off[g + 1] = row_off[g] + mat_m[g];
  }
  const long long total_nnz = nnz_off[nmat];
  if (total_nnz > 0 && (mat_rowidx == nullptr || mat_val == nullptr)) {
    if (err) *err = "null matrix arrays";
    return SG_ERR_INVALID_ARGUMENT;
  }
  // Per matrix: the rows of A and of A' in their order (sg_cluster_layout.h), then the elements,
  // each operator's column numbers replaced by the other's positions.
  std::vector<StartLen> ksl(std::max(row_off[nmat], 1LL)), tsl(std::max(col_off[nmat], 1LL));
  std::vector<int> kperm(ksl.size()), tperm(tsl.size()), slice(2 * static_cast<size_t>(nmat));
  std::vector<long long> k_off(nmat + 1, 0), t_off(nmat + 1, 0), kd_off(nmat + 1, 0),
      td_off(nmat + 1, 0);
  std::vector<StartLen> kdesc, tdesc;
  std::vector<RowOrder> korder(nmat), torder(nmat);
  std::vector<std::vector<int>> kptr(nmat);
  int max_m = 0;
  // LPs of at most 512 rows and columns take several lanes a row (kWalkLanes; 32 >> slice): 64
  // unrolled LPs of 40 x 88, 200 iterations forward and backward, 2.54 ms with a lane a row, 1.95
  // now, of 110 x 242 2.83 and 2.47; 160 solves of 60 x 120, 192 iterations, 1.82 and 1.64 in FP64,
  // 1.59 and 1.52 in FP32. (Kernels that allow for both took 1% longer on the larger ones.)
  bool small = true;
  for (int g = 0; g < nmat; ++g) {
    small = small && static_cast<long long>(mat_m[g]) + mat_n[g] <= 512;
  }
  for (int g = 0; g < nmat; ++g) {
    const int m = mat_m[g], n = mat_n[g];
    max_m = std::max(max_m, m);
    const int64_t* cp = mat_colptr + cp_off[g];
    const int32_t* ri = mat_rowidx + nnz_off[g];
    const double* va = mat_val + nnz_off[g];
    for (long long p = 0; p < cp[n]; ++p) {
      if (ri[p] < 0 || ri[p] >= m || !std::isfinite(va[p])) {
        if (err) *err = "bad matrix entry";
        return SG_ERR_INVALID_ARGUMENT;
      }
    }
    std::vector<int>& kp = kptr[g];
    kp.assign(static_cast<size_t>(m) + 1, 0);
    for (long long p = 0; p < cp[n]; ++p) ++kp[ri[p] + 1];
    for (int i = 0; i < m; ++i) kp[i + 1] += kp[i];
    std::vector<int> tp(static_cast<size_t>(n) + 1);
    for (int j = 0; j <= n; ++j) tp[j] = static_cast<int>(cp[j]);
    korder[g] = order_rows(kp.data(), m, small);
    torder[g] = order_rows(tp.data(), n, small);
    slice[2 * g] = korder[g].slice;
    slice[2 * g + 1] = torder[g].slice;
    kd_off[g + 1] = kd_off[g] + slices_of(korder[g]);
    td_off[g + 1] = td_off[g] + slices_of(torder[g]);
    kdesc.resize(kd_off[g + 1]);
    tdesc.resize(td_off[g + 1]);
    const long long kn =
        place_rows(kp.data(), korder[g], ksl.data() + row_off[g], kdesc.data() + kd_off[g]);
    const long long tn =
        place_rows(tp.data(), torder[g], tsl.data() + col_off[g], tdesc.data() + td_off[g]);
    if (kn >= std::numeric_limits<int>::max() || tn >= std::numeric_limits<int>::max()) {
      if (err) *err = "matrix too large for 32-bit offsets";
      return SG_ERR_TOO_LARGE;
    }
    k_off[g + 1] = k_off[g] + kn;
    t_off[g + 1] = t_off[g] + tn;
    std::copy(korder[g].perm.begin(), korder[g].perm.end(), kperm.begin() + row_off[g]);
    std::copy(torder[g].perm.begin(), torder[g].perm.end(), tperm.begin() + col_off[g]);
  }
  std::vector<int> kidx(std::max(k_off[nmat], 1LL)), tidx(std::max(t_off[nmat], 1LL));
  std::vector<double> kval(kidx.size()), tval(tidx.size());
  for (int g = 0; g < nmat; ++g) {
    const int n = mat_n[g];
    const int64_t* cp = mat_colptr + cp_off[g];
    const int32_t* ri = mat_rowidx + nnz_off[g];
    const double* va = mat_val + nnz_off[g];
    std::fill(kidx.begin() + k_off[g], kidx.begin() + k_off[g + 1], n);  // padding
    std::fill(tidx.begin() + t_off[g], tidx.begin() + t_off[g + 1], mat_m[g]);
    std::vector<int> done(static_cast<size_t>(mat_m[g]), 0);  // nonzeros of each row placed
    for (int j = 0; j < n; ++j) {
      const int tpos = torder[g].pos[j];
      const StartLen& ts = tsl[col_off[g] + tpos];
      for (long long p = cp[j]; p < cp[j + 1]; ++p) {
        const int kpos = korder[g].pos[ri[p]];
        const long long tq = t_off[g] + place_of(ts, static_cast<int>(p - cp[j]), torder[g]);
        tidx[tq] = kpos;
        tval[tq] = va[p];
        const long long kq =
            k_off[g] + place_of(ksl[row_off[g] + kpos], done[ri[p]]++, korder[g]);
        kidx[kq] = tpos;
        kval[kq] = va[p];
      }
    }
  }
  // Instances.
  std::vector<long long> vec_off(count + 1, 0), yrow_off(count + 1, 0), state_off(count + 1, 0);
  const size_t tsz = precision == 1 ? sizeof(float) : sizeof(double);
  for (int i = 0; i < count; ++i) {
    const int g = inst_mat[i];
    if (g < 0 || g >= nmat) {
      if (err) *err = "instance matrix out of range";
      return SG_ERR_INVALID_ARGUMENT;
    }
    const long long nt = static_cast<long long>(mat_n[g]) + mat_m[g];
    vec_off[i + 1] = vec_off[i] + nt;
    yrow_off[i + 1] = yrow_off[i] + mat_m[g];
    // Keep every instance's block 16-byte aligned.
    long long elems = instance_elements(mat_n[g], mat_m[g], slice[2 * g + 1], slice[2 * g],
                                        precision == 1);
    const long long align = 16 / static_cast<long long>(tsz);
    elems = (elems + align - 1) / align * align;
    state_off[i + 1] = state_off[i] + elems;
  }
  for (long long k = 0; k < vec_off[count]; ++k) {
    if (!std::isfinite(cost[k]) || std::isnan(lower[k]) || std::isnan(upper[k])) {
      if (err) *err = "cost or bound not valid";
      return SG_ERR_INVALID_ARGUMENT;
    }
  }
  // Largest instances first.
  std::vector<int> order(count);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) {
    const long long wa = nnz_off[inst_mat[a] + 1] - nnz_off[inst_mat[a]] + vec_off[a + 1] - vec_off[a];
    const long long wc = nnz_off[inst_mat[c] + 1] - nnz_off[inst_mat[c]] + vec_off[c + 1] - vec_off[c];
    return wa > wc;
  });
  std::vector<double> u0(std::max(max_m, 1));
  {
    // The reference's power-iteration start (pdlp.cpp:47-51).
    std::mt19937_64 rng(12345);
    std::uniform_real_distribution<double> dist(-1.0, 1.0);
    for (int i = 0; i < max_m; ++i) u0[i] = dist(rng);
  }
  int dev_count = 0;
  if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count <= 0) {
    cudaGetLastError();
    if (err) *err = "no GPU";
    return SG_ERR_NO_DEVICE;
  }
  Batch* b = new Batch();
  b->time_limit_ = time_limit;
  b->total_vec_ = vec_off[count];
  b->total_rows_ = yrow_off[count];
  b->vec_off_host_ = vec_off;
  b->inst_nt_host_.resize(count);
  b->inst_m_host_.resize(count);
  for (int i = 0; i < count; ++i) {
    b->inst_nt_host_[i] = static_cast<int>(vec_off[i + 1] - vec_off[i]);
    b->inst_m_host_[i] = mat_m[inst_mat[i]];
  }
  SG_B_CUDA(cudaStreamCreateWithFlags(&b->stream_, cudaStreamNonBlocking));
  BatchView& v = b->v_;
  v.nmat = nmat;
  v.count = count;
  auto up = [&](auto** dst, const auto* src, size_t n) -> int {
    using E = std::remove_const_t<std::remove_reference_t<decltype(*src)>>;
    E* d = nullptr;
    int rc = b->alloc(&d, n);
    if (rc != SG_OK) return rc;
    if (n > 0 && cudaMemcpy(d, src, n * sizeof(E), cudaMemcpyHostToDevice) != cudaSuccess) {
      return SG_ERR_CUDA;
    }
    *dst = d;
    return SG_OK;
  };
  int* d_mm = nullptr;
  int* d_mn = nullptr;
  long long *d_ko = nullptr, *d_to = nullptr, *d_co = nullptr, *d_ro = nullptr;
  SG_B_TRY(up(&d_mm, mat_m, nmat));
  SG_B_TRY(up(&d_mn, mat_n, nmat));
  SG_B_TRY(up(&d_ko, k_off.data(), nmat + 1));
  SG_B_TRY(up(&d_to, t_off.data(), nmat + 1));
  SG_B_TRY(up(&d_co, col_off.data(), nmat + 1));
  SG_B_TRY(up(&d_ro, row_off.data(), nmat + 1));
  v.mat_m = d_mm;
  v.mat_n = d_mn;
  v.mat_k_off = d_ko;
  v.mat_t_off = d_to;
  v.mat_col_off = d_co;
  v.mat_row_off = d_ro;
  int *d_ki = nullptr, *d_ti = nullptr, *d_kperm = nullptr, *d_tperm = nullptr, *d_sl = nullptr;
  StartLen *d_ksl = nullptr, *d_tsl = nullptr, *d_kdesc = nullptr, *d_tdesc = nullptr;
  long long *d_kdo = nullptr, *d_tdo = nullptr;
  double *d_kv0 = nullptr, *d_tv0 = nullptr;
  SG_B_TRY(up(&d_ksl, ksl.data(), ksl.size()));
  SG_B_TRY(up(&d_tsl, tsl.data(), tsl.size()));
  SG_B_TRY(up(&d_kdesc, kdesc.data(), kdesc.size()));
  SG_B_TRY(up(&d_tdesc, tdesc.data(), tdesc.size()));
  SG_B_TRY(up(&d_kdo, kd_off.data(), nmat + 1));
  SG_B_TRY(up(&d_tdo, td_off.data(), nmat + 1));
  SG_B_TRY(up(&d_kperm, kperm.data(), kperm.size()));
  SG_B_TRY(up(&d_tperm, tperm.data(), tperm.size()));
  SG_B_TRY(up(&d_sl, slice.data(), slice.size()));
  SG_B_TRY(up(&d_ki, kidx.data(), kidx.size()));
  SG_B_TRY(up(&d_ti, tidx.data(), tidx.size()));
  SG_B_TRY(up(&d_kv0, kval.data(), kval.size()));
  SG_B_TRY(up(&d_tv0, tval.data(), tval.size()));
  static_assert(sizeof(StartLen) == sizeof(int2), "row starts layout");
  v.k_sl = reinterpret_cast<const int2*>(d_ksl);
  v.t_sl = reinterpret_cast<const int2*>(d_tsl);
  v.k_desc = reinterpret_cast<const int2*>(d_kdesc);
  v.t_desc = reinterpret_cast<const int2*>(d_tdesc);
  v.mat_kd_off = d_kdo;
  v.mat_td_off = d_tdo;
  v.k_perm = d_kperm;
  v.t_perm = d_tperm;
  v.mat_slice = d_sl;
  v.k_idx = d_ki;
  v.t_idx = d_ti;
  v.k_val0 = d_kv0;
  v.t_val0 = d_tv0;
  SG_B_TRY(b->alloc(&v.k_val, kval.size()));
  SG_B_TRY(b->alloc(&v.t_val, tval.size()));
  v.fp32 = precision == 1 ? 1 : 0;
  if (v.fp32) {
    SG_B_TRY(b->alloc(&v.k_val32, kval.size()));
    SG_B_TRY(b->alloc(&v.t_val32, tval.size()));
  }
  SG_B_TRY(b->alloc(&v.cs, col_off[nmat]));
  SG_B_TRY(b->alloc(&v.rs, row_off[nmat]));
  SG_B_TRY(b->alloc(&v.ics, col_off[nmat]));
  SG_B_TRY(b->alloc(&v.irs, row_off[nmat]));
  v.spill = nullptr;
  for (int g = 0; g < nmat && v.spill == nullptr; ++g) {
    if (cluster_vector_bytes(mat_n[g], mat_m[g], slice[2 * g + 1], slice[2 * g], 1,
                             sizeof(double)) > kClusterSmemMax) {
      SG_B_TRY(b->alloc(&v.spill, col_off[nmat] + row_off[nmat] + 2 * nmat));
    }
  }
  SG_B_TRY(b->alloc(&v.info, nmat));
  const double* d_u0 = nullptr;
  SG_B_TRY(up(&d_u0, u0.data(), u0.size()));
  v.power_start = d_u0;
  int* d_im = nullptr;
  long long *d_vo = nullptr, *d_yo = nullptr, *d_so = nullptr;
  double *d_c = nullptr, *d_l = nullptr, *d_u = nullptr;
  SG_B_TRY(up(&d_im, inst_mat, count));
  SG_B_TRY(up(&d_vo, vec_off.data(), count + 1));
  SG_B_TRY(up(&d_yo, yrow_off.data(), count + 1));
  SG_B_TRY(up(&d_so, state_off.data(), count + 1));
  SG_B_TRY(up(&d_c, cost, vec_off[count]));
  SG_B_TRY(up(&d_l, lower, vec_off[count]));
  SG_B_TRY(up(&d_u, upper, vec_off[count]));
  v.inst_mat = d_im;
  v.vec_off = d_vo;
  v.row_off = d_yo;
  v.state_off = d_so;
  v.cost = d_c;
  v.lower = d_l;
  v.upper = d_u;
  unsigned char* st = nullptr;
  SG_B_TRY(b->alloc(&st, static_cast<size_t>(state_off[count]) * tsz));
  v.state = st;
  SG_B_TRY(b->alloc(&v.x_out, vec_off[count]));
  SG_B_TRY(b->alloc(&v.y_out, yrow_off[count]));
  SG_B_TRY(b->alloc(&v.results, count));
  SG_B_TRY(b->alloc(&v.queue, kModes));
  unsigned long long* dl = nullptr;
  SG_B_TRY(b->alloc(&dl, 1));
  v.deadline = dl;
  SG_B_TRY(b->alloc(&v.wait_error, 1));
  SG_B_CUDA(cudaMemset(v.wait_error, 0, sizeof(int)));
  SG_B_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&b->wait_host_), sizeof(int),
                          cudaHostAllocDefault));
  v.max_iter = max_iter;
  v.tol = tol;
  v.algorithm = algorithm == 1 || algorithm == 2 ? algorithm : 0;
  // The reference's 0.36 for its own algorithm; the Halpern iteration restarts at 0.1, as the
  // single-LP engine does (the enhanced PDHG keeps 0.36 here: measured no faster at 0.1 on the
  // batched node relaxations).
  v.art_frac = v.algorithm == 2 ? 0.1 : 0.36;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&b->sms_, cudaDevAttrMultiProcessorCount, dev);
  b->mat_m_.assign(mat_m, mat_m + nmat);
  b->mat_n_.assign(mat_n, mat_n + nmat);
  b->inst_mat_.assign(inst_mat, inst_mat + count);
  b->mat_slice_ = slice;
  b->small_ = small;
  b->mat_nnz_.resize(nmat);
  for (int g = 0; g < nmat; ++g) b->mat_nnz_[g] = nnz_off[g + 1] - nnz_off[g];
  b->order_ = std::move(order);
  SG_B_TRY(b->make_plan(Kind::kSetup, &b->setup_plan_));
  SG_B_TRY(b->make_plan(Kind::kSolve, &b->solve_plan_));
  *out = b;
  return SG_OK;
}

// Cluster size, shared memory and clusters of one kernel: the size with the shortest estimated
// finish when the instances go to the clusters largest first. The estimate of an iteration, in
// microseconds, is fitted to measured ones of random LPs (FP64 from 100 x 250, FP32 from 20 x 50, to
// 5,000 x 10,000) and facility-location LPs, 1 to 600 of them, at every size (within 20%; e.g. FP64,
// 1 LP of 1,500 x 3,000: 34.9 / 20.0 / 10.4 / 7.4 / 6.7 with 1 / 2 / 4 / 8 / 16 CTAs; 160 LPs of 500 x
// 1,200: 15.3 / 17.6 / 21.5 / 32.2 / 84.9; FP32, 1 LP of 20 x 50: 1.7 / 2.2 / 2.2 / 2.4 / 2.9, of 2,000 x
// 5,000: 14.7 / 9.0 / 5.3 / 4.0 / 3.9).
int Batch::make_plan(Kind kind, ClusterPlan* plan) {
  auto holds = [&](const ClusterPlan& p) {
    if (p.size == 1) return true;
    switch (kind) {
      case Kind::kSetup: return setup_fits(p);
      case Kind::kSolve:
        return v_.fp32 ? solve32_fits(p, v_.algorithm) : solve64_fits(p, v_.algorithm);
      default: return unroll_fits(p, kind == Kind::kAdjoint);
    }
  };
  // Smaller clusters where the device cannot hold one of the size that suits best.
  std::vector<int> lists[kModes];
  for (int most = cluster_limit();; most = plan->size / 2) {
    plan_clusters(kind, most, plan, lists);
    if (holds(*plan)) break;
  }
  return upload_lists(lists, plan);
}

// The plan with clusters of at most `most` CTAs, and its instances by mode.
void Batch::plan_clusters(Kind kind, int most, ClusterPlan* plan, std::vector<int>* lists) {
  *plan = ClusterPlan();
  const bool setup = kind == Kind::kSetup;
  const bool fp32 = kind == Kind::kSolve && v_.fp32;
  const size_t elem = fp32 ? sizeof(float) : sizeof(double);
  const int count = setup ? static_cast<int>(mat_m_.size()) : v_.count;
  const size_t limit = fp32 ? kClusterSmemMax : kClusterSmemHalf;
  auto vector_bytes = [&](int g, int size) {
    return cluster_vector_bytes(mat_n_[g], mat_m_[g], mat_slice_[2 * g + 1], mat_slice_[2 * g],
                                size, elem);
  };
  auto all_bytes = [&](int g, int size) {
    const int ks = mat_slice_[2 * g], ts = mat_slice_[2 * g + 1];
    const long long kslices = share_rows(mat_m_[g], ks, size) >> ks;
    const long long tslices = share_rows(mat_n_[g], ts, size) >> ts;
    return vector_bytes(g, size) +
           (setup                  ? 0
            : kind == Kind::kSolve ? solve_state_bytes(tslices, kslices, elem)
                                   : unroll_state_bytes(tslices, kslices, kind == Kind::kAdjoint));
  };
  std::vector<std::pair<double, int>> work(count);  // an iteration's time by one CTA, the matrix
  bool fits = true;  // every instance's gathered vectors in shared memory
  double all_work = 0.0, alone_work = 0.0;  // of LPs whose vectors leave an SM no second CTA
  for (int i = 0; i < count; ++i) {
    const int g = setup ? i : inst_mat_[i];
    const double rows = static_cast<double>(mat_m_[g]) + mat_n_[g];
    const double nnz = static_cast<double>(mat_nnz_[g]);
    work[i] = {(fp32 ? 1.5e-4 : 5.6e-4) * (2 * nnz + 5 * rows), g};
    fits = fits && vector_bytes(g, 2) <= kClusterSmemMax;
    all_work += work[i].first;
    if (vector_bytes(g, 1) > kClusterSmemHalf) alone_work += work[i].first;
  }
  std::sort(work.begin(), work.end(), std::greater<std::pair<double, int>>());
  // Two FP64 CTAs share an SM, unless most of the work is in LPs whose vectors leave no room for a
  // second one: then one of 512 threads has it (128 iterations of facility-location LPs with 256 and with 512: 16 of
  // 60 x 240 7.8 and 4.7 ms, 64 of 100 x 400 72.0 and 42.5; 256 random LPs of 5,000 x 12,500 67.3 and
  // 42.8). With less of them the others' sharing counts for more: 512 LPs of 100 to 5,000 rows, 41% of the
  // work in such ones, to 1e-4, 3.18 s as two to an SM and 3.46 otherwise, Halpern 8.24 and 12.9. FP32
  // CTAs take an SM each.
  const bool alone = !fp32 && alone_work > 0.5 * all_work;
  const int per_sm = fp32 || alone ? 1 : 2;
  // The sizes' exchanges and epilogues.
  const int sizes[5] = {1, 2, 4, 8, 16};
  const double fixed64[5] = {0.7, 2.2, 3.4, 4.2, 5.2};
  const double fixed32[5] = {1.4, 2.0, 2.1, 2.6, 3.4};
  // The setup's passes end in reductions over the cluster (the same unit: a thirtieth of it; 64
  // LPs of 500 x 1,200: 0.66 / 0.55 / 0.61 / 1.09 ms with 1 / 2 / 4 / 8 CTAs).
  const double fixed_setup[5] = {5.5, 9.0, 9.9, 10.6, 11.3};
  const double* fixed = setup ? fixed_setup : fp32 ? fixed32 : fixed64;
  plan->size = 1;
  double best_time = -1.0;
  for (int k = 0; k < 5; ++k) {
    const int size = sizes[k];
    if (size > most || (size > 1 && !fits)) break;
    // Clusters at once (SMs of a GPC left over by clusters of 8 and 16: an eighth or more; a quarter
    // with an SM to a CTA, where 16 clusters of 8 no longer run side by side).
    const int whole = per_sm * sms_ / size;
    const int slots = std::max(1, whole - (size >= 8 ? whole / (per_sm == 1 ? 4 : 8) : 0));
    const bool shared_sm = per_sm == 2 && static_cast<long long>(std::min(count, slots)) * size > sms_;
    // Largest first, each to the cluster that is free first.
    std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
    for (int c = 0; c < std::min(count, slots); ++c) free_at.push(0.0);
    double end = 0.0;
    for (const auto& w : work) {
      const double own = w.first / size;
      double t = own + fixed[k];
      // The FP64 pipe of a shared SM; a state left in device memory (160 LPs of 2,000 x 4,000:
      // 72 us with 2 CTAs, 48 with 4, which hold it).
      if (shared_sm) t = setup ? 1.25 * t : std::max(t, 1.15 * own);
      if (!setup && per_sm == 2 && all_bytes(w.second, size) > limit) t *= 1.45;
      t += free_at.top();
      free_at.pop();
      free_at.push(t);
      end = std::max(end, t);
    }
    // (Where the state stays in device memory, a larger cluster's gain is partly the memory's: 256
    // nodes of 100 x 400 in FP32 54.1 ms with clusters of four, estimated alike, 42.8 with one CTA.)
    const bool close = fp32 && all_bytes(work[0].second, size) > limit;
    if (best_time < 0 || end < (close ? 0.95 : 1.0) * best_time) {
      best_time = end;
      plan->size = size;
    }
  }
  const int best = plan->size;
  plan->clusters = std::max(1, (fp32 ? 1 : 2) * sms_ / best);
  plan->sms = sms_;
  plan->small = small_;
  if (alone) plan->threads[kVectorsShared] = plan->threads[kInDevice] = kThreads64Large;
  if (setup) {
    plan->threads[0] = alone ? kThreads64Large : kThreads64;
    // One launch for all matrices; a matrix whose vectors do not fit leaves them in device
    // memory.
    for (int g = 0; g < count; ++g) {
      const size_t vec = vector_bytes(g, best);
      if (vec <= kClusterSmemMax) plan->smem[0] = std::max(plan->smem[0], vec);
    }
    return;
  }
  // Every instance in the mode that keeps the most in shared memory, FP64 ones within half of it
  // (two CTAs to an SM) as long as their vectors allow that.
  for (int mode = 0; mode < kModes; ++mode) lists[mode].clear();
  int most_rows = 0;
  for (int i : order_) {
    const int g = inst_mat_[i];
    const size_t vec = vector_bytes(g, best);
    const size_t all = all_bytes(g, best);
    const int mode = all <= limit             ? kAllShared
                     : vec <= kClusterSmemMax ? kVectorsShared
                                              : kInDevice;
    const size_t need = mode == kAllShared ? all : mode == kVectorsShared ? vec : 0;
    lists[mode].push_back(i);
    plan->smem[mode] = std::max(plan->smem[mode], need);
    ++plan->group[mode].count;
    if (mode == kAllShared) most_rows = std::max(most_rows, (mat_m_[g] + mat_n_[g]) / best);
  }
  if (!fp32) return;
  // Threads of an FP32 CTA by the largest LP's rows and columns a CTA. Few: 256 threads, all in
  // registers (every kernel of 512 spilled, the averaging one 1,600 bytes of loads a thread, and an
  // iteration of 64 LPs of 60 x 120 took 6.9 us; so 2.3). More: 384 (256 LPs of facility location
  // 40 x 120, averaging, 192 iterations: 10.6 ms with 256, 7.1 with 384, 8.6 with 512). The Halpern
  // iteration, whose rows take fewer registers, has use for 512 from 3,000 on, to hide the loads of
  // longer rows (facility location 40 x 80 5.4 with 384, 5.3 with 512; 40 x 160 11.2 and 10.0; but
  // 160 random LPs of 1,200 x 3,000 6.8 and 7.6).
  const bool halpern = v_.algorithm == 2;
  plan->threads[kAllShared] = most_rows <= 1600             ? kThreads32Few
                              : !halpern || most_rows < 3000 ? kThreads32Mid
                                                             : kThreads32;
  plan->threads[kVectorsShared] = plan->threads[kInDevice] = kThreads32;
}

int Batch::upload_lists(const std::vector<int>* lists, ClusterPlan* plan) {
  // (Small LPs' vectors and state are 60 KB at most.)
  if (plan->small && !(lists[kInDevice].empty() && lists[kVectorsShared].empty())) {
    return SG_ERR_INTERNAL;
  }
  int used = 0;
  for (int mode = 0; mode < kModes; ++mode) {
    if (lists[mode].empty()) continue;
    ++used;
    int* d = nullptr;
    const int rc = alloc(&d, lists[mode].size());
    if (rc != SG_OK) return rc;
    if (cudaMemcpy(d, lists[mode].data(), lists[mode].size() * sizeof(int),
                   cudaMemcpyHostToDevice) != cudaSuccess) {
      return SG_ERR_CUDA;
    }
    plan->group[mode].inst = d;
  }
  if (used > 1 && groups_.fork == nullptr) {
    cudaError_t e = cudaEventCreateWithFlags(&groups_.fork, cudaEventDisableTiming);
    for (int mode = 1; mode < kModes; ++mode) {
      if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&groups_.stream[mode], cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&groups_.join[mode], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) return SG_ERR_CUDA;
  }
  return SG_OK;
}

// Waits for the stream; a wait inside a kernel that gave up is an error too.
cudaError_t Batch::finish(std::string* err) {
  cudaError_t e = cudaMemcpyAsync(wait_host_, v_.wait_error, sizeof(int), cudaMemcpyDeviceToHost,
                                  stream_);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess && *wait_host_ != 0) {
    cudaMemset(v_.wait_error, 0, sizeof(int));
    e = cudaErrorUnknown;
    if (err) *err = "an exchange between the CTAs of a cluster did not complete";
    return e;
  }
  if (e != cudaSuccess && err) *err = cudaGetErrorString(e);
  return e;
}

int Batch::solve(InstResult* results, double* x, double* y, double* device_ms, std::string* err) {
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, stream_);
  const unsigned long long budget =
      time_limit_ > 0 ? static_cast<unsigned long long>(time_limit_ * 1e9) : 0ull;
  cudaError_t e = launch_batch(v_, setup_plan_, solve_plan_, budget, groups_, stream_);
  cudaEventRecord(e1, stream_);
  std::string why;
  if (e == cudaSuccess) {
    e = finish(&why);
  } else {
    why = cudaGetErrorString(e);
  }
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (device_ms) *device_ms = ms;
  if (e != cudaSuccess) {
    if (err) *err = "batch solve: " + why;
    return SG_ERR_CUDA;
  }
  if (results) {
    e = cudaMemcpy(results, v_.results, sizeof(InstResult) * v_.count, cudaMemcpyDeviceToHost);
  }
  if (e == cudaSuccess && x) {
    e = cudaMemcpy(x, v_.x_out, sizeof(double) * total_vec_, cudaMemcpyDeviceToHost);
  }
  if (e == cudaSuccess && y && total_rows_ > 0) {
    e = cudaMemcpy(y, v_.y_out, sizeof(double) * total_rows_, cudaMemcpyDeviceToHost);
  }
  if (e != cudaSuccess) {
    if (err) *err = std::string("batch download: ") + cudaGetErrorString(e);
    return SG_ERR_CUDA;
  }
  return SG_OK;
}

int Batch::unroll(int iterations, int every, double* v_out, std::string* err) {
  if (v_.fp32) {
    if (err) *err = "the unrolled PDHG runs in FP64: create the batch with SG_PRECISION_FP64";
    return SG_ERR_INVALID_ARGUMENT;
  }
  if (iterations <= 0 || every <= 0) {
    if (err) *err = "iterations and checkpoint interval must be positive";
    return SG_ERR_INVALID_ARGUMENT;
  }
  const int count = v_.count;
  const int nck = (iterations + every - 1) / every;
  std::vector<long long> ck_off(count + 1, 0), mask_off(count + 1, 0);
  for (int i = 0; i < count; ++i) {
    const long long nt = inst_nt_host_[i];
    ck_off[i + 1] = ck_off[i] + static_cast<long long>(nck) * (2 * nt + inst_m_host_[i]);
    // Keep every instance's masks 16-byte aligned.
    mask_off[i + 1] = mask_off[i] + (static_cast<long long>(every) * nt + 15) / 16 * 16;
  }
  auto fail = [&](cudaError_t e, const char* what) {
    cudaGetLastError();  // reported here, not by the next call
    if (err) *err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? SG_ERR_OUT_OF_MEMORY : SG_ERR_CUDA;
  };
  if (u_.iterations != iterations || u_.every != every || u_.ck == nullptr) {
    // (Where an allocation below fails, neither the adjoint nor a later call finds half of them.)
    unrolled_ = false;
    u_.iterations = 0;
    for (void* p : {static_cast<void*>(u_.ck), static_cast<void*>(u_.mask),
                    const_cast<void*>(static_cast<const void*>(u_.ck_off)),
                    const_cast<void*>(static_cast<const void*>(u_.mask_off))}) {
      if (p) cudaFree(p);
    }
    u_.ck = nullptr;
    u_.mask = nullptr;
    u_.ck_off = nullptr;
    u_.mask_off = nullptr;
    double* ck = nullptr;
    unsigned char* mask = nullptr;
    long long *cko = nullptr, *mko = nullptr;
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&ck),
                               std::max<long long>(ck_off[count], 1) * sizeof(double));
    if (e == cudaSuccess) {
      e = cudaMalloc(reinterpret_cast<void**>(&mask), std::max<long long>(mask_off[count], 16));
    }
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&cko), count * sizeof(long long));
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&mko), count * sizeof(long long));
    if (e == cudaSuccess) {
      e = cudaMemcpy(cko, ck_off.data(), count * sizeof(long long), cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) {
      e = cudaMemcpy(mko, mask_off.data(), count * sizeof(long long), cudaMemcpyHostToDevice);
    }
    u_.ck = ck;
    u_.mask = mask;
    u_.ck_off = cko;
    u_.mask_off = mko;
    if (e != cudaSuccess) return fail(e, "unroll buffers");
    if (u_.grad_v == nullptr) {  // the last of them
      for (double** p : {&u_.v_out, &u_.grad_cost, &u_.grad_lower, &u_.grad_upper}) {
        const int rc = alloc(p, total_vec_);
        if (rc != SG_OK) {
          if (err) *err = "unroll buffers: out of memory";
          return rc;
        }
      }
      double* gv = nullptr;
      const int rc = alloc(&gv, total_vec_);
      if (rc != SG_OK) {
        if (err) *err = "unroll buffers: out of memory";
        return rc;
      }
      u_.grad_v = gv;
    }
    u_.iterations = iterations;
    u_.every = every;
    u_.nck = nck;
  }
  if (forward_plan_.size == 0) {
    int rc = make_plan(Kind::kForward, &forward_plan_);
    if (rc == SG_OK) rc = make_plan(Kind::kAdjoint, &adjoint_plan_);
    if (rc != SG_OK) {
      forward_plan_ = ClusterPlan();
      if (err) *err = "unroll plan: out of memory";
      return rc;
    }
  }
  std::string why;
  cudaError_t e = launch_batch_setup(v_, setup_plan_, stream_);
  if (e == cudaSuccess) e = launch_unroll(v_, u_, forward_plan_, 0, groups_, stream_);
  if (e != cudaSuccess) return fail(e, "unroll");
  e = finish(&why);
  if (e != cudaSuccess) {
    if (err) *err = "unroll: " + why;
    return SG_ERR_CUDA;
  }
  if (v_out) {
    e = cudaMemcpy(v_out, u_.v_out, sizeof(double) * total_vec_, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(e, "unroll download");
  }
  unrolled_ = true;
  return SG_OK;
}

int Batch::unroll_adjoint(const double* grad_v, double* grad_cost, double* grad_lower,
                          double* grad_upper, std::string* err) {
  if (!unrolled_) {
    if (err) *err = "sg_batch_unroll must run before its adjoint";
    return SG_ERR_NOT_READY;
  }
  if (grad_v == nullptr) {
    if (err) *err = "grad_v is required";
    return SG_ERR_INVALID_ARGUMENT;
  }
  auto fail = [&](cudaError_t e, const char* what) {
    if (err) *err = std::string(what) + ": " + cudaGetErrorString(e);
    return SG_ERR_CUDA;
  };
  cudaError_t e = cudaMemcpy(const_cast<double*>(u_.grad_v), grad_v,
                             sizeof(double) * total_vec_, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return fail(e, "adjoint upload");
  std::string why;
  e = launch_batch_setup(v_, setup_plan_, stream_);
  if (e == cudaSuccess) e = launch_unroll(v_, u_, adjoint_plan_, 1, groups_, stream_);
  if (e != cudaSuccess) return fail(e, "adjoint");
  e = finish(&why);
  if (e != cudaSuccess) {
    if (err) *err = "adjoint: " + why;
    return SG_ERR_CUDA;
  }
  const std::pair<double*, const double*> outs[3] = {
      {grad_cost, u_.grad_cost}, {grad_lower, u_.grad_lower}, {grad_upper, u_.grad_upper}};
  for (const auto& o : outs) {
    if (o.first == nullptr) continue;
    e = cudaMemcpy(o.first, o.second, sizeof(double) * total_vec_, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(e, "adjoint download");
  }
  return SG_OK;
}

}  // namespace sg

struct sg_batch {
  sg::Batch* batch = nullptr;
};

namespace {
thread_local std::string g_batch_error;
}

extern "C" {

int sg_batch_create(sg_batch** handle, int nmat, const int* mat_m, const int* mat_n,
                    const int64_t* mat_colptr, const int32_t* mat_rowidx, const double* mat_val,
                    int count, const int* inst_mat, const double* cost, const double* lower,
                    const double* upper, const sg_pdlp_opts* opts) {
  if (handle == nullptr) return SG_ERR_INVALID_ARGUMENT;
  *handle = nullptr;
  try {
    sg_pdlp_opts d;
    sg_pdlp_default_opts(&d);
    if (opts == nullptr) opts = &d;
    std::string why;
    sg::Batch* b = nullptr;
    const int rc = sg::Batch::create(&b, nmat, mat_m, mat_n, mat_colptr, mat_rowidx, mat_val,
                                     count, inst_mat, cost, lower, upper,
                                     opts->tol > 0 ? opts->tol : 1e-8, opts->max_iterations,
                                     opts->time_limit, opts->precision, opts->algorithm, &why);
    if (rc != SG_OK) {
      g_batch_error = why;
      return rc;
    }
    *handle = new sg_batch{b};
    return SG_OK;
  } catch (...) {
    g_batch_error = "unexpected exception";
    return SG_ERR_INTERNAL;
  }
}

int sg_batch_solve(sg_batch* handle, sg_batch_result* results, double* x, double* y,
                   double* device_ms) {
  if (handle == nullptr || handle->batch == nullptr) return SG_ERR_INVALID_ARGUMENT;
  try {
    std::string why;
    static_assert(sizeof(sg::InstResult) == sizeof(sg_batch_result), "result layout");
    const int rc = handle->batch->solve(reinterpret_cast<sg::InstResult*>(results), x, y,
                                        device_ms, &why);
    if (rc != SG_OK) g_batch_error = why;
    return rc;
  } catch (...) {
    g_batch_error = "unexpected exception";
    return SG_ERR_INTERNAL;
  }
}

void sg_batch_destroy(sg_batch* handle) {
  if (handle == nullptr) return;
  try {
    delete handle->batch;
  } catch (...) {
  }
  delete handle;
}

int sg_batch_unroll(sg_batch* handle, int iterations, int checkpoint_every, double* v_out) {
  if (handle == nullptr || handle->batch == nullptr) return SG_ERR_INVALID_ARGUMENT;
  try {
    std::string why;
    const int rc = handle->batch->unroll(iterations, checkpoint_every, v_out, &why);
    if (rc != SG_OK) g_batch_error = why;
    return rc;
  } catch (...) {
    g_batch_error = "unexpected exception";
    return SG_ERR_INTERNAL;
  }
}

int sg_batch_unroll_adjoint(sg_batch* handle, const double* grad_v, double* grad_cost,
                            double* grad_lower, double* grad_upper) {
  if (handle == nullptr || handle->batch == nullptr) return SG_ERR_INVALID_ARGUMENT;
  try {
    std::string why;
    const int rc =
        handle->batch->unroll_adjoint(grad_v, grad_cost, grad_lower, grad_upper, &why);
    if (rc != SG_OK) g_batch_error = why;
    return rc;
  } catch (...) {
    g_batch_error = "unexpected exception";
    return SG_ERR_INTERNAL;
  }
}

const char* sg_batch_last_error(void) { return g_batch_error.c_str(); }

}  // extern "C"
