// Batched PDLP (see sg_batch.cu): device views and the host engine.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <string>
#include <vector>

#include "sg_cluster.cuh"
#include "sg_common.cuh"

namespace sg {

struct MatInfo {
  double eta;              // 0.99 / ||[A_eq -I]||
  double a_norm_max_col;   // relative-residual scales of the original matrix
  double at_norm_max_row;
  double pad;
};

struct InstResult {
  int status;
  int pad;
  long long iterations;
  double rel_primal, rel_dual, rel_gap, primal_obj, dual_obj;
  long long restarts;
};

struct BatchView {
  int nmat, count;
  const int* mat_m;
  const int* mat_n;
  // Operators by rows (k: A, t: A'), in the layout of sg_cluster.cuh.
  const long long* mat_k_off;     // first element of a matrix's idx and val arrays
  const long long* mat_t_off;
  const long long* mat_col_off;   // first column and row of a matrix (starts, orders, scales)
  const long long* mat_row_off;
  const int* mat_slice;           // 2 per matrix: log2 of the rows of a slice (A, A')
  const long long* mat_kd_off;    // first slice of a matrix (desc)
  const long long* mat_td_off;
  const int2* k_sl;               // first nonzero and length of each row, by position
  const int2* k_desc;             // per slice (RowShare::desc)
  const int* k_perm;              // position -> row
  const int* k_idx;               // column positions
  double* k_val;
  const double* k_val0;
  float* k_val32;
  const int2* t_sl;
  const int2* t_desc;
  const int* t_perm;
  const int* t_idx;
  double* t_val;
  const double* t_val0;
  float* t_val32;
  double* cs;                     // scales and their reciprocals, by position
  double* rs;
  double* ics;
  double* irs;
  double* spill;                  // setup's gathered vectors where shared memory is too small
                                  // (null when every matrix fits)
  MatInfo* info;
  const double* power_start;
  // Instances.
  const int* inst_mat;
  const long long* vec_off;    // cost/lower/upper/x offsets (n + m each)
  const long long* row_off;    // y offsets (m each)
  const long long* state_off;  // iterate storage offsets (in elements of the storage type)
  const double* cost;
  const double* lower;
  const double* upper;
  void* state;
  double* x_out;
  double* y_out;
  InstResult* results;
  unsigned* queue;                // a position per mode
  int* wait_error;                // set to 1 when a bounded wait gave up
  long long max_iter;
  double tol;
  const unsigned long long* deadline;  // device word: %globaltimer deadline, 0 = none
  int algorithm;     // 0 reference, 1 enhanced, 2 Halpern (enhanced preconditioning)
  int fp32;
  double art_frac;   // forced restart once the iterations since the last reach this fraction
};

// Unrolled PDHG of every instance (the differentiable layer's forward and adjoint).
struct UnrollView {
  int iterations;            // K
  int every;                 // checkpoint interval
  int nck;                   // checkpoints per instance, ceil(K / every)
  const long long* ck_off;   // per instance: first double of its checkpoints
  const long long* mask_off; // per instance: first byte of its segment masks
  double* ck;                // checkpoints: nck x (v: n+m, v_bar: n+m, y: m)
  unsigned char* mask;       // every x (n+m): 0 inside, 1 at lower, 2 at upper
  double* v_out;             // v_K in the LpProblem's space (n+m per instance, vec_off)
  const double* grad_v;      // adjoint of v_K (n+m per instance, vec_off)
  double* grad_cost;         // outputs (n+m per instance, vec_off)
  double* grad_lower;
  double* grad_upper;
};

// Instances in the order they are taken (device array).
struct InstanceList {
  const int* inst = nullptr;
  int count = 0;
};

// A kernel's cluster size and number of clusters at most; its instances by mode, each group a
// launch of its own (a kernel that held every mode would spill), and a CTA's dynamic shared
// memory in each.
struct ClusterPlan {
  int size = 0;
  int clusters = 1;
  int sms = 0;  // SMs of the device
  bool small = false;  // the kernels of kWalkLanes (every instance in kAllShared)
  int threads[kModes] = {kThreads64, kThreads64, kThreads64};
  InstanceList group[kModes];
  size_t smem[kModes] = {0, 0, 0};
};

// Streams and events of the groups after the first (made when a plan has more than one).
struct GroupStreams {
  cudaStream_t stream[kModes] = {nullptr, nullptr, nullptr};
  cudaEvent_t fork = nullptr, join[kModes] = {nullptr, nullptr, nullptr};
};

// launch(mode, stream) for every group that has instances: the first on s, the others side by
// side, all after what s holds and before what s gets next.
template <typename Launch>
cudaError_t for_groups(const ClusterPlan& p, const GroupStreams& gs, cudaStream_t s,
                       cudaError_t e, const Launch& launch) {
  bool first = true;
  for (int mode = 0; mode < kModes && e == cudaSuccess; ++mode) {
    if (p.group[mode].count == 0) continue;
    if (first || gs.fork == nullptr) {
      if (first && gs.fork != nullptr) e = cudaEventRecord(gs.fork, s);
      if (e == cudaSuccess) e = launch(mode, s);
    } else {
      e = cudaStreamWaitEvent(gs.stream[mode], gs.fork, 0);
      if (e == cudaSuccess) e = launch(mode, gs.stream[mode]);
      if (e == cudaSuccess) e = cudaEventRecord(gs.join[mode], gs.stream[mode]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(s, gs.join[mode], 0);
    }
    first = false;
  }
  return e;
}

// The largest cluster an engine or batch may take: SG_MAX_CLUSTER when it is created (1: none, the
// step launches and a CTA per LP), up to kMaxCluster.
inline int cluster_limit() {
  const char* v = getenv("SG_MAX_CLUSTER");
  const int most = v == nullptr ? kMaxCluster : atoi(v);
  return most < 1 ? kMaxCluster : most < kMaxCluster ? most : kMaxCluster;
}

// The clusters that a device was found to hold with kClusterSmemMax (sg_batch_host.cu): whether this
// one is among them, after `add` it is. Safe from several threads.
bool known_to_fit(const void* kernel, int device, int size, int threads, bool add);

// Dynamic shared memory of a cluster kernel at most: a CTA's 227 KB less its static part.
constexpr size_t kClusterSmemMax = 227 * 1024 - 8 * 1024;
// FP64 kernels: a CTA's half of an SM's 228 KB (1 KB of each CTA is the system's).
constexpr size_t kClusterSmemHalf = 113 * 1024 - 8 * 1024;

// Rows of a CTA's share at most (the first CTA's), whole slices of 2^slice rows.
__host__ __device__ inline long long share_rows(long long rows, int slice, int size) {
  const long long slices = (rows + (1LL << slice) - 1) >> slice;
  return ((slices + size - 1) / size) << slice;
}
// Shared memory of one CTA for an LP of n columns and m rows, the same in every CTA of the
// cluster: the gathered vectors and masks; the solve's and the unrolled layer's state.
__host__ __device__ inline size_t cluster_vector_bytes(long long n, long long m, int tslice,
                                                       int kslice, int size, size_t elem) {
  const long long nc = share_rows(n, tslice, size);
  const long long nr = share_rows(m, kslice, size);
  const size_t masks = size > 1 ? static_cast<size_t>(nr + nc) * 2 : 0;
  return (static_cast<size_t>(n + m + 2) * elem + masks + 15) & ~static_cast<size_t>(15);
}
// The state (sg_batch_solve.cuh, sg_batch_unroll.cu) holds 32 entries per slice and array.
__host__ __device__ inline size_t solve_state_bytes(long long tslices, long long kslices,
                                                    size_t elem) {
  return static_cast<size_t>(32 * (5 * tslices + 8 * kslices)) * elem;
}
__host__ __device__ inline size_t unroll_state_bytes(long long tslices, long long kslices,
                                                     bool adjoint) {
  return static_cast<size_t>(32 * ((adjoint ? 9 : 4) * tslices + (adjoint ? 13 : 6) * kslices)) *
         sizeof(double);
}
// Device storage of an instance, in entries: gathered vectors (n + m + 2), second points (2 (n + m)),
// state.
inline long long instance_elements(long long n, long long m, int tslice, int kslice, bool fp32) {
  const long long ts = share_rows(n, tslice, 1) >> tslice;
  const long long ks = share_rows(m, kslice, 1) >> kslice;
  const long long state = 32 * (fp32 ? 5 * ts + 8 * ks : 9 * ts + 13 * ks);
  return 3 * (n + m) + 2 + state;
}

cudaError_t launch_batch(const BatchView& b, const ClusterPlan& setup, const ClusterPlan& solve,
                         unsigned long long budget_ns, const GroupStreams& gs, cudaStream_t s);
cudaError_t launch_batch_setup(const BatchView& b, const ClusterPlan& setup, cudaStream_t s);
cudaError_t launch_solve64(const BatchView& b, const ClusterPlan& p, int mode, cudaStream_t s);
cudaError_t launch_solve32(const BatchView& b, const ClusterPlan& p, int mode, cudaStream_t s);
cudaError_t launch_unroll(const BatchView& b, const UnrollView& u, const ClusterPlan& p,
                          int adjoint, const GroupStreams& gs, cudaStream_t s);
// Whether the device can hold a cluster of the plan's size of each kernel that a plan of several
// CTAs launches.
bool setup_fits(const ClusterPlan& p);
bool solve64_fits(const ClusterPlan& p, int algorithm);
bool solve32_fits(const ClusterPlan& p, int algorithm);
bool unroll_fits(const ClusterPlan& p, int adjoint);

class Batch {
 public:
  ~Batch();
  static int create(Batch** out, int nmat, const int* mat_m, const int* mat_n,
                    const int64_t* mat_colptr, const int32_t* mat_rowidx, const double* mat_val,
                    int count, const int* inst_mat, const double* cost, const double* lower,
                    const double* upper, double tol, long long max_iter, double time_limit,
                    int precision, int algorithm, std::string* err);
  int solve(InstResult* results, double* x, double* y, double* device_ms, std::string* err);
  // Differentiable layer: K fixed-step PDHG iterations of every instance (v_K out, n+m per
  // instance) and the adjoint of v_K with respect to cost, lower and upper.
  int unroll(int iterations, int every, double* v_out, std::string* err);
  int unroll_adjoint(const double* grad_v, double* grad_cost, double* grad_lower,
                     double* grad_upper, std::string* err);
  long long total_vec() const { return total_vec_; }
  long long total_rows() const { return total_rows_; }

 private:
  Batch() = default;
  BatchView v_{};
  std::vector<void*> allocs_;
  cudaStream_t stream_ = nullptr;
  int sms_ = 148;
  long long total_vec_ = 0, total_rows_ = 0;
  std::vector<int> mat_m_, mat_n_, inst_mat_, mat_slice_, order_;
  bool small_ = false;  // the layout of kWalkLanes
  std::vector<long long> mat_nnz_;
  ClusterPlan setup_plan_, solve_plan_, forward_plan_, adjoint_plan_;
  int* wait_host_ = nullptr;  // pinned copy of the wait flag
  enum class Kind { kSetup, kSolve, kForward, kAdjoint };
  int make_plan(Kind kind, ClusterPlan* plan);
  void plan_clusters(Kind kind, int most, ClusterPlan* plan, std::vector<int>* lists);
  int upload_lists(const std::vector<int>* lists, ClusterPlan* plan);
  GroupStreams groups_;
  cudaError_t finish(std::string* err);
  double time_limit_ = 0.0;
  // Unrolled PDHG: the host copies of the per-instance offsets and the device buffers.
  UnrollView u_{};
  std::vector<long long> vec_off_host_;
  std::vector<int> inst_nt_host_, inst_m_host_;
  bool unrolled_ = false;
  template <typename T>
  int alloc(T** p, size_t count);
};

}  // namespace sg
