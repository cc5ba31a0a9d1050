// The iterations between two evaluations of a small LP in one launch (see sg_chunk.cu).
#pragma once

#include "sg_cluster_layout.h"
#include "sg_kernels.cuh"

namespace sg {

constexpr int kChunkThreads = 512;

// An operator in tasks (sg_cluster_layout.h), and where a CTA keeps its block of it in shared
// memory (bytes).
template <typename T>
struct ChunkOp {
  const int* perm;   // position -> row
  const int* pos;    // row -> position
  const int2* row;   // per position: first element, log2 lanes
  const int4* task;
  const int* task_off;
  const int* elem_off;
  const int* filled;
  unsigned short* idx;
  T* val;
  int per;           // positions of a CTA
  unsigned val_at, idx_at, task_at;
};

template <typename T>
struct ChunkView {
  ChunkOp<T> K, Kt;
  T* second;        // Halpern's T(z), by position
  int n, m;
  int np, mp;       // positions of the columns and rows
  int size;         // CTAs of the cluster; 0: the LP takes step launches
  unsigned cols_at, rows_at, sums_at;  // the state of the own columns and rows, a walk's sums
  size_t smem;
  int* wait_error;  // set to 1 when a bounded wait gave up
};

// Sets the places in shared memory and smem; false when they do not fit.
template <typename T>
bool place_chunk(ChunkView<T>* v, const TaskLayout& k, const TaskLayout& t);
// Whether the device can hold the placed chunk's cluster.
template <typename T>
bool chunk_fits(const ChunkView<T>& c, bool halpern);
// The column numbers of both operators, from their CSR arrays.
template <typename T>
void launch_chunk_indices(const ChunkView<T>& c, const OpView<T>& K, const OpView<T>& Kt,
                          cudaStream_t s);
// The values of both operators, from their CSR arrays.
template <typename T>
void launch_chunk_values(const ChunkView<T>& c, const OpView<T>& K, const OpView<T>& Kt,
                         cudaStream_t s);
// The iterations up to the next evaluation.
template <typename T>
cudaError_t launch_chunk(Ctl* ctl, const ChunkView<T>& c, const IterView<T>& it, bool halpern,
                         cudaStream_t s);

// The scaling passes of a solve's setup (the reference's Ruiz, or the enhanced ones) from the given
// values in the chunk's layout.
cudaError_t launch_chunk_scale(const ChunkView<double>& c, const double* k_given,
                               const double* t_given, bool ruiz, double* cs, double* rs,
                               cudaStream_t s);
// The power iteration of a solve's setup on A_eq (the chunk's values), from u0: sigma into the
// control block (launch_power_finish takes it).
cudaError_t launch_chunk_power(Ctl* ctl, const ChunkView<double>& c, const double* u0,
                               int iterations, cudaStream_t s);

}  // namespace sg
