// The iterations between two evaluations of a small LP in one launch (see sg_chunk.cu).
#pragma once

#include "sg_kernels.cuh"

namespace sg {

// An operator in the cluster kernels' layout (sg_cluster.cuh).
template <typename T>
struct ClusterOp {
  const int2* sl;
  const int2* desc;
  const int* perm;  // position -> row
  const int* pos;   // row -> position
  int* idx;
  T* val;
  int slice;        // log2 of the rows of a slice
};

template <typename T>
struct ChunkView {
  ClusterOp<T> K, Kt;
  T* second;        // n + 2m: Halpern's T(z) by position
  int n, m;
  int size;         // CTAs of the cluster
  size_t smem;
  int* wait_error;  // set to 1 when a bounded wait gave up
};

// Shared memory of a CTA that holds its share of an LP, and whether it fits.
size_t chunk_smem_bytes(int n, int m, int tslice, int kslice, int size, size_t elem);
bool chunk_fits(size_t smem);
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

}  // namespace sg
