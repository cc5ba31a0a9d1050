// y = A x for a CSR matrix already in device memory, with no allocation of any kind.
//
// Some callers cannot call cudaMalloc: a solver running under a memory pool or budget that
// forbids driver allocations, or a plug-in living in a process whose device memory is handed
// out by another runtime. This entry point serves them: the caller passes device pointers for
// every input and output, and the only scratch the kernels need — one carry record per chunk
// of nonzeros — sits in a file-scope __device__ array that every GPU loading the library holds
// until the process exits.
//
// Work split (deterministic): the nonzeros are cut into chunks; the CTA of a chunk owns the rows
// that start inside it. Up to kOneLaunch nonzeros it sums its rows to their ends, and that is
// all. Beyond, it sums each owned row up to the chunk's end; a row that runs past its chunk is
// continued by the following CTAs, each writing one carry (row, partial sum of its slice) to the
// scratch; a second kernel adds every carried row's partials in chunk order. A row takes as many
// lanes as half the rows' average length, so that a warp sums several rows side by side, a longer
// one a warp, the longest the CTA. Same values as the engine's load-balanced tile SpMV up to
// summation order (round-off).
//
// Bound by latency: two launches, a binary search of 2 log2 m dependent loads and rows of 15
// nonzeros one after another on each warp took 24.6 us for 500 rows of 15, now 7.1; 40,000 rows of
// 15 took 32.7, now 16.4; a power-law matrix of 20,000 rows and 240,000 nonzeros 69.7, now 24.6
// (device time a call, back to back).
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "../../include/sg_pdlp.h"

namespace sg {
void set_last_error(const char* message);  // sg_capi.cpp
}  // namespace sg

namespace {

constexpr int kChunkNnz = 2048;  // nonzeros per chunk at most (what the scratch covers)
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxChunks = SG_SPMV_NOALLOC_MAX_CHUNKS;
// One launch up to here, where a single row of all the nonzeros is still only 64 steps of its CTA
// (16,200 nonzeros 6.9 us; 40,000 with the second launch 12.3).
constexpr long long kOneLaunch = 16384;
constexpr int kLongRow = 64;     // longer rows are left to a warp
constexpr int kBlockRow = 1024;  // and these to the CTA

struct Carry {
  double value;  // partial sum of the chunk's slice of the carried row
  int row;       // -1: no carried row in this chunk
  int pad;
};

// The scratch: one carry per chunk (16 bytes each).
static __device__ __align__(256) Carry g_noalloc_carry[kMaxChunks];

// First index r in [0, m) with ptr[r] >= key (m when none), by a warp: 32 probes a round.
__device__ __forceinline__ int lower_bound_ptr(const int* ptr, int m, long long key) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = m;
  while (lo < hi) {
    const int step = static_cast<int>((static_cast<unsigned>(hi - lo) + 31u) >> 5);
    const long long at = lo + static_cast<long long>(lane + 1) * step - 1;
    const bool below = at < hi && static_cast<long long>(ptr[at]) < key;
    const int c = __popc(__ballot_sync(0xffffffffu, below));
    const long long next = lo + static_cast<long long>(c + 1) * step - 1;
    lo = static_cast<int>(min(static_cast<long long>(hi), lo + static_cast<long long>(c) * step));
    if (next < hi) hi = static_cast<int>(next);
  }
  return lo;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// The products b .. e - 1, every `step`-th from b + first on.
__device__ __forceinline__ double partial(long long b, long long e, int first, int step,
                                          const int* __restrict__ idx,
                                          const double* __restrict__ val,
                                          const double* __restrict__ x) {
  double s = 0.0;
#pragma unroll 4
  for (long long q = b + first; q < e; q += step) s += val[q] * x[idx[q]];
  return s;
}

// The sum over the CTA, in thread 0 (a barrier before and after the scratch's use).
__device__ __forceinline__ double block_total(double v, double* scratch) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < kWarps; ++w) s += scratch[w];
  }
  return s;
}

// One CTA per chunk [k0, k1): owned rows (start in the chunk; the last chunk also owns the
// trailing empty rows), and, unless `whole`, the carry of the row that enters the chunk. 2^lanes
// threads to a row.
__global__ void __launch_bounds__(kThreads) spmv_chunk_kernel(int m, const int* __restrict__ ptr,
                                                              const int* __restrict__ idx,
                                                              const double* __restrict__ val,
                                                              const double* __restrict__ x,
                                                              double* __restrict__ y,
                                                              Carry* __restrict__ carry,
                                                              int chunks, int chunk_nnz,
                                                              int lanes, int whole) {
  __shared__ int range[2];
  __shared__ int longs[kChunkNnz / kLongRow + 1];  // rows that end in the chunk, and the last
  __shared__ int nlongs;
  __shared__ double scratch[kWarps];
  const int c = blockIdx.x;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // The matrix's own nonzero count decides the chunk bounds: chunks past it are empty, and the
  // last chunk runs to its end (owned rows and the carried row alike), so a grid sized from a
  // count that differs from row_ptr[m] still writes every row once.
  const long long nnz = ptr[m];
  const bool last_chunk = c == chunks - 1;
  long long k0 = static_cast<long long>(c) * chunk_nnz;
  if (k0 > nnz) k0 = nnz;
  const long long k1 = last_chunk ? nnz : (k0 + chunk_nnz < nnz ? k0 + chunk_nnz : nnz);
  // Rows starting in [k0, k1); the last chunk takes every row starting at or after k0.
  if (threadIdx.x == 0) nlongs = 0;
  if (warp == 0) {
    const int r = c == 0 ? 0 : lower_bound_ptr(ptr, m, k0);
    if (lane == 0) range[0] = r;
  } else if (warp == 1) {
    const int r = last_chunk ? m : lower_bound_ptr(ptr, m, k1);
    if (lane == 0) range[1] = r;
  }
  __syncthreads();
  const int r_begin = range[0];
  // (Unsigned: the numbers past the last row are no int beyond 2^31 - 256 rows.)
  const unsigned r_end = static_cast<unsigned>(range[1]);
  auto end_of = [&](unsigned r) {
    const long long e = ptr[r + 1];
    return e > k1 && !last_chunk && !whole ? k1 : e;
  };
  // Rows side by side, `rows` at a time; every lane of a warp stays in the loop for the shuffles.
  const int width = 1 << lanes;
  const int part = threadIdx.x & (width - 1);
  const unsigned rows = kThreads >> lanes;
  for (unsigned base = static_cast<unsigned>(r_begin); base < r_end; base += rows) {
    const unsigned r = base + (threadIdx.x >> lanes);
    const long long b = r < r_end ? ptr[r] : 0;
    const long long e = r < r_end ? end_of(r) : 0;
    // (A last chunk that runs on to a count beyond the grid's may hold more long rows than the
    // list: those are summed here.)
    int slot = 0;
    if (e - b > kLongRow && part == 0) slot = atomicAdd(&nlongs, 1) + 1;
    slot = __shfl_sync(0xffffffffu, slot, lane & ~(width - 1));
    const bool listed = slot > 0 && slot <= static_cast<int>(sizeof(longs) / sizeof(longs[0]));
    if (listed && part == 0) longs[slot - 1] = static_cast<int>(r);
    double s = listed ? 0.0 : partial(b, e, part, width, idx, val, x);
    for (int o = width >> 1; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, width);
    if (r < r_end && !listed && part == 0) y[r] = s;
  }
  __syncthreads();
  const int count = min(nlongs, static_cast<int>(sizeof(longs) / sizeof(longs[0])));
  for (int i = 0; i < count; ++i) {
    const int r = longs[i];
    const long long b = ptr[r];
    const long long e = end_of(r);
    if (e - b <= kBlockRow) continue;
    const double s = block_total(partial(b, e, threadIdx.x, kThreads, idx, val, x), scratch);
    if (threadIdx.x == 0) y[r] = s;
  }
  for (int i = warp; i < count; i += kWarps) {
    const int r = longs[i];
    const long long b = ptr[r];
    const long long e = end_of(r);
    if (e - b > kBlockRow) continue;
    const double s = warp_sum(partial(b, e, lane, 32, idx, val, x));
    if (lane == 0) y[r] = s;
  }
  if (whole) return;
  // The row entering this chunk from an earlier one (it started before k0).
  const int entering = c > 0 && r_begin > 0 && ptr[r_begin] > k0 ? r_begin - 1 : -1;
  double s = 0.0;
  if (entering >= 0) {
    const long long e_row = ptr[entering + 1];
    s = block_total(partial(k0, e_row < k1 ? e_row : k1, threadIdx.x, kThreads, idx, val, x),
                    scratch);
  }
  if (threadIdx.x == 0) {
    carry[c].row = entering;
    carry[c].value = s;
  }
}

// Adds the carried partials of each row to its owner's sum, in chunk order (one thread per
// chunk; the first chunk of a run of equal rows does the run).
__global__ void spmv_carry_kernel(double* __restrict__ y, const Carry* __restrict__ carry,
                                  int chunks) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= chunks) return;
  const int row = carry[c].row;
  if (row < 0) return;
  if (c > 0 && carry[c - 1].row == row) return;
  double s = y[row];
  for (int g = c; g < chunks && carry[g].row == row; ++g) s += carry[g].value;
  y[row] = s;
}

// The scratch's device address, looked up once per device (cudaGetSymbolAddress, with that
// device current). A cudaDeviceReset of the device unloads the module and makes the address
// stale; sg_spmv_noalloc is not meant to be called after one.
std::mutex g_setup_mutex;
Carry* g_carry_ptr[64] = {nullptr};

int scratch_for_current_device(Carry** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SG_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (g_carry_ptr[dev] == nullptr) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_carry);
    if (e != cudaSuccess || p == nullptr) return SG_ERR_CUDA;
    g_carry_ptr[dev] = static_cast<Carry*>(p);
  }
  *out = g_carry_ptr[dev];
  return SG_OK;
}

int refuse(int code, const char* message) {
  sg::set_last_error(message);
  return code;
}

}  // namespace

extern "C" int sg_spmv_noalloc(int m, long long nnz, const int* d_row_ptr, const int* d_col_idx,
                               const double* d_val, const double* d_x, double* d_y,
                               void* stream) {
  if (m < 0 || nnz < 0 || d_row_ptr == nullptr || d_y == nullptr ||
      (nnz > 0 && (d_col_idx == nullptr || d_val == nullptr || d_x == nullptr))) {
    return refuse(SG_ERR_INVALID_ARGUMENT, "sg_spmv_noalloc: negative size or NULL pointer");
  }
  const long long chunks_ll = nnz == 0 ? 1 : (nnz + kChunkNnz - 1) / kChunkNnz;
  if (chunks_ll > kMaxChunks) {
    return refuse(SG_ERR_TOO_LARGE,
                  "sg_spmv_noalloc: more nonzeros than its fixed scratch covers "
                  "(SG_SPMV_NOALLOC_MAX_CHUNKS * 2048)");
  }
  if (m == 0) return SG_OK;
  Carry* carry = nullptr;
  const int rc = scratch_for_current_device(&carry);
  if (rc != SG_OK) return refuse(rc, "sg_spmv_noalloc: no scratch address on this device");
  // Chunks small enough for about four CTAs per SM; the scratch covers the largest.
  int whole = nnz <= kOneLaunch;
  int chunk_nnz = 256;
  while (chunk_nnz < kChunkNnz && nnz > chunk_nnz * 608LL) chunk_nnz *= 2;
  int chunks = static_cast<int>(nnz == 0 ? 1 : (nnz + chunk_nnz - 1) / chunk_nnz);
  int lanes = 0;
  while (lanes < 5 && (4LL << lanes) <= nnz / m) ++lanes;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // cudaLaunchKernel reports the error of this launch only (the caller's earlier errors stay
  // where they are).
  const int* rp = d_row_ptr;
  const int* ci = d_col_idx;
  const double* va = d_val;
  const double* xv = d_x;
  double* yv = d_y;
  void* chunk_args[] = {&m,     &rp,    &ci,        &va,    &xv,   &yv,
                        &carry, &chunks, &chunk_nnz, &lanes, &whole};
  cudaError_t e = cudaLaunchKernel(reinterpret_cast<const void*>(spmv_chunk_kernel),
                                   dim3(chunks), dim3(kThreads), chunk_args, 0, s);
  if (e == cudaSuccess && !whole) {
    const Carry* cc = carry;
    void* carry_args[] = {&yv, &cc, &chunks};
    e = cudaLaunchKernel(reinterpret_cast<const void*>(spmv_carry_kernel),
                         dim3((chunks + 255) / 256), dim3(256), carry_args, 0, s);
  }
  if (e != cudaSuccess) {
    sg::set_last_error(cudaGetErrorString(e));
    return SG_ERR_CUDA;
  }
  return SG_OK;
}
