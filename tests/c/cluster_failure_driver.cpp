// Runs the batched kernels' control flow on the CPU, a host thread per CTA of a cluster, and makes
// bounded waits give up: whatever fails, every CTA must pass the same cluster barriers and none may
// store into one that has ended. The walks do nothing but wait (test_cluster_failure.py puts the
// kernels' own sources behind this file's stand-ins for the device).
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

#include "emulated_device.h"
#include "sg_cluster.cuh"

#include "sg_batch.cu"
#include "sg_batch_solve.cuh"
#include "sg_batch_unroll.cu"

namespace {

using namespace sg;

constexpr int kM = 3, kN = 4, kInstances = 2;

struct Problem {
  int m = kM, n = kN, slice[2] = {5, 5}, inst[kInstances] = {0, 0}, perm[8] = {0};
  int2 starts[8] = {};
  long long mats[2] = {0, 0}, offs[kInstances] = {0, 0};
  std::vector<double> v = std::vector<double>(4096, 1.0);
  std::vector<unsigned char> mask = std::vector<unsigned char>(4096);
  MatInfo info{1.0, 1.0, 1.0, 0.0};
  InstResult results[kInstances];
  unsigned queue[kModes] = {0, 0, 0};
  int order[kInstances] = {0, 1}, wait_error = 0;
  unsigned long long deadline = 0;
  BatchView view(int algorithm) {
    BatchView b{};
    b.nmat = 1;
    b.count = kInstances;
    b.mat_m = &m;
    b.mat_n = &n;
    b.mat_k_off = b.mat_t_off = b.mat_col_off = b.mat_row_off = b.mat_kd_off = b.mat_td_off = mats;
    b.mat_slice = slice;
    b.k_perm = b.t_perm = b.k_idx = b.t_idx = perm;
    b.k_sl = b.t_sl = b.k_desc = b.t_desc = starts;
    b.k_val0 = b.t_val0 = v.data();
    b.cs = b.rs = b.ics = b.irs = b.k_val = b.t_val = v.data();
    b.spill = v.data();
    b.info = &info;
    b.power_start = v.data();
    b.inst_mat = inst;
    b.vec_off = b.row_off = b.state_off = offs;
    b.cost = b.lower = b.upper = v.data();
    b.state = v.data();
    b.x_out = b.y_out = v.data();
    b.results = results;
    b.queue = queue;
    b.wait_error = &wait_error;
    b.max_iter = 150;
    b.tol = -1.0;
    b.deadline = &deadline;
    b.algorithm = algorithm;
    b.art_frac = 0.36;
    return b;
  }
  UnrollView unroll() {
    UnrollView u{};
    u.iterations = 20;
    u.every = 8;
    u.nck = 3;
    u.ck_off = u.mask_off = offs;
    u.ck = v.data();
    u.mask = mask.data();
    u.v_out = u.grad_cost = u.grad_lower = u.grad_upper = v.data();
    u.grad_v = v.data();
    return u;
  }
};

// One launch of `kernel` on a cluster of `size`; CTA r's waits fail from its fail_at[r]-th on.
template <typename Kernel>
bool run(unsigned size, const std::vector<int>& fail_at, const Kernel& kernel) {
  emu::cluster.reset(size);
  std::vector<std::thread> ctas;
  for (unsigned r = 0; r < size; ++r) {
    ctas.emplace_back([&, r] {
      emu::enter(r, size, fail_at[r]);
      kernel();
      emu::cluster.leave(r);
    });
  }
  for (auto& t : ctas) t.join();
  return emu::cluster.sound();
}

}  // namespace

int main() {
  int cases = 0, bad = 0;
  const unsigned size = 4;
  for (int which = 0; which < 6; ++which) {
    for (int at = 0; at < 70; at += at < 8 ? 1 : 7) {
      for (unsigned who = 0; who < size; ++who) {
        for (int later : {0, 1, 3, 40, 1 << 20}) {
          std::vector<int> fail_at(size, at + later);
          fail_at[who] = at;
          Problem p;
          const bool ok = run(size, fail_at, [&] {
            const BatchView b = p.view(which == 1 || which == 3 ? 2 : 0);
            const InstanceList list{p.order, kInstances};
            if (which < 2) batch_setup_kernel<kWalkOne, kThreads64>(b, 1u << 20);
            if (which == 2) batch_solve_kernel<double, kAllShared, false, kThreads64>(b, list);
            if (which == 3) batch_solve_kernel<double, kAllShared, true, kThreads64>(b, list);
            if (which == 4) unroll_kernel<false, kAllShared>(b, p.unroll(), list);
            if (which == 5) unroll_kernel<true, kAllShared>(b, p.unroll(), list);
          });
          const bool told = p.wait_error != 0 || !emu::cluster.failed;
          ++cases;
          if (!ok || !told) {
            if (bad++ < 5) {
              printf("kernel %d, CTA %u at wait %d, the others %d later: %s\n", which, who, at,
                     later, !ok ? "barriers" : "not reported");
            }
          }
        }
      }
    }
  }
  printf("%d cases, %d bad\n", cases, bad);
  return bad == 0 ? 0 : 1;
}
