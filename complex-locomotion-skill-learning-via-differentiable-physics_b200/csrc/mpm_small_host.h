// mpm_small_host.h -- launches of the one-CTA-per-env MPM rollouts
// (csrc/mpm_small.cu).
#pragma once
#include <cuda_runtime.h>

#include "mpm_kernels.cuh"

namespace cls {
namespace mpm {

constexpr int kSmallThreads = 512;
// Particles per env up to which one CTA takes a whole env: forward + reverse per
// substep, B200, one CTA per env / the general kernels: 1-16 envs of 400, 1000,
// 2000 particles 12 / 22, 23 / 23, 47 / 23 us (a lone CTA issues everything), 148
// envs 13 / 27, 25 / 42, 49 / 67 us (every SM has its env), 600 envs 57 / 60, 121 /
// 113, 241 / 227 us.
constexpr int kSmallParticles = 896, kSmallParticlesMany = 2048;
__host__ inline bool small_body(int E, int P) {
  return P <= kSmallParticles || (E >= 64 && E <= 296 && P <= kSmallParticlesMany);
}

template <typename R>
struct SmallFwdArgs {
  Phys<R> c;
  int steps;
  int cap;                                              // scatter table size (SmallLaunch::plan)
  const R* x0; const R* v0; const R* C0; const R* F0;   // state of step 0
  R* rec_x; R* rec_v; R* rec_C; R* rec_F;               // [step][component][E P]; step 0 is not written
  R* fin_x; R* fin_v; R* fin_C; R* fin_F;
  V4<R>* grid;                                          // [step][E][nblk 64]
  const R* act;                                         // [step][E][M]
  double* csum;                                         // [step][E][D], zeroed
};
template <typename R>
struct SmallAdjArgs {
  Phys<R> c;
  int steps;
  int cap;                                              // scatter table size (SmallLaunch::plan)
  const R* x0; const R* v0; const R* C0; const R* F0;
  const R* rec_x; const R* rec_v; const R* rec_C; const R* rec_F;
  const V4<R>* grid;
  const R* act;
  R* gact;                                              // [step][E][M], zeroed
  const R* seed_w;                                      // [step] loss weights
  const double* csum; const R* target;                  // [step][E][D]
  R pw_sum;
  R* out_ax; R* out_av; R* out_aC; R* out_aF;
};

template <typename R, int D>
struct SmallLaunch {
  // whether E envs of P particles on an n_grid^D grid fit one CTA each on
  // the current device, and the scatter tables' sizes then (raises the kernels'
  // shared-memory limits)
  static cudaError_t plan(int E, int P, int n_grid, bool* ok, int* fwd_cap, int* adj_cap);
  static cudaError_t forward(const SmallFwdArgs<R>& a, cudaStream_t s);
  static cudaError_t reverse(const SmallAdjArgs<R>& a, cudaStream_t s);
};

}  // namespace mpm
}  // namespace cls
