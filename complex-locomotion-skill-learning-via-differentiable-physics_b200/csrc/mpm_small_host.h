// mpm_small_host.h -- launches of the one-CTA-per-env MPM rollouts
// (csrc/mpm_small.cu).
#pragma once
#include <cuda_runtime.h>

#include "mpm_kernels.cuh"

namespace cls {
namespace mpm {

constexpr int kSmallThreads = 512;
// Bodies that one CTA takes whole, by dimension, envs E, particles P and the device's
// SMs.  Times over those of the general kernels with a record, forward / forward and
// reverse, B200, voxelised and random bodies (24 substeps).  2D, 32 x 32 grid: up to 512
// particles 0.41-0.60 / 0.46-0.62 at 1-148 envs, 0.75-0.97 / 0.82-0.97 at 600-1000 while
// two CTAs fit an SM (the caller checks), beyond 8 envs per SM no gain; on a
// 64 x 64 grid, one CTA per SM, 0.5-0.6 / 0.6-0.7 up to 148 envs and 0.9-1.4 / 0.9-1.5 at
// 200-600.  Up to 896: 0.63-0.96 / 0.55-1.02 at 1-148, 1.1-1.5 / 1.0-1.3 at 200 and 600.  Up
// to 2048 only with an env for most SMs: 148 envs 0.75 / 0.65, 64 1.0-1.1 / 0.95, 1 env 1.8.
// 3D (8 particles per cell, 27 sums per run): 300-512 particles and 148 envs 0.7-0.8 /
// 0.7-0.87, else 0.8-2.4 / 1.0-2.3.
__host__ inline bool small_body(int D, int E, int P, int n_sm) {
  const bool one_each = 3LL * E >= 2LL * n_sm && E <= n_sm;  // an env for most SMs
  if (D == 3) return one_each && P > 256 && P <= 512;
  return P <= 512 ? E <= 8LL * n_sm : (P <= 896 ? E <= n_sm : P <= 2048 && one_each);
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

// Loss weights of a launch, by value as the general kernels take theirs, so that a
// captured reverse pass keeps the weights of its capture.
template <typename R>
struct SeedChunk {
  static constexpr int kMax = 3840 / sizeof(R);   // kernel parameters: 4 KB
  R w[kMax];
  int n;
  R* out;
};

template <typename R, int D>
struct SmallLaunch {
  // whether E envs of P particles on an n_grid^D grid fit one CTA each on
  // the current device, and the scatter tables' sizes then (raises the kernels'
  // shared-memory limits)
  static cudaError_t plan(int E, int P, int n_grid, bool* ok, int* fwd_cap, int* adj_cap);
  static cudaError_t forward(const SmallFwdArgs<R>& a, cudaStream_t s);
  static cudaError_t reverse(const SmallAdjArgs<R>& a, cudaStream_t s);
  // w[0 .. n) into `out` on the device, for SmallAdjArgs::seed_w
  static cudaError_t seeds(const double* w, int n, R* out, cudaStream_t s);
};

}  // namespace mpm
}  // namespace cls
