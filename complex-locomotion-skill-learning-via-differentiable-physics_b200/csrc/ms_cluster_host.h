// ms_cluster_host.h -- host-side launch interface of the cluster-per-env segment
// kernels (csrc/ms_cluster.cu), compiled into their own module like the batched
// controller's kernels, so that the single-CTA kernels' code is unchanged.
#pragma once
#include <cuda_runtime.h>

#include "ms_kernels.cuh"

namespace cls {

// capacities of one launch's shared memory, in elements
struct ClusterCaps {
  int n;        // vertices of the largest robot
  int own;      // vertices of one CTA (largest share)
  int p0;       // controller input row
  int h;        // hidden layer outputs
  int o;        // controller outputs
  int oslice;   // controller outputs owned by one CTA (reverse)
  int inc;      // incidence records of one CTA (0: read from global memory)
  int log2c;    // log2 of the cluster size
};

// the share [cut(r), cut(r + 1)) of rank r out of 2^log2c: whole groups of `unit`
__host__ __device__ __forceinline__ int cluster_cut(int n, int unit, int r, int log2c) {
  const int c = unit * ((((n + unit - 1) / unit) * r) >> log2c);
  return c < n ? c : n;
}
constexpr int kVertexUnit = 4;   // 4 vertices = 12 input columns = three 16-byte groups

template <typename R>
struct ClusterLaunch {
  static int max_threads();
  // dynamic shared memory of the two kernels, and what a CTA may have
  static size_t fwd_bytes(const ClusterCaps& cap);
  static size_t rev_bytes(const ClusterCaps& cap, int cluster, int threads);
  static cudaError_t setup(int optin, size_t* fwd_max, size_t* rev_max);
  // clusters of both kernels that can be resident at once
  static cudaError_t resident(int cluster, int threads, size_t fwd_smem, size_t rev_smem, int* n);
  static cudaError_t forward(const MsArgs<R>& a, const ClusterCaps& cap, int cluster, int threads, size_t smem,
                             cudaStream_t s, int t_begin, int t_end, int mode, int src_slot);
  static cudaError_t reverse(const MsArgs<R>& a, const ClusterCaps& cap, int cluster, int threads, size_t smem,
                             cudaStream_t s, int t_begin, int t_end, int last_seg);
};

}  // namespace cls
