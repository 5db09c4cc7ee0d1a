// ms_cluster.cu -- launches of the cluster-per-env segment kernels
// (ms_cluster.cuh), in their own module (see ms_cluster_host.h).
#include <map>
#include <mutex>
#include <tuple>

#include "ms_cluster.cuh"
#include "ms_cluster_host.h"

namespace cls {

namespace {
template <typename R>
cudaLaunchConfig_t config(int items, int cluster, int threads, size_t smem, cudaStream_t s, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)(items * cluster));
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)cluster;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  c.attrs = at;
  c.numAttrs = 1;
  return c;
}
}  // namespace

template <typename R>
int ClusterLaunch<R>::max_threads() { return kClusterMaxThreads; }

template <typename R>
size_t ClusterLaunch<R>::fwd_bytes(const ClusterCaps& cap) {
  return cl::carve<R>(nullptr, cap, (cl::FwdShared<R>*)nullptr);
}
template <typename R>
size_t ClusterLaunch<R>::rev_bytes(const ClusterCaps& cap, int cluster, int threads) {
  return cl::carve<R>(nullptr, cap, cluster, threads, (cl::RevShared<R>*)nullptr);
}

template <typename R>
cudaError_t ClusterLaunch<R>::setup(int optin, size_t* fwd_max, size_t* rev_max) {
  cudaFuncAttributes fa{}, ra{};
  cudaError_t e = cudaFuncGetAttributes(&fa, ms_cluster_forward_kernel<R>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&ra, ms_cluster_reverse_kernel<R>);
  if (e != cudaSuccess) return e;
  *fwd_max = (size_t)optin - fa.sharedSizeBytes;
  *rev_max = (size_t)optin - ra.sharedSizeBytes;
  e = cudaFuncSetAttribute(ms_cluster_forward_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*fwd_max);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ms_cluster_reverse_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*rev_max);
  // clusters of 16 (8 is the portable maximum)
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ms_cluster_forward_kernel<R>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ms_cluster_reverse_kernel<R>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

template <typename R>
cudaError_t ClusterLaunch<R>::resident(int cluster, int threads, size_t fwd_smem, size_t rev_smem, int* n) {
  int dev = 0, nf = 0, nr = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nf, ms_cluster_forward_kernel<R>, threads, fwd_smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nr, ms_cluster_reverse_kernel<R>, threads, rev_smem);
  if (e != cudaSuccess) return e;
  // clusters are placed whole within a GPC, so their number follows from the
  // CTAs that an SM holds: one query (about a millisecond) per such number,
  // device and cluster size in the process
  static std::mutex lock;
  static std::map<std::tuple<int, int, int>, int> known;
  const std::tuple<int, int, int> key(dev, cluster, nf < nr ? nf : nr);
  std::lock_guard<std::mutex> hold(lock);
  const auto it = known.find(key);
  if (it != known.end()) {
    *n = it->second;
    return cudaSuccess;
  }
  cudaLaunchAttribute at{};
  if (nf < nr) {
    const cudaLaunchConfig_t c = config<R>(1, cluster, threads, fwd_smem, nullptr, &at);
    e = cudaOccupancyMaxActiveClusters(n, ms_cluster_forward_kernel<R>, &c);
  } else {
    const cudaLaunchConfig_t c = config<R>(1, cluster, threads, rev_smem, nullptr, &at);
    e = cudaOccupancyMaxActiveClusters(n, ms_cluster_reverse_kernel<R>, &c);
  }
  if (e == cudaSuccess) known[key] = *n;
  return e;
}

template <typename R>
cudaError_t ClusterLaunch<R>::forward(const MsArgs<R>& a, const ClusterCaps& cap, int cluster, int threads, size_t smem,
                                      cudaStream_t s, int t_begin, int t_end, int mode, int src_slot) {
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t c = config<R>(a.n_items, cluster, threads, smem, s, &at);
  return cudaLaunchKernelEx(&c, ms_cluster_forward_kernel<R>, a, cap, t_begin, t_end, mode, src_slot);
}

template <typename R>
cudaError_t ClusterLaunch<R>::reverse(const MsArgs<R>& a, const ClusterCaps& cap, int cluster, int threads, size_t smem,
                                      cudaStream_t s, int t_begin, int t_end, int last_seg) {
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t c = config<R>(a.n_items, cluster, threads, smem, s, &at);
  return cudaLaunchKernelEx(&c, ms_cluster_reverse_kernel<R>, a, cap, t_begin, t_end, last_seg);
}

template struct ClusterLaunch<float>;
template struct ClusterLaunch<double>;

}  // namespace cls
