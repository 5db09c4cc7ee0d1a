// ms_dense.cu -- the batched-controller kernels (ms_dense.cuh) and their
// launches, compiled into their own module (see ms_dense_host.h).
#include <algorithm>
#include <type_traits>

#include "ms_dense.cuh"
#include "ms_dense_host.h"
#include "ms_hubs_host.h"

namespace cls {

namespace {
// A launch of the substep chain: as a programmatic dependent, so that its
// prologue (launch, tables, tensor memory) runs while the launch before it ends.
// Each kernel of the chain releases its dependent at once and waits, before it
// reads what an earlier launch wrote, until all of them have finished; the tables
// read ahead of that wait are laid out when the batch is prepared.  4096 spiders, a
// training step of 80 substeps: 35.5 -> 33.8 ms; 300: 14.6 -> 14.3.  Not in FP64, where
// CTAs are larger and those that wait take the running launches' room (21 substeps and
// their adjoint of 100 / 256 / 400 / 1000 spiders with and without: 7.2 / 7.8 / 8.9 / 13.8 and
// 7.5 / 7.9 / 9.0 / 12.1 ms, of 150-vertex robots 3.7 / 4.7 / 5.1 / 6.2 and 3.9 / 4.1 / 4.2 / 5.8).
template <typename R, typename... P, typename... A>
cudaError_t chain(void (*fn)(P...), int grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t c{};
  cudaLaunchAttribute at{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = std::is_same<R, float>::value ? 1 : 0;
  return cudaLaunchKernelEx(&c, fn, P(args)...);
}
}  // namespace

template <typename R>
int DenseLaunch<R>::tile_m() { return std::is_same<R, float>::value ? umma::TM : kSimtTile; }
template <typename R>
int DenseLaunch<R>::tile_n() { return std::is_same<R, float>::value ? kDenseTN : kSimtTile; }
template <typename R>
int DenseLaunch<R>::job_n(int n_tiles, int n_sm) {
  if (!std::is_same<R, float>::value) return kSimtTile;
  return 2 * n_tiles <= n_sm ? kDenseTNSmall : kDenseTN;
}
template <typename R>
long long DenseLaunch<R>::split_floats(int rows, int tile_rows, int k) {
  return (long long)umma::split_tiles_floats(rows, tile_rows, k);
}

template <typename R>
cudaError_t DenseLaunch<R>::setup(bool hubs, size_t* fwd_static, size_t* rev_static, int optin) {
  *fwd_static = *rev_static = 0;
  cudaError_t e = cudaSuccess;
  auto prepare = [&](auto fn, size_t* st) {
    cudaFuncAttributes fa{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return;
    *st = std::max(*st, fa.sharedSizeBytes);
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)((size_t)optin - fa.sharedSizeBytes));
  };
  prepare(ms_step_fwd_kernel<R, kStepThreads, TAB_NONE>, fwd_static);
  prepare(ms_step_fwd_kernel<R, kStepThreads, TAB_ROWS>, fwd_static);
  if (hubs) prepare(HubKernels<R>::step_fwd(), fwd_static);
  prepare(ms_step_rev_kernel<R, kStepThreads, TAB_NONE>, rev_static);
  prepare(ms_step_rev_kernel<R, kStepThreads, TAB_ROWS>, rev_static);
  if (hubs) prepare(HubKernels<R>::step_rev(), rev_static);
  if constexpr (std::is_same<R, float>::value) {
    const int sm = (int)umma::BulkShape<kDenseTN, kBulkStages>::kSmemBytes;
    for (auto fn : {ms_ctrl_gemm_tc_kernel<0, kDenseTN>, ms_ctrl_gemm_tc_kernel<1, kDenseTN>,
                    ms_ctrl_gemm_tc_kernel<0, kDenseTNSmall>, ms_ctrl_gemm_tc_kernel<1, kDenseTNSmall>})
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ms_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  }
  return e;
}

template <typename R>
cudaError_t DenseLaunch<R>::step_fwd(const MsArgs<R>& a, bool hubs, int grid, int threads, size_t smem, cudaStream_t s, int t,
                              int t_first, int t_end, int mode, int src_slot, int k_prev, int k_cur) {
  auto fn = !a.imp_cap ? ms_step_fwd_kernel<R, kStepThreads, TAB_NONE>
                       : (hubs ? HubKernels<R>::step_fwd() : ms_step_fwd_kernel<R, kStepThreads, TAB_ROWS>);
  return chain<R>(fn, grid, threads, smem, s, a, t, t_first, t_end, mode, src_slot, k_prev, k_cur);
}

template <typename R>
cudaError_t DenseLaunch<R>::step_rev(const MsArgs<R>& a, bool hubs, int grid, int threads, size_t smem, cudaStream_t s, int t_post,
                              int t_pre, int t_begin, int t_end, int last_seg) {
  auto fn = !a.adj_cap ? ms_step_rev_kernel<R, kStepThreads, TAB_NONE>
                       : (hubs ? HubKernels<R>::step_rev() : ms_step_rev_kernel<R, kStepThreads, TAB_ROWS>);
  return chain<R>(fn, grid, threads, smem, s, a, t_post, t_pre, t_begin, t_end, last_seg);
}

template <typename R>
cudaError_t DenseLaunch<R>::gemm(const MsArgs<R>& a, bool adjoint, int n_jobs, int job_cols, const DenseJob* jobs,
                                 const TcJob* tc, int kslot, cudaStream_t s) {
  if constexpr (std::is_same<R, float>::value) {
    if (job_cols == kDenseTNSmall)
      return chain<R>(adjoint ? ms_ctrl_gemm_tc_kernel<1, kDenseTNSmall> : ms_ctrl_gemm_tc_kernel<0, kDenseTNSmall>, n_jobs,
                   umma::kBulkThreads, umma::BulkShape<kDenseTNSmall, kBulkStages>::kSmemBytes, s, a, tc, kslot);
    return chain<R>(adjoint ? ms_ctrl_gemm_tc_kernel<1, kDenseTN> : ms_ctrl_gemm_tc_kernel<0, kDenseTN>, n_jobs,
                 umma::kBulkThreads, umma::BulkShape<kDenseTN, kBulkStages>::kSmemBytes, s, a, tc, kslot);
  } else {
    return chain<R>(adjoint ? ms_ctrl_gemm_simt_kernel<R, 1> : ms_ctrl_gemm_simt_kernel<R, 0>, n_jobs, 256, 0, s, a, jobs,
                 kslot);
  }
}

template <typename R>
void DenseLaunch<R>::pack_weights(const R* w, R* wt, R* tiles, const TransSeg* tsegs, int n_tsegs, int n_ttiles,
                                  const SplitSeg* ssegs, int n_ssegs, long long split_total, cudaStream_t s) {
  if constexpr (std::is_same<R, float>::value) {
    if (split_total == 0) return;
    const int blocks = (int)std::min<long long>(4096, (split_total + 255) / 256);
    ms_split_weights_kernel<<<blocks, 256, 0, s>>>(w, tiles, ssegs, n_ssegs, split_total);
  } else {
    if (n_ttiles == 0) return;
    ms_transpose_weights_kernel<R><<<n_ttiles, 256, 0, s>>>(w, wt, tsegs, n_tsegs);
  }
}

template <typename R>
void DenseLaunch<R>::wgrad(const MsArgs<R>& a, int grid_x, int n_cols, int slot0, int nslots, const WgTrans* trans,
                           const WgCol* cols, int n_jobs, const WgJob* jobs, R* gw, R* gb, cudaStream_t s) {
  if constexpr (std::is_same<R, float>::value) {
    if (n_cols > 0 && nslots > 0)
      ms_wgrad_transpose_kernel<<<dim3(grid_x, n_cols, (nslots + kWgSlots - 1) / kWgSlots), 256, 0, s>>>(
          a, trans, cols, slot0, nslots);
    if (n_jobs > 0)
      ms_wgrad_tc_kernel<<<n_jobs, umma::kBulkThreads, umma::BulkShape<kDenseTN, kBulkStages>::kSmemBytes, s>>>(
          a, jobs, nslots, gw, gb);
  }
}

template struct DenseLaunch<float>;
template struct DenseLaunch<double>;

}  // namespace cls
