// ms_step.cuh -- step kernels of the batched-controller path (ms_dense.cuh).
#pragma once
#include <type_traits>

#include "ms_segment.cuh"
#include "umma_gemm.cuh"

namespace cls {

__host__ __device__ __forceinline__ int pad4(int x) { return (x + 3) & ~3; }

// ------------------------------------------------------------ step kernels
// Registers for four CTAs of 256 threads per SM, which is also what the spider's
// spring tables leave room for (54 KB per CTA).  4096 spiders, 80 substeps, forward
// / reverse step kernels: 128 threads 15.3 / 19.5 ms, 128 x 8 CTAs 11.1 / 15.9, 256 x
// 3 12.6 / 14.8, 256 x 4 10.8 / 12.8; 300 spiders differ by 10 %.
constexpr int kStepCtas = 4;
// FP64: 128 registers, four CTAs of the 128 threads it runs with (181 registers without
// the bound: 400 robots of 150 vertices, 21 substeps and their adjoint, 4.9 -> 4.2 ms).
constexpr int kStepCtas64 = 2;
// One CTA per env; the substep halves with the env's state in the CTA's
// shared memory (the fused kernels' carve with the controller buffers sized
// for the output layer only).  One warp per env
// (several envs per CTA, no CTA barrier) measured slower.

// Forward step t of a range [t_first, t_end):
//   t > t_first: controller outputs of t-1 from the output layer's record
//                (slot k_prev), then spring forces and advance of t-1;
//   t < t_end:   checkpoint / records / observables of x(t), the input row of
//                t into record slot k_cur (zero padded) and, FP32, into the
//                first GEMM's pre-split operand; state to live_x/v;
//   t == t_end:  the range's end (checkpoint, final state).
// The state comes from checkpoint slot src_slot at t == t_first, else from
// live_x/v.
template <typename R, int MAXT, int TAB>
__global__ void __launch_bounds__(MAXT, sizeof(R) == 4 ? kStepCtas : kStepCtas64)
ms_step_fwd_kernel(MsArgs<R> a, int t, int t_first, int t_end, int mode, int src_slot, int k_prev,
                   int k_cur) {
  extern __shared__ __align__(256) char smem_raw[];
  __shared__ RobotDesc rb;
  __shared__ EnvDesc ed;
  dependents_launch();
  const int item = blockIdx.x;
  if (item >= a.n_items) return;
  FwdSmem<R> s = carve_fwd<R>(smem_raw, a);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int e = a.order[item];
  load_descs<R>(a, e, rb, ed);
  dependents_wait();
  const int N = rb.n_v, L = rb.n_layers;
  CLS_PHASE_START();
  {
    const bool first = (t == t_first);
    const V4<R>* cx = first ? a.ckpt_x + (size_t)src_slot * a.v_total + ed.v_off : a.live_x + ed.v_off;
    const V4<R>* cv = first ? a.ckpt_v + (size_t)src_slot * a.v_total + ed.v_off : a.live_v + ed.v_off;
    for (int i = tid; i < N; i += nt) { s.xs[i] = cx[i]; s.vs[i] = cv[i]; }
  }
  __syncthreads();
  if (t > t_first) {
    const R* zl = a.rec_z + a.z_base[L - 1] + (size_t)k_prev * a.z_total[L - 1] + ed.z_off[L - 1];
    const R* bo = a.bias + rb.b_off[L - 1];
    for (int o = tid; o < rb.n_out; o += nt) s.buf0[o] = act_f<R>(a.act_out, zl[o] + bo[o]);
    __syncthreads();
    CLS_PHASE(a, 20);
    fwd_post<R, TAB>(a, rb, ed, s, t - 1, mode, k_prev, s.buf0);
    CLS_PHASE(a, 21);
  }
  if (t < t_end) {
    R hprev = 0;
    if ((mode & FWD_OBS) && t > 0) hprev = a.obs_height[(size_t)(t - 1) * a.n_envs + e];
    load_head_smem<R>(a, rb, ed, s, t, mode);
    fwd_pre<R>(a, rb, ed, s, e, t, t_first, mode, k_cur, true, true, hprev);
    CLS_PHASE(a, 22);
    if constexpr (std::is_same<R, float>::value) {
      // the input row as the first layer's pre-split A operand
      const umma::SplitTiles st{a.tiles + a.dense[ed.robot].ta_f[0], umma::TM, (rb.n_c + 31) / 32};
      const int j = e - rb.env_first;
      for (int q = 4 * tid; q < rb.n_c; q += 4 * nt)
        st.store4(j, q, make_float4(s.ain[q], s.ain[q + 1], s.ain[q + 2], s.ain[q + 3]));
    }
    CLS_PHASE(a, 23);
    for (int i = tid; i < N; i += nt) {
      a.live_x[ed.v_off + i] = s.xs[i];
      a.live_v[ed.v_off + i] = s.vs[i];
    }
    CLS_PHASE(a, 24);
  } else {
    fwd_finish<R>(a, rb, ed, s, t_first, t_end, mode);
  }
}

// Reverse step over a segment [t_begin, t_end):
//   t_post >= 0: adjoint of substep t_post from its controller input on
//                (d input positions in din, x(t_post) from the records);
//   t_pre >= 0:  adjoint of substep t_pre up to dZ of the output layer (and,
//                FP32, dZ as the adjoint GEMM's pre-split operand).
// The adjoint state is carried in adj_x/v/h between launches; the first
// launch of the segment (t_pre = t_end - 1) seeds it (last segment) or takes
// the carry of the later segment.
template <typename R, int MAXT, int TAB>
__global__ void __launch_bounds__(MAXT, sizeof(R) == 4 ? kStepCtas : kStepCtas64)
ms_step_rev_kernel(MsArgs<R> a, int t_post, int t_pre, int t_begin, int t_end, int last_seg) {
  extern __shared__ __align__(256) char smem_raw[];
  __shared__ RobotDesc rb;
  __shared__ EnvDesc ed;
  dependents_launch();
  const int item = blockIdx.x;
  if (item >= a.n_items) return;
  RevSmem<R> s = carve_rev<R>(smem_raw, a);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int e = a.order[item];
  load_descs<R>(a, e, rb, ed);
  dependents_wait();
  const int N = rb.n_v;
  R hcarry = 0;
  CLS_PHASE_START();
  rev_load_carry<R>(a, rb, ed, s, e, t_end, t_pre == t_end - 1 && last_seg != 0, hcarry);
  CLS_PHASE(a, 25);
  if (t_post >= 0) {
    const int kk = t_post - t_begin;
    const V4<R>* rx = a.rec_x + (size_t)kk * a.v_total + ed.v_off;
    for (int i = tid; i < N; i += nt) s.xv.lo[i] = rx[i];  // x(t_post) only: rev_post reads p
    const R* dp = a.din + (size_t)3 * ed.v_off;
    for (int q = tid; q < 3 * N; q += nt) s.bufA[q] = dp[q];
    __syncthreads();
    rev_post<R>(a, rb, ed, s, e, t_post, hcarry);
    CLS_PHASE(a, 26);
  }
  if (t_pre >= 0) {
    rev_pre<R, TAB>(a, rb, ed, s, e, t_pre, t_pre - t_begin);
    CLS_PHASE(a, 27);
    if constexpr (std::is_same<R, float>::value) {
      // dZ of the output layer as the adjoint GEMM's pre-split A operand
      const int no = rb.n_out;
      const umma::SplitTiles st{a.tiles + a.dense[ed.robot].ta_b[rb.n_layers - 1], umma::TM, (no + 31) / 32};
      const int j = e - rb.env_first;
      for (int q = 4 * tid; q < no; q += 4 * nt) {
        const float4 v = make_float4(s.dz[q], q + 1 < no ? s.dz[q + 1] : 0.f, q + 2 < no ? s.dz[q + 2] : 0.f,
                                     q + 3 < no ? s.dz[q + 3] : 0.f);
        st.store4(j, q, v);
      }
    }
    CLS_PHASE(a, 28);
  }
  rev_store_carry<R>(a, rb, ed, s, e, hcarry);
  CLS_PHASE(a, 29);
}

}  // namespace cls
