// ms_hubs.cu -- see ms_hubs_host.h.
#include "ms_dense_host.h"
#include "ms_hubs_host.h"
#include "ms_step.cuh"

namespace cls {

template <typename R>
typename HubKernels<R>::FwdFn HubKernels<R>::forward(int threads) {
  return threads <= 256 ? ms_forward_kernel<R, 256, TAB_HUBS>
                        : (threads <= 512 ? ms_forward_kernel<R, 512, TAB_HUBS> : ms_forward_kernel<R, 1024, TAB_HUBS>);
}
template <typename R>
typename HubKernels<R>::RevFn HubKernels<R>::reverse(int threads) {
  return threads <= 256 ? ms_reverse_kernel<R, 256, TAB_HUBS>
                        : (threads <= 512 ? ms_reverse_kernel<R, 512, TAB_HUBS> : ms_reverse_kernel<R, 1024, TAB_HUBS>);
}
template <typename R>
typename HubKernels<R>::StepFwdFn HubKernels<R>::step_fwd() { return ms_step_fwd_kernel<R, kStepThreads, TAB_HUBS>; }
template <typename R>
typename HubKernels<R>::StepRevFn HubKernels<R>::step_rev() { return ms_step_rev_kernel<R, kStepThreads, TAB_HUBS>; }

template struct HubKernels<float>;
template struct HubKernels<double>;

}  // namespace cls
