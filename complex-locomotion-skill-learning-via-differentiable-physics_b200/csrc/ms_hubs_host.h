// ms_hubs_host.h -- kernel instances for robots with hub vertices (kEllRows), in their
// own module (csrc/ms_hubs.cu): loaded by the first handle that has such a robot.
#pragma once
#include "ms_kernels.cuh"

namespace cls {

template <typename R>
struct HubKernels {
  using FwdFn = void (*)(MsArgs<R>, int, int, int, int);
  using RevFn = void (*)(MsArgs<R>, int, int, int);
  using StepFwdFn = void (*)(MsArgs<R>, int, int, int, int, int, int, int);
  using StepRevFn = void (*)(MsArgs<R>, int, int, int, int, int);
  static FwdFn forward(int threads);
  static RevFn reverse(int threads);
  static StepFwdFn step_fwd();
  static StepRevFn step_rev();
};

}  // namespace cls
