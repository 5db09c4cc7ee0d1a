// cls_context.h -- the id of the current CUDA context, for what outlives a handle and
// belongs to a context (ids are never reused, so a context created after
// cudaDeviceReset or cuCtxDestroy has an id of its own).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

namespace cls {

// `id` of the current context (0 when none is current); false when the driver does
// not tell.  The driver's entry points are resolved through the runtime so that the
// library does not link libcuda (it must load on machines without a driver).
inline bool current_ctx_id(unsigned long long* id) {
  typedef CUresult (*GetCurrent)(CUcontext*);
  typedef CUresult (*GetId)(CUcontext, unsigned long long*);
  static std::mutex lock;
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  *id = 0;
  {
    std::lock_guard<std::mutex> hold(lock);
    if (!get_current || !get_id) {
      void* f0 = nullptr;
      void* f1 = nullptr;
      cudaDriverEntryPointQueryResult q0, q1;
      if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f0, cudaEnableDefault, &q0) != cudaSuccess ||
          q0 != cudaDriverEntryPointSuccess || !f0)
        return false;
      if (cudaGetDriverEntryPoint("cuCtxGetId", &f1, cudaEnableDefault, &q1) != cudaSuccess ||
          q1 != cudaDriverEntryPointSuccess || !f1)
        return false;
      get_current = reinterpret_cast<GetCurrent>(f0);
      get_id = reinterpret_cast<GetId>(f1);
    }
  }
  CUcontext ctx = nullptr;
  if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return true;
  if (get_id(ctx, id) != CUDA_SUCCESS) *id = 0;
  return true;
}

}  // namespace cls
