// stream_sms.cuh - the SMs that a stream's kernels can run on: those of the
// device, or of the green context (a part of the device) that the caller's
// stream belongs to.  Host code.
#pragma once

#include <algorithm>

#include <cuda.h>
#include <cuda_runtime.h>

namespace hbtg
{
namespace
{

template <typename F>
F driver_function(const char *name)
{
  void *f = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPointByVersion(name, &f, 12040, cudaEnableDefault, &found) != cudaSuccess)
  {
    cudaGetLastError();
    return nullptr;
  }
  return found == cudaDriverEntryPointSuccess ? reinterpret_cast<F>(f) : nullptr;
}

// Zero where it cannot be told.
inline int stream_sms(cudaStream_t st, int device_sms)
{
  const auto context_of = driver_function<decltype(&cuStreamGetGreenCtx)>("cuStreamGetGreenCtx");
  const auto resource_of = driver_function<decltype(&cuGreenCtxGetDevResource)>("cuGreenCtxGetDevResource");
  if (!context_of || !resource_of)
    return device_sms; // a driver without green contexts
  CUgreenCtx part = nullptr;
  if (context_of(st, &part) != CUDA_SUCCESS)
    return 0;
  if (!part)
    return device_sms;
  CUdevResource r;
  if (resource_of(part, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
    return 0;
  return std::min(device_sms, (int)r.sm.smCount);
}

} // namespace
} // namespace hbtg
