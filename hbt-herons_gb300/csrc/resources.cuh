// resources.cuh - what a handle holds of the CUDA runtime from its creation to
// its end: streams, events, the pinned staging buffer and the scans' ticket.
// Host code only, and nothing but runtime calls.
#pragma once

#include <cstddef>

#include <cuda_runtime_api.h>

#include "../../include/hbt_unbind_gpu.h"

namespace hbtg
{

// Host-pointer calls whose arrays take at most this much go through one pinned
// buffer and one copy each way: some thirty copies of a few hundred bytes were
// 0.2 ms of a 0.65 ms call on one subhalo of 300 particles (now 0.47 ms), and of
// 4,000, the largest that fit, 1.26 ms (now 1.12).  The limit is the pinned
// memory that a handle holds: a buffer of 8 MB would still take a call on 6,000
// particles from 1.36 to 1.19 ms, on 16,000 from 1.69 to 1.52, on 32,000 from 2.03 to 1.93.
constexpr size_t kStageBytes = 256 * 1024;

struct Resources
{
  cudaStream_t stream = nullptr;
  cudaStream_t side = nullptr;         // uploads that only the epilogue needs (host-pointer calls)
  cudaStream_t side2 = nullptr;        // a second copy stream: velocities up, energies down
  cudaEvent_t copy_events[7] = {};     // host-pointer calls: copy phases and the side streams
  cudaEvent_t span[2] = {};            // first and last event of a call
  void *stage = nullptr;               // pinned staging of small host-pointer calls, then of the totals
  unsigned *ticket = nullptr;          // a device zero for the last-block scans (primitives.cuh)

  // All of them on the current device, or none: what a failure leaves is released.
  int create()
  {
    const int rc = create_each();
    if (rc != HBTG_OK)
    {
      cudaGetLastError();
      release();
    }
    return rc;
  }

  void release()
  {
    cudaFree(ticket);
    cudaFreeHost(stage);
    for (cudaEvent_t e : span)
      if (e)
        cudaEventDestroy(e);
    for (cudaEvent_t e : copy_events)
      if (e)
        cudaEventDestroy(e);
    for (cudaStream_t s : {side, side2, stream})
      if (s)
        cudaStreamDestroy(s);
    *this = Resources();
  }

private:
  int create_each()
  {
    for (cudaStream_t *s : {&stream, &side, &side2})
      if (cudaStreamCreateWithFlags(s, cudaStreamNonBlocking) != cudaSuccess)
        return HBTG_ERR_CUDA;
    void *p = nullptr;
    if (cudaMalloc(&p, 256) != cudaSuccess)
      return HBTG_ERR_NOMEM;
    ticket = static_cast<unsigned *>(p);
    // zero before any stream can reach it: the streams here do not wait for the
    // default stream, nor do the callers' own for these
    if (cudaMemsetAsync(ticket, 0, 256, stream) != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess)
      return HBTG_ERR_CUDA;
    for (cudaEvent_t &e : copy_events)
      if (cudaEventCreate(&e) != cudaSuccess)
        return HBTG_ERR_CUDA;
    for (cudaEvent_t &e : span)
      if (cudaEventCreate(&e) != cudaSuccess)
        return HBTG_ERR_CUDA;
    if (cudaMallocHost(&stage, kStageBytes + 256) != cudaSuccess)
      return HBTG_ERR_NOMEM;
    return HBTG_OK;
  }
};

} // namespace hbtg
