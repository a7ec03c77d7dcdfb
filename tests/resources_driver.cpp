// Drives csrc/resources.cuh against a runtime of its own that counts what is
// live and can fail its n-th call.  Prints "live <objects left>" for a failed
// creation, or for a whole one that was released again, and "pending <streams>":
// those with work enqueued that the creation did not wait for.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "../hbt-herons_gb300/csrc/resources.cuh"

static std::set<void *> live, pending;
static int calls = 0, fail_at = -1;

static bool fails() { return calls++ == fail_at; }
template <typename T>
static cudaError_t make(T *out)
{
  if (fails())
    return cudaErrorMemoryAllocation;
  void *p = std::malloc(16);
  live.insert(p);
  *out = reinterpret_cast<T>(p);
  return cudaSuccess;
}
static cudaError_t drop(void *p)
{
  if (p && !live.erase(p))
    std::printf("released twice\n");
  return cudaSuccess;
}

extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return make(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return make(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
cudaError_t cudaMalloc(void **p, size_t) { return make(p); }
cudaError_t cudaFree(void *p) { return drop(p); }
cudaError_t cudaMallocHost(void **p, size_t) { return make(p); }
cudaError_t cudaFreeHost(void *p) { return drop(p); }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t s)
{
  pending.insert(s);
  return fails() ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); } // asynchronous on device memory
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
  pending.erase(s);
  return fails() ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

int main(int argc, char **argv)
{
  fail_at = argc > 1 ? std::atoi(argv[1]) : -1;
  hbtg::Resources r;
  const int rc = r.create();
  const int made = calls;
  const size_t waits = pending.size();
  if (rc == HBTG_OK)
    r.release();
  std::printf("rc %d calls %d pending %zu live %zu\n", rc, made, waits, live.size());
}
