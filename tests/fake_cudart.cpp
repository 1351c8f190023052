// The CUDA calls of host_pipe.cu on host memory, for its tests without a
// device: a copy is a memcpy, every event is complete, calls are counted.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <thread>

#include "host_pipe.cuh"

namespace {
std::atomic<int> pinned_made{0}, pinned_freed{0}, event_waits{0}, worker_waits{0};
const std::thread::id caller = std::this_thread::get_id();  // (loaded by the thread that makes the calls)
}  // namespace

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
  ++pinned_made;
  *p = std::malloc(bytes);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) {
  ++pinned_freed;
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  ++event_waits;
  if (std::this_thread::get_id() != caller) ++worker_waits;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(dst, src, bytes);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}

// What the tests call. up and down return 1 when the transfer had the ring, 0
// when it was left to the driver; beside: as beside kernels, else alone.
void open_context() { pdb::host_pipe_retain(); }
void close_context() { pdb::host_pipe_release(); }
int up(void* dst, const void* src, size_t bytes, int beside) {
  pdb::HostLease lease(0, src, bytes, beside ? pdb::kPipeBeside : pdb::kPipeUpload);
  if (!lease) return 0;
  lease.upload(dst, src, bytes, nullptr);
  return lease.through(bytes) == cudaSuccess ? 1 : -1;
}
int down(void* dst, const void* src, size_t bytes, int beside) {
  pdb::HostLease lease(0, dst, bytes, beside ? pdb::kPipeBeside : pdb::kPipeDownload);
  if (!lease) return 0;
  const cudaError_t e = lease.download(dst, src, bytes, nullptr), w = lease.finish();
  return e == cudaSuccess && w == cudaSuccess ? 1 : -1;
}
int count(int what) {
  return (what == 0 ? pinned_made : what == 1 ? pinned_freed : what == 2 ? event_waits : worker_waits).load();
}
}
