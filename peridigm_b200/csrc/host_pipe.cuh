// Transfers between the device and a caller's pageable memory.
//
// The driver stages such a copy through its own pinned buffer on the calling
// thread, which also takes the page faults of a fresh destination: some 5 to 8
// GB/s against the link's 50. Here a few worker threads move the bytes between
// the caller's memory and a ring of pinned slots, beside each other, the DMA
// and the kernels. One ring and its workers serve every context of the process
// (8 MB pinned, made once the open contexts have moved enough bytes to pay for it,
// given back with the last of them); one transfer uses it at a time, and a
// transfer that finds it taken or not made yet, is small, or has pinned memory
// goes to the driver.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace pdb {

// Contexts that may use the ring.
void host_pipe_retain();
void host_pipe_release();

struct HostRing;
constexpr int kHostSlots = 16;

// The ring for the life of the object (of one call); false when the transfer
// has to go to the driver.
class HostLease {
 public:
  HostLease(int device, const void* host, size_t bytes);
  ~HostLease();
  HostLease(const HostLease&) = delete;
  HostLease& operator=(const HostLease&) = delete;
  explicit operator bool() const { return ring_ != nullptr; }

  // Copies `src` [bytes] to the device array dst on `stream`, in order;
  // through(end) issues the copies of the bytes before `end`, waiting for the
  // workers only as far as it must. All is read from src once through(bytes)
  // has returned.
  void upload(void* dst, const void* src, size_t bytes, cudaStream_t stream);
  cudaError_t through(size_t end);

  // Copies device bytes to host memory after the work on `stream`; the bytes
  // are there after finish(). (A lease serves uploads or downloads, not both.)
  cudaError_t download(void* dst, const void* src, size_t bytes, cudaStream_t stream);
  cudaError_t finish();

 private:
  HostRing* ring_ = nullptr;
  char* up_dst_ = nullptr;
  const char* up_src_ = nullptr;
  size_t up_bytes_ = 0, up_issued_ = 0, up_queued_ = 0;  // pieces (of a slot each)
  cudaStream_t up_stream_ = nullptr;
  struct Piece {
    char* dst;
    size_t bytes;
  };
  cudaError_t hand_out(size_t until);  // pieces before `until` to the workers, each when its DMA is done
  size_t down_ = 0, down_out_ = 0;     // pieces issued, handed out
  Piece down_to_[kHostSlots] = {};     // where the issued pieces go
};

}  // namespace pdb
