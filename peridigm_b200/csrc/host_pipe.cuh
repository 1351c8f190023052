// Transfers between the device and a caller's pageable memory.
//
// The driver stages such a copy through its own pinned buffer on the calling
// thread, which also takes the page faults of a fresh destination, and the
// kernels before and after it wait. Here a few worker threads move the bytes between
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

// Bytes from which a transfer takes the ring; smaller ones are the driver's.
// What it gains over the driver's copy depends on what there is to hide:
// kernels, page faults of the destination (the workers take them beside each
// other), or nothing but the copy itself, beside which their waking up (some
// tens of microseconds each) counts. Measured, driver and ring, us:
//   beside kernels (force from host buffers, coordinates in and forces out, of
//   this size each; result array reused / fresh)
//                0.6 MB  989 and 880 / 1050 and 940     2.2 MB  1390 and 1115 / 1560 and 1510
//                7.7 MB  2035 and 1340 / 2745 and 2570  24.6 MB 4200 and 2530 / 5960 and 4250
//   upload alone 2.4 MB  160 and 570     8 MB 445 and 1170      32 MB 1620 and 1750    48 MB 2570 and 2200
//   download alone (into one reused array / each of four new arrays, dropped
//   together / a new array that is kept)
//                1.5 MB  115 and 410 / 315 and 610 / 760 and 540
//                2.4 MB  160 and 215 / 425 and 500 / 1140 and 510
//                4 MB    240 and 205 / 600 and 460 / 1880 and 550
//                12 MB   650 and 455 / 2750 and 960 / 3160 and 1120
constexpr size_t kPipeBeside = size_t(1) << 20, kPipeUpload = size_t(40) << 20, kPipeDownload = size_t(3) << 20;

// The ring for the life of the object (of one call); false when the transfer
// has to go to the driver.
class HostLease {
 public:
  HostLease(int device, const void* host, size_t bytes, size_t least);  // least: one of the above
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
  // Hands the pieces before `until` to the workers. Behind kernels the calling
  // thread waits for each piece's DMA, as it does in the driver's copies: a
  // worker that did would spin beside it for as long as the kernels take. Alone,
  // there is the DMA only, and the workers wait for that: they are awake when
  // it ends (4 MB into a reused array: 205 us, 500 when handed out after it).
  cudaError_t hand_out(size_t until);
  const bool behind_kernels_;
  size_t down_ = 0, down_out_ = 0;     // pieces issued, handed out
  Piece down_to_[kHostSlots] = {};     // where the issued pieces go
};

}  // namespace pdb
