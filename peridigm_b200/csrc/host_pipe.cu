// The pinned ring and its workers (host_pipe.cuh).
#include "host_pipe.cuh"

#include <unistd.h>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <thread>
#include <vector>

namespace pdb {

namespace {
constexpr size_t kSlotBytes = size_t(512) << 10;
constexpr int kSlots = kHostSlots;
// Pieces between a worker's end of the ring and the DMA's: the other half of
// the slots is with the workers.
constexpr size_t kInFlight = kSlots / 2;
// Bytes that go to the driver before the ring is made: making it takes some 7
// ms (the pinned memory, the threads) and it saves some 36 us per MB (a force
// from host buffers of 24.6 MB each way: 6.0 ms by the driver, 4.2 ms through the
// ring), so it has paid for itself after about as much again. Only transfers
// that the ring would take count, from the first of the contexts now open: a
// program that opens one context per problem and moves a few arrays never makes
// the ring.
constexpr size_t kPipeEarned = size_t(192) << 20;
}  // namespace

struct HostRing {
  struct Job {
    void* dst;
    const void* src;
    size_t bytes;
    int slot;
    cudaEvent_t after;  // the DMA into the slot, where the worker waits for it
  };
  char* pinned = nullptr;
  cudaEvent_t ev[kSlots] = {};
  bool recorded[kSlots] = {};  // ev[k] stands for a DMA of this lease
  bool busy[kSlots] = {};      // a job on the slot is not done
  int device = -1;             // of the events
  const pid_t owner = getpid();  // a forked child has the ring's memory and none of its workers
  bool stop = false;
  cudaError_t error = cudaSuccess;  // of the workers' waits, for the lease
  std::mutex m;
  std::condition_variable work, done;
  std::deque<Job> jobs;
  std::vector<std::thread> workers;

  bool start() {
    if (cudaHostAlloc((void**)&pinned, kSlotBytes * kSlots, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      pinned = nullptr;
      return false;
    }
    const unsigned hw = std::thread::hardware_concurrency();
    const int count = (int)std::min(6u, std::max(1u, hw / 2));
    try {
      for (int k = 0; k < count; ++k) workers.emplace_back([this] { run(); });
    } catch (...) {  // as many as there could be
    }
    return !workers.empty();
  }
  void run() {
    for (;;) {
      Job j;
      int dev;
      {
        std::unique_lock<std::mutex> l(m);
        work.wait(l, [this] { return stop || !jobs.empty(); });
        if (jobs.empty()) return;
        j = jobs.front();
        jobs.pop_front();
        dev = device;
      }
      cudaError_t e = cudaSuccess;
      if (j.after) {
        cudaSetDevice(dev);
        e = cudaEventSynchronize(j.after);
      }
      if (e == cudaSuccess) std::memcpy(j.dst, j.src, j.bytes);
      {
        std::lock_guard<std::mutex> l(m);
        if (e != cudaSuccess) error = e;
        busy[j.slot] = false;
      }
      done.notify_all();
    }
  }
  void push(const Job& j) {
    {
      std::lock_guard<std::mutex> l(m);
      busy[j.slot] = true;
      jobs.push_back(j);
    }
    work.notify_one();
  }
  // The slot's last piece has been copied by its worker.
  void wait(int slot) {
    std::unique_lock<std::mutex> l(m);
    done.wait(l, [&] { return !busy[slot]; });
  }
  cudaError_t failure() {
    std::lock_guard<std::mutex> l(m);
    return error;
  }
  // The slot's last DMA is done (the calling thread waits).
  cudaError_t dma_done(int slot) {
    if (!recorded[slot]) return cudaSuccess;
    const cudaError_t e = cudaEventSynchronize(ev[slot]);
    if (e == cudaSuccess) recorded[slot] = false;
    return e;
  }
  // Nothing of a lease left in flight, in the workers or the DMA.
  void drain() {
    std::unique_lock<std::mutex> l(m);
    done.wait(l, [&] { return jobs.empty() && std::none_of(busy, busy + kSlots, [](bool b) { return b; }); });
    l.unlock();
    for (int k = 0; k < kSlots; ++k) {
      dma_done(k);
      recorded[k] = false;
    }
    error = cudaSuccess;
  }
  bool on(int dev) {  // events of this device
    if (device == dev) return true;
    drop_events();
    for (auto& e : ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        drop_events();
        return false;
      }
    device = dev;
    return true;
  }
  void drop_events() {
    for (auto& e : ev) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    device = -1;
  }
  ~HostRing() {
    {
      std::lock_guard<std::mutex> l(m);
      stop = true;
    }
    work.notify_all();
    for (auto& t : workers) t.join();
    drop_events();
    if (pinned) cudaFreeHost(pinned);
  }
};

namespace {
// (plain objects that no exit handler destroys: contexts may outlive statics)
struct Shared {
  std::mutex count_m;  // users and the ring's life
  std::mutex lease_m;  // held by the lease
  int users = 0;
  HostRing* ring = nullptr;
  bool failed = false;
  size_t passed = 0;  // bytes offered without a ring since there was no context
};
Shared& shared() {
  static Shared* s = new Shared();
  return *s;
}
}  // namespace

void host_pipe_retain() {
  Shared& s = shared();
  std::lock_guard<std::mutex> l(s.count_m);
  ++s.users;
}

void host_pipe_release() {
  Shared& s = shared();
  HostRing* r = nullptr;
  {
    std::lock_guard<std::mutex> l(s.count_m);
    if (--s.users > 0) return;
    r = s.ring;  // (no context is left that could hold a lease)
    s.ring = nullptr;
    s.failed = false;
    s.passed = 0;
  }
  if (r && r->owner == getpid()) delete r;
}

HostLease::HostLease(int device, const void* host, size_t bytes, size_t least) : behind_kernels_(least == kPipeBeside) {
  if (!host || bytes < least) return;
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (a.type != cudaMemoryTypeUnregistered) return;
  Shared& s = shared();
  if (!s.lease_m.try_lock()) return;
  HostRing* r = nullptr;
  {
    std::lock_guard<std::mutex> l(s.count_m);
    if (!s.ring && !s.failed && (s.passed += bytes) >= kPipeEarned) {
      try {
        s.ring = new HostRing();
        if (!s.ring->start()) {
          delete s.ring;
          s.ring = nullptr;
        }
      } catch (...) {
        s.ring = nullptr;
      }
      s.failed = s.ring == nullptr;
    }
    r = s.ring;
  }
  if (!r || r->owner != getpid() || !r->on(device)) {
    s.lease_m.unlock();
    return;
  }
  ring_ = r;
}

HostLease::~HostLease() {
  if (!ring_) return;
  ring_->drain();
  shared().lease_m.unlock();
}

void HostLease::upload(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  up_dst_ = static_cast<char*>(dst);
  up_src_ = static_cast<const char*>(src);
  up_bytes_ = bytes;
  up_issued_ = up_queued_ = 0;
  up_stream_ = stream;
}

cudaError_t HostLease::through(size_t end) {
  const size_t pieces = (up_bytes_ + kSlotBytes - 1) / kSlotBytes;
  const size_t need = std::min(pieces, (end + kSlotBytes - 1) / kSlotBytes);
  while (up_issued_ < need) {
    // the workers run ahead; a slot's last DMA ends before it is filled again
    for (; up_queued_ < pieces && up_queued_ < up_issued_ + kInFlight; ++up_queued_) {
      const int k = (int)(up_queued_ % kSlots);
      const size_t off = up_queued_ * kSlotBytes;
      const cudaError_t e = ring_->dma_done(k);
      if (e != cudaSuccess) return e;
      ring_->push({ring_->pinned + k * kSlotBytes, up_src_ + off, std::min(kSlotBytes, up_bytes_ - off), k, nullptr});
    }
    const int k = (int)(up_issued_ % kSlots);
    const size_t off = up_issued_ * kSlotBytes;
    ring_->wait(k);
    cudaError_t e = cudaMemcpyAsync(up_dst_ + off, ring_->pinned + k * kSlotBytes, std::min(kSlotBytes, up_bytes_ - off),
                                    cudaMemcpyHostToDevice, up_stream_);
    if (e == cudaSuccess) e = cudaEventRecord(ring_->ev[k], up_stream_);
    if (e != cudaSuccess) return e;
    ring_->recorded[k] = true;
    ++up_issued_;
  }
  return cudaSuccess;
}

cudaError_t HostLease::hand_out(size_t until) {
  for (; down_out_ < until; ++down_out_) {
    const int k = (int)(down_out_ % kSlots);
    if (behind_kernels_) {
      const cudaError_t e = ring_->dma_done(k);
      if (e != cudaSuccess) return e;
    }
    ring_->push({down_to_[k].dst, ring_->pinned + k * kSlotBytes, down_to_[k].bytes, k,
                 behind_kernels_ ? nullptr : ring_->ev[k]});
  }
  return cudaSuccess;
}

cudaError_t HostLease::download(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  for (size_t off = 0; off < bytes; off += kSlotBytes) {
    const int k = (int)(down_ % kSlots);
    const size_t len = std::min(kSlotBytes, bytes - off);
    // (alone, every piece is with a worker already)
    cudaError_t e = hand_out(down_ < kInFlight ? 0 : std::max(down_out_, down_ - kInFlight));
    if (e != cudaSuccess) return e;
    ring_->wait(k);  // the slot's last piece has been taken out
    e = cudaMemcpyAsync(ring_->pinned + k * kSlotBytes, static_cast<const char*>(src) + off, len, cudaMemcpyDeviceToHost,
                        stream);
    if (e == cudaSuccess) e = cudaEventRecord(ring_->ev[k], stream);
    if (e != cudaSuccess) return e;
    ring_->recorded[k] = true;
    down_to_[k] = {static_cast<char*>(dst) + off, len};
    ++down_;
    if (!behind_kernels_) hand_out(down_);
  }
  return cudaSuccess;
}

cudaError_t HostLease::finish() {
  cudaError_t e = hand_out(down_);
  for (int k = 0; k < kSlots; ++k) ring_->wait(k);
  return e != cudaSuccess ? e : ring_->failure();
}

}  // namespace pdb
