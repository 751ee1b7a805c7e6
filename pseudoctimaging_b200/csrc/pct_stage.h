// Copies between pageable host memory and the device through pinned slots filled and emptied by
// several host threads.
//
// A copy from or to pageable memory runs at the rate of the one driver thread that moves it through
// the driver's own pinned buffer (about 11 GB/s), a fifth of what the link carries, and for a drop-in
// call on the caller's arrays that is longer than the fusion it feeds. Here the caller names all its
// uploads first; worker threads copy them, in order and slot by slot, into pinned memory ahead of
// the calling thread, which issues each slot's transfer on its stream as soon as it is filled.
// 176x208x96, 6 atlases, NH 11 from pageable arrays: 12.0 ms against 19.2 (the fusion takes 9.9); three
// workers and 2 MB slots, which also keep 20 MB calls from losing (six workers 12.1 and 5 % slower
// there; sleeping instead of polling waits 14.8).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <atomic>
#include <memory>
#include <thread>
#include <vector>

namespace pct {

class HostStager {
 public:
  struct Job {
    const void *src;
    size_t bytes;
  };
  HostStager();
  ~HostStager();

  // Whether p is plain pageable memory (pinned, managed and device memory are copied directly).
  static bool pageable(const void *p);

  // Starts staging `jobs` in order, once the work that `s` (the stream of the transfers, or the one
  // they follow) already has is done. False (nothing started, the caller copies directly) when they
  // are too small to gain, no slots are at hand and too little was copied yet to pin some, or the
  // slots or threads cannot be had.
  bool begin(int device, const std::vector<Job> &jobs, cudaStream_t s);
  bool active() const { return !threads_.empty(); }
  // The next job's transfer, enqueued on s. Jobs must be taken in the order given to begin.
  cudaError_t copy(void *dst, const void *src, size_t bytes, cudaStream_t s);
  // Ends the staging (all jobs taken, or an error on the way): joins the workers. Transfers may
  // still be in flight from the slots; the next begin or download waits for them.
  void end();

  // Whether a download of this size to p is worth staging.
  static bool takes(const void *p, size_t bytes) { return bytes >= kMinBytes && pageable(p); }
  // Ends a call: has slots pinned for later ones if it asked for them.
  void pin_ahead();

  // Device to pageable host memory, complete on return; waits for the work that s already has first.
  // Falls back to one direct copy (and waits for it) where the slots or threads cannot be had.
  cudaError_t download(int device, void *dst, const void *src, size_t bytes, cudaStream_t s);

  static constexpr int kSlots = 8;
  static constexpr size_t kSlotBytes = 2u << 20;
  static constexpr size_t kMinBytes = 12u << 20;  // below, thread start and hand-over eat the gain
  // A stager without slots copies directly until it has been asked for kPinBytes: pinning slots takes
  // 2.6 ms and staging gains 0.04 to 0.065 ms per MB. From then on a call of kPinCall or more, which
  // gains about what they cost, pins them itself. After a smaller call a thread of its own does, for
  // later calls, which copy directly until it has. (20 MB calls take 1.4 ms; one that pinned in its own
  // time took 3.1. Now a call that comes while the thread pins takes 2.3, for the driver's lock, and one
  // that comes 5 ms later 1.4.)
  static constexpr size_t kPinBytes = 60u << 20, kPinCall = 48u << 20;

  struct Block {  // pinned slots and the events of their transfers
    int device;
    char *slots;
    cudaEvent_t ev[kSlots];
  };

 private:
  struct Chunk {
    const char *src;
    char *dst;
    size_t bytes;
  };
  // The slots come from a process-wide list of at most two blocks that stagers leave behind and go
  // back to it; the last stager frees the list. Slots are huge pages registered with the device: 2.6
  // ms for 16 MB, where cudaHostAlloc takes 8 to 20 (a new handle's first call on 21 MB of arrays
  // took 17 ms with it, 4.9 with direct copies as now).
  bool reserve(int device, size_t bytes);
  bool take(const Block &b);
  void release();
  bool start(int device, bool uploads);
  void work(int device, bool uploads);
  int worker_count() const;

  int device_ = -1;
  char *slots_ = nullptr;
  size_t asked_ = 0;  // bytes that would have been staged while there were no slots
  int pin_device_ = -1;  // pin_ahead pins slots for it
  std::thread pinner_;   // makes pinning_, then sets pinned_
  Block pinning_{};
  std::atomic<bool> pinned_{false};
  cudaEvent_t ev_[kSlots] = {};
  bool used_[kSlots] = {};  // a transfer was recorded on ev_[k]

  std::vector<Chunk> chunks_;
  std::vector<Job> jobs_;
  size_t job_ = 0, chunk_ = 0;  // next job and chunk of the calling thread
  std::atomic<size_t> next_{0};
  std::vector<std::thread> threads_;
  std::unique_ptr<std::atomic<char>[]> staged_;  // chunk filled (uploads) or emptied by a worker
  size_t staged_size_ = 0;
  std::atomic<size_t> issued_{0};  // chunks whose transfer is enqueued
  std::atomic<bool> cancel_{false};
  std::atomic<int> error_{(int)cudaSuccess};
};

}  // namespace pct
