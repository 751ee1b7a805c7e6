// See pct_stage.h. Hand-over: chunk i uses slot i % kSlots. Upload: a worker waits until chunk
// i - kSlots has been issued and its transfer (the slot's event) is done, fills the slot and marks
// the chunk staged; the calling thread issues chunks in order. Download: the calling thread waits
// until chunk i - kSlots has been emptied, issues chunk i into the slot and records the event; a
// worker waits for it and empties the slot. Workers take chunks in order, so the oldest open chunk
// always has someone working on it and nobody waits for a later one. A chunk is 40 us of the link,
// about what a sleeping thread takes to wake, so the waits poll and yield. That is for the transfers
// alone: what the stream has before them (a fusion of many milliseconds) is waited for before the
// workers start. (Workers started at once: a tensor-core call of 132 ms took 530 ms of CPU time, 180 now.)
#include "pct_stage.h"

#include <stdint.h>
#include <string.h>
#include <sys/mman.h>

#include <algorithm>
#include <chrono>
#include <mutex>

namespace pct {
namespace {

// Polls, and after 200 us (a transfer held up behind a repack that waits for the SMs) looks every 20 us
// only: 222x222x112, 10 atlases, NH 11 takes the same 28.6 ms and 68 ms of CPU time instead of 95.
template <class F>
void poll_until(F &&done) {
  using Clock = std::chrono::steady_clock;
  Clock::time_point since{};
  for (int i = 0; !done(); ++i) {
    if (i <= 64) continue;
    if (i == 65) since = Clock::now();
    if (Clock::now() - since < std::chrono::microseconds(200))
      std::this_thread::yield();
    else
      std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
}

// Pinned blocks that no stager holds, guarded by the mutex; freed with the last stager.
using Block = HostStager::Block;
constexpr size_t kMaxSpare = 2;
std::mutex spare_mutex;
std::vector<Block> spare;
int stagers = 0;

constexpr size_t kHuge = 2u << 20, kBlockBytes = HostStager::kSlots * HostStager::kSlotBytes;

// kBlockBytes of host memory registered with the current device; nullptr if it cannot be had. Not
// inherited by a fork: pages shared with a child would be copied away from the registration. (In one
// piece: eight take 3 ms more.)
char *pin_block() {
  char *map = static_cast<char *>(mmap(nullptr, kBlockBytes + kHuge, PROT_READ | PROT_WRITE,
                                       MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  if (map == MAP_FAILED) return nullptr;
  const size_t lead = (kHuge - reinterpret_cast<uintptr_t>(map) % kHuge) % kHuge;
  char *p = map + lead;
  if (lead) munmap(map, lead);
  if (kHuge - lead) munmap(p + kBlockBytes, kHuge - lead);
  madvise(p, kBlockBytes, MADV_HUGEPAGE);
  memset(p, 0, kBlockBytes);  // (two thirds of the time, and not inside the driver)
  if (madvise(p, kBlockBytes, MADV_DONTFORK) == 0 &&
      cudaHostRegister(p, kBlockBytes, cudaHostRegisterDefault) == cudaSuccess)
    return p;
  cudaGetLastError();
  munmap(p, kBlockBytes);
  return nullptr;
}

void free_block(const Block &b) {
  for (cudaEvent_t e : b.ev)
    if (e) cudaEventDestroy(e);
  if (!b.slots) return;
  cudaHostUnregister(b.slots);
  munmap(b.slots, kBlockBytes);
}

// A new block; without slots if it cannot be had. May run beside another thread's stream capture.
Block make_block(int device) {
  Block b{device, nullptr, {}};
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaSetDevice(device) == cudaSuccess && cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess) {
    bool whole = (b.slots = pin_block()) != nullptr;
    for (cudaEvent_t &e : b.ev)
      whole = whole && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!whole) {
      free_block(b);
      b = Block{device, nullptr, {}};
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
  if (!b.slots) cudaGetLastError();
  return b;
}

}  // namespace

HostStager::HostStager() {
  std::lock_guard<std::mutex> lock(spare_mutex);
  ++stagers;
}

HostStager::~HostStager() {
  release();
  std::lock_guard<std::mutex> lock(spare_mutex);
  if (--stagers > 0) return;
  for (const Block &b : spare) free_block(b);
  spare.clear();
}

bool HostStager::pageable(const void *p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

int HostStager::worker_count() const {
  const unsigned hw = std::thread::hardware_concurrency();
  return (int)std::min(3u, std::max(1u, hw / 2));
}

bool HostStager::take(const Block &b) {
  if (!b.slots) return false;
  device_ = b.device;
  slots_ = b.slots;
  std::copy(b.ev, b.ev + kSlots, ev_);
  std::fill(used_, used_ + kSlots, false);
  return true;
}

bool HostStager::reserve(int device, size_t bytes) {
  if (slots_) return true;
  // (a call that is worth slots by itself waits for those being pinned)
  if (pinner_.joinable() && (bytes >= kPinCall || pinned_.load(std::memory_order_acquire))) {
    pinner_.join();
    if (take(pinning_)) return true;
  }
  {
    std::lock_guard<std::mutex> lock(spare_mutex);
    for (size_t i = 0; i < spare.size(); ++i) {
      if (spare[i].device != device) continue;
      const Block b = spare[i];
      spare.erase(spare.begin() + i);
      return take(b);
    }
  }
  asked_ += bytes;
  if (asked_ < kPinBytes || pinner_.joinable()) return false;
  asked_ = 0;  // (tried again after as much if it fails)
  if (bytes >= kPinCall) return take(make_block(device));
  pin_device_ = device;
  return false;
}

void HostStager::pin_ahead() {
  const int device = pin_device_;
  pin_device_ = -1;
  if (device < 0 || pinner_.joinable()) return;
  pinned_ = false;
  try {
    pinner_ = std::thread([this, device] {
      pinning_ = make_block(device);
      pinned_.store(true, std::memory_order_release);
    });
  } catch (...) {  // (no thread to be had)
  }
}

// Waits for the transfers of its own slots, then leaves them on the list or frees them.
void HostStager::release() {
  end();
  if (pinner_.joinable()) {
    pinner_.join();
    if (!slots_)
      take(pinning_);
    else
      free_block(pinning_);
  }
  if (!slots_) return;
  Block b{device_, slots_, {}};
  bool whole = true;
  for (int k = 0; k < kSlots; ++k) {
    if (used_[k] && cudaEventSynchronize(ev_[k]) != cudaSuccess) whole = false;
    b.ev[k] = ev_[k];
    ev_[k] = nullptr;
    used_[k] = false;
  }
  slots_ = nullptr;
  std::lock_guard<std::mutex> lock(spare_mutex);
  try {
    if (whole && spare.size() < kMaxSpare) {
      spare.push_back(b);
      return;
    }
  } catch (...) {
  }
  free_block(b);
}

// Starts the workers on chunks_.
bool HostStager::start(int device, bool uploads) {
  job_ = chunk_ = 0;
  issued_ = 0;
  next_ = 0;
  cancel_ = false;
  error_ = (int)cudaSuccess;
  try {
    if (staged_size_ < chunks_.size()) {
      staged_.reset(new std::atomic<char>[chunks_.size()]);
      staged_size_ = chunks_.size();
    }
    for (size_t i = 0; i < chunks_.size(); ++i) staged_[i] = 0;
    const int n = (int)std::min<size_t>(worker_count(), chunks_.size());
    threads_.reserve(n);
    for (int k = 0; k < n; ++k) threads_.emplace_back([this, device, uploads] { work(device, uploads); });
  } catch (...) {
    if (threads_.empty()) return false;  // (fewer workers than asked for are enough)
  }
  return true;
}

bool HostStager::begin(int device, const std::vector<Job> &jobs, cudaStream_t s) {
  end();
  try {
    size_t total = 0;
    for (const Job &j : jobs) total += j.bytes;
    if (total < kMinBytes) return false;
    for (const Job &j : jobs)
      if (!pageable(j.src)) return false;
    if (!reserve(device, total)) return false;
    chunks_.clear();
    jobs_ = jobs;
    for (const Job &j : jobs)
      for (size_t o = 0; o < j.bytes; o += kSlotBytes)
        chunks_.push_back(Chunk{static_cast<const char *>(j.src) + o, nullptr,
                                std::min(kSlotBytes, j.bytes - o)});
    if (cudaStreamSynchronize(s) != cudaSuccess) return false;  // (the direct copies meet the error)
    return start(device, true);
  } catch (...) {  // out of host memory
    end();
    return false;
  }
}

void HostStager::work(int device, bool uploads) {
  cudaError_t bad = cudaSetDevice(device);
  for (;;) {
    const size_t i = next_.fetch_add(1);
    if (i >= chunks_.size()) return;
    const int slot = (int)(i % kSlots);
    char *mem = slots_ + slot * kSlotBytes;
    const size_t need = uploads ? (i >= kSlots ? i - kSlots + 1 : 0) : i + 1;
    poll_until([&] { return cancel_.load() || issued_.load(std::memory_order_acquire) >= need; });
    if (cancel_) return;
    // (uploads: also a transfer of an earlier call may still read the slot)
    if (bad == cudaSuccess && (!uploads || used_[slot]))
      poll_until([&] {
        bad = cudaEventQuery(ev_[slot]);
        return bad != cudaErrorNotReady || cancel_.load();
      });
    if (cancel_) return;
    if (bad == cudaSuccess) {
      const Chunk &c = chunks_[i];
      if (uploads)
        memcpy(mem, c.src, c.bytes);
      else
        memcpy(c.dst, mem, c.bytes);
    }
    if (bad != cudaSuccess) error_ = (int)bad;
    staged_[i].store(1, std::memory_order_release);
  }
}

cudaError_t HostStager::copy(void *dst, const void *src, size_t bytes, cudaStream_t s) {
  if (!active() || job_ >= jobs_.size() || jobs_[job_].src != src || jobs_[job_].bytes != bytes)
    return cudaErrorInvalidValue;
  ++job_;
  for (size_t o = 0; o < bytes; o += kSlotBytes, ++chunk_) {
    const size_t i = chunk_;
    const int slot = (int)(i % kSlots);
    poll_until([&] { return staged_[i].load(std::memory_order_acquire) != 0; });
    if (error_ != (int)cudaSuccess) return (cudaError_t)error_.load();
    cudaError_t e = cudaMemcpyAsync(static_cast<char *>(dst) + o, slots_ + slot * kSlotBytes,
                                    chunks_[i].bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaEventRecord(ev_[slot], s);
    if (e != cudaSuccess) return e;
    used_[slot] = true;
    issued_.store(i + 1, std::memory_order_release);
  }
  return cudaSuccess;
}

void HostStager::end() {
  cancel_ = true;
  for (std::thread &t : threads_) t.join();
  threads_.clear();
}

cudaError_t HostStager::download(int device, void *dst, const void *src, size_t bytes,
                                 cudaStream_t s) {
  end();
  bool staged = bytes >= kMinBytes && pageable(dst) && reserve(device, bytes);
  if (staged) {
    try {
      chunks_.clear();
      jobs_.clear();
      for (size_t o = 0; o < bytes; o += kSlotBytes)
        chunks_.push_back(Chunk{static_cast<const char *>(src) + o, static_cast<char *>(dst) + o,
                                std::min(kSlotBytes, bytes - o)});
      const cudaError_t e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return e;
      staged = start(device, false);
    } catch (...) {
      end();
      staged = false;
    }
  }
  if (!staged) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
  }
  cudaError_t e = cudaSuccess;
  for (size_t i = 0; i < chunks_.size() && e == cudaSuccess; ++i) {
    const int slot = (int)(i % kSlots);
    if (i >= kSlots) poll_until([&] { return staged_[i - kSlots].load(std::memory_order_acquire) != 0; });
    e = (cudaError_t)error_.load();
    // (a slot's earlier upload runs before this on the device only if the streams are ordered)
    if (e == cudaSuccess && i < kSlots && used_[slot]) e = cudaEventSynchronize(ev_[slot]);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(slots_ + slot * kSlotBytes, chunks_[i].src, chunks_[i].bytes,
                          cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaEventRecord(ev_[slot], s);
    if (e != cudaSuccess) break;
    used_[slot] = true;
    issued_.store(i + 1, std::memory_order_release);
  }
  if (e == cudaSuccess) {
    for (size_t i = 0; i < chunks_.size(); ++i)
      poll_until([&] { return staged_[i].load(std::memory_order_acquire) != 0; });
    e = (cudaError_t)error_.load();
  }
  end();
  return e;
}

}  // namespace pct
