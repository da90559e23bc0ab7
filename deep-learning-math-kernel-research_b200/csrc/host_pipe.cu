// See host_pipe.hpp.  Why: a cudaMemcpyAsync from or to pageable memory is one thread copying through the driver's
// pinned buffer, about 13 GB/s on the measured box, in both directions one after the other -- 1.1 ms for the 16 MB
// of a 64-image INT8 1x1 layer whose kernel takes 9 us, where the bus would take 0.25 ms.
#include "host_pipe.hpp"

#include <sys/mman.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <new>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace elb {

namespace {
inline void relax() {
#if defined(__x86_64__)
  _mm_pause();
#else
  std::this_thread::yield();
#endif
}
}  // namespace

HostPipe::Events::~Events() {
  for (int i = 0; i < SLOTS; ++i) {
    if (in[i]) cudaEventDestroy(in[i]);
    if (out[i]) cudaEventDestroy(out[i]);
  }
}

std::shared_ptr<HostPipe> HostPipe::get(bool make) {
  static std::mutex m;
  static std::weak_ptr<HostPipe> current;
  std::lock_guard<std::mutex> lock(m);
  std::shared_ptr<HostPipe> p = current.lock();
  if (!p && make) {
    p.reset(new (std::nothrow) HostPipe());
    if (!p || !p->start()) return nullptr;
    current = p;
  }
  return p;
}

bool HostPipe::start() {
  // Mapped into every device's context: plans of several GPUs share the slots.  On huge pages, where there are any:
  // touching and pinning 16 MB takes 3.5 ms, from cudaHostAlloc 7 to 20.
  constexpr size_t HUGE_PAGE = size_t(2) << 20, bytes = 2 * SLOTS * SLOT_BYTES;
  slots_ = static_cast<unsigned char *>(std::aligned_alloc(HUGE_PAGE, bytes));
  if (!slots_) return false;
  madvise(slots_, bytes, MADV_HUGEPAGE);
  std::memset(slots_, 0, bytes);
  pinned_ = cudaHostRegister(slots_, bytes, cudaHostRegisterPortable) == cudaSuccess;
  if (!pinned_) {
    cudaGetLastError();
    return false;
  }
  // the calling thread copies too; half of the cores at most, and no more than saturate the memory
  const int n = std::min(6, static_cast<int>(std::thread::hardware_concurrency()) / 2 - 1);
  try {
    for (int i = 0; i < n; ++i) threads_.emplace_back([this] { helper(); });
  } catch (...) {      // fewer threads, or none: the calling thread does the rest
  }
  return true;
}

HostPipe::~HostPipe() {
  {
    std::lock_guard<std::mutex> lock(m_);
    stop_ = true;
  }
  cv_.notify_all();
  for (std::thread &t : threads_) t.join();
  if (pinned_) cudaHostUnregister(slots_);
  std::free(slots_);
}

void HostPipe::begin() {
  {
    std::lock_guard<std::mutex> lock(m_);
    active_ = 1;
  }
  cv_.notify_all();
}
void HostPipe::end() {
  std::lock_guard<std::mutex> lock(m_);
  active_ = 0;
}

void HostPipe::submit(void *dst, const void *src, size_t bytes, std::atomic<int> *left) {
  const int parts = static_cast<int>((bytes + PART - 1) / PART);
  left->store(parts, std::memory_order_relaxed);
  std::lock_guard<std::mutex> lock(m_);
  for (size_t at = 0; at < bytes; at += PART)
    tasks_[(first_task_ + queued_++) % MAX_TASKS] = {static_cast<char *>(dst) + at, static_cast<const char *>(src) + at,
                                                     bytes - at < PART ? bytes - at : PART, left};
  ready_.fetch_add(parts, std::memory_order_release);
}

bool HostPipe::run_one() {
  if (ready_.load(std::memory_order_acquire) <= 0) { relax(); return false; }
  Task t;
  {
    std::lock_guard<std::mutex> lock(m_);
    if (queued_ == 0) return false;
    t = tasks_[first_task_];
    first_task_ = (first_task_ + 1) % MAX_TASKS;
    --queued_;
    ready_.fetch_sub(1, std::memory_order_relaxed);
  }
  std::memcpy(t.dst, t.src, t.bytes);
  t.left->fetch_sub(1, std::memory_order_release);
  return true;
}

// Helpers sleep between calls and poll during one: its pauses are shorter than a wake-up.
void HostPipe::helper() {
  while (true) {
    {
      std::unique_lock<std::mutex> lock(m_);
      cv_.wait(lock, [this] { return stop_ || active_; });
      if (stop_) return;
    }
    while (active_.load(std::memory_order_relaxed) && !stop_.load(std::memory_order_relaxed))
      if (!run_one())
        for (int i = 0; i < 16; ++i) relax();
  }
}

}  // namespace elb
