// Copies between pageable host memory and the device for waiting calls (host_pipe.cu): a ring of pinned slots that
// helper threads fill and empty while the copy engines and the kernels work on the others.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

namespace elb {

class HostPipe {
 public:
  static constexpr size_t SLOT_BYTES = size_t(1) << 20;
  static constexpr int SLOTS = 8;              // per direction
  // What a plan moves the plain way before it asks for a pipe to be made: making and giving back one (pinning, threads)
  // takes about 5 ms, what the pipe then saves about 25 us per MB, so a plan that runs a few times and goes never pays it.
  static constexpr size_t EARN_BYTES = size_t(192) << 20;
  // The process's pipe, shared by all plans that hold it and given back (threads joined, memory freed) with the last
  // of them.  Null when there is none and `make` is false, or when it cannot be had.
  static std::shared_ptr<HostPipe> get(bool make);
  ~HostPipe();

  // One piece of a transfer: `bytes` <= SLOT_BYTES
  struct Piece {
    void *host, *dev;
    size_t bytes;
    int chunk;
  };
  // What a plan keeps for its device: one event per slot.
  struct Events {
    cudaEvent_t in[SLOTS] = {}, out[SLOTS] = {};
    ~Events();
  };
  // Run one call: every piece of `in` host -> device on s_in, `launch(chunk)` once a chunk's pieces have been enqueued,
  // every piece of `out` device -> host on s_out behind its chunk's launch (launch() orders the streams).  Returns when
  // everything has arrived.  One call at a time: under try_lock().
  template <typename Launch>
  cudaError_t run(Events &ev, const std::vector<Piece> &in, const std::vector<Piece> &out, int chunks, cudaStream_t s_in,
                  cudaStream_t s_out, Launch launch);
  std::unique_lock<std::mutex> try_lock() { return std::unique_lock<std::mutex>(busy_, std::try_to_lock); }

 private:
  HostPipe() = default;
  static constexpr size_t PART = size_t(128) << 10;      // a slot is filled by several threads, in parts of this size
  static constexpr int MAX_TASKS = 2 * SLOTS * static_cast<int>(SLOT_BYTES / PART);
  struct Task {
    void *dst;
    const void *src;
    size_t bytes;
    std::atomic<int> *left;
  };
  bool start();
  bool run_one();                              // take one task if there is one
  void submit(void *dst, const void *src, size_t bytes, std::atomic<int> *left);
  void begin();
  void end();
  void helper();

  std::mutex busy_;
  unsigned char *slots_ = nullptr;             // pinned: SLOTS for each direction
  bool pinned_ = false;
  std::vector<std::thread> threads_;
  std::mutex m_;
  std::condition_variable cv_;
  Task tasks_[MAX_TASKS];                      // a ring: from first_task_, queued_ of them (it never allocates)
  int first_task_ = 0, queued_ = 0;
  std::atomic<int> ready_{0}, active_{0};
  std::atomic<bool> stop_{false};
};

template <typename Launch>
cudaError_t HostPipe::run(Events &ev, const std::vector<Piece> &in, const std::vector<Piece> &out, int chunks, cudaStream_t s_in,
                          cudaStream_t s_out, Launch launch) {
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < SLOTS && e == cudaSuccess; ++i) {
    if (!ev.in[i]) e = cudaEventCreateWithFlags(&ev.in[i], cudaEventDisableTiming);
    if (e == cudaSuccess && !ev.out[i]) e = cudaEventCreateWithFlags(&ev.out[i], cudaEventDisableTiming);
  }
  if (e != cudaSuccess) return e;
  auto slot_in = [&](size_t i) { return slots_ + (i % SLOTS) * SLOT_BYTES; };
  auto slot_out = [&](size_t i) { return slots_ + (SLOTS + i % SLOTS) * SLOT_BYTES; };
  std::atomic<int> in_left[SLOTS], out_left[SLOTS];
  for (int i = 0; i < SLOTS; ++i) { in_left[i] = 0; out_left[i] = 0; }
  // counters over the pieces, each only ever ahead of the next
  size_t filled = 0, sent = 0, in_free = 0;                 // input: handed to the helpers, enqueued, slot free again
  size_t fetched = 0, landed = 0, emptied = 0;              // output: enqueued, on the host (handed to the helpers), done
  int launched = 0;
  auto over = [](cudaEvent_t x, cudaError_t &err) {
    const cudaError_t q = cudaEventQuery(x);
    if (q == cudaSuccess) return true;
    if (q != cudaErrorNotReady) err = q;
    return false;
  };
  begin();
  while (e == cudaSuccess && (launched < chunks || emptied < out.size())) {
    bool moved = false;
    while (in_free < sent && over(ev.in[in_free % SLOTS], e)) { ++in_free; moved = true; }
    while (filled < in.size() && filled < in_free + SLOTS) {
      submit(slot_in(filled), in[filled].host, in[filled].bytes, &in_left[filled % SLOTS]);
      ++filled;
      moved = true;
    }
    while (e == cudaSuccess && sent < filled && in_left[sent % SLOTS].load(std::memory_order_acquire) == 0) {
      // (a chunk without input of its own cannot occur: every chunk has at least one image)
      if (in[sent].chunk > launched) break;
      e = cudaMemcpyAsync(in[sent].dev, slot_in(sent), in[sent].bytes, cudaMemcpyHostToDevice, s_in);
      if (e == cudaSuccess) e = cudaEventRecord(ev.in[sent % SLOTS], s_in);
      ++sent;
      moved = true;
      if (e == cudaSuccess && (sent == in.size() || in[sent].chunk != launched)) { e = launch(launched); ++launched; }
    }
    if (in.empty())
      while (e == cudaSuccess && launched < chunks) { e = launch(launched); ++launched; moved = true; }
    while (e == cudaSuccess && fetched < out.size() && out[fetched].chunk < launched && fetched < emptied + SLOTS) {
      e = cudaMemcpyAsync(slot_out(fetched), out[fetched].dev, out[fetched].bytes, cudaMemcpyDeviceToHost, s_out);
      if (e == cudaSuccess) e = cudaEventRecord(ev.out[fetched % SLOTS], s_out);
      ++fetched;
      moved = true;
    }
    while (e == cudaSuccess && landed < fetched && over(ev.out[landed % SLOTS], e)) {
      submit(out[landed].host, slot_out(landed), out[landed].bytes, &out_left[landed % SLOTS]);
      ++landed;
      moved = true;
    }
    while (emptied < landed && out_left[emptied % SLOTS].load(std::memory_order_acquire) == 0) { ++emptied; moved = true; }
    if (!moved) run_one();
  }
  // (after an error too, nobody may still write the slots or the caller's tensors)
  while (run_one()) {}
  for (int i = 0; i < SLOTS; ++i)
    while (in_left[i].load(std::memory_order_acquire) || out_left[i].load(std::memory_order_acquire)) std::this_thread::yield();
  end();
  const cudaError_t e1 = cudaStreamSynchronize(s_in), e2 = cudaStreamSynchronize(s_out);
  return e != cudaSuccess ? e : e1 != cudaSuccess ? e1 : e2;
}

}  // namespace elb
