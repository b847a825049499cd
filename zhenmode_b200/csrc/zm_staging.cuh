// Host copies of a state that lives in ordinary (pageable) memory.
//
// The driver stages a pageable copy itself, on the calling thread, at the speed of
// one core's memcpy, and the first touch of a fresh result array (page faults and
// their zeroing) falls into the same serial copy.  Here several threads stage the
// chunks through pinned slots of their own, two each, so that a thread fills or
// empties one slot while the other is on the bus, and they let the kernel map the
// result's pages while the device computes.  A whole host step on one machine, copied
// directly and staged (six threads): 8 MB of state 1.53 and 1.21 ms, 15 MB 6.8 and
// 1.77, 31 MB 8.2 and 4.0.  How long the driver's own staging takes differs from
// machine to machine (31 MB: 5 to 12 ms).
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

namespace zm {

class HostStage {
 public:
  struct Piece {
    char* host;
    char* dev;
    size_t bytes;
  };
  static constexpr size_t CHUNK = 512 << 10;
  static constexpr int MAX_WORKERS = 6;
  // Making the slots costs the handle's first staged call 1.3 ms.  A call of 20 MB gains that at once (31 MB: 6.6 ms
  // with it, 10 to 13 copied directly; 15 MB 4.1, and 3.8 to 8 directly); from 3 MB on a handle gains 0.04 ms a MB in
  // each call and makes them when it has moved 32 MB (8 MB: 1.21 ms staged, 1.53 directly, 3.5 with the slots);
  // below, both take the same time.
  static constexpr size_t LEAST = 3u << 20, AT_ONCE = 20u << 20, IN_ALL = 32u << 20;

  HostStage() = default;
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;
  ~HostStage() { release(); }

  // Whether every array is pageable host memory that the driver knows nothing of.
  static bool pageable(const void* const* p, int n) {
    for (int q = 0; q < n; ++q) {
      cudaPointerAttributes a{};
      if (cudaPointerGetAttributes(&a, p[q]) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
      }
      if (a.type != cudaMemoryTypeUnregistered) return false;
    }
    return true;
  }

  // Whether a call with pageable arrays of this many bytes is staged.
  bool wanted(size_t bytes) {
    moved_ = std::min(moved_, IN_ALL) + bytes;
    return bytes >= LEAST && (pin_ || bytes >= AT_ONCE || moved_ >= IN_ALL);
  }

  // Pinned slots and events, kept with the solver; false where they cannot be had.
  bool ready() {
    if (pin_) return true;
    workers_ = std::max(1, std::min(MAX_WORKERS, (int)std::thread::hardware_concurrency() / 2));
    if (!pin(2 * CHUNK * workers_)) return false;
    for (int w = 0; w < workers_; ++w)
      for (cudaEvent_t& e : ev_[w])
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
          e = nullptr;
          (void)cudaGetLastError();
          release();
          return false;
        }
    return true;
  }

  // Fields in[0 .. n) -> device on `cs`; then compute(), which queues the work and makes `cs` wait for it and
  // returns whether to go on; then device -> out[0 .. n).  Returns the first CUDA error of the copies; on any
  // return nothing of this call is in flight on `cs` any more.  Throws only what compute() throws.
  template <class Compute>
  cudaError_t run(int device, cudaStream_t cs, const Piece* in, const Piece* out, int n, Compute&& compute) {
    Job job(device, cs, in, out, n);
    std::thread team[MAX_WORKERS];
    try {
      for (int w = 1; w < workers_; ++w)
        team[w] = std::thread([this, &job, w] {
          note(job, cudaSetDevice(job.device));
          upload(job, w);
          populate(job);
          {
            std::unique_lock<std::mutex> lock(job.m);
            job.turn.wait(lock, [&job] { return job.phase.load() != 0; });
          }
          if (job.phase.load() == 1) download(job, w);
        });
    } catch (...) {  // fewer threads, or none, do the same work
    }
    bool go = false;
    try {
      upload(job, 0);
      while (job.sent.load(std::memory_order_acquire) < job.up.count && !job.err.load()) std::this_thread::yield();
      go = !job.err.load() && compute();
    } catch (...) {
      finish(job, team);
      throw;
    }
    if (go) {
      note(job, cudaStreamSynchronize(cs));  // one thread waits for the device; the others sleep
      begin(job, 1);
      download(job, 0);
    }
    finish(job, team);
    return (cudaError_t)job.err.load();
  }

 private:
  // The chunks of some fields, in order.
  struct Chunks {
    const Piece* field;
    size_t count = 0;
    Chunks(const Piece* f, int n) : field(f) {
      for (int q = 0; q < n; ++q) count += (f[q].bytes + CHUNK - 1) / CHUNK;
    }
    Piece operator[](size_t c) const {
      const Piece* f = field;
      for (size_t m; c >= (m = (f->bytes + CHUNK - 1) / CHUNK); c -= m) ++f;
      const size_t o = c * CHUNK;
      return {f->host + o, f->dev + o, std::min(CHUNK, f->bytes - o)};
    }
  };
  struct Job {
    int device;
    cudaStream_t cs;
    Chunks up, down;
    std::atomic<size_t> next_up{0}, sent{0}, next_page{0}, next_down{0};
    std::atomic<int> phase{0};  // 1: the results may be fetched, 2: there are none
    std::atomic<int> err{0};
    std::mutex m;
    std::condition_variable turn;
    Job(int dv, cudaStream_t s, const Piece* in, const Piece* out, int n) : device(dv), cs(s), up(in, n), down(out, n) {}
  };

  static void note(Job& job, cudaError_t e) {
    int none = 0;
    if (e != cudaSuccess) job.err.compare_exchange_strong(none, (int)e);
  }
  // Page-locked memory of huge pages: the first host step of a handle pays for it.  cudaHostAlloc
  // of 6 MB took 2.2 to 11 ms, a mapping of huge pages and its registration take 0.8.
  bool pin(size_t bytes) {
    constexpr size_t HUGE_PAGE = 2u << 20;
    const size_t len = (bytes + HUGE_PAGE - 1) / HUGE_PAGE * HUGE_PAGE + HUGE_PAGE;
    void* m = mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED) return false;
    char* p = reinterpret_cast<char*>(((uintptr_t)m + HUGE_PAGE - 1) / HUGE_PAGE * HUGE_PAGE);
#ifdef MADV_HUGEPAGE
    (void)madvise(p, len - HUGE_PAGE, MADV_HUGEPAGE);  // where there are none, ordinary pages
#endif
    if (cudaHostRegister(p, bytes, cudaHostRegisterDefault) != cudaSuccess) {
      (void)cudaGetLastError();
      munmap(m, len);
      return false;
    }
    map_ = m;
    map_len_ = len;
    pin_ = p;
    return true;
  }
  void release() {
    for (auto& w : ev_)
      for (cudaEvent_t& e : w) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
      }
    if (!pin_) return;
    (void)cudaHostUnregister(pin_);
    munmap(map_, map_len_);
    pin_ = nullptr;
  }

  char* slot(int w, int s) const { return pin_ + (size_t)(2 * w + s) * CHUNK; }

  void upload(Job& job, int w) {
    bool used[2] = {false, false};
    int s = 0;
    for (size_t c; !job.err.load() && (c = job.next_up.fetch_add(1)) < job.up.count; s ^= 1) {
      const Piece p = job.up[c];
      if (used[s]) note(job, cudaEventSynchronize(ev_[w][s]));
      std::memcpy(slot(w, s), p.host, p.bytes);
      note(job, cudaMemcpyAsync(p.dev, slot(w, s), p.bytes, cudaMemcpyHostToDevice, job.cs));
      note(job, cudaEventRecord(ev_[w][s], job.cs));
      used[s] = true;
      job.sent.fetch_add(1, std::memory_order_release);
    }
    for (int q = 0; q < 2; ++q)
      if (used[q]) note(job, cudaEventSynchronize(ev_[w][q]));
  }

  // Maps the whole pages of the results; their contents stay as they are, and where the system knows no
  // such request the download faults them in.
  void populate(Job& job) {
#ifdef MADV_POPULATE_WRITE
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    for (size_t c; job.phase.load() == 0 && (c = job.next_page.fetch_add(1)) < job.down.count;) {
      const Piece p = job.down[c];
      const uintptr_t a = ((uintptr_t)p.host + page - 1) / page * page;
      const uintptr_t b = ((uintptr_t)p.host + p.bytes) / page * page;
      if (b > a && madvise(reinterpret_cast<void*>(a), b - a, MADV_POPULATE_WRITE) != 0) return;
    }
#else
    (void)job;
#endif
  }

  void download(Job& job, int w) {
    Piece pending{nullptr, nullptr, 0};
    int s = 0;
    for (;;) {
      const size_t c = job.err.load() ? job.down.count : job.next_down.fetch_add(1);
      const bool more = c < job.down.count;
      const Piece p = more ? job.down[c] : Piece{nullptr, nullptr, 0};
      if (more) {
        note(job, cudaMemcpyAsync(slot(w, s), p.dev, p.bytes, cudaMemcpyDeviceToHost, job.cs));
        note(job, cudaEventRecord(ev_[w][s], job.cs));
      }
      if (pending.bytes) {
        note(job, cudaEventSynchronize(ev_[w][s ^ 1]));
        if (!job.err.load()) std::memcpy(pending.host, slot(w, s ^ 1), pending.bytes);
      }
      pending = p;
      if (!more) return;
      s ^= 1;
    }
  }

  static void begin(Job& job, int phase) {
    std::lock_guard<std::mutex> lock(job.m);
    job.phase.store(phase);
    job.turn.notify_all();
  }
  void finish(Job& job, std::thread (&team)[MAX_WORKERS]) {
    if (job.phase.load() == 0) begin(job, 2);
    for (std::thread& t : team)
      if (t.joinable()) t.join();
    note(job, cudaStreamSynchronize(job.cs));
  }

  size_t moved_ = 0;     // bytes of the calls so far
  void* map_ = nullptr;  // the mapping that holds the slots
  size_t map_len_ = 0;
  char* pin_ = nullptr;
  int workers_ = 1;
  cudaEvent_t ev_[MAX_WORKERS][2] = {};
};

}  // namespace zm
