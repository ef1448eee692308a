// af_xfer.cu -- host<->device row-block copies at the link's rate from
// pinned or pageable host memory (see af_xfer.h).
#include "af_xfer.h"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace af {
namespace {

constexpr int kBufs = 8;                // pinned buffers: chunks in flight
constexpr size_t kBufBytes = 4u << 20;  // each: the longest chunk
// The size of a chunk; a quarter of it is one thread's turn at the host side.
// A short copy wants the first chunk on its way soon and a ring that stays in
// the caches (8 MB to the device: 1 MB chunks 0.45 ms, 4 MB 0.49; from it 0.35
// and 0.51), a long one few calls (537 MB to the device: 1 MB chunks 15.9 ms,
// 2 MB 12.1, 4 MB 12.0, but 60 MB 1.8, 1.6 and 2.3), and one into memory touched
// for the first time long turns, as the threads meet in its pages (a 2731 x
// 2747 grid's three fields: 1 MB chunks 11.8 ms, 2 MB 10.3, 4 MB 9.6; 8192 x
// 8192: 102, 92 and 87).  Rows want two or more to a chunk (211 rows of 1.6 MB
// from the device: 2 MB 8.6 ms, 4 MB 7.0).
size_t chunk_bytes(size_t width, size_t rows, bool to_device) {
  if (width > 512u << 10) return kBufBytes;
  return width * rows < (24u << 20) ? 1u << 20 : to_device ? 2u << 20 : 4u << 20;
}
// Smaller copies go the driver's own way, which is as quick (2 MB 0.14 ms).
constexpr size_t kMinStaged = 2u << 20;
// A worker that has run out of pieces looks for the next copy for this long
// before it sleeps: waking a sleeping one can take a few tenths of a
// millisecond, as long as a copy of several MB, and copies come in series (the
// fields of a grid, the members of an ensemble).
constexpr std::chrono::microseconds kLinger(200);

// The host side of one copy: rows x width bytes between the caller's memory and
// the ring of buffers, cut into chunks of `rpc` rows (chunk c in buffer c %
// kBufs) and pieces of `rpp` rows.  Threads take pieces in order, none of a
// chunk at or past `limit`, which the calling thread moves as buffers become
// free (to the device) or arrive (from it).
struct Job {
  char* host;
  size_t pitch, width, rows, rpc, rpp;
  char* ring;
  size_t stride;  // of the ring's buffers
  bool to_device;
  size_t pieces_per_chunk, chunks;
  std::atomic<size_t> next{0}, limit{0};
  std::unique_ptr<std::atomic<unsigned>[]> done;  // pieces of each chunk

  size_t pieces_of(size_t c) const {
    return (std::min(rpc, rows - c * rpc) + rpp - 1) / rpp;
  }
  // Takes and copies one piece; false when none may be taken now.
  bool turn() {
    size_t i = next.load(std::memory_order_relaxed);
    for (;;) {
      const size_t c = i / pieces_per_chunk;
      if (c >= chunks || c >= limit.load(std::memory_order_acquire)) return false;
      if (i % pieces_per_chunk >= pieces_of(c)) {  // a last, shorter chunk
        if (next.compare_exchange_weak(i, (c + 1) * pieces_per_chunk)) i = (c + 1) * pieces_per_chunk;
        continue;
      }
      if (next.compare_exchange_weak(i, i + 1)) break;
    }
    const size_t c = i / pieces_per_chunk, k = i % pieces_per_chunk;
    const size_t r0 = c * rpc + k * rpp, r1 = std::min({r0 + rpp, (c + 1) * rpc, rows});
    char* buf = ring + (c % kBufs) * stride + k * rpp * width;
    char* mem = host + r0 * pitch;
    if (pitch == width) {
      std::memcpy(to_device ? buf : mem, to_device ? mem : buf, (r1 - r0) * width);
    } else {
      for (size_t r = r0; r < r1; r++, buf += width, mem += pitch)
        std::memcpy(to_device ? buf : mem, to_device ? mem : buf, width);
    }
    done[c].fetch_add(1, std::memory_order_release);
    return true;
  }
  bool chunk_done(size_t c) const {
    return done[c].load(std::memory_order_acquire) == pieces_of(c);
  }
  bool over() const { return next.load(std::memory_order_relaxed) >= chunks * pieces_per_chunk; }
};

// Worker threads that take turns at the current copy.  The calling thread takes
// turns too and never waits for a worker that is not in the middle of one.
class CopyPool {
 public:
  explicit CopyPool(int workers) {
    try {
      for (int k = 0; k < workers; k++) th_.emplace_back([this] { loop(); });
    } catch (const std::system_error&) {  // no more threads: those there are, or the caller alone
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> g(mu_);
      stop_ = true;
      gen_++;
    }
    cv_.notify_all();
    for (auto& t : th_) t.join();
  }
  void post(std::shared_ptr<Job> job) {
    bool wake;
    {
      std::lock_guard<std::mutex> g(mu_);
      job_ = std::move(job);
      gen_++;
      wake = asleep_ > 0;
    }
    if (wake) cv_.notify_all();
  }
  // The workers drop the copy (a piece in hand is finished by its own thread;
  // the job and its counters live until the last of them lets go).
  void retire() {
    std::lock_guard<std::mutex> g(mu_);
    job_.reset();
  }

 private:
  void loop() {
    unsigned long long seen = 0;
    for (;;) {
      std::shared_ptr<Job> job;
      const auto until = std::chrono::steady_clock::now() + kLinger;
      while (gen_.load(std::memory_order_acquire) == seen &&
             std::chrono::steady_clock::now() < until)
        std::this_thread::yield();
      {
        std::unique_lock<std::mutex> l(mu_);
        if (gen_.load() == seen) {
          asleep_++;
          cv_.wait(l, [&] { return stop_ || gen_.load() != seen; });
          asleep_--;
        }
        if (stop_) return;
        seen = gen_.load();
        job = job_;
      }
      while (job && !job->over())
        if (!job->turn()) std::this_thread::yield();
    }
  }
  std::mutex mu_;
  std::condition_variable cv_;
  std::shared_ptr<Job> job_;  // under mu_, as stop_ and asleep_
  std::atomic<unsigned long long> gen_{0};
  int asleep_ = 0;
  bool stop_ = false;
  std::vector<std::thread> th_;
};

// The process's pinned buffers and copy threads, made on first use.
// Never freed: they live until the process exits (CUDA's own teardown at
// exit makes freeing pinned memory from a static destructor unsafe).
struct Staging {
  std::mutex mu;  // one staged copy at a time
  char* ring = nullptr;
  CopyPool* pool = nullptr;
  bool tried = false;
  pid_t pid = 0;
};

Staging& staging() {
  static Staging* s = new Staging;
  return *s;
}

// Under s.mu.  A forked child starts over (its parent's threads are gone).
bool ready(Staging& s) {
  if (s.pid != getpid()) {
    s.pid = getpid();
    s.ring = nullptr;
    s.pool = nullptr;
    s.tried = false;
  }
  if (!s.tried) {
    s.tried = true;
    void* p = nullptr;
    if (cudaHostAlloc(&p, kBufs * kBufBytes, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    s.ring = static_cast<char*>(p);
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
    if (p) s.pool = new CopyPool(std::max(0, std::min(7, hw - 1)));
  }
  return s.ring != nullptr;
}

// Pageable host memory: the driver cannot DMA it directly.  A pointer CUDA
// cannot classify goes to the driver, which reports the error.
bool pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// One block of rows; rows without gaps on either side as one run.
cudaError_t copy_rows(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                      size_t rows, cudaMemcpyKind kind, cudaStream_t st) {
  if (dpitch == width && spitch == width)
    return cudaMemcpyAsync(dst, src, width * rows, kind, st);
  return cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows, kind, st);
}

// The staged copy between `host` (pageable) and `dev`.
cudaError_t staged(Staging& S, char* dev, size_t dpitch, char* host, size_t hpitch, size_t width,
                   size_t rows, bool to_device, cudaStream_t st) {
  auto job = std::make_shared<Job>();
  Job& J = *job;
  J.host = host;
  J.pitch = hpitch;
  J.width = width;
  J.rows = rows;
  J.stride = chunk_bytes(width, rows, to_device);
  J.rpp = std::max<size_t>(1, J.stride / 4 / width);
  J.rpc = std::max<size_t>(1, J.stride / width / J.rpp) * J.rpp;  // whole pieces
  J.ring = S.ring;
  J.to_device = to_device;
  J.pieces_per_chunk = (J.rpc + J.rpp - 1) / J.rpp;
  J.chunks = (rows + J.rpc - 1) / J.rpc;
  J.done.reset(new std::atomic<unsigned>[J.chunks]);
  for (size_t c = 0; c < J.chunks; c++) J.done[c].store(0);

  cudaEvent_t ev[kBufs] = {};
  cudaError_t e = cudaSuccess;
  for (size_t b = 0; b < kBufs && b < J.chunks && e == cudaSuccess; b++)
    e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
  size_t issued = 0;  // chunks whose device copy has been issued ...
  size_t moved = 0;   // ... and has been seen to finish
  auto issue = [&]() {
    const size_t c = issued, r = c * J.rpc, n = std::min(J.rpc, rows - r);
    char* buf = S.ring + (c % kBufs) * J.stride;
    e = to_device
            ? copy_rows(dev + r * dpitch, dpitch, buf, width, width, n, cudaMemcpyHostToDevice, st)
            : copy_rows(buf, width, dev + r * dpitch, dpitch, width, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaEventRecord(ev[c % kBufs], st);
    issued++;
  };
  auto look = [&]() {  // whether the oldest issued copy has finished
    const cudaError_t q = cudaEventQuery(ev[moved % kBufs]);
    if (q == cudaErrorNotReady) return false;
    if (q != cudaSuccess) e = q;
    moved++;
    return true;
  };
  if (e == cudaSuccess) {
    if (to_device) {
      J.limit.store(kBufs, std::memory_order_release);
      S.pool->post(job);
      while (issued < J.chunks && e == cudaSuccess) {
        if (J.chunk_done(issued)) {
          issue();
        } else if (moved < issued && look()) {
          J.limit.store(moved + kBufs, std::memory_order_release);
        } else if (!J.turn()) {
          std::this_thread::yield();
        }
      }
    } else {
      while (issued < J.chunks && issued < kBufs && e == cudaSuccess) issue();
      // What the stream had to do before this copy is waited for here: the
      // threads are asked when there is something to drain.
      if (e == cudaSuccess) e = cudaEventSynchronize(ev[0]);
      if (e == cudaSuccess) S.pool->post(job);
      size_t drained = 0;
      while (drained < J.chunks && e == cudaSuccess) {
        if (moved < issued && look()) {
          J.limit.store(moved, std::memory_order_release);
        } else if (drained < moved && J.chunk_done(drained)) {
          drained++;
          if (issued < J.chunks) issue();
        } else if (!J.turn()) {
          std::this_thread::yield();
        }
      }
    }
  }
  // Nobody touches the caller's memory or the ring past here: every piece
  // handed out is done (after an error too), every device copy has finished.
  if (e != cudaSuccess) {
    const size_t handed = J.next.exchange(J.chunks * J.pieces_per_chunk);
    for (size_t i = 0; i < handed; i++) {
      const size_t c = i / J.pieces_per_chunk;
      if (i % J.pieces_per_chunk >= J.pieces_of(c)) continue;
      const size_t upto =
          std::min(handed - c * J.pieces_per_chunk, J.pieces_of(c));  // handed out of chunk c
      while (J.done[c].load(std::memory_order_acquire) < upto) std::this_thread::yield();
      i = (c + 1) * J.pieces_per_chunk - 1;
    }
  }
  S.pool->retire();
  for (int b = 0; b < kBufs; b++)
    if (ev[b]) {
      const cudaError_t e2 = cudaEventSynchronize(ev[b]);
      if (e == cudaSuccess) e = e2;
      cudaEventDestroy(ev[b]);
    }
  return e;
}

cudaError_t copy2d(char* dev, size_t dpitch, char* host, size_t hpitch, size_t width, size_t rows,
                   bool to_device, cudaStream_t st) {
  if (rows == 0 || width == 0) return cudaSuccess;
  const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  auto direct = [&] {
    return to_device ? copy_rows(dev, dpitch, host, hpitch, width, rows, kind, st)
                     : copy_rows(host, hpitch, dev, dpitch, width, rows, kind, st);
  };
  if (width * rows < kMinStaged || !pageable(host)) return direct();
  Staging& S = staging();
  std::lock_guard<std::mutex> g(S.mu);
  if (!ready(S)) return direct();
  const bool dense = dpitch == width && hpitch == width;
  if (!dense && width <= kBufBytes)
    return staged(S, dev, dpitch, host, hpitch, width, rows, to_device, st);
  // One run without gaps, or rows longer than a buffer one by one: what divides
  // into blocks through the ring, the rest straight.
  constexpr size_t kBlock = 256u << 10;
  const size_t run = dense ? width * rows : width, whole = run / kBlock, rest = run % kBlock;
  for (size_t r = 0; r < (dense ? 1 : rows); r++) {
    char *d = dev + r * dpitch, *h = host + r * hpitch;
    cudaError_t e = staged(S, d, kBlock, h, kBlock, kBlock, whole, to_device, st);
    d += whole * kBlock, h += whole * kBlock;
    if (e == cudaSuccess && rest)
      e = cudaMemcpyAsync(to_device ? d : h, to_device ? h : d, rest, kind, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t copy2d_h2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                       size_t rows, cudaStream_t st) {
  return copy2d(static_cast<char*>(dst), dpitch, static_cast<char*>(const_cast<void*>(src)), spitch,
                width, rows, true, st);
}

cudaError_t copy2d_d2h(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                       size_t rows, cudaStream_t st) {
  return copy2d(static_cast<char*>(const_cast<void*>(src)), spitch, static_cast<char*>(dst), dpitch,
                width, rows, false, st);
}

}  // namespace af
