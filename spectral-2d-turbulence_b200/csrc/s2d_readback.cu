// s2d_readback.cu -- device fields into the caller's pageable memory.
//
// A copy straight into pageable memory runs at 4-5 GB/s on a fresh array: one thread of the
// driver touches each page for the first time and copies it, behind every transfer.  Here the
// transfers go through pinned slots at link speed, and up to four threads (each with two slots,
// one filling while it empties the other) share the page faults and the copies.  B200 host, 16
// cores, into a fresh array: 8 MB 1.85 -> 0.8 ms, 33 MB 7.6 -> 2.2 ms, 134 MB 29 -> 9.8 ms;
// one thread with two slots takes 0.8, 3.4 and 22 ms.
#include "s2d_readback.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace s2d {
namespace {

constexpr int kThreads = 4;
constexpr size_t kSlot = size_t(1) << 20;
// a second thread pays from two slots' worth of bytes on (its start takes ~20 us); below
// kDirect a plain copy takes no longer than the staged one
constexpr size_t kPerThread = 2 * kSlot, kDirect = size_t(256) << 10;
// making the slots and giving them back takes 4-6 ms, as long as some 16 MB of plain copies: a
// program that reads less than that from its solvers never pays for them (512^2 solver read
// once: 5-10 ms against 1.1 ms)
constexpr size_t kMakeFrom = size_t(16) << 20;

struct Staging {
  int refs = 0;
  std::mutex busy;   // one read at a time; a read that finds it taken copies directly
  bool tried = false;
  size_t read = 0;   // bytes asked for so far
  char* pinned = nullptr;
  cudaStream_t stream[kThreads] = {};
  cudaEvent_t filled[2 * kThreads] = {}, ready = nullptr;

  bool make(size_t bytes) {   // once it pays, by the holder of `busy`
    if (tried) return pinned != nullptr;
    if (read < kMakeFrom) read += bytes;
    if (read < kMakeFrom) return false;
    tried = true;
    bool ok = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) == cudaSuccess;
    for (cudaStream_t& s : stream) ok = ok && cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    for (cudaEvent_t& e : filled) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (ok && cudaHostAlloc(&pinned, 2 * kThreads * kSlot, cudaHostAllocDefault) != cudaSuccess) pinned = nullptr;
    cudaGetLastError();
    return pinned != nullptr;
  }
  ~Staging() {
    if (pinned) cudaFreeHost(pinned);
    for (cudaStream_t s : stream)
      if (s) cudaStreamDestroy(s);
    for (cudaEvent_t e : filled)
      if (e) cudaEventDestroy(e);
    if (ready) cudaEventDestroy(ready);
  }

  // thread t of `threads`: chunks t, t + threads, ... (chunk <= kSlot)
  cudaError_t share(int t, int threads, size_t chunk, char* dst, const char* src, size_t bytes) {
    char* const slot[2] = {pinned + 2 * t * kSlot, pinned + (2 * t + 1) * kSlot};
    const size_t chunks = (bytes + chunk - 1) / chunk;
    auto fill = [&](size_t c, int b) {
      const size_t lo = c * chunk;
      const cudaError_t e = cudaMemcpyAsync(slot[b], src + lo, std::min(chunk, bytes - lo), cudaMemcpyDeviceToHost, stream[t]);
      return e == cudaSuccess ? cudaEventRecord(filled[2 * t + b], stream[t]) : e;
    };
    cudaError_t e = cudaStreamWaitEvent(stream[t], ready, 0);
    int b = 0;
    if (e == cudaSuccess && (size_t)t < chunks) e = fill(t, 0);
    for (size_t c = t; e == cudaSuccess && c < chunks; c += threads, b ^= 1) {
      if (c + threads < chunks) e = fill(c + threads, b ^ 1);
      if (e == cudaSuccess) e = cudaEventSynchronize(filled[2 * t + b]);
      if (e == cudaSuccess) std::memcpy(dst + c * chunk, slot[b], std::min(chunk, bytes - c * chunk));
    }
    if (e != cudaSuccess) cudaStreamSynchronize(stream[t]);   // no transfer into a slot outlives the read
    return e;
  }
};

std::mutex g_mu;
std::map<int, std::shared_ptr<Staging>> g_staging;   // by device

cudaError_t read_direct(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
  return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
}

}  // namespace

void readback_retain(int dev) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_staging.find(dev);
  if (it == g_staging.end()) {
    try {
      it = g_staging.emplace(dev, std::make_shared<Staging>()).first;
    } catch (const std::bad_alloc&) {
      return;   // fields are then copied directly
    }
  }
  ++it->second->refs;
}

void readback_release(int dev) {
  std::shared_ptr<Staging> last;   // destroyed outside the lock
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_staging.find(dev);
  if (it != g_staging.end() && --it->second->refs == 0) {
    last = std::move(it->second);
    g_staging.erase(it);
  }
}

cudaError_t read_back(int dev, void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaPointerAttributes at{};
  // pageable destinations only (others are the copy engine's), and not inside a capture
  if (bytes < kDirect || cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone ||
      cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type != cudaMemoryTypeUnregistered) {
    cudaGetLastError();
    return read_direct(dst, src, bytes, stream);
  }
  std::shared_ptr<Staging> s;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_staging.find(dev);
    if (it != g_staging.end()) s = it->second;
  }
  std::unique_lock<std::mutex> busy;
  if (s) busy = std::unique_lock<std::mutex>(s->busy, std::try_to_lock);
  if (!s || !busy.owns_lock() || !s->make(bytes)) return read_direct(dst, src, bytes, stream);
  cudaError_t e = cudaEventRecord(s->ready, stream);
  if (e != cudaSuccess) return e;
  const int cores = std::max(1, (int)std::thread::hardware_concurrency());
  int threads = (int)std::min<size_t>(std::min(kThreads, cores), std::max<size_t>(1, bytes / kPerThread));
  // four chunks a thread at least, so that a short read overlaps its transfer with its copies
  const size_t chunk = std::min(kSlot, std::max(size_t(64) << 10, bytes / (4 * threads) & ~size_t(4095)));
  char* const d = static_cast<char*>(dst);
  const char* const p = static_cast<const char*>(src);
  cudaError_t err[kThreads] = {};
  std::thread team[kThreads];
  int started = 1;
  auto run = [&](int t) {
    cudaError_t r = t ? cudaSetDevice(dev) : cudaSuccess;
    if (r == cudaSuccess) r = s->share(t, threads, chunk, d, p, bytes);
    err[t] = r;
  };
  for (; started < threads; ++started) {
    try {
      team[started] = std::thread([&run, t = started] {
        // what a capture on another thread forbids is for the caller's thread, in its mode, to meet
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        run(t);
      });
    } catch (...) {   // no thread to be had, or no memory for one: its share is done below
      break;
    }
  }
  run(0);
  for (int t = started; t < threads; ++t) run(t);   // shares of threads that did not start
  for (int t = 1; t < started; ++t) team[t].join();
  for (int t = 0; t < threads; ++t)
    if (err[t] != cudaSuccess) return err[t];
  return cudaSuccess;
}

}  // namespace s2d
