// copyout.cu -- results from device memory to the caller's host memory.
//
// A copy to pageable memory goes through the driver's staging on one host
// thread, which also takes the page faults of a freshly allocated result
// array: parents and levels of rMat 2^20 (8 MB into new arrays) were 1.7 ms
// of a 1.8 ms call.  Large results for pageable memory go through a pinned
// ring here instead: the device copies piece after piece into it and several
// host threads move each piece on, so the faults are taken in parallel and
// overlap the link: rMat 2^20 2.0 -> 0.99 ms a call, randLocal 6,000,001 (48 MB
// of results) 13.2 -> 5.6 ms.  The line (MIN_STAGED): results of 5.6 MB in all
// mostly go to arrays whose pages the process has already (0.75 ms plain,
// 1.03 through the ring, whose threads cost 0.1-0.2 ms to start and wake);
// from about 6.4 MB the allocator maps them anew (3.4 ms plain, 1.3 ms).
// Pinned destinations get the plain copy, at the link's rate.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "internal.cuh"

namespace pbg {
namespace {

constexpr size_t PIECE = 2ull << 20;
constexpr int RING = 8;                       // pieces in flight: 16 MiB of pinned memory
constexpr size_t MIN_STAGED = 6ull << 20;     // pageable bytes of a call; see below
constexpr size_t MIN_PART = 1ull << 20;       // bytes a thread is started for
constexpr unsigned MAX_THREADS = 8;

// The ring is pinned on first use (a few ms) and kept for the process, as the
// file transfers' pieces are; a call that finds it in use copies plainly.
struct Ring {
  std::mutex mu;
  char* mem = nullptr;
  cudaEvent_t ev[RING] = {};
  int device = -1;  // of the events
};
Ring g_ring;

bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

struct Piece {
  char* dst;
  const char* src;
  size_t len;
};

// Events and memory for the current device; false: not to be had.
bool ring_ready(Ring& r) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (!r.mem && cudaHostAlloc(&r.mem, PIECE * RING, cudaHostAllocPortable) != cudaSuccess) {
    r.mem = nullptr;
    cudaGetLastError();
    return false;
  }
  if (r.device != dev) {
    for (auto& e : r.ev) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    r.device = -1;
    for (auto& e : r.ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        cudaGetLastError();
        return false;
      }
    r.device = dev;
  }
  return true;
}

// Moves the pieces through the ring; every piece is on the host on return.
cudaError_t move_pieces(Ring& r, const std::vector<Piece>& pieces, cudaStream_t s) {
  const size_t n = pieces.size();
  size_t bytes = 0;
  for (const Piece& p : pieces) bytes += p.len;
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  unsigned parts = (unsigned)std::min<size_t>(std::min(MAX_THREADS, hw), bytes / MIN_PART);
  if (parts < 1) parts = 1;
  std::mutex mu;
  std::condition_variable cv;
  size_t ready = 0;  // pieces that have arrived in the ring
  bool stop = false;
  std::vector<std::atomic<unsigned>> done(n);  // parts of each piece moved on
  for (auto& d : done) d.store(0);
  auto move_part = [&](size_t i, unsigned k, unsigned of) {
    const Piece& p = pieces[i];
    const size_t a = p.len * k / of, b = p.len * (k + 1) / of;
    std::memcpy(p.dst + a, r.mem + (i % RING) * PIECE + a, b - a);
    done[i].fetch_add(1, std::memory_order_release);
  };
  std::atomic<unsigned> team{parts};  // threads that share a piece, fixed before the first one is ready
  auto work = [&](unsigned k) {
    for (size_t i = 0; i < n; i++) {
      {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return ready > i || stop; });
        if (ready <= i) return;
      }
      move_part(i, k, team.load(std::memory_order_relaxed));
    }
  };
  std::vector<std::thread> th;
  th.reserve(parts);
  try {
    for (unsigned k = 1; k < parts; k++) th.emplace_back(work, k);
  } catch (const std::system_error&) {  // no more threads: the ones there are share the pieces
    team.store((unsigned)th.size() + 1);
  }
  const unsigned of = team.load();
  cudaError_t e = cudaSuccess;
  size_t issued = 0;
  for (size_t i = 0; i < n && e == cudaSuccess; i++) {
    while (issued < n && issued < i + RING && e == cudaSuccess) {
      if (issued >= RING) {  // its slot's previous piece has been moved on
        while (done[issued - RING].load(std::memory_order_acquire) < of) {
          if (issued > i) break;
          std::this_thread::yield();
        }
        if (done[issued - RING].load(std::memory_order_acquire) < of) break;
      }
      const Piece& p = pieces[issued];
      e = cudaMemcpyAsync(r.mem + (issued % RING) * PIECE, p.src, p.len, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaEventRecord(r.ev[issued % RING], s);
      if (e == cudaSuccess) issued++;
    }
    if (e == cudaSuccess) e = cudaEventSynchronize(r.ev[i % RING]);
    if (e != cudaSuccess) break;
    {
      std::lock_guard<std::mutex> lk(mu);
      ready = i + 1;
    }
    cv.notify_all();
    move_part(i, 0, of);
  }
  {
    std::lock_guard<std::mutex> lk(mu);
    if (e != cudaSuccess) stop = true;
  }
  cv.notify_all();
  for (auto& t : th) t.join();
  if (e != cudaSuccess) cudaStreamSynchronize(s);  // no copy into the ring is left in flight
  return e;
}

}  // namespace

int copy_out(const HostCopy* copies, int count, cudaStream_t s) {
  std::vector<Piece> pieces;
  size_t total = 0;
  for (int i = 0; i < count; i++) total += copies[i].dst ? copies[i].bytes : 0;
  for (int i = 0; i < count; i++) {
    const HostCopy& c = copies[i];
    if (!c.dst || !c.bytes) continue;
    if (total < MIN_STAGED || !pageable(c.dst)) {
      PBG_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, s));
      continue;
    }
    for (size_t o = 0; o < c.bytes; o += PIECE)
      pieces.push_back({static_cast<char*>(c.dst) + o, static_cast<const char*>(c.src) + o,
                        std::min(PIECE, c.bytes - o)});
  }
  if (!pieces.empty()) {
    std::unique_lock<std::mutex> lk(g_ring.mu, std::try_to_lock);
    if (lk.owns_lock() && ring_ready(g_ring)) {
      const cudaError_t e = move_pieces(g_ring, pieces, s);
      if (e != cudaSuccess) return cuda_fail(e, "result copy");
    } else {
      for (const Piece& p : pieces)
        PBG_CUDA(cudaMemcpyAsync(p.dst, p.src, p.len, cudaMemcpyDeviceToHost, s));
    }
  }
  PBG_CUDA(cudaStreamSynchronize(s));
  return PBG_OK;
}

}  // namespace pbg
