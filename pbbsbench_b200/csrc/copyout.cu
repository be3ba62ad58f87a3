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
#include <mutex>
#include <vector>

#include "hostmove.h"
#include "internal.cuh"

namespace pbg {
namespace {

using hostmove::Moved;
using hostmove::PIECE;
using hostmove::Piece;
using hostmove::RING;
constexpr size_t MIN_STAGED = 6ull << 20;  // bytes of a call; see above

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

// The device's copies into the ring, on stream s.
struct RingLink {
  Ring& r;
  cudaStream_t s;
  cudaError_t e = cudaSuccess;
  bool issue(const Piece& p, int slot) {
    e = cudaMemcpyAsync(r.mem + slot * PIECE, p.src, p.len, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaEventRecord(r.ev[slot], s);
    return e == cudaSuccess;
  }
  bool wait(int slot) {
    e = cudaEventSynchronize(r.ev[slot]);
    return e == cudaSuccess;
  }
};

// The pageable copies' pieces; false when there is no memory for the list.
bool cut(const HostCopy* copies, int count, std::vector<Piece>* out) {
  try {
    for (int i = 0; i < count; i++) {
      const HostCopy& c = copies[i];
      if (!c.dst || !pageable(c.dst)) continue;
      for (size_t o = 0; o < c.bytes; o += PIECE)
        out->push_back({static_cast<char*>(c.dst) + o, static_cast<const char*>(c.src) + o, std::min(PIECE, c.bytes - o)});
    }
  } catch (...) {
    return false;
  }
  return true;
}

}  // namespace

int copy_out(const HostCopy* copies, int count, cudaStream_t s) {
  size_t total = 0;
  for (int i = 0; i < count; i++) total += copies[i].dst ? copies[i].bytes : 0;
  const bool large = total >= MIN_STAGED;
  auto plain = [&](bool pageables) -> int {
    for (int i = 0; i < count; i++) {
      const HostCopy& c = copies[i];
      if (c.dst && c.bytes && (!large || pageable(c.dst)) == pageables)
        PBG_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, s));
    }
    return PBG_OK;
  };
  bool staged = false;
  if (large) {
    const int rc = plain(false);
    if (rc) return rc;
    std::vector<Piece> pieces;
    std::unique_lock<std::mutex> lk(g_ring.mu, std::defer_lock);
    if (cut(copies, count, &pieces) && !pieces.empty() && lk.try_lock() && ring_ready(g_ring)) {
      RingLink link{g_ring, s};
      const Moved m = hostmove::move_pieces(pieces, g_ring.mem, link);
      if (m == Moved::LINK_FAILED) {
        cudaStreamSynchronize(s);  // no copy into the ring is left in flight
        return cuda_fail(link.e, "result copy");
      }
      staged = m == Moved::ALL;
    }
  }
  if (!staged) {
    const int rc = plain(true);
    if (rc) return rc;
  }
  PBG_CUDA(cudaStreamSynchronize(s));
  return PBG_OK;
}

}  // namespace pbg
