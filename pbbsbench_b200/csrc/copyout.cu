// copyout.cu -- results from device memory to the caller's host memory.
//
// A copy to pageable memory goes through the driver's staging on one host
// thread, which also takes the page faults of a freshly allocated result
// array: parents and levels of rMat 2^20 (8 MB into new arrays) were 1.7 ms
// of a 1.8 ms call.  Results that are large, or whose memory has no pages yet
// (worth_ring in hostmove.h: the lines and what they measured), go through a
// pinned ring here instead: the device copies piece after piece into it and
// several host threads move each piece on, so the faults are taken in parallel
// and overlap the link: rMat 2^20 into new arrays 2.0 -> 0.99 ms a call,
// randLocal 6,000,001 (48 MB of results) 13.2 -> 5.6 ms.  Pinned destinations
// get the plain copy, at the link's rate.
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

// The pieces of the copies marked in `ring`; false when there is no memory for
// the list.
bool cut(const HostCopy* copies, int count, const bool* ring, std::vector<Piece>* out) {
  try {
    for (int i = 0; i < count; i++)
      for (size_t o = 0; ring[i] && o < copies[i].bytes; o += PIECE)
        out->push_back({static_cast<char*>(copies[i].dst) + o, static_cast<const char*>(copies[i].src) + o,
                        std::min(PIECE, copies[i].bytes - o)});
  } catch (...) {
    return false;
  }
  return true;
}

}  // namespace

int copy_out(const HostCopy* copies, int count, cudaStream_t s) {
  constexpr int MAX = 2;
  if (count > MAX) return fail(PBG_ERR_ARG, "copy_out: too many copies");
  hostmove::Range to[MAX];
  bool ring[MAX] = {};  // the pageable ones, where the call takes the ring
  size_t total = 0;
  int nto = 0;
  for (int i = 0; i < count; i++) total += copies[i].dst ? copies[i].bytes : 0;
  for (int i = 0; i < count && total >= hostmove::MIN_RING; i++) {
    ring[i] = copies[i].dst && copies[i].bytes && pageable(copies[i].dst);
    if (ring[i]) to[nto++] = {copies[i].dst, copies[i].bytes};
  }
  const bool worth = hostmove::worth_ring(to, nto);
  auto plain = [&](bool want) -> int {
    for (int i = 0; i < count; i++)
      if (copies[i].dst && copies[i].bytes && (worth && ring[i]) == want)
        PBG_CUDA(cudaMemcpyAsync(copies[i].dst, copies[i].src, copies[i].bytes, cudaMemcpyDeviceToHost, s));
    return PBG_OK;
  };
  int rc = plain(false);
  if (rc) return rc;
  if (worth) {
    std::vector<Piece> pieces;
    std::unique_lock<std::mutex> lk(g_ring.mu, std::defer_lock);
    Moved m = Moved::NOT_BEGUN;
    if (cut(copies, count, ring, &pieces) && lk.try_lock() && ring_ready(g_ring)) {
      RingLink link{g_ring, s};
      m = hostmove::move_pieces(pieces, g_ring.mem, link);
      if (m == Moved::LINK_FAILED) {
        cudaStreamSynchronize(s);  // no copy into the ring is left in flight
        return cuda_fail(link.e, "result copy");
      }
    }
    if (m == Moved::NOT_BEGUN) {
      rc = plain(true);
      if (rc) return rc;
    }
  }
  PBG_CUDA(cudaStreamSynchronize(s));
  return PBG_OK;
}

}  // namespace pbg
