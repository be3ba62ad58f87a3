// hostmove.h -- the host side of copyout.cu: which results are worth a ring of
// host buffers, and the pieces that arrive in it, moved on to the caller's
// memory by several threads.  No CUDA in here; the link that fills the ring is
// the template's argument.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace pbg {
namespace hostmove {

constexpr size_t PIECE = 2ull << 20;
constexpr int RING = 8;                  // pieces in flight: 16 MiB of host memory
constexpr size_t MIN_PART = 1ull << 20;  // bytes a thread is started for
constexpr unsigned MAX_THREADS = 8;

// When a call's results to pageable memory go through the ring.  It takes the
// page faults of memory that has no pages yet with several threads, and moves
// large results faster than the driver's one; its own threads cost 0.2-0.4 ms
// to start and wake.  ms a call, plain copies / ring, parents and levels
// together:
//   all pages present  6.5 MB 0.73 / 0.87-1.0   8 MB 0.83 / 1.1   12 MB 1.06 /
//                      1.13   16 MB 1.30 / 1.25   24 MB 1.80 / 1.5   64 MB 4.2 / 3.0
//   no page present    5.6 MB 0.75 / 1.03 (mostly pages from the heap after
//                      all)   6.5 MB 3.7-4.1 / 1.6   16 MB 8.6 / 3.1
//   8 MB, 0.5 MB without pages 1.2-1.3 / 1.3-1.4, 1 MB 1.4-1.6 / 1.4, 2 MB
//                      1.8-2.1 / 1.3-1.4
constexpr size_t MIN_RING = 6ull << 20;           // below: never
constexpr size_t MIN_RING_PRESENT = 16ull << 20;  // from here on: always
constexpr size_t MIN_ABSENT = 1ull << 20;         // between: when so much has no pages

struct Range {
  const void* p;
  size_t bytes;
};

// Bytes of the range's whole pages that have no memory yet; counts no further
// once `enough` are found.  0 where the system does not say.
inline size_t absent_bytes(const Range& r, size_t enough) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  const uintptr_t first = ((uintptr_t)r.p + page - 1) / page * page, end = ((uintptr_t)r.p + r.bytes) / page * page;
  size_t absent = 0;
  unsigned char present[512];
  for (uintptr_t at = first; at < end && absent < enough;) {
    const size_t pages = std::min<size_t>(sizeof(present), (end - at) / page);
    if (mincore((void*)at, pages * page, present) != 0) return 0;
    for (size_t i = 0; i < pages; i++)
      if (!(present[i] & 1)) absent += page;
    at += pages * page;
  }
  return absent;
}

// Whether the results that go to these ranges of pageable memory take the ring.
inline bool worth_ring(const Range* r, int count) {
  size_t total = 0, absent = 0;
  for (int i = 0; i < count; i++) total += r[i].bytes;
  if (total < MIN_RING || total >= MIN_RING_PRESENT) return total >= MIN_RING;
  for (int i = 0; i < count && absent < MIN_ABSENT; i++) absent += absent_bytes(r[i], MIN_ABSENT - absent);
  return absent >= MIN_ABSENT;
}

struct Piece {
  char* dst;
  const char* src;
  size_t len;  // at most PIECE
};

enum class Moved {
  ALL,       // every piece is at its destination
  NOT_BEGUN, // no memory for the move itself; the link was not used
  LINK_FAILED
};

// Moves the pieces through `ring` (RING * PIECE bytes).  link.issue(piece,
// slot) starts bringing piece.src into the slot, link.wait(slot) returns when
// it is there; both return false on an error, and the move then ends.  Never
// throws: the callers are C entry points.  Threads that cannot be started
// are done without.
template <class Link>
Moved move_pieces(const std::vector<Piece>& pieces, char* ring, Link& link) noexcept {
  const size_t n = pieces.size();
  size_t bytes = 0;
  for (const Piece& p : pieces) bytes += p.len;
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  const unsigned parts = std::max(1u, (unsigned)std::min<size_t>(std::min(MAX_THREADS, hw), bytes / MIN_PART));
  std::mutex mu;
  std::condition_variable cv;
  size_t ready = 0;  // pieces that have arrived in the ring
  bool stop = false;
  std::vector<std::atomic<unsigned>> done;  // parts of each piece moved on
  std::vector<std::thread> th;
  try {
    done = std::vector<std::atomic<unsigned>>(n);
    th.reserve(parts);
  } catch (...) {
    return Moved::NOT_BEGUN;
  }
  for (auto& d : done) d.store(0);
  auto move_part = [&](size_t i, unsigned k, unsigned of) {
    const Piece& p = pieces[i];
    const size_t a = p.len * k / of, b = p.len * (k + 1) / of;
    std::memcpy(p.dst + a, ring + (i % RING) * PIECE + a, b - a);
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
  try {
    for (unsigned k = 1; k < parts; k++) th.emplace_back(work, k);
  } catch (...) {  // no thread, or no memory for one: those that are there share the pieces
    team.store((unsigned)th.size() + 1);
  }
  const unsigned of = team.load();
  bool ok = true;
  size_t issued = 0;
  for (size_t i = 0; i < n && ok; i++) {
    while (issued < n && issued < i + RING && ok) {
      if (issued >= RING) {  // its slot's previous piece has been moved on
        while (done[issued - RING].load(std::memory_order_acquire) < of) {
          if (issued > i) break;
          std::this_thread::yield();
        }
        if (done[issued - RING].load(std::memory_order_acquire) < of) break;
      }
      ok = link.issue(pieces[issued], (int)(issued % RING));
      if (ok) issued++;
    }
    if (ok) ok = link.wait((int)(i % RING));
    if (!ok) break;
    {
      std::lock_guard<std::mutex> lk(mu);
      ready = i + 1;
    }
    cv.notify_all();
    move_part(i, 0, of);
  }
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!ok) stop = true;
  }
  cv.notify_all();
  for (auto& t : th) t.join();
  return ok ? Moved::ALL : Moved::LINK_FAILED;
}

}  // namespace hostmove
}  // namespace pbg
