// hostmove.h -- the host side of copyout.cu: pieces that arrive in a ring of
// host buffers, moved on to the caller's memory by several threads.  No CUDA
// in here; the link that fills the ring is the template's argument.
#pragma once

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
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
