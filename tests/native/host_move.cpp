// The host side of large result copies without a GPU: a link that copies
// within host memory, allocations and thread starts that fail on demand.
// Prints one line a case; a wrong byte, a wrong verdict or an abort fails it.
#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <new>

#include "../../pbbsbench_b200/csrc/hostmove.h"

using namespace pbg::hostmove;

static thread_local long alloc_budget = -1;  // allocations of this thread that succeed; -1: all
static thread_local long failed_allocs = 0;
void* operator new(size_t n) {
  if (alloc_budget == 0) {
    failed_allocs++;
    throw std::bad_alloc();
  }
  if (alloc_budget > 0) alloc_budget--;
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static long thread_budget = -1;  // threads that may be started; -1: all
static long refused_threads = 0;
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  if (thread_budget == 0) {
    refused_threads++;
    return EAGAIN;
  }
  if (thread_budget > 0) thread_budget--;
  return real(t, a, f, arg);
}

// early: the piece is in the slot as soon as it is issued (a slot given out
// too early is overwritten); late: only when it is waited for (a piece moved
// on too early is stale).
struct Link {
  char* ring;
  bool early;
  long fail_at;  // calls until one fails; -1: none
  size_t issued = 0;
  Piece in_slot[RING] = {};
  bool step() { return fail_at < 0 || fail_at-- > 0; }
  bool issue(const Piece& p, int slot) {
    if (!step()) return false;
    issued++;
    in_slot[slot] = p;
    if (early) std::memcpy(ring + slot * PIECE, p.src, p.len);
    return true;
  }
  bool wait(int slot) {
    if (!step()) return false;
    if (!early) std::memcpy(ring + slot * PIECE, in_slot[slot].src, in_slot[slot].len);
    return true;
  }
};

static int bad = 0;
static void expect(bool ok, const char* what, size_t a, long b) {
  if (!ok) {
    std::printf("FAILED %s (%zu, %ld)\n", what, a, b);
    bad = 1;
  }
}

int main() {
  char* ring = (char*)std::malloc(PIECE * RING);
  const size_t sizes[] = {1, PIECE - 1, PIECE, PIECE + 1, 6 * PIECE + 5, RING * PIECE, RING * PIECE + 3, 21 * PIECE + 777};
  const size_t most = 21 * PIECE + 777;
  char* src = (char*)std::malloc(most);
  char* dst = (char*)std::malloc(most + 1);
  for (size_t i = 0; i < most; i++) src[i] = (char)(i * 2654435761u >> 13);
  for (size_t bytes : sizes) {
    std::vector<Piece> pieces;
    for (size_t o = 0; o < bytes; o += PIECE) pieces.push_back({dst + o, src + o, std::min(PIECE, bytes - o)});
    auto go = [&](bool early, long fail_at, size_t* issued = nullptr) {
      std::memset(dst, 0x5A, bytes + 1);
      Link link{ring, early, fail_at};
      const Moved m = move_pieces(pieces, ring, link);
      if (issued) *issued = link.issued;
      return m;
    };
    auto right = [&] { return std::memcmp(dst, src, bytes) == 0 && dst[bytes] == 0x5A; };
    for (bool early : {true, false}) expect(go(early, -1) == Moved::ALL && right(), "plain", bytes, early);
    // every allocation of the move fails in its turn
    for (long k = 0;; k++) {
      size_t issued = 0;
      alloc_budget = k;
      failed_allocs = 0;
      const Moved m = go(true, -1, &issued);
      alloc_budget = -1;
      expect(m == Moved::ALL ? right() : m == Moved::NOT_BEGUN && issued == 0, "allocation", bytes, k);
      if (failed_allocs == 0) break;
    }
    // no thread, one, two ... can be started
    for (long k = 0;; k++) {
      thread_budget = k;
      refused_threads = 0;
      const Moved m = go(false, -1);
      thread_budget = -1;
      expect(m == Moved::ALL && right(), "threads", bytes, k);
      if (refused_threads == 0) break;
    }
    // the link fails at each of its calls
    for (long k = 0; k < (long)(2 * pieces.size()); k++) expect(go(k & 1, k) == Moved::LINK_FAILED, "link", bytes, k);
    std::printf("%zu bytes\n", bytes);
  }
  std::puts(bad ? "failed" : "all right");
  return bad;
}
