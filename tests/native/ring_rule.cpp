// Which results are worth the ring, on memory with and without pages.
#include <cstdio>
#include <cstdlib>

#include "../../pbbsbench_b200/csrc/hostmove.h"

using namespace pbg::hostmove;

static char* fresh(size_t bytes) {
  void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED) std::abort();
  madvise(p, bytes, MADV_NOHUGEPAGE);
  return static_cast<char*>(p);
}
static void touch(char* p, size_t bytes) {
  for (size_t i = 0; i < bytes; i += 4096) p[i] = 1;
}

static int bad = 0;
static void expect(bool got, bool want, const char* what, size_t bytes) {
  if (got != want) {
    std::printf("FAILED %s: %zu bytes\n", what, bytes);
    bad = 1;
  }
}
static bool one(const void* p, size_t bytes) {
  const Range r{p, bytes};
  return worth_ring(&r, 1);
}

int main() {
  const size_t MB = 1 << 20;
  for (size_t bytes : {6 * MB, 8 * MB, 16 * MB - 4096}) {
    char* p = fresh(bytes);
    expect(one(p, bytes), true, "no page", bytes);
    touch(p, bytes - MB + 4096);
    expect(one(p, bytes), false, "all but a little less than a MiB", bytes);
    touch(p, bytes);
    expect(one(p, bytes), false, "all pages", bytes);
    madvise(p + 2 * MB, MB, MADV_DONTNEED);
    expect(one(p, bytes), true, "a hole of a MiB", bytes);
    expect(one(p + 3, bytes - 3 < 6 * MB ? 0 : bytes - 3), bytes > 6 * MB, "odd start", bytes);
    touch(p, bytes);
    expect(one(p + 3, bytes - 8), false, "odd start, all pages", bytes);
  }
  char* p = fresh(40 * MB);
  expect(one(p, 6 * MB - 1), false, "small", 6 * MB - 1);
  expect(one(p, 40 * MB), true, "large, no page", 40 * MB);
  touch(p, 40 * MB);
  expect(one(p, 40 * MB), true, "large, all pages", 40 * MB);
  expect(one(p, 16 * MB), true, "the upper line, all pages", 16 * MB);
  // two arrays: the sum counts, in size and in pages
  char* q = fresh(4 * MB);
  const Range half[2] = {{p, 4 * MB}, {q, 4 * MB}};
  expect(worth_ring(half, 2), true, "one of two without pages", 8 * MB);
  touch(q, 4 * MB);
  expect(worth_ring(half, 2), false, "both with pages", 8 * MB);
  expect(worth_ring(half, 0), false, "none", 0);
  // memory that is not there is the copy's to report
  munmap(q, 4 * MB);
  expect(worth_ring(half, 2), false, "unmapped", 8 * MB);
  std::puts(bad ? "failed" : "all right");
  return bad;
}
