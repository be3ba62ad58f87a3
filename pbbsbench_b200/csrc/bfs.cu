// bfs.cu -- single-source, direction-optimizing BFS as ONE persistent
// cooperative kernel per search (sm_100a).
//
// Replaces the hot loop of backForwardBFS
// (benchmarks/breadthFirstSearch/backForwardBFS/BFS.C:38-61) and the two
// edge_map bodies of common/ligraLight.h:
//   * top-down   = edge_map_sparse (ligraLight.h:70-85): the frontier is a
//     queue; every frontier edge (u, v) tries to claim v;
//   * bottom-up  = edge_map_dense (ligraLight.h:87-112): every unvisited v
//     scans N(v) for a frontier vertex and stops at the first one;
//   * the switch = edge_map::operator() (ligraLight.h:114-136): go bottom-up
//     when |F| + sum deg(F) > m / alpha, stay bottom-up while |F| > n / beta.
//
// Device layout (all in HBM, resident across calls on the handle):
//   offsets u32[n+1], edges u32[m]     CSR, read through the read-only path
//   parent  u32[n]                     output (0xFFFFFFFF = unvisited)
//   level   u32[n]                     optional output
//   bm[2]   u32[nwords]                visited bitmaps (2 MiB at n = 2^24, L2-resident)
//   q[2]    u32[n]                     frontier queues of short lists (deg < chunk_min_degree),
//                                      expanded 32 lists per warp, one per lane
//   qbig[2] uint4[big_cap]             (v, begin, end, first chunk) of longer lists, cut
//                                      in 256-edge pieces that any warp of the grid expands
//   ctrl                               counters, barrier, statistics
//
// Invariant: at the start of level L, bm[cur] holds every vertex of level <= L
// (plus degree-0 vertices of symmetric graphs and the padding bits past n, so
// whole words can be skipped).  Bottom-up therefore needs no separate frontier
// bitmap: an unvisited v whose neighbour u is in bm[cur] has level(u) == L.
//
// Parent rules:
//   ANY: claim by atomicOr on bm[cur] in place; the winner writes parent.
//   MIN/MAX: every frontier edge into a vertex not in bm[cur] (read-only this
//     level) does atomicMin/atomicMax on parent; the claim that decides who
//     enqueues v goes to bm[cur^1], which holds level <= L-1 and receives the
//     frontier's own bits from the threads expanding it; then cur flips.
//   Bottom-up scans N(v) ascending (MAX: descending) and stops at the first
//   frontier neighbour, which is the min (max) because lists are sorted.
//
// One grid barrier per level.  Every barrier wait is bounded by a
// %globaltimer budget; on expiry the kernel sets an error bit and all blocks
// return, the host reports PBG_ERR_TIMEOUT.
//
// Graphs whose largest degree is below the chunk degree run bfs_lean, the
// same search without the chunk queue, and small graphs bfs_small, one block
// with its state in shared memory (see their comments).
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "device_util.cuh"
#include "internal.cuh"

namespace pbg {
namespace {

using dev::block_sum;
using dev::FULL;
using dev::globaltimer;
using dev::ld_relaxed_u64;
constexpr uint32_t CHUNK = 256;  // edges per chunk task: 8 per lane of a warp
constexpr int PER_LANE = 8;      // independent loads each lane keeps in flight
constexpr uint32_t CONV = 3;     // BfsCtrl::conv as a slot index
static_assert(offsetof(BfsCtrl, conv) == offsetof(BfsCtrl, slot) + CONV * sizeof(LevelSlot), "conv follows the slots");
constexpr unsigned long long BIG_SHIFT = 40;
constexpr unsigned long long BIG_MASK = (1ull << BIG_SHIFT) - 1;

enum { MODE_ANY = 0, MODE_MIN = 1, MODE_MAX = 2 };

struct BfsArgs {
  const uint32_t* __restrict__ offsets;
  const uint32_t* __restrict__ edges;
  const uint32_t* __restrict__ iso;
  uint32_t* parent;
  uint32_t* level;
  uint32_t* bm0;
  uint32_t* bm1;
  uint32_t* q0;
  uint32_t* q1;
  uint2* qr0;  // adjacency range (begin, end) of each q entry
  uint2* qr1;
  uint4* qb0;
  uint4* qb1;
  BfsCtrl* ctrl;
  unsigned long long m;
  uint32_t n;
  uint32_t nwords;
  uint32_t big_cap;
  uint32_t src;
  uint32_t alpha;
  uint32_t beta;
  uint32_t policy;
  uint32_t chunk_deg;
  uint32_t symmetric;
};

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Fills x[0, n) with 0xFFFFFFFF, 16 bytes per store where aligned.
__device__ __forceinline__ void init_fill(uint32_t* x, uint32_t n, unsigned long long tid, unsigned long long nth) {
  const uint32_t mis = (uint32_t)(((16 - (reinterpret_cast<uintptr_t>(x) & 15)) & 15) / 4);
  const uint32_t head = mis < n ? mis : n;
  for (unsigned long long i = tid; i < head; i += nth) x[i] = PBG_NONE;
  uint4* x4 = reinterpret_cast<uint4*>(x + head);
  const unsigned long long n4 = (n - head) / 4;
  const uint4 f = make_uint4(PBG_NONE, PBG_NONE, PBG_NONE, PBG_NONE);
  for (unsigned long long i = tid; i < n4; i += nth) x4[i] = f;
  for (unsigned long long i = head + n4 * 4 + tid; i < n; i += nth) x[i] = PBG_NONE;
}

// The adjacency ranges of the candidates v[i] (set bits of `act`), loaded
// before their claims are issued, so the winners' ranges, which the append
// needs, arrive during the claims' round trip instead of after it.
__device__ __forceinline__ void load_ranges(const BfsArgs& a, const uint32_t (&v)[PER_LANE], unsigned act,
                                            uint32_t (&ob)[PER_LANE], uint32_t (&oe)[PER_LANE]) {
#pragma unroll
  for (int i = 0; i < PER_LANE; i++) {
    ob[i] = ((act >> i) & 1u) ? __ldg(a.offsets + v[i]) : 0u;
    oe[i] = ((act >> i) & 1u) ? __ldg(a.offsets + v[i] + 1) : 0u;
  }
}

// Which of the paired arrays a level reads and writes, as bits of one word:
// the pointers are selected from the launch arguments where they are used,
// which costs a select each and keeps some 20 registers free for the loops.
// The 1024-thread kernels are held to 64 registers: with this and 32-bit
// per-thread sums they spill 136-140 bytes (bfs_lean 72) instead of 244-280
// (196-240).  us a search, before and now, same box, runs within 0.2%: rMat
// 2^24 561 / 551, 2^20 64.4 / 61.5; bfs_lean, ANY: torus 160^3 1659 / 1600,
// 100^3 881 / 877, 60^3 507 / 505, 40^3 356 / 327, 20^3 163 / 166; random-local
// 100 k 302 / 303, 1 M 622 / 636, 8 M 2615 / 2660: wide levels of short lists
// pay the selects without having had spills in the way.  Carrying the queue
// pointers again there costs the lattices more (torus 160^3 1659).
struct Level {
  uint32_t bits;  // 0: output queues are q0/qr0/qb0 (else q1/qr1/qb1); 1: bm1 is the visited bitmap
  uint32_t slot;  // counters of the frontier produced (3: conv)
  uint32_t next;  // level number of what is found
  __device__ __forceinline__ LevelSlot* out(const BfsArgs& a) const { return a.ctrl->slot + slot; }
  __device__ __forceinline__ uint32_t* q(const BfsArgs& a) const { return (bits & 1u) ? a.q0 : a.q1; }
  __device__ __forceinline__ uint2* qr(const BfsArgs& a) const { return (bits & 1u) ? a.qr0 : a.qr1; }
  __device__ __forceinline__ uint4* qb(const BfsArgs& a) const { return (bits & 1u) ? a.qb0 : a.qb1; }
  __device__ __forceinline__ const uint32_t* qin(const BfsArgs& a) const { return (bits & 1u) ? a.q1 : a.q0; }
  __device__ __forceinline__ const uint2* qrin(const BfsArgs& a) const { return (bits & 1u) ? a.qr1 : a.qr0; }
  __device__ __forceinline__ const uint4* qbin(const BfsArgs& a) const { return (bits & 1u) ? a.qb1 : a.qb0; }
  __device__ __forceinline__ const uint32_t* vis(const BfsArgs& a) const { return (bits & 2u) ? a.bm1 : a.bm0; }
  // ANY claims in the visited bitmap itself, MIN/MAX in the other one
  template <int MODE>
  __device__ __forceinline__ uint32_t* claim(const BfsArgs& a) const {
    return ((bits & 2u) != 0) == (MODE == MODE_ANY) ? a.bm1 : a.bm0;
  }
};

// Warp-collective append of up to K vertices per lane (cand[i] for the set
// bits i of `win`) to the next frontier.  Vertices with degree >= chunk_deg
// go to the chunk queue as (v, begin, end, first chunk) with their number of
// CHUNK-edge pieces; the rest to the main queue.  (ob[i], oe[i]) is cand[i]'s
// adjacency range (load_ranges).  Positions come from warp
// prefix sums and one atomic per queue per warp: entries of one warp are
// contiguous, and chunk numbering follows slot order across warps because
// slot and chunk counters move in one 64-bit atomic.
template <int K>
__device__ __forceinline__ void emit_k(const BfsArgs& a, const Level& lv, const uint32_t (&cand)[K], unsigned win,
                                       uint32_t& degacc, const uint32_t (&ob)[K],
                                       const uint32_t (&oe)[K]) {
  if (!__any_sync(FULL, win != 0)) return;
  const int lane = threadIdx.x & 31;
  // pass 1: classify (only a bit per candidate stays live)
  uint32_t ns = 0, nc = 0, nch = 0;
  unsigned chunked = 0;
#pragma unroll
  for (int i = 0; i < K; i++) {
    if ((win >> i) & 1u) {
      const uint32_t d = oe[i] - ob[i];
      degacc += d;
      if (d >= a.chunk_deg) {
        chunked |= 1u << i;
        nc++;
        nch += (d + CHUNK - 1) / CHUNK;
      } else {
        ns++;
      }
    }
  }
  const uint32_t ps = warp_incl_scan(ns), pc = warp_incl_scan(nc), pch = warp_incl_scan(nch);
  const uint32_t ts = __shfl_sync(FULL, ps, 31), tc = __shfl_sync(FULL, pc, 31), tch = __shfl_sync(FULL, pch, 31);
  unsigned long long bs = 0, bc = 0;
  if (lane == 0) {
    if (ts) bs = atomicAdd(&lv.out(a)->nmain, (unsigned long long)ts);
    if (tc) bc = atomicAdd(&lv.out(a)->big, ((unsigned long long)tc << BIG_SHIFT) | tch);
  }
  bs = __shfl_sync(FULL, bs, 0);
  bc = __shfl_sync(FULL, bc, 0);
  uint32_t ps_pos = (uint32_t)bs + ps - ns;
  uint32_t pc_pos = (uint32_t)(bc >> BIG_SHIFT) + pc - nc;
  uint32_t chunk = (uint32_t)(bc & BIG_MASK) + pch - nch;
  // pass 2: write
#pragma unroll
  for (int i = 0; i < K; i++) {
    if ((win >> i) & 1u) {
      const uint32_t b = ob[i], e = oe[i];
      if ((chunked >> i) & 1u) {
        if (pc_pos < a.big_cap)
          lv.qb(a)[pc_pos] = make_uint4(cand[i], b, e, chunk);
        else
          atomicOr(&a.ctrl->sync.error, ERR_QUEUE);
        pc_pos++;
        chunk += (e - b + CHUNK - 1) / CHUNK;
      } else {
        lv.q(a)[ps_pos] = cand[i];
        lv.qr(a)[ps_pos] = make_uint2(b, e);
        ps_pos++;
        // the next level reads this list: start it on its way from HBM to L2
        if (e > b) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.edges + b));
      }
    }
  }
}

// Top-down claims of up to K neighbours v[i] (set bits of `act`) by the
// lane's vertex u, and the adjacency ranges (ob, oe) of the candidates that
// may be won.  Every load and atomic of the K candidates is issued before
// any store that depends on one, so the K round trips overlap instead of
// running one after another.  Returns the bits of the candidates this lane
// enqueues.
// MIN/MAX test the read-only snapshot of the level's visited set first and
// load ranges for the unvisited only: large levels are bound by the L1's rate
// of about one request a clock and SM, and most of their edges lead to visited
// vertices.  The claim on the bitmap is issued before the reduction on the
// parent, which nothing waits for.  us a search, before and now: directed 2 M
// vertices (22.8 M edges, MAX) 613 / 506, 4 M (MIN) 1486 / 1177, 20 k 129 /
// 114; torus 100^3 (MIN) 993 / 928.  Letting the reduction that finds the parent
// unset be the claim saves an atomic, but waits for a word of a large array
// instead of the bitmap's: 555, 1151, 147, 1179.
template <int MODE, int K>
__device__ __forceinline__ unsigned td_claim_k(const BfsArgs& a, const Level& lv, uint32_t u,
                                               const uint32_t (&v)[K], unsigned act, uint32_t (&ob)[K],
                                               uint32_t (&oe)[K]) {
  uint32_t old[K];
  unsigned win = 0;
  if (MODE == MODE_ANY) {
    load_ranges(a, v, act, ob, oe);
#pragma unroll
    for (int i = 0; i < K; i++) old[i] = ((act >> i) & 1u) ? atomicOr(lv.claim<MODE>(a) + (v[i] >> 5), 1u << (v[i] & 31)) : FULL;
#pragma unroll
    for (int i = 0; i < K; i++)
      if (!((old[i] >> (v[i] & 31)) & 1u)) win |= 1u << i;
#pragma unroll
    for (int i = 0; i < K; i++)
      if ((win >> i) & 1u) a.parent[v[i]] = u;
  } else {
    unsigned live = act;
    uint32_t w[K];
#pragma unroll
    for (int i = 0; i < K; i++) w[i] = ((act >> i) & 1u) ? lv.vis(a)[v[i] >> 5] : 0u;
#pragma unroll
    for (int i = 0; i < K; i++)
      if ((w[i] >> (v[i] & 31)) & 1u) live &= ~(1u << i);
    load_ranges(a, v, live, ob, oe);
#pragma unroll
    for (int i = 0; i < K; i++)
      old[i] = ((live >> i) & 1u) ? atomicOr(lv.claim<MODE>(a) + (v[i] >> 5), 1u << (v[i] & 31)) : FULL;
#pragma unroll
    for (int i = 0; i < K; i++) {
      if ((live >> i) & 1u) {
        if (MODE == MODE_MIN)
          atomicMin(a.parent + v[i], u);
        else
          atomicMax(reinterpret_cast<int*>(a.parent) + v[i], (int)u);
      }
    }
#pragma unroll
    for (int i = 0; i < K; i++)
      if (!((old[i] >> (v[i] & 31)) & 1u)) win |= 1u << i;
  }
  if (a.level && win) {
#pragma unroll
    for (int i = 0; i < K; i++)
      if ((win >> i) & 1u) a.level[v[i]] = lv.next;
  }
  return win;
}

// One CHUNK-edge piece of a long list, expanded by a whole warp.
template <int MODE>
__device__ __forceinline__ void td_chunk(const BfsArgs& a, const uint4& ent, uint32_t c_local, const Level& lv,
                                         uint32_t& degacc) {
  const int lane = threadIdx.x & 31;
  const uint32_t u = ent.x;
  const uint32_t cb = ent.y + c_local * CHUNK;
  const uint32_t len = min(ent.z - cb, CHUNK);  // positions counted from cb: a list may end at 2^32 - 1
  if (MODE != MODE_ANY && c_local == 0 && lane == 0) atomicOr(lv.claim<MODE>(a) + (u >> 5), 1u << (u & 31));
  uint32_t v[PER_LANE];
  unsigned act = 0;
#pragma unroll
  for (int i = 0; i < PER_LANE; i++) {
    v[i] = 0;
    if (i * 32 + lane < len) {
      v[i] = __ldg(a.edges + (cb + i * 32 + lane));
      act |= 1u << i;
    }
  }
  uint32_t ob[PER_LANE], oe[PER_LANE];
  const unsigned win = td_claim_k<MODE, PER_LANE>(a, lv, u, v, act, ob, oe);
  emit_k<PER_LANE>(a, lv, v, win, degacc, ob, oe);
}

// 32 short lists (degree < chunk_deg), one per lane, PER_LANE edges a step.
template <int MODE>
__device__ __forceinline__ void td_small(const BfsArgs& a, uint32_t tile, uint32_t nmain, const Level& lv,
                                         uint32_t& degacc) {
  const int lane = threadIdx.x & 31;
  const uint32_t idx = tile * 32 + lane;  // n < 2^31
  uint32_t u = 0, b = 0, e = 0;
  if (idx < nmain) {
    u = lv.qin(a)[idx];
    const uint2 r = lv.qrin(a)[idx];  // range stored by the claimer: no offsets load
    b = r.x;
    e = r.y;
    if (MODE != MODE_ANY) atomicOr(lv.claim<MODE>(a) + (u >> 5), 1u << (u & 31));
  }
  const uint32_t maxd = __reduce_max_sync(FULL, e - b);
  for (uint32_t k0 = 0; k0 < maxd; k0 += PER_LANE) {
    uint32_t v[PER_LANE];
    unsigned act = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; i++) {
      const uint32_t j = b + k0 + i;
      v[i] = 0;
      if (j < e) {
        v[i] = __ldg(a.edges + j);
        act |= 1u << i;
      }
    }
    uint32_t ob[PER_LANE], oe[PER_LANE];
    const unsigned win = td_claim_k<MODE, PER_LANE>(a, lv, u, v, act, ob, oe);
    emit_k<PER_LANE>(a, lv, v, win, degacc, ob, oe);
  }
}

// Top-down level: chunk tasks first (edge-balanced over every warp of the
// grid), then 32-entry tiles of short lists.
template <int MODE>
__device__ void td_level(const BfsArgs& a, uint32_t nmain, uint32_t nbig, uint32_t nchunks, const Level& lv,
                         uint32_t& degacc) {
  // tasks go round-robin over blocks first, so a small level still uses
  // every SM's load/store pipeline
  const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint32_t tw = (gridDim.x * blockDim.x) >> 5;
  const unsigned long long tasks = (unsigned long long)nchunks + (nmain + 31) / 32;
  for (unsigned long long t = gw; t < tasks; t += tw) {
    if (t < nchunks) {
      const uint32_t c = (uint32_t)t;
      uint32_t lo = 0, hi = nbig - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (lv.qbin(a)[mid].w <= c)
          lo = mid;
        else
          hi = mid - 1;
      }
      const uint4 ent = lv.qbin(a)[lo];
      td_chunk<MODE>(a, ent, c - ent.w, lv, degacc);
    } else {
      td_small<MODE>(a, (uint32_t)(t - nchunks), nmain, lv, degacc);
    }
  }
}

// Bottom-up over bitmap words, one warp per word, one lane per vertex.  Each
// unvisited lane probes the first LSHARE neighbours of its own list, PROBES
// independent loads a step (ascending; MAX: descending), while any lane of
// the warp is still unresolved; lists that are longer and still unresolved
// are then scanned by the whole warp, 32 neighbours per step, one list after
// another, the first frontier neighbour in scan order winning (the early
// exit of ligraLight.h:99-105).  A lane share of 16 in steps of 4 was the
// fastest of shares 4-64 and steps 1-8 on rMat 2^20 and 2^24: one probe a
// step leaves most of a warp's misses to the serial warp scan, wide steps
// issue requests a lane rarely needs.  The word loop is software-pipelined three deep: the
// bitmap word two steps ahead and the offsets one step ahead are in flight
// while the current word's probes run.  Counts and degree sums stay in
// registers.
template <int MODE>
__device__ __forceinline__ void bu_word(const BfsArgs& a, const uint32_t* vin, uint32_t* vout, uint32_t next_level,
                                        uint32_t w, uint32_t word, uint32_t b, uint32_t e, uint32_t& cnt,
                                        uint32_t& degacc) {
  constexpr int PROBES = 4;
  constexpr uint32_t LSHARE = 16;
  const int lane = threadIdx.x & 31;
  if (word == FULL) {
    if (lane == 0) vout[w] = word;
    return;
  }
  const uint32_t v = w * 32 + lane;
  const uint32_t deg = e - b;  // 0 for visited lanes
  bool found = false;
  uint32_t p = 0;
  for (uint32_t k0 = 0; k0 < LSHARE; k0 += PROBES) {
    if (!__any_sync(FULL, !found && deg > k0)) break;
    uint32_t cu[PROBES], cw[PROBES];
#pragma unroll
    for (int i = 0; i < PROBES; i++) {
      cu[i] = 0;
      if (!found && k0 + i < deg) cu[i] = __ldg(a.edges + ((MODE == MODE_MAX) ? (e - 1 - k0 - i) : (b + k0 + i)));
    }
#pragma unroll
    for (int i = 0; i < PROBES; i++) cw[i] = (!found && k0 + i < deg) ? vin[cu[i] >> 5] : 0u;
#pragma unroll
    for (int i = 0; i < PROBES; i++) {
      if (!found && k0 + i < deg && ((cw[i] >> (cu[i] & 31)) & 1u)) {
        found = true;
        p = cu[i];
      }
    }
  }
  unsigned mm = __ballot_sync(FULL, !found && deg > LSHARE);
  while (mm) {
    const int l = __ffs(mm) - 1;
    mm &= mm - 1;
    const uint32_t bb = __shfl_sync(FULL, b, l);
    const uint32_t ee = __shfl_sync(FULL, e, l);
    uint32_t hit = 0;
    bool got = false;
    if (MODE == MODE_MAX) {
      for (long long top = (long long)ee - LSHARE; top > (long long)bb && !got; top -= 32) {
        const long long j = top - 1 - lane;
        uint32_t x = 0;
        bool h = false;
        if (j >= (long long)bb) {
          x = __ldg(a.edges + j);
          h = (vin[x >> 5] >> (x & 31)) & 1u;
        }
        const unsigned hb = __ballot_sync(FULL, h);
        if (hb) {
          got = true;
          hit = __shfl_sync(FULL, x, __ffs(hb) - 1);
        }
      }
    } else {
      for (uint32_t k = LSHARE; k < ee - bb && !got; k += 32) {  // counted from bb: a list may end at 2^32 - 1
        uint32_t x = 0;
        bool h = false;
        if (k + lane < ee - bb) {
          x = __ldg(a.edges + (bb + k + lane));
          h = (vin[x >> 5] >> (x & 31)) & 1u;
        }
        const unsigned hb = __ballot_sync(FULL, h);
        if (hb) {
          got = true;
          hit = __shfl_sync(FULL, x, __ffs(hb) - 1);
        }
      }
    }
    if (lane == l && got) {
      found = true;
      p = hit;
    }
  }
  const unsigned nb = __ballot_sync(FULL, found);
  if (lane == 0) vout[w] = word | nb;
  if (found) {
    a.parent[v] = p;
    if (a.level) a.level[v] = next_level;
    cnt += 1;
    degacc += deg;
  }
}

template <int MODE>
__device__ void bu_level(const BfsArgs& a, const uint32_t* vin, uint32_t* vout, uint32_t next_level,
                         uint32_t& cnt, uint32_t& degacc) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t tw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t nw = a.nwords;
  uint32_t w0 = gw, w1 = gw + tw;
  uint32_t word0 = (w0 < nw) ? vin[w0] : FULL;
  uint32_t word1 = (w1 < nw) ? vin[w1] : FULL;
  uint32_t b0 = 0, e0 = 0;
  if (!((word0 >> lane) & 1u)) {
    b0 = __ldg(a.offsets + w0 * 32 + lane);
    e0 = __ldg(a.offsets + w0 * 32 + lane + 1);
  }
  while (w0 < nw) {
    const uint32_t w2 = w1 + tw;
    const uint32_t word2 = (w2 < nw) ? vin[w2] : FULL;
    uint32_t b1 = 0, e1 = 0;
    if (!((word1 >> lane) & 1u)) {
      b1 = __ldg(a.offsets + w1 * 32 + lane);
      e1 = __ldg(a.offsets + w1 * 32 + lane + 1);
    }
    bu_word<MODE>(a, vin, vout, next_level, w0, word0, b0, e0, cnt, degacc);
    w0 = w1;
    word0 = word1;
    b0 = b1;
    e0 = e1;
    w1 = w2;
    word1 = word2;
  }
}

// Rebuilds the frontier queues from the bitmap difference after a bottom-up
// level (the sparse form of the dense frontier, as pack_index does in
// ligraLight.h:132).  Lane l of a warp handles word w0 + l.
__device__ void dense_to_queue(const BfsArgs& a, const uint32_t* before, const uint32_t* after, const Level& lv) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint32_t tw = (gridDim.x * blockDim.x) >> 5;
  uint32_t dummy = 0;
  for (uint32_t w0 = gw * 32; w0 < a.nwords; w0 += tw * 32) {
    const uint32_t w = w0 + lane;
    uint32_t diff = (w < a.nwords) ? (after[w] & ~before[w]) : 0u;
    while (__any_sync(FULL, diff != 0)) {
      uint32_t v[PER_LANE];
      unsigned act = 0;
#pragma unroll
      for (int i = 0; i < PER_LANE; i++) {
        v[i] = 0;
        if (diff) {
          v[i] = w * 32 + (__ffs(diff) - 1);
          diff &= diff - 1;
          act |= 1u << i;
        }
      }
      uint32_t ob[PER_LANE], oe[PER_LANE];
      load_ranges(a, v, act, ob, oe);
      emit_k<PER_LANE>(a, lv, v, act, dummy, ob, oe);
    }
  }
}

// BLOCK = 256 runs 4 blocks per SM at <= 64 registers, 512 one block at
// <= 128 registers (no spills), 1024 one block at <= 64 registers.
template <int MODE, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == 256 ? 4 : 1) bfs_persistent(BfsArgs a) {
  BfsCtrl* c = a.ctrl;
  __shared__ unsigned long long s_in[3];
  unsigned long long bar_epoch = 0;  // barriers passed (thread 0's count matters)

  // ---- init: parent/level = NONE, bitmaps = degree-0 + padding bits, source.
  {
    const unsigned long long tid = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long nth = (unsigned long long)gridDim.x * blockDim.x;
    if (tid == 0) c->t_start = globaltimer();
    init_fill(a.parent, a.n, tid, nth);
    if (a.level) init_fill(a.level, a.n, tid, nth);
    const uint32_t sw = a.src >> 5, sbit = 1u << (a.src & 31);
    for (unsigned long long w = tid; w < a.nwords; w += nth) {
      const uint32_t x = a.iso[w];
      a.bm0[w] = (w == sw) ? (x | sbit) : x;
      a.bm1[w] = (MODE == MODE_ANY && w == sw) ? (x | sbit) : x;
    }
    if (tid == 0) {
      const uint32_t b = __ldg(a.offsets + a.src), e = __ldg(a.offsets + a.src + 1);
      const uint32_t deg = e - b;
      for (int s = 0; s < 3; s++) c->slot[s] = LevelSlot{0, 0, 0, 0};
      c->conv = LevelSlot{0, 0, 0, 0};
      if (deg >= a.chunk_deg) {
        a.qb0[0] = make_uint4(a.src, b, e, 0u);
        c->slot[0].big = (1ull << BIG_SHIFT) | ((deg + CHUNK - 1) / CHUNK);
      } else {
        a.q0[0] = a.src;
        a.qr0[0] = make_uint2(b, e);
        c->slot[0].nmain = 1;
      }
      c->slot[0].deg = deg;
    }
  }
  // the source's own entries, after every block has filled
  if (!dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.parent[a.src] = a.src;
    if (a.level) a.level[a.src] = 0;
  }
  bool ok = dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch);

  uint32_t cur = 0;
  bool prev_bu = false;
  unsigned long long visited = 0, reached = 0, bumask = 0;
  uint32_t tdl = 0, bul = 0;
  uint32_t L = 0;
  while (ok) {
    LevelSlot* in = &c->slot[L % 3];
    LevelSlot* out = &c->slot[(L + 1) % 3];
    if (threadIdx.x == 0) {
      s_in[0] = ld_relaxed_u64(&in->nmain);
      s_in[1] = ld_relaxed_u64(&in->big);
      s_in[2] = ld_relaxed_u64(&in->deg);
    }
    __syncthreads();
    unsigned long long nmain = s_in[0], big = s_in[1];
    const unsigned long long fdeg = s_in[2];
    __syncthreads();
    const unsigned long long nf = nmain + (big >> BIG_SHIFT);
    if (nf == 0) break;
    if (L >= a.n) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&c->sync.error, ERR_LEVEL_LIMIT);
      break;
    }

    bool bu;
    if (a.policy == PBG_DIR_TOPDOWN || !a.symmetric)
      bu = false;
    else if (a.policy == PBG_DIR_BOTTOMUP)
      bu = true;
    else if (!prev_bu)
      bu = (nf + fdeg) > a.m / a.alpha;
    else
      bu = nf > (unsigned long long)(a.n / a.beta);

    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->slot[(L + 2) % 3] = LevelSlot{0, 0, 0, 0};
      if (bu) c->conv = LevelSlot{0, 0, 0, 0};
      if (L < PBG_TRACE_LEVELS) {
        c->t_ns[L] = globaltimer();
        c->t_nf[L] = nf;
        c->t_deg[L] = fdeg;
        c->t_bu[L] = bu ? 1u : 0u;
      }
      visited += nf;
      reached += fdeg;
      if (bu) {
        bul++;
        if (L < 64) bumask |= 1ull << L;
      } else {
        tdl++;
      }
    }

    uint32_t* bcur = cur ? a.bm1 : a.bm0;
    uint32_t* both = cur ? a.bm0 : a.bm1;
    if (bu) {
      uint32_t cnt = 0, degacc = 0;
      bu_level<MODE>(a, bcur, both, L + 1, cnt, degacc);
      const unsigned long long bc = block_sum(cnt);
      const unsigned long long bd = block_sum(degacc);
      if (threadIdx.x == 0) {
        if (bc) atomicAdd(&out->nmain, bc);
        if (bd) atomicAdd(&out->deg, bd);
      }
      cur ^= 1u;
    } else {
      if (prev_bu) {
        // the frontier came from a bottom-up level: build its queues first
        dense_to_queue(a, both, bcur, Level{(L & 1u) ^ 1u, CONV, L});
        ok = dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch);
        if (!ok) break;
        if (threadIdx.x == 0) {
          s_in[0] = ld_relaxed_u64(&c->conv.nmain);
          s_in[1] = ld_relaxed_u64(&c->conv.big);
        }
        __syncthreads();
        nmain = s_in[0];
        big = s_in[1];
        __syncthreads();
      }
      const uint32_t nbig = (uint32_t)(big >> BIG_SHIFT);
      if (nbig > a.big_cap || nmain > a.n) {  // cannot happen: each vertex enters one frontier once
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&c->sync.error, ERR_QUEUE);
        break;
      }
      uint32_t degacc = 0;
      td_level<MODE>(a, (uint32_t)nmain, nbig, (uint32_t)(big & BIG_MASK),
                     Level{(L & 1u) | (cur << 1), (L + 1) % 3, L + 1}, degacc);
      const unsigned long long bd = block_sum(degacc);
      if (threadIdx.x == 0 && bd) atomicAdd(&out->deg, bd);
      if (MODE != MODE_ANY) cur ^= 1u;
    }
    prev_bu = bu;
    L++;
    ok = dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (L <= PBG_TRACE_LEVELS) c->t_ns[L] = globaltimer();
    c->t_end = globaltimer();
    c->levels = L;
    c->td_levels = tdl;
    c->bu_levels = bul;
    c->final_bm = cur;
    c->visited = visited;
    c->edges_reached = reached;
    c->bu_mask = bumask;
  }
}

// ---------------------------------------------------------------- lean kernel
// For graphs whose every list is shorter than the chunk degree (a lattice, a
// road-like or random-local graph): the same direction-optimizing search as
// bfs_persistent without the chunk queue and its tasks, and with each warp
// adding its frontier degree (bottom-up: and count) to the level's counters
// itself instead of a block reduction; on the 3-D torus 160^3 about 20%
// faster a level.
// Bottom-up levels and the rebuild of queues after them are
// bfs_persistent's (bu_level, dense_to_queue).

// Appends the winners (bits of `win`) of a step to the next queue, one atomic
// per warp.
__device__ __forceinline__ void lean_emit(const BfsArgs& a, const Level& lv,
                                          const uint32_t (&cand)[PER_LANE], unsigned win,
                                          uint32_t& degacc, const uint32_t (&ob)[PER_LANE],
                                          const uint32_t (&oe)[PER_LANE]) {
  if (!__any_sync(FULL, win != 0)) return;
  const int lane = threadIdx.x & 31;
  const uint32_t ns = __popc(win);
  const uint32_t ps = warp_incl_scan(ns);
  const uint32_t ts = __shfl_sync(FULL, ps, 31);
  unsigned long long b0 = 0;
  if (lane == 0) b0 = atomicAdd(&lv.out(a)->nmain, (unsigned long long)ts);
  unsigned long long pos = __shfl_sync(FULL, b0, 0) + ps - ns;
#pragma unroll
  for (int i = 0; i < PER_LANE; i++) {
    if ((win >> i) & 1u) {
      const uint32_t b = ob[i], e = oe[i];
      degacc += e - b;
      lv.q(a)[pos] = cand[i];
      lv.qr(a)[pos] = make_uint2(b, e);
      pos++;
      // the next level reads this list: start it on its way from HBM to L2
      if (e > b) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.edges + b));
    }
  }
}

// 32 queue entries, one per lane, PER_LANE edges a step.
template <int MODE>
__device__ __forceinline__ void lean_tile(const BfsArgs& a, uint32_t tile, uint32_t nq, const Level& lv,
                                          uint32_t& degacc) {
  const int lane = threadIdx.x & 31;
  const uint32_t idx = tile * 32 + lane;  // n < 2^31
  uint32_t u = 0, b = 0, e = 0;
  if (idx < nq) {
    u = lv.qin(a)[idx];
    const uint2 r = lv.qrin(a)[idx];  // range stored by the claimer: no offsets load
    b = r.x;
    e = r.y;
    if (MODE != MODE_ANY) atomicOr(lv.claim<MODE>(a) + (u >> 5), 1u << (u & 31));
  }
  const uint32_t maxd = __reduce_max_sync(FULL, e - b);
  for (uint32_t k0 = 0; k0 < maxd; k0 += PER_LANE) {
    uint32_t v[PER_LANE];
    unsigned act = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; i++) {
      const uint32_t j = b + k0 + i;
      v[i] = 0;
      if (j < e) {
        v[i] = __ldg(a.edges + j);
        act |= 1u << i;
      }
    }
    uint32_t ob[PER_LANE], oe[PER_LANE];
    const unsigned win = td_claim_k<MODE, PER_LANE>(a, lv, u, v, act, ob, oe);
    lean_emit(a, lv, v, win, degacc, ob, oe);
  }
}

template <int MODE>
__global__ void __launch_bounds__(1024, 1) bfs_lean(BfsArgs a) {
  BfsCtrl* c = a.ctrl;
  __shared__ unsigned long long s_in[3];
  unsigned long long bar_epoch = 0;
  {
    const unsigned long long tid = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long nth = (unsigned long long)gridDim.x * blockDim.x;
    if (tid == 0) c->t_start = globaltimer();
    init_fill(a.parent, a.n, tid, nth);
    if (a.level) init_fill(a.level, a.n, tid, nth);
    const uint32_t sw = a.src >> 5, sbit = 1u << (a.src & 31);
    for (unsigned long long w = tid; w < a.nwords; w += nth) {
      const uint32_t x = a.iso[w];
      a.bm0[w] = (w == sw) ? (x | sbit) : x;
      a.bm1[w] = (MODE == MODE_ANY && w == sw) ? (x | sbit) : x;
    }
    if (tid == 0) {
      const uint32_t b = __ldg(a.offsets + a.src), e = __ldg(a.offsets + a.src + 1);
      for (int s = 0; s < 3; s++) c->slot[s] = LevelSlot{0, 0, 0, 0};
      c->conv = LevelSlot{0, 0, 0, 0};
      a.q0[0] = a.src;
      a.qr0[0] = make_uint2(b, e);
      c->slot[0].nmain = 1;
      c->slot[0].deg = e - b;
    }
  }
  if (!dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.parent[a.src] = a.src;
    if (a.level) a.level[a.src] = 0;
  }
  bool ok = dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch);
  uint32_t cur = 0;
  bool prev_bu = false;
  unsigned long long visited = 0, reached = 0, bumask = 0;
  uint32_t tdl = 0, bul = 0;
  uint32_t L = 0;
  while (ok) {
    LevelSlot* in = &c->slot[L % 3];
    LevelSlot* out = &c->slot[(L + 1) % 3];
    if (threadIdx.x == 0) {
      s_in[0] = ld_relaxed_u64(&in->nmain);
      s_in[1] = ld_relaxed_u64(&in->deg);
    }
    __syncthreads();
    unsigned long long nq = s_in[0];
    const unsigned long long nf = nq, fdeg = s_in[1];
    __syncthreads();
    if (nf == 0) break;
    if (L >= a.n) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&c->sync.error, ERR_LEVEL_LIMIT);
      break;
    }
    bool bu;
    if (a.policy == PBG_DIR_TOPDOWN || !a.symmetric)
      bu = false;
    else if (a.policy == PBG_DIR_BOTTOMUP)
      bu = true;
    else if (!prev_bu)
      bu = (nf + fdeg) > a.m / a.alpha;
    else
      bu = nf > (unsigned long long)(a.n / a.beta);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->slot[(L + 2) % 3] = LevelSlot{0, 0, 0, 0};
      if (bu) c->conv = LevelSlot{0, 0, 0, 0};
      if (L < PBG_TRACE_LEVELS) {
        c->t_ns[L] = globaltimer();
        c->t_nf[L] = nf;
        c->t_deg[L] = fdeg;
        c->t_bu[L] = bu ? 1u : 0u;
      }
      visited += nf;
      reached += fdeg;
      if (bu) {
        bul++;
        if (L < 64) bumask |= 1ull << L;
      } else {
        tdl++;
      }
    }
    uint32_t* bcur = cur ? a.bm1 : a.bm0;
    uint32_t* both = cur ? a.bm0 : a.bm1;
    uint32_t cnt = 0, degacc = 0;
    if (bu) {
      bu_level<MODE>(a, bcur, both, L + 1, cnt, degacc);
      cur ^= 1u;
    } else {
      if (prev_bu) {
        // the frontier came from a bottom-up level: build its queue first
        // (every list is short, so nothing goes to the chunk queue)
        dense_to_queue(a, both, bcur, Level{(L & 1u) ^ 1u, CONV, L});
        ok = dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch);
        if (!ok) break;
        if (threadIdx.x == 0) s_in[0] = ld_relaxed_u64(&c->conv.nmain);
        __syncthreads();
        nq = s_in[0];
        __syncthreads();
      }
      if (nq > a.n) {  // cannot happen: each vertex enters one frontier once
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&c->sync.error, ERR_QUEUE);
        break;
      }
      const Level lv{(L & 1u) | (cur << 1), (L + 1) % 3, L + 1};
      // tiles go round-robin over blocks first, so a small level still uses
      // every SM's load/store pipeline
      const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
      const uint32_t tw = (gridDim.x * blockDim.x) >> 5;
      const unsigned long long tiles = (nq + 31) / 32;
      for (unsigned long long t = gw; t < tiles; t += tw)
        lean_tile<MODE>(a, (uint32_t)t, (uint32_t)nq, lv, degacc);
      if (MODE != MODE_ANY) cur ^= 1u;
    }
    // per warp: one reduction atomic per counter (no block barrier)
    cnt = __reduce_add_sync(FULL, cnt);
    degacc = __reduce_add_sync(FULL, degacc);
    if ((threadIdx.x & 31) == 0) {
      if (bu && cnt) atomicAdd(&out->nmain, (unsigned long long)cnt);  // a count: the frontier is the bitmap difference
      if (degacc) atomicAdd(&out->deg, (unsigned long long)degacc);
    }
    prev_bu = bu;
    L++;
    ok = dev::grid_barrier(&c->sync, ERR_BARRIER_TIMEOUT, bar_epoch);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (L <= PBG_TRACE_LEVELS) c->t_ns[L] = globaltimer();
    c->t_end = globaltimer();
    c->levels = L;
    c->td_levels = tdl;
    c->bu_levels = bul;
    c->final_bm = cur;
    c->visited = visited;
    c->edges_reached = reached;
    c->bu_mask = bumask;
  }
}

// ---------------------------------------------------------------- small graphs
// Graphs of at most SMALL_N vertices whose search one block finishes sooner
// than the grid (small_graph): the same search with the bitmaps, the parents,
// the levels and the queue in shared memory.  Such a search is a chain of
// round trips: a level of the grid-wide kernels costs 4-7 us (claims, queue
// positions, entries and the barrier all through L2), a top-down level here
// about 2; only offsets and edges are read from memory.
constexpr uint32_t SMALL_N = 5120;
constexpr uint64_t SMALL_M = 1u << 18;
constexpr uint32_t SMALL_T = 1024;
constexpr uint32_t SMALL_PAD = 64;  // words past the starts that are read, never a start
constexpr uint16_t NO_LEVEL = 0xFFFF;

// Where the line lies: one SM walks 2-4 edges a ns, so levels of many edges
// are the grid's (SMALL_M), and so are levels that probe for many unvisited
// vertices (SMALL_N).  Grid / one block, us a search: rMat 2^10, 8n 44.6 / 22.3;
// 2^12, 16n 53.0 / 29.7; 2^12, 30n 49.2 / 31.8; torus 17^3 131 / 73; randLocal
// 5101, 3 edges within 60 420 / 130, 8 within 700 69.6 / 58.3, 20 within 700
// 81.6 / 70.2, 25 within 100 257 / 162; directed 5101, 61 k edges 70.9 / 70.3,
// 121 k 125 / 104.  Past the line, grid / one block built with a limit of 8,192
// (whose wider bottom-up step spills 50-96 bytes): randLocal 6001, 8 edges
// within 700 79 / 87; 7001, 8 within 900 68 / 85, 20 within 700 98 / 98; 8001, 8
// within 1000 73 / 85; rMat 2^13, 14n 39 / 40; directed 8001, 96 k edges 97 /
// 103; but graphs of many small levels gain there too: torus 18^3 152 / 83,
// 20^3 166 / 98, randLocal 6001, 3 within 60 438 / 153.  Vertices and edges do
// not tell the two kinds apart, so the line is where no kind loses.
bool small_graph(const pbg_graph* g) { return g->n <= SMALL_N && g->m <= SMALL_M; }

size_t small_bytes(uint32_t n, uint32_t nwords) {
  // parents, queue; bitmaps; starts, list begins and vertices of a queue chunk; levels
  return sizeof(uint32_t) * (2 * (size_t)n + 2 * nwords + 3 * SMALL_T + SMALL_PAD) + sizeof(uint16_t) * (size_t)n;
}

struct SmallState {
  uint32_t* parent;  // [n]
  uint32_t* q;       // [n]: every vertex enters one frontier, so all of them follow one another
  uint32_t* vis;     // [nwords]
  uint32_t* fresh;   // [nwords] found this level (bottom-up, MIN/MAX)
  // a chunk of the queue, its entries with edges:
  uint32_t* start;  // [SMALL_T + SMALL_PAD] first position of an entry, PBG_NONE past the last
  uint32_t* begin;  // [SMALL_T] its list begin less that
  uint32_t* ent;    // [SMALL_T] its vertex
  uint16_t* level;   // [n]
  uint32_t* tail;
};

// Appends the lanes' found vertices (bits k of `win`: v[k]) to the queue.
template <int K>
__device__ __forceinline__ void small_append(const SmallState& s, const uint32_t (&v)[K], unsigned win) {
  const uint32_t total = __reduce_add_sync(FULL, __popc(win));
  if (total == 0) return;
  const int lane = threadIdx.x & 31;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(s.tail, total);
  at = __shfl_sync(FULL, at, 0);
#pragma unroll
  for (int k = 0; k < K; k++) {
    const unsigned b = __ballot_sync(FULL, (win >> k) & 1u);
    if ((win >> k) & 1u) s.q[at + __popc(b & ((1u << lane) - 1u))] = v[k];
    at += __popc(b);
  }
}

// (1 << SMALL_SHIFT | degree) of a queue entry with edges, 0 of one without:
// one sum counts both (degrees sum to at most SMALL_M, entries to SMALL_T).
constexpr uint32_t SMALL_SHIFT = 20, SMALL_DEG = (1u << SMALL_SHIFT) - 1;
static_assert(SMALL_M <= SMALL_DEG && SMALL_T < (1u << (32 - SMALL_SHIFT)), "packed sums");
__device__ __forceinline__ uint32_t small_pack(uint32_t d) { return d ? (1u << SMALL_SHIFT) | d : 0u; }

// Exclusive prefix sum of x over the block (two syncs); *total = the sum.
__device__ __forceinline__ uint32_t small_scan(uint32_t x, uint32_t* s_part, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t incl = warp_incl_scan(x);
  if (lane == 31) s_part[wid] = incl;
  __syncthreads();
  const uint32_t part = s_part[lane];
  const uint32_t sum = warp_incl_scan(part);
  *total = __shfl_sync(FULL, sum, 31);
  const uint32_t before = __shfl_sync(FULL, sum - part, wid);
  __syncthreads();
  return before + incl - x;
}

// Expands the queue chunk in s.start / begin / ent: `total` positions, a run
// of consecutive ones per warp, 32 * K a step.  The entry of a run's first
// position is searched; from there each window counts the entries that start
// in it (at most 32: none is empty).
template <int MODE>
__device__ __forceinline__ void small_expand(const BfsArgs& a, const SmallState& s, uint32_t total, uint32_t next) {
  constexpr int K = 4;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t run = (total + SMALL_T - 1) / SMALL_T * 32;
  const uint32_t p0 = (threadIdx.x >> 5) * run, p1 = min(total, p0 + run);
  if (p0 >= total) return;  // warp-uniform
  uint32_t own = 0;
#pragma unroll
  for (uint32_t step = SMALL_T / 2; step; step >>= 1)
    if (s.start[own + step] <= p0) own += step;
  for (uint32_t wb = p0; wb < p1; wb += 32 * K) {
    uint32_t v[K], u[K];
    unsigned act = 0, win = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t w = wb + 32 * k;
      u[k] = v[k] = 0;
      if (w >= p1) continue;  // warp-uniform
      const uint32_t rel = s.start[own + 1 + lane] - (w + 1);
      const unsigned starts = __reduce_or_sync(FULL, rel < 32 ? 1u << rel : 0u);  // bit j: at position w + 1 + j
      if (w + lane < p1) {
        const uint32_t my = own + __popc(starts & ((1u << lane) - 1u));
        u[k] = s.ent[my];
        v[k] = __ldg(a.edges + (s.begin[my] + w + lane));  // begin - start may have wrapped: add in 32 bits
        act |= 1u << k;
      }
      own += __popc(starts);
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t bit = 1u << (v[k] & 31);
      if (!((act >> k) & 1u) || (s.vis[v[k] >> 5] & bit)) continue;
      bool won;
      if (MODE == MODE_ANY) {
        won = !(atomicOr(s.vis + (v[k] >> 5), bit) & bit);
        if (won) s.parent[v[k]] = u[k];
      } else {
        const uint32_t old = MODE == MODE_MIN
                                 ? atomicMin(s.parent + v[k], u[k])
                                 : (uint32_t)atomicMax(reinterpret_cast<int*>(s.parent) + v[k], (int)u[k]);
        won = old == PBG_NONE;
        if (won) atomicOr(s.fresh + (v[k] >> 5), bit);
      }
      if (won) {
        s.level[v[k]] = (uint16_t)next;
        win |= 1u << k;
      }
    }
    small_append<K>(s, v, win);
  }
}

// Bottom-up level: a warp takes G bitmap words (all of them in one round of
// the block), a lane one vertex of each, the first LSHARE neighbours by the lane and the rest of longer lists
// by the warp, as in bu_word.
template <int MODE>
__device__ __forceinline__ void small_bottom_up(const BfsArgs& a, const SmallState& s, uint32_t next) {
  constexpr int G = SMALL_N / SMALL_T, PROBES = 2;
  constexpr uint32_t LSHARE = 64;
  const uint32_t lane = threadIdx.x & 31;
  auto hit = [&](uint32_t x) { return (s.vis[x >> 5] >> (x & 31)) & 1u; };
  constexpr uint32_t WARPS = SMALL_T / 32;
  static_assert(G * WARPS * 32 >= SMALL_N, "one round takes every word");
  const uint32_t w0 = threadIdx.x >> 5, nw = (a.n + 31) / 32;  // words w0, w0 + WARPS, ...
  if (w0 < nw) {
    uint32_t b[G], e[G], v[G], p[G];
    unsigned todo = 0, found = 0;
#pragma unroll
    for (int g = 0; g < G; g++) {
      v[g] = (w0 + WARPS * g) * 32 + lane;
      b[g] = e[g] = p[g] = 0;
      if (w0 + WARPS * g < nw && !((s.vis[w0 + WARPS * g] >> lane) & 1u)) {  // the padding past n is marked visited
        b[g] = __ldg(a.offsets + v[g]);
        e[g] = __ldg(a.offsets + v[g] + 1);
        todo |= 1u << g;
      }
    }
    for (uint32_t k0 = 0; k0 < LSHARE; k0 += PROBES) {
      bool any = false;
#pragma unroll
      for (int g = 0; g < G; g++) any |= ((todo & ~found) >> g & 1u) && e[g] - b[g] > k0;
      if (!__any_sync(FULL, any)) break;
      uint32_t x[G][PROBES];
#pragma unroll
      for (int g = 0; g < G; g++)
#pragma unroll
        for (int i = 0; i < PROBES; i++) {
          x[g][i] = PBG_NONE;
          if (w0 + WARPS * g < nw && ((todo & ~found) >> g & 1u) && k0 + i < e[g] - b[g])
            x[g][i] = __ldg(a.edges + (MODE == MODE_MAX ? e[g] - 1 - k0 - i : b[g] + k0 + i));
        }
#pragma unroll
      for (int g = 0; g < G; g++)
#pragma unroll
        for (int i = 0; i < PROBES; i++)
          if (w0 + WARPS * g < nw && x[g][i] != PBG_NONE && !((found >> g) & 1u) && hit(x[g][i])) {
            found |= 1u << g;
            p[g] = x[g][i];
          }
    }
#pragma unroll
    for (int g = 0; g < G; g++) {
      if (w0 + WARPS * g >= nw) break;  // warp-uniform
      unsigned mm = __ballot_sync(FULL, ((todo & ~found) >> g & 1u) && e[g] - b[g] > LSHARE);
      for (; mm; mm &= mm - 1) {
        const int l = __ffs(mm) - 1;
        const uint32_t bb = __shfl_sync(FULL, b[g], l), len = __shfl_sync(FULL, e[g], l) - bb;
        for (uint32_t j = LSHARE; j < len; j += 32) {  // position in scan order (MAX: from the end)
          const uint32_t q = j + lane;
          uint32_t x = 0;
          bool h = false;
          if (q < len) {
            x = __ldg(a.edges + (MODE == MODE_MAX ? bb + len - 1 - q : bb + q));
            h = hit(x);
          }
          const unsigned hb = __ballot_sync(FULL, h);
          if (hb) {
            const uint32_t f = __shfl_sync(FULL, x, __ffs(hb) - 1);
            if (lane == l) {
              found |= 1u << g;
              p[g] = f;
            }
            break;
          }
        }
      }
      const unsigned nb = __ballot_sync(FULL, (found >> g) & 1u);
      if (lane == 0 && nb) s.fresh[w0 + WARPS * g] = nb;
      if ((found >> g) & 1u) {
        s.parent[v[g]] = p[g];
        s.level[v[g]] = (uint16_t)next;
      }
    }
    small_append<G>(s, v, found);
  }
}

template <int MODE>
__global__ void __launch_bounds__(SMALL_T, 1) bfs_small(BfsArgs a) {
  extern __shared__ uint32_t s_mem[];
  __shared__ uint32_t s_tail, s_part[32];
  const uint32_t n = a.n, nw = a.nwords, tid = threadIdx.x;
  SmallState s;
  s.parent = s_mem;
  s.q = s.parent + n;
  s.vis = s.q + n;
  s.fresh = s.vis + nw;
  s.start = s.fresh + nw;
  s.begin = s.start + SMALL_T + SMALL_PAD;
  s.ent = s.begin + SMALL_T;
  s.level = reinterpret_cast<uint16_t*>(s.ent + SMALL_T);
  s.tail = &s_tail;
  BfsCtrl* c = a.ctrl;
  if (tid == 0) c->t_start = globaltimer();
  for (uint32_t v = tid; v < n; v += SMALL_T) {
    s.parent[v] = PBG_NONE;
    s.level[v] = NO_LEVEL;
  }
  for (uint32_t w = tid; w < nw; w += SMALL_T) {
    s.vis[w] = a.iso[w] | (w == a.src >> 5 ? 1u << (a.src & 31) : 0u);
    s.fresh[w] = 0;
  }
  if (tid < SMALL_PAD) s.start[SMALL_T + tid] = PBG_NONE;
  __syncthreads();
  if (tid == 0) {
    s.parent[a.src] = a.src;
    s.level[a.src] = 0;
    s.q[0] = a.src;
    s_tail = 1;
  }
  __syncthreads();
  uint32_t head = 0, L = 0, tdl = 0, bul = 0;
  unsigned long long reached = 0, bumask = 0;
  bool prev_bu = false;
  for (;;) {
    const uint32_t tail = s_tail, nf = tail - head;
    if (nf == 0) break;
    // the first SMALL_T entries' lists (all of them, mostly), and the
    // frontier's out-degree
    uint32_t u = 0, b = 0, d = 0, rest = 0;
    if (tid < nf) {
      u = s.q[head + tid];
      b = __ldg(a.offsets + u);
      d = __ldg(a.offsets + u + 1) - b;
    }
    for (uint32_t i = SMALL_T + tid; i < nf; i += SMALL_T) {
      const uint32_t x = s.q[head + i];
      rest += __ldg(a.offsets + x + 1) - __ldg(a.offsets + x);
    }
    uint32_t total = 0, more = 0;
    uint32_t at = small_scan(small_pack(d), s_part, &total);
    if (nf > SMALL_T) small_scan(rest, s_part, &more);
    const uint32_t fdeg = (total & SMALL_DEG) + more;
    bool bu;
    if (a.policy == PBG_DIR_TOPDOWN || !a.symmetric)
      bu = false;
    else if (a.policy == PBG_DIR_BOTTOMUP)
      bu = true;
    else if (!prev_bu)
      bu = (unsigned long long)nf + fdeg > a.m / a.alpha;
    else
      bu = nf > a.n / a.beta;
    // A level that the switch takes bottom-up while its frontier holds few of
    // the edges is found from the frontier's side all the same: the vertices are
    // the same, and so are MIN and MAX parents, and unvisited vertices that probe
    // in vain for a frontier of a few dozen cost one SM 18-43 us on rMat 2^12
    // (5-12 k frontier edges of 97 k), the frontier's edges 4-6 us; level with
    // each other at a quarter.  The switch goes on from its own choice (bu); what
    // is reported is what ran.
    const bool up = bu && !(a.policy == PBG_DIR_AUTO && 4ull * fdeg <= a.m);
    if (tid == 0) {
      if (L < PBG_TRACE_LEVELS) {
        c->t_ns[L] = globaltimer();
        c->t_nf[L] = nf;
        c->t_deg[L] = fdeg;
        c->t_bu[L] = up ? 1u : 0u;
      }
      reached += fdeg;
      if (up) {
        bul++;
        if (L < 64) bumask |= 1ull << L;
      } else {
        tdl++;
      }
    }
    if (up) {
      small_bottom_up<MODE>(a, s, L + 1);
    } else {
      for (uint32_t c0 = 0; c0 < nf; c0 += SMALL_T) {
        if (c0) {  // a later chunk of a long queue
          d = 0;
          if (c0 + tid < nf) {
            u = s.q[head + c0 + tid];
            b = __ldg(a.offsets + u);
            d = __ldg(a.offsets + u + 1) - b;
          }
          at = small_scan(small_pack(d), s_part, &total);  // its syncs also end the chunk before
        }
        const uint32_t entries = total >> SMALL_SHIFT;
        if (tid >= entries) s.start[tid] = PBG_NONE;
        if (d) {
          const uint32_t r = at >> SMALL_SHIFT, p = at & SMALL_DEG;
          s.start[r] = p;
          s.begin[r] = b - p;
          s.ent[r] = u;
        }
        __syncthreads();
        small_expand<MODE>(a, s, total & SMALL_DEG, L + 1);
      }
    }
    __syncthreads();
    if (up || MODE != MODE_ANY) {
      for (uint32_t w = tid; w < nw; w += SMALL_T) {
        const uint32_t f = s.fresh[w];
        if (f) {
          s.vis[w] |= f;
          s.fresh[w] = 0;
        }
      }
      __syncthreads();
    }
    prev_bu = bu;
    head = tail;
    L++;
  }
  for (uint32_t v = tid; v < n; v += SMALL_T) {
    a.parent[v] = s.parent[v];
    if (a.level) a.level[v] = s.level[v] == NO_LEVEL ? PBG_NONE : (uint32_t)s.level[v];
  }
  if (tid == 0) {
    if (L <= PBG_TRACE_LEVELS) c->t_ns[L] = globaltimer();
    c->t_end = globaltimer();
    c->levels = L;
    c->td_levels = tdl;
    c->bu_levels = bul;
    c->final_bm = 0;
    c->visited = head;
    c->edges_reached = reached;
    c->bu_mask = bumask;
    c->sync.error = 0;
  }
}

template <int MODE>
int launch_small(const BfsArgs& a, cudaStream_t s) {
  static std::mutex mu;
  static int dev_of = -1;
  int dev = 0;
  PBG_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev_of != dev) {
      PBG_CUDA(cudaFuncSetAttribute(bfs_small<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)small_bytes(SMALL_N, SMALL_N / 32)));
      dev_of = dev;
    }
  }
  bfs_small<MODE><<<1, SMALL_T, small_bytes(a.n, a.nwords), s>>>(a);
  PBG_CUDA(cudaGetLastError());
  return PBG_OK;
}

template <int MODE>
int launch_lean(const BfsArgs& a, int num_sms, cudaStream_t s) {
  static std::mutex mu;
  static int grid = 0, dev_of = -1;
  int dev = 0;
  PBG_CUDA(cudaGetDevice(&dev));
  int g;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev_of != dev) {
      int per_sm = 0;
      PBG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bfs_lean<MODE>, 1024, 0));
      if (per_sm < 1) return fail(PBG_ERR_CUDA, "BFS kernel cannot be resident with this block size");
      grid = per_sm * num_sms;
      dev_of = dev;
    }
    g = grid;
  }
  BfsArgs args = a;
  void* params[] = {&args};
  PBG_CUDA(cudaLaunchCooperativeKernel((const void*)bfs_lean<MODE>, dim3(g), dim3(1024), params, 0, s));
  return PBG_OK;
}

template <int MODE, int BLOCK>
int launch_shape(const BfsArgs& a, int num_sms, cudaStream_t s) {
  static std::mutex mu;
  static int grid = 0, dev_of = -1;
  int dev = 0;
  PBG_CUDA(cudaGetDevice(&dev));
  int g;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev_of != dev) {
      int per_sm = 0;
      PBG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bfs_persistent<MODE, BLOCK>, BLOCK, 0));
      if (per_sm < 1) return fail(PBG_ERR_CUDA, "BFS kernel cannot be resident with this block size");
      grid = per_sm * num_sms;
      dev_of = dev;
    }
    g = grid;
  }
  BfsArgs args = a;
  void* params[] = {&args};
  PBG_CUDA(cudaLaunchCooperativeKernel((const void*)bfs_persistent<MODE, BLOCK>, dim3(g), dim3(BLOCK), params, 0, s));
  return PBG_OK;
}

template <int MODE>
int launch_mode(const BfsArgs& a, int block, int num_sms, cudaStream_t s) {
  if (block == 256) return launch_shape<MODE, 256>(a, num_sms, s);
  if (block == 1024) return launch_shape<MODE, 1024>(a, num_sms, s);
  return launch_shape<MODE, 512>(a, num_sms, s);
}

}  // namespace

void resolve_opts(const pbg_bfs_opts* in, pbg_bfs_opts* o) {
  if (in)
    *o = *in;
  else
    pbg_bfs_opts_default(o);
  if (o->alpha == 0) o->alpha = 20;
  if (o->beta == 0) o->beta = 20;
  if (o->block_threads == 0) o->block_threads = 1024;
  if (o->chunk_min_degree == 0) o->chunk_min_degree = 32;
}

void resolve_graph_opts(const pbg_graph* g, const pbg_bfs_opts* in, bool multi, pbg_bfs_opts* o) {
  if (!in && g && (multi ? g->has_tuned_multi : g->has_tuned))
    resolve_opts(multi ? &g->tuned_multi : &g->tuned, o);
  else
    resolve_opts(in, o);
  // the lanes of a tile step together, so a short list's position runs up to
  // the chunk degree past its end (td_small, lean_tile): not past 2^32
  if (g && !multi && g->m + o->chunk_min_degree + PER_LANE > (1ull << 32)) o->chunk_min_degree = 32;
}

int bfs_ensure_workspace(pbg_graph* g, const pbg_bfs_opts& o) {
  BfsWorkspace& w = g->ws;
  if (w.ready && w.big_min_degree <= o.chunk_min_degree) return PBG_OK;
  bfs_free_workspace(g);
  const size_t n = g->n ? g->n : 1;
  const uint32_t big_cap = (uint32_t)std::min<uint64_t>(n, g->m / o.chunk_min_degree + 1);
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 2 && e == cudaSuccess; i++) {
    e = cudaMalloc(&w.bm[i], sizeof(uint32_t) * g->nwords);
    if (e == cudaSuccess) e = cudaMalloc(&w.q[i], sizeof(uint32_t) * n);
    if (e == cudaSuccess) e = cudaMalloc(&w.qr[i], sizeof(uint2) * n);
    if (e == cudaSuccess) e = cudaMalloc(&w.qbig[i], sizeof(uint4) * big_cap);
  }
  if (e == cudaSuccess) e = cudaMalloc(&w.ctrl, sizeof(BfsCtrl));
  if (e == cudaSuccess) e = cudaMemset(w.ctrl, 0, sizeof(BfsCtrl));
  if (e == cudaSuccess && !w.ev0) e = cudaEventCreate(&w.ev0);
  if (e == cudaSuccess && !w.ev1) e = cudaEventCreate(&w.ev1);
  if (e != cudaSuccess) {
    bfs_free_workspace(g);
    cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? PBG_ERR_OOM : PBG_ERR_CUDA,
                std::string("BFS workspace: ") + cudaGetErrorString(e));
  }
  w.big_cap = big_cap;
  w.big_min_degree = o.chunk_min_degree;
  w.ready = true;
  return PBG_OK;
}

void bfs_free_workspace(pbg_graph* g) {
  BfsWorkspace& w = g->ws;
  for (int i = 0; i < 2; i++) {
    cudaFree(w.bm[i]);
    cudaFree(w.q[i]);
    cudaFree(w.qr[i]);
    w.qr[i] = nullptr;
    cudaFree(w.qbig[i]);
    w.bm[i] = nullptr;
    w.q[i] = nullptr;
    w.qbig[i] = nullptr;
  }
  cudaFree(w.ctrl);
  w.ctrl = nullptr;
  cudaFree(w.parent);
  cudaFree(w.level);
  w.parent = nullptr;
  w.level = nullptr;
  w.ready = false;
}

// Launches the persistent kernel on caller-provided state arrays (used by the
// allocation-free entry point in noalloc.cu; the handle path above builds the
// same arguments from its workspace).
int bfs_launch_on(const BfsOnArgs& r, const pbg_bfs_opts& o, int num_sms, cudaStream_t s) {
  BfsArgs a;
  a.offsets = r.offsets;
  a.edges = r.edges;
  a.iso = r.iso;
  a.parent = r.parent;
  a.level = r.level;
  a.bm0 = r.bm0;
  a.bm1 = r.bm1;
  a.q0 = r.q0;
  a.q1 = r.q1;
  a.qr0 = r.qr0;
  a.qr1 = r.qr1;
  a.qb0 = r.qb0;
  a.qb1 = r.qb1;
  a.ctrl = r.ctrl;
  a.m = r.m;
  a.n = r.n;
  a.nwords = r.nwords;
  a.big_cap = r.big_cap;
  a.src = r.src;
  a.alpha = o.alpha;
  a.beta = o.beta;
  a.policy = o.direction;
  a.chunk_deg = o.chunk_min_degree;
  a.symmetric = r.symmetric;
  switch (o.parent_mode) {
    case PBG_PARENT_ANY: return launch_mode<MODE_ANY>(a, (int)o.block_threads, num_sms, s);
    case PBG_PARENT_MIN: return launch_mode<MODE_MIN>(a, (int)o.block_threads, num_sms, s);
    default: return launch_mode<MODE_MAX>(a, (int)o.block_threads, num_sms, s);
  }
}

int bfs_launch(pbg_graph* g, uint32_t src, const pbg_bfs_opts& o, uint32_t* d_parent, uint32_t* d_level,
               cudaStream_t s) {
  if (o.parent_mode > PBG_PARENT_MAX) return fail(PBG_ERR_ARG, "unknown parent_mode");
  if (o.direction > PBG_DIR_BOTTOMUP) return fail(PBG_ERR_ARG, "unknown direction policy");
  if (o.direction == PBG_DIR_BOTTOMUP && !(g->flags & PBG_GRAPH_SYMMETRIC))
    return fail(PBG_ERR_ARG, "bottom-up needs a symmetric graph");
  if (o.block_threads != 256 && o.block_threads != 512 && o.block_threads != 1024)
    return fail(PBG_ERR_ARG, "block_threads must be 256, 512 or 1024");
  if (o.chunk_min_degree < 1) return fail(PBG_ERR_ARG, "chunk_min_degree must be >= 1");
  if (g->m > PBG_MAX_SEARCH_EDGES) return fail(PBG_ERR_ARG, "searches take at most PBG_MAX_SEARCH_EDGES edges");
  int rc = bfs_ensure_workspace(g, o);
  if (rc) return rc;
  BfsWorkspace& w = g->ws;
  BfsArgs a;
  a.offsets = g->d_offsets;
  a.edges = g->d_edges;
  a.iso = g->d_iso;
  a.parent = d_parent;
  a.level = d_level;
  a.bm0 = w.bm[0];
  a.bm1 = w.bm[1];
  a.q0 = w.q[0];
  a.q1 = w.q[1];
  a.qr0 = w.qr[0];
  a.qr1 = w.qr[1];
  a.qb0 = w.qbig[0];
  a.qb1 = w.qbig[1];
  a.ctrl = w.ctrl;
  a.m = g->m;
  a.n = g->n;
  a.nwords = g->nwords;
  a.big_cap = w.big_cap;
  a.src = src;
  a.alpha = o.alpha;
  a.beta = o.beta;
  a.policy = o.direction;
  a.chunk_deg = o.chunk_min_degree;
  a.symmetric = (g->flags & PBG_GRAPH_SYMMETRIC) ? 1u : 0u;
  const bool small = small_graph(g);
  if (!small) PBG_CUDA(cudaMemsetAsync(w.ctrl, 0, sizeof(BfsCtrl), s));  // bfs_small writes what is read of it
  PBG_CUDA(cudaEventRecord(w.ev0, s));
  if (small) {
    switch (o.parent_mode) {
      case PBG_PARENT_ANY: rc = launch_small<MODE_ANY>(a, s); break;
      case PBG_PARENT_MIN: rc = launch_small<MODE_MIN>(a, s); break;
      default: rc = launch_small<MODE_MAX>(a, s); break;
    }
  } else if (g->max_degree < o.chunk_min_degree) {  // every list short: no chunk queue (bfs_lean)
    switch (o.parent_mode) {
      case PBG_PARENT_ANY: rc = launch_lean<MODE_ANY>(a, g->num_sms, s); break;
      case PBG_PARENT_MIN: rc = launch_lean<MODE_MIN>(a, g->num_sms, s); break;
      default: rc = launch_lean<MODE_MAX>(a, g->num_sms, s); break;
    }
  } else {
    switch (o.parent_mode) {
      case PBG_PARENT_ANY: rc = launch_mode<MODE_ANY>(a, (int)o.block_threads, g->num_sms, s); break;
      case PBG_PARENT_MIN: rc = launch_mode<MODE_MIN>(a, (int)o.block_threads, g->num_sms, s); break;
      default: rc = launch_mode<MODE_MAX>(a, (int)o.block_threads, g->num_sms, s); break;
    }
  }
  if (rc) return rc;
  PBG_CUDA(cudaEventRecord(w.ev1, s));
  g->stats_pending = true;
  return PBG_OK;
}

int bfs_read_trace(pbg_graph* g, pbg_level_trace* out, uint32_t cap, uint32_t* count) {
  int rc = bfs_read_stats(g, nullptr);
  if (!g->ws.ready) {  // no search: an error, or no levels (bfs_read_stats)
    if (!rc && count) *count = 0;
    return rc;
  }
  if (rc && rc != PBG_ERR_TIMEOUT && rc != PBG_ERR_STATE) return rc;
  BfsCtrl* c = new BfsCtrl;
  cudaError_t e = cudaMemcpy(c, g->ws.ctrl, sizeof(BfsCtrl), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    delete c;
    return cuda_fail(e, "trace copy");
  }
  uint32_t nl = std::min<uint32_t>(c->levels, PBG_TRACE_LEVELS);
  uint32_t k = std::min(nl, cap);
  for (uint32_t L = 0; L < k; L++) {
    out[L].level = L;
    out[L].bottom_up = c->t_bu[L];
    out[L].frontier = c->t_nf[L];
    out[L].frontier_degree = c->t_deg[L];
    out[L].ms = (c->t_ns[L + 1] - c->t_ns[L]) * 1e-6;
  }
  if (count) *count = k;
  delete c;
  return PBG_OK;
}

// The last search's statistics; all zero on a handle that so far only ran an
// independent set.
int bfs_read_stats(pbg_graph* g, pbg_bfs_stats* st) {
  if (!g->ws.ready && !g->mis_ran) return fail(PBG_ERR_STATE, "no BFS has run on this graph");
  if (g->stats_pending) {
    BfsCtrl c;
    PBG_CUDA(cudaEventSynchronize(g->ws.ev1));
    PBG_CUDA(cudaMemcpy(&c, g->ws.ctrl, sizeof(BfsCtrl), cudaMemcpyDeviceToHost));
    pbg_bfs_stats& s = g->last;
    s.levels = c.levels;
    s.topdown_levels = c.td_levels;
    s.bottomup_levels = c.bu_levels;
    s.error = c.sync.error;
    s.visited = c.visited;
    s.edges_reached = c.edges_reached;
    s.bottomup_mask = c.bu_mask;
    float ms = 0.f;
    PBG_CUDA(cudaEventElapsedTime(&ms, g->ws.ev0, g->ws.ev1));
    s.device_ms = ms;
    s.init_ms = (c.levels > 0 && c.t_ns[0] > c.t_start) ? (float)((c.t_ns[0] - c.t_start) * 1e-6) : 0.f;
    s.kernel_ms = (c.t_end > c.t_start) ? (float)((c.t_end - c.t_start) * 1e-6) : 0.f;
    g->stats_pending = false;
  }
  if (st) *st = g->last;
  if (g->last.error & ERR_BARRIER_TIMEOUT) return fail(PBG_ERR_TIMEOUT, "BFS: a grid barrier wait ran out");
  if (g->last.error) return fail(PBG_ERR_STATE, "BFS: device error word set");
  return PBG_OK;
}

}  // namespace pbg
