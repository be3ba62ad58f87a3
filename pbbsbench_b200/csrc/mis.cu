// mis.cu -- maximal independent set on a resident graph (sm_100a): the
// frontier engine of the BFS path reused for PBBS's maximalIndependentSet
// benchmark (benchmarks/maximalIndependentSet/bench/MIS.h:8).
//
// The set computed is the one serialMIS returns
// (maximalIndependentSet/serialMIS/MIS.C:33-47): vertices are taken in id
// order and v joins unless a vertex already in the set is among its
// neighbours (a self loop keeps v out).  That greedy set is the unique one
// in which
//     v is in  <=>  no out-neighbour u < v is in, and v has no self loop,
// and this rule can be evaluated in parallel: v is decided OUT as soon as one
// earlier neighbour is IN, IN as soon as every earlier neighbour is OUT, and
// waits otherwise.  Decisions are final and correct whatever the order in
// which other vertices were decided, so threads may read flags that others
// are writing.  The result is deterministic and bit-exact with
// serialMIS, and a valid maximal independent set on symmetric graphs (the
// test of MISCheck.C:39-66), the contract of the nondeterministic ndMIS
// (ndMIS/MIS.C:41-80) as well.
//
// One cooperative launch, one pass.  The warps of the (fully resident) grid
// take 32-vertex tiles in id order and stay with a tile until its vertices are
// decided: a lane walks its list up to the first undecided earlier neighbour,
// looks at that neighbour's flag until it is decided, and walks on, so no
// list entry is walked twice.  A vertex waits for smaller ids only, and the
// earliest unfinished tile is always held by a warp whose earlier tiles are
// done, so its smallest undecided vertex decides at its next look: the pass
// ends.  In flight are the 32 * warps ids of the warps' current tiles (more
// when warps run ahead); nearly all of a list's other entries are decided
// when it is walked.  The wait is bounded: a warp that neither progresses nor
// sees any other warp progress for BARRIER_TIMEOUT_NS sets the error word.
//
// Rounds over a queue of undecided vertices with a grid barrier each, as
// before, walked everything that was undecided again and again (19 M queue
// entries on rMat 2^24), and a dependency chain cost a round a link: rMat 2^24
// 1.065 -> 0.814 ms, 2^18 118 -> 59 us, 2^11 45 -> 23 us; torus 150^3 160 -> 90
// us; randLocal 4,000,001, whose chains run along the ids, 13.6 -> 1.04 ms.
//
// Each lane walks its list in steps of MK entries, LANE_SHARE of them at
// most; a list still clear after those is walked on by the whole warp, 32 a
// step.  When the graph's lists are ascending (checked once per graph), a walk
// stops at the first neighbour above v.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "device_util.cuh"
#include "internal.cuh"

namespace pbg {
namespace {

using dev::FULL;
constexpr int MK = 4;  // loads per lane per step
constexpr uint8_t UNDECIDED = 0, IN_SET = 1, OUT_SET = 2;
constexpr uint8_t MORE = 3;      // walk result: clear so far, list goes on past the lane's share
// Entries a lane walks before the warp takes over (rMat 2^24, ms: 16 0.95, 32
// 0.814, 64 0.96, 128 1.01: a warp waits for its longest walk, and walks long
// lists one after another); MK 2 and 8 are slower elsewhere (torus 150^3 with 8
// 102 us).
constexpr uint32_t LANE_SHARE = 32;

struct MisArgs {
  const uint32_t* __restrict__ offsets;
  const uint32_t* __restrict__ edges;
  uint8_t* flags;  // UNDECIDED at the start
  BfsCtrl* ctrl;
  uint32_t* done;  // per warp of the grid: its last finished tile + 1 (0 at the start)
  uint32_t n;
  uint32_t sorted;
};

__device__ __forceinline__ uint8_t ld_flag_fresh(const uint8_t* p) {
  uint16_t v;
  asm volatile("ld.relaxed.gpu.global.u8 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return (uint8_t)v;
}

// A neighbour's flag, through L1.  A flag changes once per call, from
// UNDECIDED to its final value, so a line cached earlier holds the final
// value or an UNDECIDED that only makes the reader look again (settle, from
// L2).  Hub flags, read by many lists on one SM, then come from L1: rMat 2^18
// 87 us with L2 reads of ids that may be undecided, 60 us with L1 reads.
__device__ __forceinline__ uint8_t ld_flag(const uint8_t* p) {
  uint16_t v;
  asm volatile("ld.global.ca.u8 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return (uint8_t)v;
}

// Lane-serial walk of v's list from position j, up to LANE_SHARE entries, MK
// loads a step.
// Returns OUT_SET; UNDECIDED with *cur set to the first undecided earlier
// neighbour; IN_SET when the list is clear to its end (or to a larger
// neighbour in an ascending list); MORE with *cur at the first entry not
// walked when the share is clear and the list goes on.
__device__ __forceinline__ uint8_t walk_lane(const MisArgs& a, uint32_t v, uint32_t j, uint32_t e, uint32_t* cur) {
  const uint32_t share = min(e - j, LANE_SHARE);  // counted from j: a list may end at 2^32 - 1
  uint32_t first_wait = e;
  bool stop = false;
  for (uint32_t k = 0; k < share; k += MK) {
    uint32_t u[MK];
#pragma unroll
    for (int i = 0; i < MK; i++) u[i] = (k + i < share) ? __ldg(a.edges + j + k + i) : v + 1;
    uint8_t f[MK];
#pragma unroll
    for (int i = 0; i < MK; i++) f[i] = (u[i] < v) ? ld_flag(a.flags + u[i]) : OUT_SET;
#pragma unroll
    for (int i = 0; i < MK; i++) {
      if (k + i >= share) break;
      if (u[i] == v || f[i] == IN_SET) return OUT_SET;  // a self loop, or an earlier neighbour in the set
      if (u[i] < v && f[i] == UNDECIDED && first_wait == e) first_wait = j + k + i;
      if (u[i] > v && a.sorted) stop = true;
    }
    // A step with an undecided neighbour ends the walk: the rest of the list
    // is read when that neighbour has decided.
    if (stop || first_wait < e) break;
  }
  if (first_wait < e) {
    *cur = first_wait;
    return UNDECIDED;
  }
  if (!stop && share < e - j) {
    *cur = j + share;
    return MORE;
  }
  return IN_SET;
}

// Warp-cooperative walk of one long list (every lane calls it with the same
// v, j, e; j < e).
__device__ __forceinline__ uint8_t walk_warp(const MisArgs& a, uint32_t v, uint32_t j, uint32_t e, uint32_t* cur) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t first_wait = e;
  for (;; j += 32) {
    const bool have = lane < e - j;
    uint32_t u = v + 1;
    uint8_t f = OUT_SET;
    if (have) {
      u = __ldg(a.edges + j + lane);
      if (u < v) f = ld_flag(a.flags + u);
    }
    const bool out = have && (u == v || f == IN_SET);
    if (__any_sync(FULL, out)) return OUT_SET;
    const unsigned w = __ballot_sync(FULL, have && u < v && f == UNDECIDED);
    if (w) {  // as in walk_lane: resume at the first undecided neighbour
      first_wait = j + __ffs(w) - 1;
      break;
    }
    if (a.sorted && __any_sync(FULL, have && u > v)) break;
    if (e - j <= 32) break;
  }
  if (first_wait < e) {
    *cur = first_wait;
    return UNDECIDED;
  }
  return IN_SET;
}

// Whether any warp has finished a tile since *seen was taken (then updated):
// the order-free sum of the warps' words, which start at 0 and grow with every
// tile.  Whole warp.
__device__ bool progressed(const MisArgs& a, uint32_t warps, uint32_t* seen) {
  uint32_t s = 0;
  for (uint32_t i = threadIdx.x & 31; i < warps; i += 32) s += *reinterpret_cast<volatile uint32_t*>(a.done + i);
  s = __reduce_add_sync(FULL, s);
  const bool moved = s != *seen;
  *seen = s;
  return moved;
}

// One vertex per lane (valid when `have`; list [j, e)): walks and waits until
// all are decided.  False when the wait was given up.
__device__ __forceinline__ bool settle(const MisArgs& a, uint32_t v, uint32_t j, uint32_t e, bool have,
                                       uint32_t warps, uint32_t& in_count) {
  const int lane = threadIdx.x & 31;
  bool pending = have;
  uint32_t cur = j, waits_for = PBG_NONE;  // not walked yet
  unsigned long long t0 = 0;
  uint32_t seen = 0;
  for (uint32_t it = 1; __any_sync(FULL, pending); it++) {
    uint8_t res = UNDECIDED;
    bool walk = false;
    if (pending) {
      if (waits_for == PBG_NONE) {
        walk = true;
      } else {
        const uint8_t f = ld_flag_fresh(a.flags + waits_for);
        if (f == IN_SET) {
          res = OUT_SET;
        } else if (f == OUT_SET) {
          cur++;
          walk = true;
        }
      }
    }
    if (walk) res = walk_lane(a, v, cur, e, &cur);
    for (unsigned lm = __ballot_sync(FULL, res == MORE); lm; lm &= lm - 1) {
      const int l = __ffs(lm) - 1;
      const uint32_t lv = __shfl_sync(FULL, v, l), lj = __shfl_sync(FULL, cur, l), le = __shfl_sync(FULL, e, l);
      uint32_t lc = lj;
      const uint8_t r = walk_warp(a, lv, lj, le, &lc);
      if (lane == l) {
        res = r;
        cur = lc;
      }
    }
    if (walk && res == UNDECIDED) waits_for = __ldg(a.edges + cur);  // as read: perhaps decided by now
    if (pending && res != UNDECIDED) {
      *reinterpret_cast<volatile uint8_t*>(a.flags + v) = res;
      if (res == IN_SET) in_count++;
      pending = false;
    }
    if ((it & 255) == 0) {  // bounded while nothing moves anywhere
      // a vote: another warp may set the word between two lanes' loads, and
      // the collectives here and after the pass need every lane
      if (__any_sync(FULL, dev::ld_acquire_u32(&a.ctrl->sync.error) != 0)) return false;
      const unsigned long long now = dev::globaltimer();
      if (it == 256) {
        t0 = now;
        progressed(a, warps, &seen);
      } else if (__any_sync(FULL, now - t0 > dev::BARRIER_TIMEOUT_NS)) {
        if (!progressed(a, warps, &seen)) {
          if (lane == 0) atomicOr(&a.ctrl->sync.error, ERR_BARRIER_TIMEOUT);
          return false;
        }
        t0 = now;
      }
    }
  }
  return true;
}

// Two blocks per SM at <= 40 registers (no spills): 48 resident warps a SM
// hide more of each walk's load latency than one 1024-thread block's 32.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 2) mis_one_pass(MisArgs a) {
  BfsCtrl* c = a.ctrl;
  const uint32_t lane = threadIdx.x & 31;
  // tiles go round-robin over blocks first, so a small graph still uses every SM
  const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint32_t tw = (gridDim.x * blockDim.x) >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    c->t_start = c->t_ns[0] = dev::globaltimer();
    c->t_nf[0] = a.n;
    c->levels = 1;
  }
  const uint32_t tiles = (a.n + 31) / 32;  // n < 2^31
  uint32_t in_count = 0;
  uint32_t b = 0, e = 0;
  if (gw * 32 + lane < a.n) {
    b = __ldg(a.offsets + gw * 32 + lane);
    e = __ldg(a.offsets + gw * 32 + lane + 1);
  }
  for (uint32_t t = gw; t < tiles; t += tw) {
    const uint32_t v = t * 32 + lane;
    uint32_t nb = 0, ne = 0;  // the next tile's lists, on their way while this one settles
    if (t + tw < tiles && v + 32 * tw < a.n) {
      nb = __ldg(a.offsets + v + 32 * tw);
      ne = __ldg(a.offsets + v + 32 * tw + 1);
    }
    if (!settle(a, v, b, e, v < a.n, tw, in_count)) break;
    if (lane == 0) *reinterpret_cast<volatile uint32_t*>(a.done + gw) = t + 1;
    b = nb;
    e = ne;
  }
  const unsigned long long bin = dev::block_sum(in_count);
  if (threadIdx.x == 0) {
    if (bin) atomicAdd(&c->visited, bin);
    const unsigned long long now = dev::globaltimer();
    atomicMax(&c->t_end, now);
    atomicMax(&c->t_ns[1], now);
  }
}

// One warp per vertex: is every list ascending?  (bad set when one is not)
__global__ void k_lists_sorted(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edg, uint32_t n,
                               unsigned* bad) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = w; v < n; v += nw) {
    const uint32_t b = off[v], e = off[v + 1];
    bool unsorted = false;
    for (uint64_t j = (uint64_t)b + 1 + lane; j < e; j += 32) unsorted |= edg[j - 1] > edg[j];
    if (__any_sync(FULL, unsorted)) {
      if (lane == 0) atomicOr(bad, 1u);
    }
  }
}

constexpr int MIS_BLOCK = 768;

int mis_grid(int num_sms, int* grid_out) {
  static std::mutex mu;
  static int grid = 0, dev_of = -1;
  int dev = 0;
  PBG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev_of != dev) {
    int per_sm = 0;
    PBG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mis_one_pass<MIS_BLOCK>, MIS_BLOCK, 0));
    if (per_sm < 1) return fail(PBG_ERR_CUDA, "MIS kernel cannot be resident");
    grid = per_sm * num_sms;
    dev_of = dev;
  }
  *grid_out = grid;
  return PBG_OK;
}

// Whether every list of g is ascending, found once per graph.
int lists_sorted(pbg_graph* g, uint32_t* sorted) {
  if (g->lists_sorted >= 0) {
    *sorted = (uint32_t)g->lists_sorted;
    return PBG_OK;
  }
  unsigned* d_bad = nullptr;
  unsigned bad = 0;
  PBG_CUDA(cudaMalloc(&d_bad, sizeof(unsigned)));
  cudaError_t e = cudaMemsetAsync(d_bad, 0, sizeof(unsigned), g->stream);
  if (e == cudaSuccess) {
    k_lists_sorted<<<grid_for((uint64_t)g->n * 32, g->num_sms), 256, 0, g->stream>>>(g->d_offsets, g->d_edges, g->n,
                                                                                      d_bad);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, sizeof(unsigned), cudaMemcpyDeviceToHost, g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  cudaFree(d_bad);
  if (e != cudaSuccess) return cuda_fail(e, "list order check");
  g->lists_sorted = bad ? 0 : 1;
  *sorted = (uint32_t)g->lists_sorted;
  return PBG_OK;
}

}  // namespace

int mis_launch(pbg_graph* g, uint8_t* d_flags, cudaStream_t s) {
  uint32_t sorted = 0;
  int rc = lists_sorted(g, &sorted);
  if (rc) return rc;
  int grid = 0;
  rc = mis_grid(g->num_sms, &grid);
  if (rc) return rc;
  const size_t ctrl_bytes = sizeof(BfsCtrl) + sizeof(uint32_t) * (size_t)grid * (MIS_BLOCK / 32);
  if (!g->mis_ctrl) {
    // the control block, then the warps' progress words
    cudaError_t e = cudaMalloc(&g->mis_ctrl, ctrl_bytes);
    if (e == cudaSuccess && !g->mis_ev0) e = cudaEventCreate(&g->mis_ev0);
    if (e == cudaSuccess && !g->mis_ev1) e = cudaEventCreate(&g->mis_ev1);
    if (e != cudaSuccess) {
      cudaFree(g->mis_ctrl);
      g->mis_ctrl = nullptr;
      return cuda_fail(e, "MIS control block");
    }
  }
  // as many blocks as there are tiles, at most all that are resident
  const int blocks = (int)std::min<uint64_t>((uint64_t)grid, ((uint64_t)g->n + 31) / 32);
  MisArgs a;
  a.offsets = g->d_offsets;
  a.edges = g->d_edges;
  a.flags = d_flags;
  a.ctrl = g->mis_ctrl;
  a.done = reinterpret_cast<uint32_t*>(g->mis_ctrl + 1);
  a.n = g->n;
  a.sorted = sorted;
  PBG_CUDA(cudaEventRecord(g->mis_ev0, s));
  PBG_CUDA(cudaMemsetAsync(g->mis_ctrl, 0, ctrl_bytes, s));
  PBG_CUDA(cudaMemsetAsync(d_flags, UNDECIDED, g->n, s));
  void* params[] = {&a};
  PBG_CUDA(cudaLaunchCooperativeKernel((const void*)mis_one_pass<MIS_BLOCK>, dim3(blocks), dim3(MIS_BLOCK), params,
                                       0, s));
  PBG_CUDA(cudaEventRecord(g->mis_ev1, s));
  g->mis_pending = true;
  return PBG_OK;
}

int mis_read_stats(pbg_graph* g, pbg_mis_stats* st) {
  if (!g->mis_ctrl || !g->mis_ran) return fail(PBG_ERR_STATE, "no MIS has run on this graph");
  if (g->mis_pending) {
    BfsCtrl c;
    PBG_CUDA(cudaEventSynchronize(g->mis_ev1));
    PBG_CUDA(cudaMemcpy(&c, g->mis_ctrl, sizeof(BfsCtrl), cudaMemcpyDeviceToHost));
    pbg_mis_stats& m = g->mis_last;
    m.rounds = c.levels;
    m.error = c.sync.error;
    m.in_set = c.visited;
    float ms = 0.f;
    PBG_CUDA(cudaEventElapsedTime(&ms, g->mis_ev0, g->mis_ev1));
    m.device_ms = ms;
    m.kernel_ms = (c.t_end > c.t_start) ? (float)((c.t_end - c.t_start) * 1e-6) : 0.f;
    g->mis_pending = false;
  }
  if (st) *st = g->mis_last;
  if (g->mis_last.error & ERR_BARRIER_TIMEOUT) return fail(PBG_ERR_TIMEOUT, "MIS: a wait for a neighbour's decision ran out");
  if (g->mis_last.error) return fail(PBG_ERR_STATE, "MIS: device error word set");
  return PBG_OK;
}

// Trace of the last MIS (one entry, the pass): the vertices walked and its
// device time.
int mis_read_trace(pbg_graph* g, pbg_level_trace* out, uint32_t cap, uint32_t* count) {
  int rc = mis_read_stats(g, nullptr);
  if (rc && rc != PBG_ERR_TIMEOUT && rc != PBG_ERR_STATE) return rc;
  if (!g->mis_ctrl || !g->mis_ran) return fail(PBG_ERR_STATE, "no MIS has run on this graph");
  BfsCtrl* c = new BfsCtrl;
  cudaError_t e = cudaMemcpy(c, g->mis_ctrl, sizeof(BfsCtrl), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    delete c;
    return cuda_fail(e, "trace copy");
  }
  const uint32_t k = std::min(std::min<uint32_t>(c->levels, PBG_TRACE_LEVELS), cap);
  for (uint32_t r = 0; r < k; r++) {
    out[r].level = r;
    out[r].bottom_up = 0;
    out[r].frontier = c->t_nf[r];
    out[r].frontier_degree = 0;
    out[r].ms = (c->t_ns[r + 1] - c->t_ns[r]) * 1e-6;
  }
  if (count) *count = k;
  delete c;
  return PBG_OK;
}

}  // namespace pbg

using namespace pbg;

extern "C" int pbg_mis_device(pbg_graph* g, uint8_t* d_flags, void* stream) {
  if (!g) return fail(PBG_ERR_ARG, "graph is NULL");
  if (!d_flags) return fail(PBG_ERR_ARG, "d_flags is NULL");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int rc = mis_launch(g, d_flags, s);
  if (rc) return rc;
  g->mis_ran = true;
  return PBG_OK;
}

extern "C" int pbg_mis(pbg_graph* g, uint8_t* flags_out, pbg_mis_stats* st) {
  if (!g) return fail(PBG_ERR_ARG, "graph is NULL");
  if (!flags_out) return fail(PBG_ERR_ARG, "flags_out is NULL");
  if (!g->mis_flags) {
    cudaError_t e = cudaMalloc(&g->mis_flags, (size_t)g->n + 16);
    if (e != cudaSuccess) {
      g->mis_flags = nullptr;
      return cuda_fail(e, "MIS flags");
    }
  }
  int rc = mis_launch(g, g->mis_flags, g->stream);
  if (rc) return rc;
  g->mis_ran = true;
  const HostCopy out{flags_out, g->mis_flags, g->n};
  rc = copy_out(&out, 1, g->stream);
  if (rc) return rc;
  pbg_mis_stats tmp;
  return mis_read_stats(g, st ? st : &tmp);
}

extern "C" int pbg_mis_stats_get(pbg_graph* g, pbg_mis_stats* st) {
  if (!g || !st) return fail(PBG_ERR_ARG, "NULL argument");
  return mis_read_stats(g, st);
}

extern "C" int pbg_mis_trace(pbg_graph* g, pbg_level_trace* out, uint32_t cap, uint32_t* count) {
  if (!g || (!out && cap)) return fail(PBG_ERR_ARG, "NULL argument");
  return mis_read_trace(g, out, cap, count);
}
