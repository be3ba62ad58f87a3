// check.cu -- the BFS checker on the device.
//
// pbg_bfs_check restates checkBFS (benchmarks/breadthFirstSearch/bench/
// BFSCheck.C:39-90): levels by pointer doubling on the parent tree
// (level_number, :39-56: (0, v) for a root or an unreached vertex, else
// (1, parent); (c, p) <- (c + c[p], p[p]) until nothing changes; a vertex
// whose root has no parent gets level n), then every vertex but the start
// must have level = (minimum neighbour level) + 1, or level n with every
// neighbour at level n, and the start must be its own parent (:66-78).  The
// reference loops until a fixed point; its counts are 32-bit and wrap, so
// even a cycle in the parent array settles (its counts reach 0 after about
// 33 doublings) and the predicate then finds a failing vertex.  Here the
// counts wrap the same way and the doubling stops after MAX_ROUNDS rounds;
// one that has not settled by then fails with bad vertex n.  PBG_CHECK_EDGES
// adds the
// edge test: each parent must be a neighbour of its vertex (found during the
// same neighbour scan).  pbg_levels_check applies the same level predicate
// to uint8 level rows (255 = unreached) of batched searches.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.cuh"
#include "msbfs.cuh"

using namespace pbg;

namespace {

using dev::FULL;
constexpr uint32_t SERIAL = 64;
static_assert(SERIAL == MS_PULL_SERIAL, "list tails are the pull chunk table's pieces");
constexpr uint32_t AHEAD = 6;  // rounds enqueued per look at their words (trees of depth 32 settle in six)
constexpr uint32_t MAX_ROUNDS = 64;  // doubling rounds (a valid tree of depth d settles in log2 d + 1)

// Also records the smallest vertex whose parent is neither PBG_NONE nor a
// vertex (checked before anything else, as the oracle does).
__global__ void jump_init(const uint32_t* __restrict__ parent, uint32_t n, uint32_t* __restrict__ cnt,
                          uint32_t* __restrict__ ptr, uint32_t* bad_parent) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t p = parent[v];
    if (p != PBG_NONE && p >= n) atomicMin(bad_parent, v);
    const bool root = p == PBG_NONE || p == v || p >= n;
    cnt[v] = root ? 0u : 1u;
    ptr[v] = root ? v : p;
  }
}

// Doubling round i: changed[i] is set when any pair moves.  Does nothing once
// a round has moved none, so the host may enqueue rounds ahead and look at
// the words once: a look after every round cost as much as the rounds (rMat
// 2^20, four rounds: 0.05 ms less a check).
__global__ void jump_step(const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ ptr, uint32_t n,
                          uint32_t* __restrict__ cnt2, uint32_t* __restrict__ ptr2, unsigned* changed, uint32_t i) {
  if (i > 0 && changed[i - 1] == 0) return;
  bool moved = false;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t p = ptr[v];
    const uint32_t c = cnt[v] + cnt[p];
    const uint32_t q = ptr[p];
    cnt2[v] = c;
    ptr2[v] = q;
    moved |= (c != cnt[v] || q != p);
  }
  if (__any_sync(FULL, moved) && (threadIdx.x & 31) == 0) atomicOr(changed + i, 1u);
}

// Level of each vertex from the settled pairs (n = unreached tree).
__global__ void jump_finish(const uint32_t* __restrict__ parent, const uint32_t* __restrict__ cnt,
                            const uint32_t* __restrict__ ptr, uint32_t n, uint32_t* __restrict__ level) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    level[v] = (parent[ptr[v]] == PBG_NONE) ? n : cnt[v];
}

// Level of vertex v in row r: uint32 levels (lv32, n = unreached) or uint8
// rows (lv8, 255 = unreached, mapped to n).
struct Levels {
  const uint32_t* lv32;
  const uint8_t* lv8;
  uint32_t n;
  __device__ __forceinline__ uint32_t at(uint32_t r, uint32_t v) const {
    if (lv32) return lv32[v];
    const uint8_t x = lv8[(size_t)r * n + v];
    return x == 255 ? n : x;
  }
};

// The neighbour minimum over the tails of lists longer than SERIAL (the
// graph's pull chunk table: (vertex, first, end, degree) pieces of
// MS_PULL_CHUNK edges), one warp a piece, any warp of the grid: tmin[v]
// (initially all ones) takes the smallest level with atomicMin, tadj[v] is
// set when the piece holds v's parent.  A hub's list is then spread over the
// grid instead of walked by the one warp that holds the vertex.
__global__ void check_tails(const uint4* __restrict__ chunks, uint32_t nchunks, const uint32_t* __restrict__ edges,
                            const uint32_t* __restrict__ level, const uint32_t* __restrict__ parent,
                            uint32_t* __restrict__ tmin, uint8_t* __restrict__ tadj) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < nchunks; c += nw) {
    const uint4 ent = chunks[c];
    const uint32_t pv = parent[ent.x];
    uint32_t m = 0xFFFFFFFFu;
    bool adj = false;
#pragma unroll
    for (uint32_t k = 0; k < MS_PULL_CHUNK / 32; k++) {
      if (k * 32 + lane < ent.z - ent.y) {  // counted from ent.y: a list may end at 2^32 - 1
        const uint32_t u = edges[ent.y + k * 32 + lane];
        m = min(m, level[u]);
        adj |= (u == pv);
      }
    }
    m = __reduce_min_sync(FULL, m);
    adj = __any_sync(FULL, adj);
    if (lane == 0) {
      if (m != 0xFFFFFFFFu) atomicMin(tmin + ent.x, m);
      if (adj) tadj[ent.x] = 1;
    }
  }
}

// The predicate for 32 consecutive vertices of row r per warp: neighbour
// minimum by one lane for the first SERIAL neighbours, the rest of longer
// lists from check_tails' tmin/tadj when given (one row), else by the whole
// warp; the smallest failing (row, vertex) goes into
// *bad as (row << 32 | vertex), with the level and neighbour minimum.
__global__ void check_rows(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edges, Levels L,
                           const uint32_t* __restrict__ srcs, uint32_t rows, const uint32_t* __restrict__ parent,
                           uint32_t check_edges, unsigned long long* bad, uint32_t* bad_info,
                           const uint32_t* __restrict__ tmin, const uint8_t* __restrict__ tadj) {
  const uint32_t n = L.n;
  const int lane = threadIdx.x & 31;
  const unsigned long long tiles = (unsigned long long)rows * ((n + 31) / 32);
  const unsigned long long nw = (unsigned long long)gridDim.x * (blockDim.x >> 5);
  for (unsigned long long t = (unsigned long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tiles;
       t += nw) {
    const uint32_t r = (uint32_t)(t / ((n + 31) / 32));
    const uint32_t v = (uint32_t)(t % ((n + 31) / 32)) * 32 + lane;
    const bool active = v < n;
    const uint32_t src = srcs[r];
    uint32_t b = 0, e = 0, lv = n, pv = PBG_NONE;
    if (active) {
      b = off[v];
      e = off[v + 1];
      lv = L.at(r, v);
      if (parent) pv = parent[v];
    }
    uint32_t mn = n;
    bool padj = false;
    const uint32_t es = (e - b > SERIAL) ? b + SERIAL : e;
#pragma unroll 4
    for (uint32_t j = b; j < es; j++) {
      const uint32_t u = edges[j];
      mn = min(mn, L.at(r, u));
      padj |= (u == pv);
    }
    if (tmin && e - b > SERIAL) {
      mn = min(mn, tmin[v]);  // all ones when no tail piece saw a smaller level
      padj |= tadj[v] != 0;
    }
    unsigned big = tmin ? 0u : __ballot_sync(FULL, e - b > SERIAL);
    while (big) {
      const int l = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t bb = __shfl_sync(FULL, b, l) + SERIAL, ee = __shfl_sync(FULL, e, l);
      const uint32_t pl = __shfl_sync(FULL, pv, l);
      uint32_t m2 = n;
      bool a2 = false;
      for (uint32_t k = 0; k < ee - bb; k += 32) {  // counted from bb: a list may end at 2^32 - 1
        if (k + lane < ee - bb) {
          const uint32_t u = edges[bb + k + lane];
          m2 = min(m2, L.at(r, u));
          a2 |= (u == pl);
        }
      }
      m2 = __reduce_min_sync(FULL, m2);
      a2 = __any_sync(FULL, a2);
      if (lane == l) {
        mn = min(mn, m2);
        padj |= a2;
      }
    }
    bool ok = true;
    if (active) {
      if (v == src) {
        ok = parent ? (pv == v) : (lv == 0);
      } else {
        ok = (lv == n && mn == n) || (mn < n && lv == mn + 1);
        if (ok && check_edges && parent && pv != PBG_NONE) ok = padj;
      }
    }
    if (!ok) {
      const unsigned long long key = ((unsigned long long)r << 32) | v;
      const unsigned long long old = atomicMin(bad, key);
      if (key < old) {
        bad_info[0] = lv;
        bad_info[1] = mn;
      }
    }
  }
}

// ------------------------------------------------ many level rows at once
// check_rows reads every list once per row.  For batches of rows the levels
// are first transposed to vertex-major strips of S = 4 * W * LPV bytes, one
// byte a row, so that one gather of a neighbour's strip serves S rows and
// the byte minima run four to an instruction; the lists are then read once
// per S rows.  LPV lanes share a vertex, each with W words of the strip.
// A byte passes when its neighbour minimum is one less (want, below), with
// no smaller neighbour; list tails report those two facts as bits, so their
// pieces need no byte-wise atomic minimum.  n >= 256 is assumed: 255 in a
// strip is "unreached" and nothing else.
//
// Bound by instruction issue: the byte minima and compares (four bytes an
// instruction, several instructions each) keep the ALU pipe 67-70% busy, with
// the gathers' L2 traffic at 12-25% of its rate.  64 rows on rMat 2^20 (m = 31.4
// M): 21.2 ms a row at a time, now 0.58 ms (the transpose 0.067, tails 0.26,
// lists 0.24).

// rows [0, rows) of n bytes -> strips of `stride` bytes; rows past the last
// read as 255.  One block: 128 vertices, through shared memory.
__global__ void __launch_bounds__(256) strip_rows(const uint8_t* __restrict__ lv, uint32_t n, uint32_t rows,
                                                  uint32_t stride, uint8_t* __restrict__ strips) {
  __shared__ __align__(16) uint8_t s[64][132];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (unsigned long long v0 = (unsigned long long)blockIdx.x * 128; v0 < n;
       v0 += (unsigned long long)gridDim.x * 128) {
    for (uint32_t r = wid; r < stride; r += 8) {
      const uint8_t* p = lv + (size_t)r * n + v0 + 4 * lane;
      uint32_t x = 0xFFFFFFFFu;
      if (r < rows) {
        if ((reinterpret_cast<uintptr_t>(p) & 3) == 0 && v0 + 4 * lane + 4 <= n) {
          x = *reinterpret_cast<const uint32_t*>(p);
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (v0 + 4 * lane + i < n) x = (x & ~(0xFFu << (8 * i))) | ((uint32_t)p[i] << (8 * i));
        }
      }
      *reinterpret_cast<uint32_t*>(&s[r][4 * lane]) = x;
    }
    __syncthreads();
    // thread -> (vertex, word of its strip), a strip's words on consecutive lanes
    const uint32_t words = stride / 4;
    for (uint32_t t = threadIdx.x; t < 128 * words; t += 256) {
      const uint32_t dv = t / words, w = t % words;
      if (v0 + dv < n) {
        const uint32_t x = (uint32_t)s[4 * w][dv] | ((uint32_t)s[4 * w + 1][dv] << 8) |
                           ((uint32_t)s[4 * w + 2][dv] << 16) | ((uint32_t)s[4 * w + 3][dv] << 24);
        *reinterpret_cast<uint32_t*>(strips + (v0 + dv) * stride + 4 * w) = x;
      }
    }
    __syncthreads();
  }
}

template <int W>
struct Words {
  uint32_t x[W];
};

template <int W>
__device__ __forceinline__ Words<W> ld_words(const uint8_t* p) {  // 4 * W bytes, aligned
  Words<W> r;
  if constexpr (W == 4) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
    r.x[0] = q.x;
    r.x[1] = q.y;
    r.x[2] = q.z;
    r.x[3] = q.w;
  } else {
#pragma unroll
    for (int i = 0; i < W; i++) r.x[i] = __ldg(reinterpret_cast<const uint32_t*>(p) + i);
  }
  return r;
}

// The neighbour minimum that a level byte needs: one less; 255 for 255 (and
// for 0, which only a row's source may have: callers test it).
__device__ __forceinline__ uint32_t want_of(uint32_t lv) {
  const uint32_t none = __vcmpeq4(lv, 0xFFFFFFFFu);
  return __vsub4(lv, 0x01010101u) | none;
}

// Minimum strip words over the neighbours j, j + step, ... < e (j < e).  What
// is left of the list is compared, not j + step: e may be 2^32 - 1.
template <int W, int LPV>
__device__ __forceinline__ void strip_min(const uint32_t* __restrict__ edges, const uint8_t* __restrict__ strips,
                                          uint32_t part, uint32_t j, uint32_t e, uint32_t step, Words<W>& mn) {
  constexpr uint32_t S = 4 * W * LPV;
  constexpr int K = 4;  // gathers in flight a lane
  for (;; j += K * step) {
    const uint32_t left = e - j;
    const uint32_t* p = edges + j;
    uint32_t u[K];
#pragma unroll
    for (int k = 0; k < K; k++) u[k] = (k * step < left) ? __ldg(p + k * step) : PBG_NONE;
    Words<W> x[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (u[k] != PBG_NONE) {
        x[k] = ld_words<W>(strips + (size_t)u[k] * S + part * 4 * W);
      } else {
#pragma unroll
        for (int i = 0; i < W; i++) x[k].x[i] = 0xFFFFFFFFu;
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
      for (int i = 0; i < W; i++) mn.x[i] = __vminu4(mn.x[i], x[k].x[i]);
    if (left <= K * step) break;
  }
}

// Bits of a word's byte mask (0xFF or 0x00 a byte).
__device__ __forceinline__ uint32_t byte_bits(uint32_t m) {
  return (((m & 0x08040201u) * 0x01010101u) >> 24) & 0xFu;
}

// List tails (the graph's pull chunk table), one warp a piece: bit r of
// low[v] = a neighbour of v in the piece has a smaller level in row r than
// v may have, of hit[v] = the piece has the neighbour level that v needs.
template <int W, int LPV>
__global__ void strip_tails(const uint4* __restrict__ chunks, uint32_t nchunks, const uint32_t* __restrict__ edges,
                            const uint8_t* __restrict__ strips, unsigned long long* __restrict__ low,
                            unsigned long long* __restrict__ hit) {
  constexpr uint32_t S = 4 * W * LPV;
  const uint32_t lane = threadIdx.x & 31, part = lane % LPV, grp = lane / LPV;
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < nchunks; c += nw) {
    const uint4 ent = chunks[c];
    const Words<W> lv = ld_words<W>(strips + (size_t)ent.x * S + part * 4 * W);
    Words<W> mn;
#pragma unroll
    for (int i = 0; i < W; i++) mn.x[i] = 0xFFFFFFFFu;
    if (grp < ent.z - ent.y) strip_min<W, LPV>(edges, strips, part, ent.y + grp, ent.z, 32 / LPV, mn);
    unsigned long long lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < W; i++) {
#pragma unroll
      for (int o = LPV; o < 32; o <<= 1) mn.x[i] = __vminu4(mn.x[i], __shfl_xor_sync(FULL, mn.x[i], o));
      const uint32_t want = want_of(lv.x[i]);
      const int sh = (part * W + i) * 4;
      lo |= (unsigned long long)byte_bits(__vcmpltu4(mn.x[i], want)) << sh;
      hi |= (unsigned long long)byte_bits(__vcmpeq4(mn.x[i], want)) << sh;
    }
#pragma unroll
    for (int o = 1; o < LPV; o <<= 1) {
      lo |= __shfl_xor_sync(FULL, lo, o);
      hi |= __shfl_xor_sync(FULL, hi, o);
    }
    if (lane == 0) {
      if (lo) atomicOr(low + ent.x, lo);
      if (hi) atomicOr(hit + ent.x, hi);
    }
  }
}

// The predicate for `rows` rows (first one row0) of every vertex: the first
// SERIAL neighbours here, longer lists with the tails' bits.  The smallest
// failing (row, vertex) goes into *bad.
template <int W, int LPV>
__global__ void __launch_bounds__(256) strip_check(const uint32_t* __restrict__ off,
                                                   const uint32_t* __restrict__ edges, uint32_t n,
                                                   const uint8_t* __restrict__ strips,
                                                   const uint32_t* __restrict__ srcs, uint32_t row0, uint32_t rows,
                                                   const unsigned long long* __restrict__ low,
                                                   const unsigned long long* __restrict__ hit,
                                                   unsigned long long* bad) {
  constexpr uint32_t S = 4 * W * LPV, VPB = 256 / LPV;
  const uint32_t part = threadIdx.x % LPV;
  if (blockIdx.x == 0)  // a row's source must be at level 0
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
      const uint32_t v = srcs[row0 + r];
      if (strips[(size_t)v * S + r] != 0) atomicMin(bad, ((unsigned long long)(row0 + r) << 32) | v);
    }
  for (unsigned long long vb = (unsigned long long)blockIdx.x * VPB; vb < n;
       vb += (unsigned long long)gridDim.x * VPB) {
    const unsigned long long vv = vb + threadIdx.x / LPV;
    if (vv >= n) continue;
    const uint32_t v = (uint32_t)vv;
    const uint32_t b = __ldg(off + v), e = __ldg(off + v + 1);
    const bool tail = e - b > SERIAL;
    const Words<W> lv = ld_words<W>(strips + (size_t)v * S + part * 4 * W);
    Words<W> mn;
#pragma unroll
    for (int i = 0; i < W; i++) mn.x[i] = 0xFFFFFFFFu;
    if (b < e) strip_min<W, LPV>(edges, strips, part, b, tail ? b + SERIAL : e, 1, mn);
    unsigned long long tl = 0, th = 0;
    if (tail) {
      tl = low[v];
      th = hit[v];
    }
#pragma unroll
    for (int i = 0; i < W; i++) {
      const uint32_t want = want_of(lv.x[i]);
      const int sh = (part * W + i) * 4;
      const uint32_t differ = byte_bits(__vcmpne4(mn.x[i], want) | __vcmpeq4(lv.x[i], 0u));
      uint32_t fail = differ;
      if (tail) {
        const uint32_t under = byte_bits(__vcmpltu4(mn.x[i], want) | __vcmpeq4(lv.x[i], 0u));
        fail = under | (differ & ~(uint32_t)(th >> sh)) | (uint32_t)(tl >> sh);
        fail &= 0xFu;
      }
      while (fail) {  // rare: a source, or a fault
        const uint32_t k = __ffs(fail) - 1, r = sh + k;
        fail &= fail - 1;
        if (r < rows && srcs[row0 + r] != v) {
          const unsigned long long key = ((unsigned long long)(row0 + r) << 32) | v;
          if (key < *reinterpret_cast<volatile unsigned long long*>(bad)) atomicMin(bad, key);
        }
      }
    }
  }
}

// Level and neighbour minimum of the failing (row, vertex) in *bad.
__global__ void strip_report(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edges, Levels L,
                             const unsigned long long* bad, uint32_t* info) {
  if (*bad == ~0ull) return;
  const uint32_t r = (uint32_t)(*bad >> 32), v = (uint32_t)*bad;
  __shared__ uint32_t s_mn;
  if (threadIdx.x == 0) s_mn = L.n;
  __syncthreads();
  uint32_t mn = L.n;
  for (unsigned long long j = (unsigned long long)off[v] + threadIdx.x; j < off[v + 1]; j += blockDim.x)
    mn = min(mn, L.at(r, edges[j]));
  atomicMin(&s_mn, mn);
  __syncthreads();
  if (threadIdx.x == 0) {
    info[0] = L.at(r, v);
    info[1] = s_mn;
  }
}

int grid_for(uint32_t n) { return (int)std::min<uint64_t>((n + 255) / 256, 148 * 16); }

// Level checks give scratch above this back when they are done (a parent
// check's 25 bytes a vertex stay).
constexpr size_t CHECK_KEEP = 512ull << 20;

// Scratch of at least `bytes` for a check on g, kept on the handle for later
// checks (a larger request replaces it; every check waits for its kernels
// before returning, so none is still using the old one).
int check_scratch(pbg_graph* g, size_t bytes, void** out) {
  if (g->check_bytes < bytes) {
    cudaFree(g->check_buf);
    g->check_buf = nullptr;
    g->check_bytes = 0;
    const cudaError_t e = cudaMalloc(&g->check_buf, bytes);
    if (e != cudaSuccess) {
      g->check_buf = nullptr;
      cudaGetLastError();
      return fail(e == cudaErrorMemoryAllocation ? PBG_ERR_OOM : PBG_ERR_CUDA,
                  std::string("check scratch: ") + cudaGetErrorString(e));
    }
    g->check_bytes = bytes;
  }
  *out = g->check_buf;
  return PBG_OK;
}

// The verdict words ((row << 32 | vertex) or all ones, then level and
// neighbour minimum) back on the host.
int read_verdict(const unsigned long long* d_bad, pbg_check_result* res, cudaStream_t s) {
  unsigned long long h[2];
  PBG_CUDA(cudaMemcpyAsync(h, d_bad, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  PBG_CUDA(cudaStreamSynchronize(s));
  const uint32_t* hi = reinterpret_cast<const uint32_t*>(&h[1]);
  if (h[0] == ~0ull) {
    res->bad_vertex = PBG_NONE;
    res->row = 0;
    res->level = 0;
    res->min_neighbor_level = 0;
  } else {
    res->bad_vertex = (uint32_t)(h[0] & 0xFFFFFFFFu);
    res->row = (uint32_t)(h[0] >> 32);
    res->level = hi[0];
    res->min_neighbor_level = hi[1];
  }
  return PBG_OK;
}

int run_check(pbg_graph* g, Levels L, const uint32_t* d_srcs, uint32_t rows, const uint32_t* d_parent,
              uint32_t check_edges, pbg_check_result* res, cudaStream_t s, unsigned long long* d_bad,
              const uint32_t* tmin = nullptr, const uint8_t* tadj = nullptr) {
  uint32_t* info = reinterpret_cast<uint32_t*>(d_bad + 1);
  PBG_CUDA(cudaMemsetAsync(d_bad, 0xFF, sizeof(unsigned long long), s));
  PBG_CUDA(cudaMemsetAsync(info, 0, 2 * sizeof(uint32_t), s));
  const unsigned long long tiles = (unsigned long long)rows * ((g->n + 31) / 32);
  const int blocks = (int)std::min<unsigned long long>((tiles + 7) / 8, 148ull * 8);
  check_rows<<<std::max(blocks, 1), 256, 0, s>>>(g->d_offsets, g->d_edges, L, d_srcs, rows, d_parent, check_edges,
                                                  d_bad, info, tmin, tadj);
  PBG_CUDA(cudaGetLastError());
  return read_verdict(d_bad, res, s);
}

// Checks the rows in strips of up to 64 (see strip_rows).  scratch: per
// vertex `stride` bytes of strips and 16 of tail bits.
template <int W, int LPV>
int run_strips(pbg_graph* g, const uint8_t* d_levels, const uint32_t* d_srcs, uint32_t rows, char* scratch,
               unsigned long long* d_bad, pbg_check_result* res, cudaStream_t s) {
  constexpr uint32_t S = 4 * W * LPV;
  const uint32_t n = g->n;
  unsigned long long* low = reinterpret_cast<unsigned long long*>(scratch);
  unsigned long long* hit = low + n;
  uint8_t* strips = reinterpret_cast<uint8_t*>(scratch + ((16ull * n + 255) & ~255ull));
  PBG_CUDA(cudaMemsetAsync(d_bad, 0xFF, sizeof(unsigned long long), s));
  PBG_CUDA(cudaMemsetAsync(d_bad + 1, 0, sizeof(unsigned long long), s));
  const int tb = (int)std::min<uint64_t>(((uint64_t)n + 127) / 128, (uint64_t)g->num_sms * 16);
  const int cb = (int)std::min<uint64_t>(((uint64_t)g->n_pull_chunks + 7) / 8, (uint64_t)g->num_sms * 16);
  const int vb = (int)std::min<uint64_t>(((uint64_t)n * LPV + 255) / 256, (uint64_t)g->num_sms * 32);
  for (uint32_t r0 = 0; r0 < rows; r0 += S) {
    const uint32_t k = std::min(S, rows - r0);
    strip_rows<<<tb, 256, 0, s>>>(d_levels + (size_t)r0 * n, n, k, S, strips);
    if (cb) {
      PBG_CUDA(cudaMemsetAsync(low, 0, 16ull * n, s));
      strip_tails<W, LPV><<<cb, 256, 0, s>>>(g->d_pull_chunks, g->n_pull_chunks, g->d_edges, strips, low, hit);
    }
    strip_check<W, LPV><<<vb, 256, 0, s>>>(g->d_offsets, g->d_edges, n, strips, d_srcs, r0, k, low, hit, d_bad);
    PBG_CUDA(cudaGetLastError());
  }
  strip_report<<<1, 1024, 0, s>>>(g->d_offsets, g->d_edges, Levels{nullptr, d_levels, n}, d_bad,
                                  reinterpret_cast<uint32_t*>(d_bad + 1));
  PBG_CUDA(cudaGetLastError());
  return read_verdict(d_bad, res, s);
}

}  // namespace

extern "C" int pbg_bfs_check(pbg_graph* g, uint32_t src, const uint32_t* d_parent, uint32_t flags,
                             pbg_check_result* res) {
  if (!g || !d_parent || !res) return fail(PBG_ERR_ARG, "NULL argument");
  if (src >= g->n) return fail(PBG_ERR_ARG, "source vertex out of range");
  if (flags & ~PBG_CHECK_EDGES) return fail(PBG_ERR_ARG, "unknown check flags");
  const uint32_t n = g->n;
  cudaStream_t s = g->stream;
  int rc = ms_pull_chunks(g);  // the tails of lists longer than SERIAL, in pieces
  if (rc) return rc;
  // cnt, ptr, cnt2, ptr2, level, tmin (n each), the source; the result words;
  // tadj (n bytes)
  const size_t words = 6 * (size_t)n + 1;
  const size_t head = (sizeof(uint32_t) * words + 15) & ~15ull;
  // the verdict (16 bytes), the smallest bad parent, the rounds' words
  const size_t tail = (head + 2 * sizeof(unsigned long long) + sizeof(uint32_t) * (1 + MAX_ROUNDS) + 15) & ~15ull;
  void* sp = nullptr;
  rc = check_scratch(g, tail + n, &sp);
  if (rc) return rc;
  uint32_t* cnt = static_cast<uint32_t*>(sp);
  uint32_t* ptr = cnt + n;
  uint32_t* cnt2 = ptr + n;
  uint32_t* ptr2 = cnt2 + n;
  uint32_t* level = ptr2 + n;
  uint32_t* tmin = level + n;
  uint32_t* d_src = tmin + n;
  uint8_t* tadj = static_cast<uint8_t*>(sp) + tail;
  unsigned long long* d_bad = reinterpret_cast<unsigned long long*>(static_cast<char*>(sp) + head);
  uint32_t* bad_parent = reinterpret_cast<uint32_t*>(d_bad + 2);
  unsigned* changed = bad_parent + 1;
  PBG_CUDA(cudaMemcpyAsync(d_src, &src, sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  PBG_CUDA(cudaMemsetAsync(bad_parent, 0xFF, sizeof(uint32_t), s));
  PBG_CUDA(cudaMemsetAsync(changed, 0, sizeof(unsigned) * MAX_ROUNDS, s));
  const int grid = grid_for(n);
  jump_init<<<grid, 256, 0, s>>>(d_parent, n, cnt, ptr, bad_parent);
  PBG_CUDA(cudaGetLastError());
  bool settled = false;
  for (uint32_t i0 = 0; i0 < MAX_ROUNDS && !settled; i0 += AHEAD) {
    const uint32_t rounds = std::min(AHEAD, MAX_ROUNDS - i0);
    for (uint32_t i = 0; i < rounds; i++) {
      const bool odd = i & 1;
      jump_step<<<grid, 256, 0, s>>>(odd ? cnt2 : cnt, odd ? ptr2 : ptr, n, odd ? cnt : cnt2, odd ? ptr : ptr2,
                                     changed, i0 + i);
      PBG_CUDA(cudaGetLastError());
    }
    uint32_t h[1 + MAX_ROUNDS];  // a vertex whose parent is none, then the rounds' words
    PBG_CUDA(cudaMemcpyAsync(h, bad_parent, sizeof(h), cudaMemcpyDeviceToHost, s));
    PBG_CUDA(cudaStreamSynchronize(s));
    if (h[0] != PBG_NONE) {
      *res = pbg_check_result{h[0], 0, n, n};
      return PBG_OK;
    }
    uint32_t done = 0;  // rounds that ran: up to the first that moved nothing
    while (done < rounds && !settled) settled = h[1 + i0 + done++] == 0;
    if (done & 1) {
      std::swap(cnt, cnt2);
      std::swap(ptr, ptr2);
    }
  }
  if (!settled) {  // a cycle in the parent array
    *res = pbg_check_result{n, 0, n, n};
    return PBG_OK;
  }
  jump_finish<<<grid, 256, 0, s>>>(d_parent, cnt, ptr, n, level);
  PBG_CUDA(cudaGetLastError());
  PBG_CUDA(cudaMemsetAsync(tmin, 0xFF, sizeof(uint32_t) * n, s));
  PBG_CUDA(cudaMemsetAsync(tadj, 0, n, s));
  if (g->n_pull_chunks) {
    const int tb = (int)std::min<uint64_t>(((uint64_t)g->n_pull_chunks + 7) / 8, 148 * 16);
    check_tails<<<tb, 256, 0, s>>>(g->d_pull_chunks, g->n_pull_chunks, g->d_edges, level, d_parent, tmin, tadj);
    PBG_CUDA(cudaGetLastError());
  }
  return run_check(g, Levels{level, nullptr, n}, d_src, 1, d_parent, (flags & PBG_CHECK_EDGES) ? 1u : 0u, res, s,
                   d_bad, tmin, tadj);
}

extern "C" int pbg_levels_check(pbg_graph* g, const uint32_t* srcs, uint32_t rows, const uint8_t* d_levels,
                                pbg_check_result* res) {
  if (!g || !srcs || !d_levels || !res) return fail(PBG_ERR_ARG, "NULL argument");
  if (rows < 1) return fail(PBG_ERR_ARG, "rows must be >= 1");
  for (uint32_t i = 0; i < rows; i++)
    if (srcs[i] >= g->n) return fail(PBG_ERR_ARG, "source vertex out of range");
  cudaStream_t s = g->stream;
  // the strip width: as many rows as there are, up to 64, halved while the
  // scratch does not fit in memory; graphs under 256 vertices, where 255 is
  // not the only byte for "unreached" (n is one too), keep check_rows
  const size_t head = (sizeof(uint32_t) * (size_t)rows + 15 + 2 * sizeof(unsigned long long) + 255) & ~255ull;
  uint32_t stride = g->n < 256 ? 0 : rows > 32 ? 64 : rows > 16 ? 32 : rows > 4 ? 16 : 4;
  const size_t kept = g->check_bytes;
  void* sp = nullptr;
  int rc = PBG_OK;
  if (stride) {  // check_rows needs no table of the list tails: it is what runs where that does not fit
    rc = ms_pull_chunks(g);
    if (rc && rc != PBG_ERR_OOM) return rc;
    if (rc) stride = 0;
    for (; stride; stride = stride > 16 ? stride / 2 : stride > 4 ? 4 : 0) {
      rc = check_scratch(g, head + ((16ull * g->n + 255) & ~255ull) + (size_t)stride * g->n, &sp);
      if (rc != PBG_ERR_OOM) break;
    }
    if (rc && rc != PBG_ERR_OOM) return rc;
  }
  if (!stride) {
    rc = check_scratch(g, head, &sp);
    if (rc) return rc;
  }
  unsigned long long* d_bad = static_cast<unsigned long long*>(sp);
  uint32_t* d_srcs = reinterpret_cast<uint32_t*>(d_bad + 2);
  PBG_CUDA(cudaMemcpyAsync(d_srcs, srcs, sizeof(uint32_t) * rows, cudaMemcpyHostToDevice, s));
  char* strips = static_cast<char*>(sp) + head;
  switch (stride) {
    case 64: rc = run_strips<4, 4>(g, d_levels, d_srcs, rows, strips, d_bad, res, s); break;
    case 32: rc = run_strips<4, 2>(g, d_levels, d_srcs, rows, strips, d_bad, res, s); break;
    case 16: rc = run_strips<4, 1>(g, d_levels, d_srcs, rows, strips, d_bad, res, s); break;
    case 4: rc = run_strips<1, 1>(g, d_levels, d_srcs, rows, strips, d_bad, res, s); break;
    default: rc = run_check(g, Levels{nullptr, d_levels, g->n}, d_srcs, rows, nullptr, 0, res, s, d_bad);
  }
  if (g->check_bytes > std::max(kept, CHECK_KEEP)) {  // every kernel that used it is done
    cudaFree(g->check_buf);
    g->check_buf = nullptr;
    g->check_bytes = 0;
  }
  return rc;
}
