// graph.cu -- device-resident CSR graphs: upload, validation, and the seeded
// synthetic generators built on the device.
//
// CSR as graph<int,uint> (common/graph.h:104-152): offsets u32[n+1] with
// offsets[n] = m, edges u32[m].  Degrees are offsets[v+1] - offsets[v]; the
// reference's optional degrees[] (graph.h:130-133) is not stored.
//
// Generators restate testData/graphData/{rMatGraph,gridGraph,randLocalGraph}.C
// with SplitMix64's output mix as the hash (parlay::hash64 is unavailable),
// and build the symmetric CSR of common/graphUtils.h:54-94: no self loops,
// both directions, lists ascending, no duplicates.  The sorts are
// cub::DeviceRadixSort over packed keys (keys_to_graph).
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "internal.cuh"

namespace pbg {
namespace {

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

uint32_t prob_threshold(double p) {
  double t = p * 2147483648.0 + 0.5;
  if (t < 0) t = 0;
  if (t > 4294967295.0) t = 4294967295.0;
  return (uint32_t)t;
}

uint32_t ceil_log2(uint64_t x) {
  uint32_t r = 0;
  while ((1ull << r) < x) r++;
  return r;
}

// What is found about a new graph (the handle's `found` words).
struct Found {
  unsigned bad;         // FOUND_* bits
  unsigned max_degree;  // the largest degree
  unsigned asym;        // k_symmetric's bits
  unsigned pad;
  unsigned long long down, up;  // k_symmetric's edge counts
};
enum : unsigned { FOUND_ORDER = 1u, FOUND_ENDS = 2u, FOUND_TARGET = 4u };

// Validation (offsets[0] = 0, non-decreasing, offsets[n] = m, edges < n), the
// largest degree, and the bitmap of vertices that can never be reached or
// scanned: degree-0 vertices of a symmetric graph, and the padding bits past
// n.  One pass over each array: a lane per vertex, whose warp's ballot is the
// bitmap word, and 16 bytes of ids a load.  2^24 vertices, 520.8 M edges: 0.98
// ms in two kernels with 4-byte loads and a thread per bitmap word, 0.34 ms
// now (6.4 TB/s).
__global__ void k_validate(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edg, uint32_t n,
                           uint64_t m, uint32_t nwords, int symmetric, uint32_t* __restrict__ iso,
                           Found* __restrict__ found) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  uint32_t md = 0, err = 0;
  for (uint64_t v = tid; v < 32ull * nwords; v += nth) {  // whole warps
    bool dead = true;
    if (v < n) {
      const uint32_t b = off[v], e = off[v + 1];
      if (b > e)
        err |= FOUND_ORDER;
      else
        md = max(md, e - b);
      dead = symmetric && b == e;
    }
    const uint32_t word = __ballot_sync(FULL, dead);
    if ((threadIdx.x & 31) == 0) iso[v / 32] = word;
  }
  if (tid == 0 && (off[0] != 0 || (uint64_t)off[n] != m)) err |= FOUND_ENDS;
  const uint4* e4 = reinterpret_cast<const uint4*>(edg);  // the array starts on 16 bytes
  uint32_t top = 0;                                       // the largest id of this thread's
#pragma unroll 4
  for (uint64_t i = tid; i < m / 4; i += nth) {
    const uint4 x = __ldg(e4 + i);
    top = max(top, max(max(x.x, x.y), max(x.z, x.w)));
  }
  for (uint64_t i = m / 4 * 4 + tid; i < m; i += nth) top = max(top, edg[i]);
  if (m && top >= n) err |= FOUND_TARGET;
  md = __reduce_max_sync(FULL, md);
  err = __reduce_or_sync(FULL, err);
  if ((threadIdx.x & 31) == 0) {
    if (md) atomicMax(&found->max_degree, md);
    if (err) atomicOr(&found->bad, err);
  }
}

// The bitmap of a graph found not to be symmetric: the padding bits only.
__global__ void k_padding_bits(uint32_t n, uint32_t nwords, uint32_t* __restrict__ iso) {
  const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  const uint64_t first = (uint64_t)w * 32;
  iso[w] = first + 32 <= n ? 0u : first >= n ? 0xFFFFFFFFu : 0xFFFFFFFFu << (n - first);
}

// The generators write one key per drawn edge, smaller end first: (min << shift
// | max).  A self loop becomes `sentinel`, the key of the loop at vertex n - 1,
// which no edge has and no key exceeds, so it sorts last.
__device__ __forceinline__ uint64_t edge_key(uint32_t u, uint32_t v, uint32_t shift, uint64_t sentinel) {
  return u == v ? sentinel : ((uint64_t)min(u, v) << shift) | max(u, v);
}

// rMat draw for edge i (rMatGraph.C:53-69): start/stride keys from i and the
// seed hash, one 31-bit draw per level, top level first.  The quadrant's two
// bits come from comparisons without branches: the arms are drawn at random,
// so a warp took every one of them at every level (2^28 draws of 24 levels:
// 8.7 ms with branches, 7.5 ms without).
__global__ void k_gen_rmat(uint64_t m, uint64_t h, uint32_t logn, uint32_t ta, uint32_t tab, uint32_t tabc,
                           uint32_t shift, uint64_t sentinel, uint64_t* __restrict__ keys) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = tid; i < m; i += nth) {
    uint64_t x = mix64((2 * i) * h);
    const uint64_t st = mix64((2 * i + 1) * h);
    uint32_t u = 0, v = 0;
#pragma unroll 4
    for (uint32_t k = 0; k < logn; k++) {
      const uint32_t r = (uint32_t)(mix64(x) & 0x7FFFFFFFu);
      x += st;
      const uint32_t low = r >= tab;  // the lower half of the rows
      u = 2 * u + low;
      v = 2 * v + ((low ? r >= tabc : r >= ta) ? 1u : 0u);
    }
    keys[i] = edge_key(u, v, shift, sentinel);
  }
}

__device__ __forceinline__ uint32_t relabel(const uint32_t* perm, uint32_t x) { return perm ? perm[x] : x; }

// 3-D torus (gridGraph.C:57-72): vertex l = (i*dn + j)*dn + k, edges to the
// +1 neighbour along each axis with wraparound; optional relabelling.
__global__ void k_gen_torus(uint32_t dn, const uint32_t* __restrict__ perm, uint32_t shift, uint64_t sentinel,
                            uint64_t* __restrict__ keys) {
  const uint64_t nn = (uint64_t)dn * dn * dn;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t l = tid; l < nn; l += nth) {
    const uint64_t i = l / ((uint64_t)dn * dn), j = (l / dn) % dn, k = l % dn;
    uint64_t nb[3] = {(((i + 1) % dn) * dn + j) * dn + k, (i * dn + (j + 1) % dn) * dn + k,
                      (i * dn + j) * dn + (k + 1) % dn};
    const uint32_t u = relabel(perm, (uint32_t)l);
    for (int d = 0; d < 3; d++) keys[3 * l + d] = edge_key(u, relabel(perm, (uint32_t)nb[d]), shift, sentinel);
  }
}

// Random-local: `deg` out-edges of vertex i at (i + off) mod n, off uniform in
// [-w, w], redrawn (by rehashing) while it lands on i (randLocalGraph.C:46-57).
__global__ void k_gen_randlocal(uint32_t n, uint32_t deg, uint32_t w, uint64_t hs, uint32_t shift,
                                uint64_t sentinel, uint64_t* __restrict__ keys) {
  const uint64_t total = (uint64_t)n * deg;
  const uint64_t span = 2 * (uint64_t)w + 1;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = tid; t < total; t += nth) {
    const uint64_t i = t / deg;
    uint64_t x = mix64(hs + t);
    uint32_t j = 0;
    for (;;) {
      const int64_t offv = (int64_t)(x % span) - (int64_t)w;
      int64_t q = ((int64_t)i + offv) % (int64_t)n;
      if (q < 0) q += n;
      j = (uint32_t)q;
      if (j != i) break;
      x = mix64(x);
    }
    keys[t] = edge_key((uint32_t)i, j, shift, sentinel);
  }
}

__global__ void k_perm_keys(uint32_t n, uint64_t hs, uint64_t* __restrict__ keys) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = tid; i < n; i += nth) keys[i] = (mix64(hs + i) & 0xFFFFFFFF00000000ull) | i;
}

__global__ void k_perm_scatter(uint32_t n, const uint64_t* __restrict__ sorted, uint32_t* __restrict__ new_id) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t p = tid; p < n; p += nth) new_id[(uint32_t)(sorted[p] & 0xFFFFFFFFu)] = (uint32_t)p;
}

// Symmetry test: every list ascending, and every edge (u, v) has (v, u).
// found->asym: bit 1 = an unsorted list, bit 2 = a missing reverse edge;
// down / up = distinct edges from a heavier to a lighter vertex / from a
// lighter to a heavier one, in the total order (degree, id).  Only the
// heavy-to-light edges are looked up, in the lighter end's (shorter) list.
// When all of them have their reverse, reversal maps them one to one into the
// light-to-heavy edges, so equal counts mean that those have theirs too.
//
// A warp takes SYM_SEG consecutive edges, 32 at a time: a hub's list is
// spread over the grid, the ids are read coalesced, and each lane finds its
// edge's source by binary search between the segment's first and last
// sources (a window of the offsets that stays in L1).  Bound by the L1
// requests of the lookups (two offsets and a few probes an edge, for half
// the edges).  One thread a vertex, searching for every edge, left the hubs'
// lists to single threads: rMat 2^20 (20.5 M edges) 78.3 ms, now 0.37 ms.
constexpr uint32_t SYM_SEG = 1024;

// Last vertex v in [lo, hi] with off[v] <= j (off[lo] <= j).
__device__ __forceinline__ uint32_t edge_source(const uint32_t* __restrict__ off, uint32_t lo, uint32_t hi,
                                                uint64_t j) {
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo + 1) / 2;
    if (__ldg(off + mid) <= j)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

__global__ void k_symmetric(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edg, uint32_t n,
                            uint64_t m, Found* __restrict__ found) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t segs = (m + SYM_SEG - 1) / SYM_SEG;
  uint32_t down = 0, up = 0;  // at most 2^32 edges over all lanes of the grid
  unsigned err = 0;
  for (uint64_t s = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < segs; s += nw) {
    const uint64_t j0 = s * SYM_SEG, j1 = min(m, j0 + SYM_SEG);
    uint32_t u = 0;
    if (lane < 2) u = edge_source(off, 0, n - 1, lane ? j1 - 1 : j0);
    const uint32_t last = __shfl_sync(FULL, u, 1);
    u = __shfl_sync(FULL, u, 0);
    for (uint64_t j = j0 + lane; j < j1; j += 32) {
      u = edge_source(off, u, last, j);
      const uint32_t v = __ldg(edg + j), b = __ldg(off + u), e = __ldg(off + u + 1);
      if (j > b) {
        const uint32_t w = __ldg(edg + j - 1);
        if (w > v) err |= 1u;
        if (w == v) continue;  // a duplicate: counted once
      }
      if (v == u) continue;  // its own reverse
      uint32_t lo = __ldg(off + v), hi = __ldg(off + v + 1);
      const uint32_t du = e - b, dv = hi - lo, end = hi;
      if (du < dv || (du == dv && u < v)) {
        up++;
        continue;
      }
      down++;
      while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(edg + mid) < u)
          lo = mid + 1;
        else
          hi = mid;
      }
      if (lo == end || __ldg(edg + lo) != u) err |= 2u;
    }
    __syncwarp();
  }
  down = __reduce_add_sync(FULL, down);
  up = __reduce_add_sync(FULL, up);
  err = __reduce_or_sync(FULL, err);
  if (lane == 0) {
    if (down) atomicAdd(&found->down, (unsigned long long)down);
    if (up) atomicAdd(&found->up, (unsigned long long)up);
    if (err) atomicOr(&found->asym, err);
  }
}

// first[v] = index of the first of the `cnt` sorted keys whose vertex (the
// key's upper end when HIGH, else its lower bits) is v or above, for v in
// [0, n].  Key i (i = cnt: the end) fills the vertices after its
// predecessor's up to its own; the whole warp calls, and fills a long run of
// vertices without keys together.  Returns key i's vertex.
template <bool HIGH>
__device__ __forceinline__ uint32_t fill_first(const uint64_t* __restrict__ keys, uint64_t cnt, uint32_t n,
                                               uint32_t shift, uint64_t i, uint32_t* __restrict__ first) {
  constexpr uint32_t FULL = 0xFFFFFFFFu, RUN = 32;
  const uint64_t vmask = (1ull << shift) - 1;
  auto vertex = [&](uint64_t k) { return (uint32_t)(HIGH ? k >> shift : k & vmask); };
  uint32_t v = n, lo = 1, hi = 0;  // nothing to fill past the end
  if (i <= cnt) {
    if (i < cnt) v = vertex(keys[i]);
    lo = i ? vertex(keys[i - 1]) + 1 : 0;
    hi = v + 1;
  }
  const bool longrun = hi > lo && hi - lo > RUN;
  if (!longrun)
    for (uint32_t w = lo; w < hi; w++) first[w] = (uint32_t)i;
  for (unsigned mm = __ballot_sync(FULL, longrun); mm; mm &= mm - 1) {
    const int l = __ffs(mm) - 1;
    const uint32_t b = __shfl_sync(FULL, lo, l), e = __shfl_sync(FULL, hi, l), x = __shfl_sync(FULL, (uint32_t)i, l);
    for (uint32_t w = b + (threadIdx.x & 31); w < e; w += 32) first[w] = x;
  }
  return v;
}

// Keys in (lower end, upper end) order: where each lower end's begin, and a
// copy of the keys for the second sort.
__global__ void k_first_lower(const uint64_t* __restrict__ keys, uint64_t cnt, uint32_t n, uint32_t shift,
                              uint32_t* __restrict__ first, uint64_t* __restrict__ copy) {
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; b <= cnt; b += nth) {
    const uint64_t i = b + (threadIdx.x & 31);
    fill_first<true>(keys, cnt, n, shift, i, first);
    if (i < cnt) copy[i] = keys[i];
  }
}

// Keys in (upper end, lower end) order: where each upper end's begin, and
// the first part of every list, the neighbours below the vertex.  The list
// of v starts at below[v] + above[v], so key i's lower end goes to
// i - below[v] past that, i + above[v].
__global__ void k_lists_below(const uint64_t* __restrict__ keys, uint64_t cnt, uint32_t n, uint32_t shift,
                              const uint32_t* __restrict__ above, uint32_t* __restrict__ below,
                              uint32_t* __restrict__ edg) {
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; b <= cnt; b += nth) {
    const uint64_t i = b + (threadIdx.x & 31);
    const uint32_t v = fill_first<false>(keys, cnt, n, shift, i, below);
    if (i < cnt) edg[i + above[v]] = (uint32_t)(keys[i] >> shift);
  }
}

// The rest of every list, the neighbours above the vertex (keys in (lower,
// upper) order): past the list's below[v + 1] - below[v] first entries, key
// i's upper end goes to i + below[v + 1].  Also the offsets.
__global__ void k_lists_above(const uint64_t* __restrict__ keys, uint64_t cnt, uint32_t n, uint32_t shift,
                              const uint32_t* __restrict__ above, const uint32_t* __restrict__ below,
                              uint32_t* __restrict__ off, uint32_t* __restrict__ edg) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t vmask = (1ull << shift) - 1;
  for (uint64_t v = tid; v <= n; v += nth) off[v] = above[v] + below[v];
  for (uint64_t i = tid; i < cnt; i += nth) {
    const uint64_t k = keys[i];
    edg[i + below[(k >> shift) + 1]] = (uint32_t)(k & vmask);
  }
}

}  // namespace

int grid_for(uint64_t work, int num_sms) {
  uint64_t g = (work + 255) / 256;
  uint64_t cap = (uint64_t)num_sms * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

int new_handle(uint32_t n, uint64_t m, uint32_t flags, pbg_graph** out) {
  if (!out) return fail(PBG_ERR_ARG, "out is NULL");
  if (n == 0) return fail(PBG_ERR_ARG, "graph has no vertices");
  if (n > PBG_MAX_VERTICES)
    return fail(PBG_ERR_ARG, "n must be below 2^31: vertex ids are int (bench/BFS.h:5)");
  if (m > 0xFFFFFFFFull) return fail(PBG_ERR_ARG, "m must fit in 32 bits (uint offsets)");
  pbg_graph* g = new pbg_graph();
  g->n = n;
  g->m = m;
  g->flags = flags;
  g->nwords = (uint32_t)((((uint64_t)n + 31) / 32 + 31) / 32 * 32);
  cudaError_t e = cudaGetDevice(&g->device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g->num_sms, cudaDevAttrMultiProcessorCount, g->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking);
  // one allocation: offsets, edges, bitmap, the words that validation fills
  // (an allocation costs a third of a millisecond).  4 ids of padding after
  // the edges: 16-byte loads of aligned 4-edge groups may cover up to 3 ids
  // past the last list
  auto up = [](uint64_t bytes) { return (bytes + 255) & ~255ull; };
  const uint64_t ob = up(sizeof(uint32_t) * ((uint64_t)n + 1)), eb = up(sizeof(uint32_t) * (m + 4)),
                 ib = up(sizeof(uint32_t) * (uint64_t)g->nwords);
  char* mem = nullptr;
  if (e == cudaSuccess) e = cudaMalloc(&mem, ob + eb + ib + sizeof(Found));
  if (e == cudaSuccess) {
    g->d_offsets = reinterpret_cast<uint32_t*>(mem);
    g->d_edges = reinterpret_cast<uint32_t*>(mem + ob);
    g->d_iso = reinterpret_cast<uint32_t*>(mem + ob + eb);
  }
  if (e != cudaSuccess) {
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
    cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? PBG_ERR_OOM : PBG_ERR_CUDA,
                std::string("graph allocation: ") + cudaGetErrorString(e));
  }
  *out = g;
  return PBG_OK;
}

// Validates the CSR now on the device, derives the degree-0 bitmap and the
// largest degree, and decides symmetry when asked.
int finish_graph(pbg_graph* g) {
  Found* d = reinterpret_cast<Found*>(reinterpret_cast<char*>(g->d_iso) +
                                      ((sizeof(uint32_t) * (size_t)g->nwords + 255) & ~(size_t)255));
  Found f;
  const bool detect = g->flags & PBG_GRAPH_DETECT_SYMMETRIC;
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(Found), g->stream);
  if (e == cudaSuccess) {
    k_validate<<<grid_for(std::max<uint64_t>(g->m / 4, 32ull * g->nwords), g->num_sms), 256, 0, g->stream>>>(
        g->d_offsets, g->d_edges, g->n, g->m, g->nwords, detect || (g->flags & PBG_GRAPH_SYMMETRIC), g->d_iso, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&f, d, sizeof(f), cudaMemcpyDeviceToHost, g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  if (e != cudaSuccess) return cuda_fail(e, "graph validation");
  if (f.bad & FOUND_ENDS) return fail(PBG_ERR_ARG, "offsets[0] must be 0 and offsets[n] must equal m");
  if (f.bad & FOUND_ORDER) return fail(PBG_ERR_ARG, "offsets must be non-decreasing");
  if (f.bad & FOUND_TARGET) return fail(PBG_ERR_ARG, "an edge target is >= n");
  g->max_degree = f.max_degree;
  if (detect) {
    k_symmetric<<<grid_for(g->m / SYM_SEG * 32 + 1, g->num_sms), 256, 0, g->stream>>>(g->d_offsets, g->d_edges, g->n,
                                                                                       g->m, d);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&f, d, sizeof(f), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) return cuda_fail(e, "symmetry test");
    const bool sym = f.asym == 0 && f.down == f.up;
    g->flags = (g->flags & ~PBG_GRAPH_DETECT_SYMMETRIC) | (sym ? PBG_GRAPH_SYMMETRIC : 0u);
    if (!(g->flags & PBG_GRAPH_SYMMETRIC)) {
      k_padding_bits<<<(g->nwords + 255) / 256, 256, 0, g->stream>>>(g->n, g->nwords, g->d_iso);
      PBG_CUDA(cudaGetLastError());
      PBG_CUDA(cudaStreamSynchronize(g->stream));
    }
  }
  return PBG_OK;
}

namespace {

struct DevBuf {
  void* p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
  cudaError_t alloc(size_t bytes) { return cudaMalloc(&p, bytes ? bytes : 1); }
  template <class T>
  T* as() {
    return static_cast<T*>(p);
  }
};

// The symmetric CSR of the drawn edges: each edge once (keys, smaller end
// first), sorted by (lower, upper) end with duplicates dropped, then stably
// by the upper end alone, which gives every vertex's neighbours below it;
// those above it are the first order's.  Half the keys of a sort of both
// directions, and the second sort has the upper end's bits only; all scratch
// is one allocation of two key arrays (keys is the first; the list array, as
// long as one, is the second sort's third), not four of both directions, since
// mapping and unmapping memory costs milliseconds a GB.  rMat 2^24 with 2^28
// draws: 76 ms before, 47 ms now (24 ms of it the sorts' nine passes); 2^12 with 2^16
// draws, where the allocations count: 2.3 ms before, 1.4 ms now.
struct KeyScratch {
  DevBuf buf;
  uint64_t* keys = nullptr;  // the generator's output: nkeys entries
  uint64_t* other = nullptr;
  uint32_t* above = nullptr;  // n + 1 entries each
  uint32_t* below = nullptr;
  unsigned long long* count = nullptr;
  void* tmp = nullptr;
  size_t tmp_bytes = 0;
};

int key_scratch(uint64_t nkeys, uint32_t n, uint32_t shift, KeyScratch* ks) {
  size_t t1 = 0, t2 = 0, t3 = 0;
  cub::DoubleBuffer<uint64_t> db;
  uint64_t *in = nullptr, *out = nullptr;
  unsigned long long* cnt = nullptr;
  PBG_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, t1, db, nkeys, 0, (int)(2 * shift)));
  PBG_CUDA(cub::DeviceSelect::Unique(nullptr, t2, in, out, cnt, nkeys));
  PBG_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, t3, db, nkeys, 0, (int)shift));
  ks->tmp_bytes = std::max(t1, std::max(t2, t3));
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t kb = up(sizeof(uint64_t) * nkeys), ob = up(sizeof(uint32_t) * ((size_t)n + 1));
  if (ks->buf.alloc(2 * kb + 2 * ob + 256 + ks->tmp_bytes) != cudaSuccess) {
    cudaGetLastError();
    return fail(PBG_ERR_OOM, "generator: key buffer allocation failed");
  }
  char* p = ks->buf.as<char>();
  ks->keys = reinterpret_cast<uint64_t*>(p);
  ks->other = reinterpret_cast<uint64_t*>(p + kb);
  ks->above = reinterpret_cast<uint32_t*>(p + 2 * kb);
  ks->below = reinterpret_cast<uint32_t*>(p + 2 * kb + ob);
  ks->count = reinterpret_cast<unsigned long long*>(p + 2 * kb + 2 * ob);
  ks->tmp = p + 2 * kb + 2 * ob + 256;
  return PBG_OK;
}

int keys_to_graph(KeyScratch& ks, uint64_t nkeys, uint32_t n, uint32_t shift, uint64_t sentinel, pbg_graph** out,
                  cudaStream_t s, int num_sms) {
  cub::DoubleBuffer<uint64_t> db(ks.keys, ks.other);
  size_t tb = ks.tmp_bytes;
  PBG_CUDA(cub::DeviceRadixSort::SortKeys(ks.tmp, tb, db, nkeys, 0, (int)(2 * shift), s));
  uint64_t* uniq = db.Alternate();  // in (lower, upper) order
  tb = ks.tmp_bytes;
  PBG_CUDA(cudaMemsetAsync(ks.count, 0, sizeof(*ks.count), s));
  PBG_CUDA(cub::DeviceSelect::Unique(ks.tmp, tb, db.Current(), uniq, ks.count, nkeys, s));
  unsigned long long cnt = 0;
  PBG_CUDA(cudaMemcpyAsync(&cnt, ks.count, sizeof(cnt), cudaMemcpyDeviceToHost, s));
  PBG_CUDA(cudaStreamSynchronize(s));
  if (cnt > 0) {
    uint64_t last = 0;
    PBG_CUDA(cudaMemcpyAsync(&last, uniq + (cnt - 1), sizeof(last), cudaMemcpyDeviceToHost, s));
    PBG_CUDA(cudaStreamSynchronize(s));
    if (last == sentinel) cnt--;
  }
  pbg_graph* g = nullptr;
  int rc = new_handle(n, 2 * cnt, PBG_GRAPH_SYMMETRIC, &g);
  if (rc) return rc;
  auto build = [&]() -> int {
    uint64_t* upper = db.Current();  // its keys are done with: in (upper, lower) order from here on
    uint64_t* lists = reinterpret_cast<uint64_t*>(g->d_edges);  // 2 * cnt ids, not written yet
    const bool odd = ((shift + 7) / 8) & 1;  // passes: the second sort ends in `upper` either way
    cub::DoubleBuffer<uint64_t> d2(odd ? lists : upper, odd ? upper : lists);
    k_first_lower<<<grid_for(cnt + 1, num_sms), 256, 0, s>>>(uniq, cnt, n, shift, ks.above, d2.Current());
    PBG_CUDA(cudaGetLastError());
    size_t t = ks.tmp_bytes;
    if (cnt) PBG_CUDA(cub::DeviceRadixSort::SortKeys(ks.tmp, t, d2, cnt, 0, (int)shift, s));
    if (cnt && d2.Current() != upper)  // a small input's sort may take other passes
      PBG_CUDA(cudaMemcpyAsync(upper, d2.Current(), sizeof(uint64_t) * cnt, cudaMemcpyDeviceToDevice, s));
    k_lists_below<<<grid_for(cnt + 1, num_sms), 256, 0, s>>>(upper, cnt, n, shift, ks.above, ks.below, g->d_edges);
    PBG_CUDA(cudaGetLastError());
    k_lists_above<<<grid_for(std::max<uint64_t>(cnt, n), num_sms), 256, 0, s>>>(uniq, cnt, n, shift, ks.above,
                                                                               ks.below, g->d_offsets, g->d_edges);
    PBG_CUDA(cudaGetLastError());
    PBG_CUDA(cudaStreamSynchronize(s));
    return finish_graph(g);
  };
  rc = build();
  if (rc) {
    pbg_graph_free(g);
    return rc;
  }
  *out = g;
  return PBG_OK;
}

}  // namespace
}  // namespace pbg

using namespace pbg;

extern "C" int pbg_graph_upload(const uint32_t* offsets, const uint32_t* edges, uint32_t n, uint64_t m,
                                uint32_t flags, pbg_graph** out) {
  if (!offsets || (m && !edges)) return fail(PBG_ERR_ARG, "offsets/edges is NULL");
  if (!out) return fail(PBG_ERR_ARG, "out is NULL");
  pbg_graph* g = nullptr;
  int rc = new_handle(n, m, flags, &g);
  if (rc) return rc;
  cudaError_t e = cudaMemcpyAsync(g->d_offsets, offsets, sizeof(uint32_t) * ((uint64_t)n + 1),
                                  cudaMemcpyHostToDevice, g->stream);
  if (e == cudaSuccess && m)
    e = cudaMemcpyAsync(g->d_edges, edges, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, g->stream);
  if (e != cudaSuccess) {
    pbg_graph_free(g);
    return cuda_fail(e, "graph upload");
  }
  rc = finish_graph(g);
  if (rc) {
    pbg_graph_free(g);
    return rc;
  }
  *out = g;
  return PBG_OK;
}

extern "C" int pbg_graph_upload_device(const uint32_t* d_offsets, const uint32_t* d_edges, uint32_t n, uint64_t m,
                                       uint32_t flags, pbg_graph** out) {
  if (!d_offsets || (m && !d_edges)) return fail(PBG_ERR_ARG, "offsets/edges is NULL");
  if (!out) return fail(PBG_ERR_ARG, "out is NULL");
  pbg_graph* g = nullptr;
  int rc = new_handle(n, m, flags, &g);
  if (rc) return rc;
  // on the default stream: after whatever fills the arrays there or on a
  // stream that it waits for (the handle's own stream waits for none)
  cudaError_t e = cudaMemcpyAsync(g->d_offsets, d_offsets, sizeof(uint32_t) * ((uint64_t)n + 1),
                                  cudaMemcpyDeviceToDevice, cudaStreamLegacy);
  if (e == cudaSuccess && m)
    e = cudaMemcpyAsync(g->d_edges, d_edges, sizeof(uint32_t) * m, cudaMemcpyDeviceToDevice, cudaStreamLegacy);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
  if (e != cudaSuccess) {
    pbg_graph_free(g);
    return cuda_fail(e, "graph upload");
  }
  rc = finish_graph(g);
  if (rc) {
    pbg_graph_free(g);
    return rc;
  }
  *out = g;
  return PBG_OK;
}

extern "C" int pbg_graph_generate(const pbg_gen_params* p, pbg_graph** out) {
  if (!p || !out) return fail(PBG_ERR_ARG, "NULL argument");
  uint64_t n = 0, nkeys = 0;
  if (p->kind == PBG_GEN_RMAT) {
    if (p->logn < 1 || p->logn > 30) return fail(PBG_ERR_ARG, "rmat: logn must be in [1, 30]");
    if (!(p->a >= 0 && p->b >= 0 && p->c >= 0 && p->a + p->b + p->c <= 1.0))
      return fail(PBG_ERR_ARG, "rmat: a + b + c must be <= 1 (rMatGraph.C:44-47)");
    n = 1ull << p->logn;
    nkeys = p->samples;
  } else if (p->kind == PBG_GEN_TORUS3D) {
    if (p->dn < 1) return fail(PBG_ERR_ARG, "torus: dn must be >= 1");
    n = (uint64_t)p->dn * p->dn * p->dn;
    nkeys = 3 * n;
  } else if (p->kind == PBG_GEN_RANDLOCAL) {
    if (p->n < 2) return fail(PBG_ERR_ARG, "randlocal: n must be >= 2");
    if (p->window < 1) return fail(PBG_ERR_ARG, "randlocal: window must be >= 1");
    n = p->n;
    nkeys = (uint64_t)p->n * p->degree;
  } else {
    return fail(PBG_ERR_ARG, "unknown generator kind");
  }
  if (n > PBG_MAX_VERTICES)
    return fail(PBG_ERR_ARG, "n must be below 2^31: vertex ids are int (bench/BFS.h:5)");
  const uint32_t shift = std::max<uint32_t>(1, ceil_log2(n));
  const uint64_t sentinel = ((n - 1) << shift) | (n - 1);

  int dev = 0, num_sms = 0;
  PBG_CUDA(cudaGetDevice(&dev));
  PBG_CUDA(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
  cudaStream_t s = nullptr;
  PBG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } sg{s};

  DevBuf perm;
  KeyScratch ks;
  const int rc = key_scratch(nkeys, (uint32_t)n, shift, &ks);
  if (rc) return rc;
  const int grid = grid_for(nkeys + 1, num_sms);
  if (p->kind == PBG_GEN_RMAT) {
    const uint64_t h = mix64(p->seed);
    k_gen_rmat<<<grid, 256, 0, s>>>(p->samples, h, p->logn, prob_threshold(p->a), prob_threshold(p->a + p->b),
                                    prob_threshold(p->a + p->b + p->c), shift, sentinel, ks.keys);
  } else if (p->kind == PBG_GEN_TORUS3D) {
    if (p->permute) {
      DevBuf pk, ps, tmp;
      PBG_CUDA(pk.alloc(sizeof(uint64_t) * n));
      PBG_CUDA(ps.alloc(sizeof(uint64_t) * n));
      PBG_CUDA(perm.alloc(sizeof(uint32_t) * n));
      k_perm_keys<<<grid_for(n, num_sms), 256, 0, s>>>((uint32_t)n, mix64(p->perm_seed), pk.as<uint64_t>());
      size_t tb = 0;
      PBG_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tb, pk.as<uint64_t>(), ps.as<uint64_t>(), n, 0, 64, s));
      PBG_CUDA(tmp.alloc(tb));
      PBG_CUDA(cub::DeviceRadixSort::SortKeys(tmp.p, tb, pk.as<uint64_t>(), ps.as<uint64_t>(), n, 0, 64, s));
      k_perm_scatter<<<grid_for(n, num_sms), 256, 0, s>>>((uint32_t)n, ps.as<uint64_t>(), perm.as<uint32_t>());
      PBG_CUDA(cudaGetLastError());
      PBG_CUDA(cudaStreamSynchronize(s));
    }
    k_gen_torus<<<grid, 256, 0, s>>>(p->dn, perm.as<uint32_t>(), shift, sentinel, ks.keys);
  } else {
    k_gen_randlocal<<<grid, 256, 0, s>>>(p->n, p->degree, p->window, mix64(p->seed), shift, sentinel,
                                         ks.keys);
  }
  PBG_CUDA(cudaGetLastError());
  return keys_to_graph(ks, nkeys, (uint32_t)n, shift, sentinel, out, s, num_sms);
}

extern "C" int pbg_graph_info(const pbg_graph* g, uint32_t* n, uint64_t* m, const uint32_t** d_offsets,
                              const uint32_t** d_edges) {
  if (!g) return fail(PBG_ERR_ARG, "graph is NULL");
  if (n) *n = g->n;
  if (m) *m = g->m;
  if (d_offsets) *d_offsets = g->d_offsets;
  if (d_edges) *d_edges = g->d_edges;
  return PBG_OK;
}

extern "C" int pbg_graph_flags(const pbg_graph* g, uint32_t* flags) {
  if (!g || !flags) return fail(PBG_ERR_ARG, "NULL argument");
  *flags = g->flags;
  return PBG_OK;
}

extern "C" int pbg_graph_download(const pbg_graph* g, uint32_t* offsets, uint32_t* edges) {
  if (!g || !offsets) return fail(PBG_ERR_ARG, "NULL argument");
  PBG_CUDA(cudaMemcpyAsync(offsets, g->d_offsets, sizeof(uint32_t) * ((uint64_t)g->n + 1), cudaMemcpyDeviceToHost,
                           g->stream));
  if (g->m && edges)
    PBG_CUDA(cudaMemcpyAsync(edges, g->d_edges, sizeof(uint32_t) * g->m, cudaMemcpyDeviceToHost, g->stream));
  PBG_CUDA(cudaStreamSynchronize(g->stream));
  return PBG_OK;
}

extern "C" int pbg_graph_free(pbg_graph* g) {
  if (!g) return PBG_OK;
  if (g->stream) cudaStreamSynchronize(g->stream);
  bfs_free_workspace(g);
  pbg_msbfs_free(g->ms_ws);
  pbg_batch_free(g->ms_batch);
  if (g->ws.ev0) cudaEventDestroy(g->ws.ev0);
  if (g->ws.ev1) cudaEventDestroy(g->ws.ev1);
  cudaFree(g->d_offsets);  // and with it the edges and the bitmap (new_handle)
  cudaFree(g->d_pull_chunks);
  cudaFree(g->mis_flags);
  cudaFree(g->mis_ctrl);
  cudaFree(g->check_buf);
  if (g->mis_ev0) cudaEventDestroy(g->mis_ev0);
  if (g->mis_ev1) cudaEventDestroy(g->mis_ev1);
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
  return PBG_OK;
}
