// The maximal independent set's launch with its control block in the test's
// hands: mis.cu compiled into a library of its own, beside a hand-made graph
// handle.  Only what the kernel can meet is set up (a preset error word, an
// old call's progress words); every wait in it ends.
#include "../../pbbsbench_b200/csrc/mis.cu"

namespace pbg {
int fail(int code, const std::string&) { return code; }
int cuda_fail(cudaError_t, const char*) { return PBG_ERR_CUDA; }
int grid_for(uint64_t work, int num_sms) { return (int)std::max<uint64_t>(1, std::min<uint64_t>((work + 255) / 256, (uint64_t)num_sms * 16)); }
int copy_out(const HostCopy*, int, cudaStream_t) { return PBG_ERR_STATE; }
}  // namespace pbg

namespace {
int make(pbg_graph* g, const uint32_t* d_off, const uint32_t* d_edg, uint32_t n, uint64_t m) {
  g->n = n;
  g->m = m;
  g->d_offsets = const_cast<uint32_t*>(d_off);
  g->d_edges = const_cast<uint32_t*>(d_edg);
  if (cudaDeviceGetAttribute(&g->num_sms, cudaDevAttrMultiProcessorCount, 0) != cudaSuccess) return PBG_ERR_CUDA;
  return PBG_OK;
}
}  // namespace

// One pass with the error word set before it starts: the number of vertices
// left undecided into *left.  Returns the device error word, or -1.
extern "C" int mis_with_error_set(const uint32_t* d_off, const uint32_t* d_edg, uint32_t n, uint64_t m,
                                  uint8_t* d_flags, unsigned bit) {
  pbg_graph g;
  int grid = 0;
  if (make(&g, d_off, d_edg, n, m) || pbg::mis_grid(g.num_sms, &grid)) return -1;
  pbg::BfsCtrl* c = nullptr;
  const size_t bytes = sizeof(pbg::BfsCtrl) + sizeof(uint32_t) * (size_t)grid * (pbg::MIS_BLOCK / 32);
  if (cudaMalloc(&c, bytes) != cudaSuccess || cudaMemset(c, 0, bytes) != cudaSuccess) return -1;
  cudaMemcpy(&c->sync.error, &bit, sizeof(bit), cudaMemcpyHostToDevice);
  cudaMemset(d_flags, 0, n);
  pbg::MisArgs a{d_off, d_edg, d_flags, c, reinterpret_cast<uint32_t*>(c + 1), n, 1u};
  const int blocks = (int)std::min<uint64_t>((uint64_t)grid, ((uint64_t)n + 31) / 32);
  void* params[] = {&a};
  unsigned word = 0;
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)pbg::mis_one_pass<pbg::MIS_BLOCK>, dim3(blocks),
                                              dim3(pbg::MIS_BLOCK), params, 0, nullptr);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(&word, &c->sync.error, sizeof(word), cudaMemcpyDeviceToHost);
  cudaFree(c);
  return e == cudaSuccess ? (int)word : -1;
}

// Two calls on one handle, the words after the control block filled with
// `stale` between them: the second call's progress words into done[0 ..
// *words).
extern "C" int mis_progress_words(const uint32_t* d_off, const uint32_t* d_edg, uint32_t n, uint64_t m,
                                  uint8_t* d_flags, int stale, uint32_t* done, uint32_t* words) {
  pbg_graph g;
  int grid = 0;
  if (make(&g, d_off, d_edg, n, m) || pbg::mis_grid(g.num_sms, &grid)) return -1;
  *words = (uint32_t)grid * (pbg::MIS_BLOCK / 32);
  int rc = pbg::mis_launch(&g, d_flags, nullptr);
  if (!rc && cudaMemset(g.mis_ctrl + 1, stale, sizeof(uint32_t) * *words) != cudaSuccess) rc = -1;
  if (!rc) rc = pbg::mis_launch(&g, d_flags, nullptr);
  if (!rc && cudaDeviceSynchronize() != cudaSuccess) rc = -1;
  if (!rc && cudaMemcpy(done, g.mis_ctrl + 1, sizeof(uint32_t) * *words, cudaMemcpyDeviceToHost) != cudaSuccess) rc = -1;
  cudaFree(g.mis_ctrl);
  if (g.mis_ev0) cudaEventDestroy(g.mis_ev0);
  if (g.mis_ev1) cudaEventDestroy(g.mis_ev1);
  return rc;
}
