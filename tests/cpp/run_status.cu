// Status of a run whose grid barrier gave up: what a launch leaves behind for
// the host, and what the host makes of it.  Nothing here waits for a block
// that does not come: a block that "gave up" returns, and the barrier's error
// word is set by a copy.
#include "sssp_cc.cu"

#include <cstdio>
#include <cstdlib>

#define EXPECT(cond)                                                            \
  do {                                                                          \
    if (!(cond)) {                                                              \
      std::fprintf(stderr, "line %d: expectation failed: %s\n", __LINE__, #cond); \
      std::exit(1);                                                             \
    }                                                                           \
  } while (0)

// A run whose block `leaves` stops at its last barrier.
__global__ void run_kernel(eng::ReportRef report, sygraph::detail::GridBarrier* bar, uint32_t leaves) {
  if (!sygraph::detail::grid_sync(bar)) return;
  if (blockIdx.x == leaves) return;
  eng::report_run(report, bar, 1, 2, 3, 4, 5);
}

static void report_needs_every_block() {
  eng::RunReport report;
  EXPECT(report.alloc() == SG_OK);
  sygraph::detail::GridBarrier* bar = nullptr;
  EXPECT(cudaMalloc(&bar, sizeof(*bar)) == cudaSuccess);
  const uint32_t blocks = 8;
  for (uint32_t leaves : {blocks, 0u, 1u, blocks, 7u, blocks}) {
    eng::ReportRef ref = report.next();
    uint32_t who = leaves;
    void* args[] = {&ref, &bar, &who};
    EXPECT(cudaMemset(bar, 0, sizeof(*bar)) == cudaSuccess);
    EXPECT(cudaLaunchCooperativeKernel((const void*)run_kernel, dim3(blocks), dim3(64), args, 0, 0) == cudaSuccess);
    EXPECT(cudaDeviceSynchronize() == cudaSuccess);
    EXPECT(report.finished() == (leaves == blocks));
    if (leaves == blocks)
      for (uint32_t i = 0; i < 5; i++) EXPECT(report.host->v[i] == i + 1);
  }
  report.release();
  cudaFree(bar);
}

// Labels are not handed out after a run that gave up, with either method, and
// are after the next run; replays of a captured run do not confuse the status.
static void labels_of_an_unfinished_run() {
  const uint32_t ro[] = {0, 1, 3, 5, 6, 6}, col[] = {1, 0, 2, 1, 3, 2};
  cudaStream_t st;
  EXPECT(cudaStreamCreate(&st) == cudaSuccess);
  sg_graph g = nullptr;
  EXPECT(sg_graph_create_csr(ro, col, nullptr, SG_WEIGHT_NONE, 5, 6, 0, st, &g) == SG_OK);
  sg_cc_handle c = nullptr;
  EXPECT(sg_cc_create(g, &c) == SG_OK);
  uint32_t labels[5];
  for (int method : {SG_CC_UNION_FIND, SG_CC_PROPAGATION}) {
    EXPECT(sg_cc_set_method(c, method) == SG_OK);
    EXPECT(sg_cc_run_async(c) == SG_OK);
    EXPECT(sg_cc_get_labels(c, labels) == SG_OK && labels[0] == 3 && labels[3] == 3 && labels[4] == 4);
    EXPECT(sg_cc_run_async(c) == SG_OK);
    EXPECT(cudaMemsetAsync(&c->ws.bar->error, 1, 1, st) == cudaSuccess);
    EXPECT(sg_cc_get_labels(c, labels) == SG_ERR_TIMEOUT);
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    EXPECT(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess);
    EXPECT(sg_cc_run_async(c) == SG_OK);
    EXPECT(cudaStreamEndCapture(st, &graph) == cudaSuccess);
    EXPECT(cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess);
    EXPECT(sg_cc_run(c, nullptr) == SG_OK);
    EXPECT(cudaMemsetAsync(c->labels, 0, sizeof(labels), st) == cudaSuccess);
    EXPECT(cudaGraphLaunch(exec, st) == cudaSuccess);
    labels[0] = 0;
    EXPECT(sg_cc_get_labels(c, labels) == SG_OK && labels[0] == 3 && labels[4] == 4);
    EXPECT(sg_cc_run(c, nullptr) == SG_OK);
    EXPECT(cudaGraphExecDestroy(exec) == cudaSuccess && cudaGraphDestroy(graph) == cudaSuccess);
  }
  EXPECT(sg_cc_destroy(c) == SG_OK && sg_graph_destroy(g) == SG_OK);
  EXPECT(cudaStreamDestroy(st) == cudaSuccess);
}

int main() {
  labels_of_an_unfinished_run();
  report_needs_every_block();
  std::puts("ALL OK");
  return 0;
}
