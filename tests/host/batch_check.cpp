// rbk_batch.cu over fakes of the CUDA runtime, the planned launches and the
// engine's sweep: a run whose large instance fails leaves no work in flight, so
// that the batch can be run again or destroyed at once.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "rbk.h"
#include "rbk_adjoint.h"
#include "rbk_kernels.h"
#include "rbk_small_adjoint.h"

static bool g_in_flight = false, g_sweep_fails = false;
static std::string g_error;

static void fail(const char* what) { std::printf("FAILED: %s\n", what); std::exit(1); }
static void idle(const char* what) { if (g_in_flight) fail(what); }

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void* p) { if (p) idle("cudaFree with work in flight"); std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { if (p) idle("cudaFreeHost with work in flight"); std::free(p); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t)
{
  idle("launched again with work in flight");
  g_in_flight = true;
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t) { g_in_flight = false; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { g_in_flight = false; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = reinterpret_cast<cudaGraph_t>(1); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = reinterpret_cast<cudaGraphExec_t>(1); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { idle("graph destroyed with work in flight"); return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
const char* rbk_last_error(void) { return g_error.c_str(); }
}

namespace rbk {
int set_last_error(int code, const char* m) { g_error = m; return code; }
bool sa_plan(int n, const rbk_circuit_gate*, int, int, const char*, const double*, sa_program& out) { out.n = n; return true; }
static double g_zero[4] = {};
sa_set::~sa_set() = default;
int sa_set::assign(int, const std::vector<const sa_program*>& list, const double*, int, cudaStream_t)
{
  insts_.resize(list.size());
  slot_begin_.assign(list.size(), 0);
  h_out_ = g_zero;
  return RBK_OK;
}
int sa_set::launch(const double*, int, cudaStream_t, const std::vector<cudaStream_t>&, const std::vector<cudaEvent_t>&) { return RBK_OK; }
int sa_set::fetch(cudaStream_t) { return RBK_OK; }
struct adjoint_workspace {};
int adjoint_workspace_create(int, int, int, adjoint_workspace** out) { *out = new adjoint_workspace; return RBK_OK; }
void adjoint_workspace_destroy(adjoint_workspace* w) { delete w; }
int adjoint_workspace_set_shape(adjoint_workspace*, int) { return RBK_OK; }
int adjoint_run(adjoint_workspace*, const rbk_circuit_gate*, int, const double*, int, int, const char*, const double*, double*, double*)
{
  return g_sweep_fails ? set_last_error(RBK_ERR_INVALID, "refused") : RBK_OK;
}
}  // namespace rbk

int main()
{
  const double coeffs[2] = {1, 0};
  const std::string z4(4, 'Z'), z16(16, 'Z');
  const rbk_batch_instance instances[2] = {{4, 0, nullptr, 0, 1, z4.c_str(), coeffs}, {16, 0, nullptr, 0, 1, z16.c_str(), coeffs}};
  double energies[2];
  rbk_batch* b = nullptr;
  if (rbk_batch_create(RBK_C128, 0, 2, instances, &b) != RBK_OK) fail(rbk_last_error());
  for (const bool fails : {false, true, true, false, true}) {
    g_sweep_fails = fails;
    if (rbk_batch_run(b, nullptr, energies, nullptr) != (fails ? RBK_ERR_INVALID : RBK_OK)) fail("wrong status");
  }
  rbk_batch_destroy(b);
  std::printf("ALL OK\n");
  return 0;
}
