// rbk_capi.cpp over a fake CUDA runtime, in which device and pinned memory are
// host memory, copies are memcpy and one chosen allocation fails: a call that
// met the failure reports it, and the next call on the same object works.
// Every copy and every buffer handed to a launch must be live memory.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "rbk.h"
#include "rbk_adjoint.h"
#include "rbk_kernels.h"
#include "rbk_small_adjoint.h"

static int g_allocs = 0, g_fail_at = 0;

static void fail(const char* what) { std::printf("FAILED: %s\n", what); std::exit(1); }

static cudaError_t alloc(void** p, size_t bytes)
{
  *p = nullptr;
  if (++g_allocs == g_fail_at) return cudaErrorMemoryAllocation;
  *p = std::calloc(bytes ? bytes : 1, 1);
  return cudaSuccess;
}

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) { return alloc(p, bytes); }
cudaError_t cudaMallocHost(void** p, size_t bytes) { return alloc(p, bytes); }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t)
{
  if (!to || !from) fail("copy to or from a null pointer");
  std::memcpy(to, from, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t)
{
  if (!p) fail("memset of a null pointer");
  std::memset(p, v, bytes);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

// The launches that the calls below reach: they touch the buffers they are given.
namespace rbk {
static void touch(const void* p) { if (!p) fail("launch on a null pointer"); else (void)*static_cast<const volatile char*>(p); }

template <typename Real> cudaError_t launch_set_basis(void* a, int, uint64_t, cudaStream_t) { touch(a); return cudaSuccess; }
template <typename Real> cudaError_t launch_tile_pass(void* a, int, const dev_pass&, int, cudaStream_t) { touch(a); return cudaSuccess; }
template <typename Real> cudaError_t launch_inner(const void* a, const void* b, int, double* partials, double* out, cudaStream_t)
{
  touch(a); touch(b); touch(partials); touch(out);
  return cudaSuccess;
}
template <typename Real> cudaError_t launch_pauli_apply_tiled(const void* a, void* b, int, const pauli_sum&, cudaStream_t)
{
  touch(a); touch(b);
  return cudaSuccess;
}
template <typename Real> cudaError_t launch_zsum2(const void* a, const void* b, int, const zsum2_set&, double* partials, double* out, cudaStream_t)
{
  touch(a); touch(b); touch(partials); touch(out);
  return cudaSuccess;
}
template <typename Real>
cudaError_t launch_pair_rotate(void* a, void* b, int, const pair_rotate_set& set, double* partials, size_t begin,
                               std::vector<pair_rotate_result>& results, size_t* used, cudaStream_t)
{
  touch(a); touch(b); touch(partials);
  *used = size_t(set.g.nflips);
  for (size_t i = 0; i < *used; ++i) partials[begin + i] = 1.0;
  for (int f = 0; f < set.g.nflips; ++f)
    if (set.flip[f].out_slot >= 0) results.push_back({begin, 1, set.g.nflips, f, -1, set.flip[f].out_slot, 0, 1.0});
  return cudaSuccess;
}
cudaError_t launch_finish_pair_rotate(const double* partials, const pair_rotate_result* r, int count, double* out, cudaStream_t)
{
  if (!partials || !r || !out) fail("launch on a null pointer");
  for (int i = 0; i < count; ++i) out[2 * r[i].slot + 1] = partials[r[i].begin + size_t(r[i].column)];
  return cudaSuccess;
}
cudaError_t launch_unitary_tf32x3(void* a, int, int, const float* w, int* flag, int, const tc_layout&, cudaStream_t)
{
  touch(a); touch(w); touch(flag);
  return cudaSuccess;
}
size_t tc_w_split_floats(int k) { return size_t(8) << (2 * k); }
size_t overlaps_partials_doubles() { return 64; }
size_t pair_overlaps_partials_doubles() { return 64; }
size_t tile_overlaps_partials_doubles(int, int) { return 64; }
size_t pair_rotate_partials_doubles() { return 64; }
bool sa_plan(int, const rbk_circuit_gate*, int, int, const char*, const double*, sa_program&) { return false; }
sa_set::~sa_set() = default;
int sa_set::assign(int, const std::vector<const sa_program*>&, const double*, int, cudaStream_t) { return RBK_ERR_STATE; }
int sa_set::launch(const double*, int, cudaStream_t, const std::vector<cudaStream_t>&, const std::vector<cudaEvent_t>&) { return RBK_ERR_STATE; }
int sa_set::fetch(cudaStream_t) { return RBK_ERR_STATE; }

#define RBK_FAKES(Real) \
  template cudaError_t launch_set_basis<Real>(void*, int, uint64_t, cudaStream_t); \
  template cudaError_t launch_tile_pass<Real>(void*, int, const dev_pass&, int, cudaStream_t); \
  template cudaError_t launch_inner<Real>(const void*, const void*, int, double*, double*, cudaStream_t); \
  template cudaError_t launch_pauli_apply_tiled<Real>(const void*, void*, int, const pauli_sum&, cudaStream_t); \
  template cudaError_t launch_zsum2<Real>(const void*, const void*, int, const zsum2_set&, double*, double*, cudaStream_t); \
  template cudaError_t launch_pair_rotate<Real>(void*, void*, int, const pair_rotate_set&, double*, size_t, \
                                                std::vector<pair_rotate_result>&, size_t*, cudaStream_t);
RBK_FAKES(double)
RBK_FAKES(float)
}  // namespace rbk

// `call` once with each of its allocations failing, and once more after each.
static void sweep(const char* name, const std::function<std::function<int()>()>& make)
{
  g_fail_at = 0;
  auto first = make();
  g_allocs = 0;
  if (first() != RBK_OK) fail(rbk_last_error());
  const int count = g_allocs;
  for (int at = 1; at <= count; ++at) {
    auto call = make();
    g_allocs = 0;
    g_fail_at = at;
    const int rc = call();
    g_fail_at = 0;
    if (rc != RBK_ERR_OOM) fail("an allocation that failed was not reported");
    if (call() != RBK_OK) fail(rbk_last_error());
  }
  std::printf("%s: %d allocations\n", name, count);
}

int main()
{
  constexpr int n = 14;
  std::vector<rbk_circuit_gate> gates;
  for (int layer = 0; layer < 2; ++layer)
    for (int q = 0; q < n; ++q)
      for (int kind : {RBK_GATE_EY, RBK_GATE_EZ}) {
        rbk_circuit_gate g{};
        g.kind = kind;
        g.qubits[0] = q;
        g.param = int(gates.size());
        g.scale = -0.5;
        gates.push_back(g);
      }
  const int params = int(gates.size());
  std::vector<double> theta(gates.size(), 0.3), grad(gates.size());
  std::string strings(2 * n, 'I');
  strings[0] = strings[1] = 'Z';
  strings[n] = 'X';
  const double coeffs[4] = {1, 0, 0.5, 0};
  double energy = 0;
  for (int precision : {RBK_C128, RBK_C64}) {
    sweep("gradient", [&] {
      rbk::adjoint_workspace* w = nullptr;
      if (rbk::adjoint_workspace_create(n, precision, 0, &w) != RBK_OK) fail(rbk_last_error());
      const std::shared_ptr<rbk::adjoint_workspace> held(w, rbk::adjoint_workspace_destroy);
      return [&, held] {
        return rbk::adjoint_run(held.get(), gates.data(), params, theta.data(), params, 2, strings.data(), coeffs, &energy, grad.data());
      };
    });
  }
  // A dense unitary of 5 qubits on the tensor cores.
  std::vector<double> u(2 * 32 * 32, 0.0);
  for (int r = 0; r < 32; ++r) u[2 * (33 * r)] = 1.0;
  const uint32_t qubits[5] = {0, 1, 2, 3, 4};
  sweep("unitary", [&] {
    rbk_state* s = nullptr;
    if (rbk_state_create(n, RBK_C64, 0, 0, &s) != RBK_OK) fail(rbk_last_error());
    const std::shared_ptr<rbk_state> held(s, rbk_state_destroy);
    return [&, held] { return rbk_apply_unitary(held.get(), u.data(), qubits, 5); };
  });
  std::printf("ALL OK\n");
  return 0;
}
