// rbk_batch.cu -- energies and adjoint gradients of many parametrised circuits
// of uneven size in one call (rbk_batch_* of include/rbk.h).
//
// Instances whose two state vectors fit the shared memory of one CTA (up to 12
// qubits) or of one cluster (up to 15) run in one set of launches
// (rbk_small_adjoint.cu), one launch per size class on streams of their own, which
// do the whole job of every instance and are captured with their copies in a CUDA
// graph that every parameter vector replays.  The CTA size is picked by an autotuner that times the
// candidates on the batch's own instances.  Larger instances run through the
// engine's adjoint sweep (rbk_adjoint_gradient) on worker threads, with the
// fused passes' tile shape (their fusion width) picked per qubit count by a
// second autotuner.
//
// The reference has no differentiation or batching; the gate arithmetic is
// ket's (exponential_pauli_y.hpp:40-85, exponential_pauli_z.hpp:40-78,
// phase_shift.hpp:660-709 and :1200-1254), the same matrices as the engine's.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "rbk.h"
#include "rbk_adjoint.h"
#include "rbk_kernels.h"
#include "rbk_small_adjoint.h"

namespace {

int fail(int code, const std::string& m) { return rbk::set_last_error(code, m.c_str()); }

struct dev_free {
  void operator()(void* p) const { if (p) cudaFree(p); }
};
template <typename T>
using dptr = std::unique_ptr<T, dev_free>;

template <typename T>
T* dalloc(size_t count)
{
  void* p = nullptr;
  if (cudaMalloc(&p, sizeof(T) * (count ? count : 1)) != cudaSuccess) throw std::bad_alloc();
  return static_cast<T*>(p);
}

}  // namespace

struct rbk_batch {
  int precision = RBK_C128;
  int device = 0;
  int num_instances = 0;
  int total_params = 0;
  std::vector<int> param_begin, num_params;
  // instances of at most kSmallAdjointBits qubits: one set of launches
  std::vector<int> set_index;  // instance of each of the set's programs
  std::vector<rbk::sa_program> programs;  // their overlaps' parameters (the gates live on the device)
  rbk::sa_set set;
  int threads = 256;
  dptr<double> d_theta;
  double* h_theta = nullptr;  // pinned staging
  cudaStream_t stream = nullptr;
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> events;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  // large instances: the engine's adjoint sweep
  std::vector<int> large;
  std::vector<std::vector<rbk_circuit_gate>> large_gates;
  std::vector<std::string> large_strings;
  std::vector<std::vector<double>> large_coeffs;
  rbk_batch_stats stats{};
  // Worker threads for the large instances, each with its own workspaces by size.
  int workers = 8;
  std::vector<std::map<int, rbk::adjoint_workspace*>> pools;
  // Tile shape of the fused passes per qubit count of the large instances (the
  // fusion width: 2^11 or 2^12 amplitudes per tile), picked by timing.
  std::map<int, int> shape_of;

  ~rbk_batch()
  {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);  // a call that ended early may have left its launches
    for (auto& pool : pools)
      for (auto& kv : pool) rbk::adjoint_workspace_destroy(kv.second);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (h_theta) cudaFreeHost(h_theta);
    for (cudaEvent_t e : events) cudaEventDestroy(e);
    for (cudaStream_t q : side) cudaStreamDestroy(q);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

// Records the job of the set's instances (parameters in, the launches, results out) on b->stream.
int record_small(rbk_batch* b)
{
  if (cudaMemcpyAsync(b->d_theta.get(), b->h_theta, sizeof(double) * static_cast<size_t>(b->total_params), cudaMemcpyHostToDevice,
                      b->stream) != cudaSuccess)
    return fail(RBK_ERR_CUDA, "batch copies");
  if (int rc = b->set.launch(b->d_theta.get(), b->threads, b->stream, b->side, b->events)) return rc;
  return b->set.fetch(b->stream);
}

// Whether the engine's sweep refuses what the planned instance asks for
// (rbk_adjoint_gradient: phase exponents above n, more than 128 strings or 64 flip
// patterns).
bool sweep_refuses(const rbk_batch_instance& I, const rbk::sa_program& P)
{
  for (int k = 0; k < I.num_gates; ++k)
    if (I.gates[k].kind == RBK_GATE_U && std::abs(I.gates[k].angles[0]) >= I.num_qubits + 1) return true;
  int flips = P.terms.empty() ? 0 : 1;
  for (size_t t = 1; t < P.terms.size(); ++t) flips += P.terms[t].flip != P.terms[t - 1].flip ? 1 : 0;
  return P.terms.size() > static_cast<size_t>(rbk::kMaxSumTerms) || flips > rbk::kMaxSumGroups;
}

int sync_bounded(cudaStream_t s)
{
  const char* env = std::getenv("RBK_TIMEOUT_S");
  const double limit = env ? std::atof(env) : 600.0;
  const auto t0 = std::chrono::steady_clock::now();
  while (true) {
    const cudaError_t e = cudaStreamQuery(s);
    if (e == cudaSuccess) return RBK_OK;
    if (e != cudaErrorNotReady) return fail(RBK_ERR_CUDA, std::string("batch: ") + cudaGetErrorString(e));
    if (std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() > limit)
      return fail(RBK_ERR_TIMEOUT, "batch: device wait timed out");
    std::this_thread::yield();
  }
}

// Fusion width of the large instances: for every qubit count from
// kTuneMinQubits up, one instance of that size is run through the sweep with
// each tile shape (2^11 amplitudes per tile in 4 CTAs per SM, 2^12 in 2, and
// 2^11 in 3 persistent CTAs that prefetch), and the fastest shape is kept for
// all instances of that size.  Below that size the default shape is kept: the
// sweeps there are bound by launches, not by the passes.
constexpr int kTuneMinQubits = 16;
int tune_shapes(rbk_batch* b)
{
  std::map<int, size_t> rep;  // qubit count -> index into b->large of the first instance of that size
  for (size_t k = 0; k < b->large.size(); ++k) {
    const int nt = static_cast<int>(b->large_coeffs[k].size() / 2);
    const int nq = static_cast<int>(b->large_strings[k].size() / static_cast<size_t>(nt));
    if (nq >= kTuneMinQubits && !rep.count(nq)) rep.emplace(nq, k);
  }
  for (const auto& kv : rep) {
    const int nq = kv.first;
    const size_t k = kv.second;
    const int i = b->large[k];
    const auto& gs = b->large_gates[k];
    const int nt = static_cast<int>(b->large_coeffs[k].size() / 2);
    std::vector<double> theta(static_cast<size_t>(std::max(1, b->num_params[i])), 0.1);
    std::vector<double> grad(theta.size());
    double energy = 0.0;
    rbk::adjoint_workspace* w = nullptr;
    if (int rc = rbk::adjoint_workspace_create(nq, b->precision, b->device, &w)) return rc;
    double best = 1e300;
    int best_shape = 2;
    int rc = RBK_OK;
    for (int shape : {2, 0, 3}) {
      rc = rbk::adjoint_workspace_set_shape(w, shape);
      double ms = 1e300;
      for (int r = 0; rc == RBK_OK && r < 3; ++r) {  // the first run warms up
        const auto t0 = std::chrono::steady_clock::now();
        rc = rbk::adjoint_run(w, gs.data(), static_cast<int>(gs.size()), theta.data(), b->num_params[i], nt,
                              b->large_strings[k].data(), b->large_coeffs[k].data(), &energy, grad.data());
        const double t = 1e3 * std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (r > 0) ms = std::min(ms, t);
      }
      if (rc != RBK_OK) break;
      if (ms < best) { best = ms; best_shape = shape; }
    }
    rbk::adjoint_workspace_destroy(w);
    if (rc != RBK_OK) return rc;
    b->shape_of[nq] = best_shape;
  }
  return RBK_OK;
}

}  // namespace

extern "C" int rbk_batch_tuned_shape(const rbk_batch* b, int num_qubits, int* shape)
{
  if (!b || !shape) return fail(RBK_ERR_INVALID, "null argument");
  const auto it = b->shape_of.find(num_qubits);
  *shape = it == b->shape_of.end() ? -1 : it->second;
  return RBK_OK;
}

extern "C" int rbk_batch_create(int precision, int device, int num_instances, const rbk_batch_instance* instances,
                                rbk_batch** out)
{
  try {
    if (!out || num_instances < 0 || (num_instances > 0 && !instances)) return fail(RBK_ERR_INVALID, "bad batch arguments");
    if (precision != RBK_C128 && precision != RBK_C64) return fail(RBK_ERR_INVALID, "unknown precision");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(RBK_ERR_CUDA, "no CUDA device available");
    if (device < 0 || device >= ndev) return fail(RBK_ERR_INVALID, "device out of range");
    if (cudaSetDevice(device) != cudaSuccess) return fail(RBK_ERR_CUDA, "cudaSetDevice");
    auto b = std::make_unique<rbk_batch>();
    b->precision = precision;
    b->device = device;
    b->num_instances = num_instances;
    const int small_limit = precision == RBK_C128 ? 12 : 13;
    for (int i = 0; i < num_instances; ++i) {
      const auto& I = instances[i];
      if (I.num_qubits < 1 || I.num_qubits > 33 || I.num_gates < 0 || (I.num_gates > 0 && !I.gates) || I.num_params < 0 ||
          I.num_terms < 1 || !I.strings || !I.coeffs)
        return fail(RBK_ERR_INVALID, "instance " + std::to_string(i) + ": bad arguments");
      for (int k = 0; k < I.num_gates; ++k) {
        const auto& g = I.gates[k];
        const bool two = g.kind == RBK_GATE_CNOT || g.kind == RBK_GATE_CZ || g.kind == RBK_GATE_U || g.kind == RBK_GATE_SWAP;
        if (g.qubits[0] < 0 || g.qubits[0] >= I.num_qubits || (two && (g.qubits[1] < 0 || g.qubits[1] >= I.num_qubits ||
                                                                      g.qubits[1] == g.qubits[0])))
          return fail(RBK_ERR_INVALID, "instance " + std::to_string(i) + ": qubit out of range");
        if (g.param >= I.num_params) return fail(RBK_ERR_INVALID, "instance " + std::to_string(i) + ": parameter out of range");
        if (g.param >= 0 && g.kind != RBK_GATE_EX && g.kind != RBK_GATE_EY && g.kind != RBK_GATE_EZ)
          return fail(RBK_ERR_UNSUPPORTED, "only EX, EY and EZ gates take parameters");
        if (g.kind < RBK_GATE_H || g.kind > RBK_GATE_SWAP) return fail(RBK_ERR_INVALID, "instance " + std::to_string(i) + ": unknown gate kind");
      }
      b->param_begin.push_back(b->total_params);
      b->num_params.push_back(I.num_params);
      b->total_params += I.num_params;
      if (I.num_qubits > rbk::kSmallAdjointBits) {
        b->large.push_back(i);
        continue;
      }
      b->programs.emplace_back();
      const bool planned = rbk::sa_plan(I.num_qubits, I.gates, I.num_gates, I.num_terms, I.strings, I.coeffs, b->programs.back());
      if (!planned && I.num_qubits <= small_limit) return fail(RBK_ERR_INVALID, "Pauli strings use the characters I, X, Y, Z");
      if (I.num_qubits > small_limit && (!planned || sweep_refuses(I, b->programs.back()))) {
        b->programs.pop_back();  // the sweep refuses it when the batch runs
        b->large.push_back(i);
        continue;
      }
      b->programs.back().theta_begin = b->param_begin.back();
      b->set_index.push_back(i);
      ++(I.num_qubits <= small_limit ? b->stats.num_small : b->stats.num_large);
    }
    std::stable_sort(b->large.begin(), b->large.end(),
                     [&](int x, int y) { return instances[x].num_qubits > instances[y].num_qubits; });
    for (int li : b->large) {
      const auto& I = instances[li];
      b->large_gates.emplace_back(I.gates, I.gates + I.num_gates);
      b->large_strings.emplace_back(I.strings, static_cast<size_t>(I.num_terms) * I.num_qubits);
      b->large_coeffs.emplace_back(I.coeffs, I.coeffs + 2 * I.num_terms);
    }
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(RBK_ERR_CUDA, "stream");
    const size_t np = static_cast<size_t>(b->total_params);
    if (cudaMallocHost(reinterpret_cast<void**>(&b->h_theta), sizeof(double) * (np ? np : 1)) != cudaSuccess)
      return fail(RBK_ERR_OOM, "pinned host memory");
    std::memset(b->h_theta, 0, sizeof(double) * (np ? np : 1));
    b->stats.num_large += static_cast<int>(b->large.size());
    if (!b->programs.empty()) {
      b->d_theta.reset(dalloc<double>(np));
      // A side stream for each size class after the first, and an event more.  Those of
      // all six classes whatever the sizes made creating a batch of one class 1 ms longer
      // (four instances of 12 qubits: 5.4 ms, now 4.5 to 4.9).
      std::set<int> classes;
      for (const auto& P : b->programs) classes.insert(rbk::sa_set::size_class(P.n));
      for (size_t k = 1; k < classes.size(); ++k) {
        cudaStream_t q;
        if (cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking) != cudaSuccess) return fail(RBK_ERR_CUDA, "stream");
        b->side.push_back(q);
      }
      for (size_t k = 0; k < classes.size(); ++k) {
        cudaEvent_t ev;
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return fail(RBK_ERR_CUDA, "event");
        b->events.push_back(ev);
      }
      std::vector<const rbk::sa_program*> list;
      for (const auto& P : b->programs) list.push_back(&P);
      if (int rc = b->set.assign(precision, list, nullptr, 0, b->stream)) return rc;
      for (auto& P : b->programs) {  // on the device from here on
        P.ops = {};
        P.phases = {};
        P.rots = {};
        P.terms = {};
      }
      // Autotuner: time each CTA size on the batch's own small instances (theta = 0) and keep the fastest.
      cudaEvent_t e0, e1;
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      float best = 1e30f;
      bool warmed = false;
      int best_threads = 256;
      for (int threads : {512, 256, 128}) {
        b->threads = threads;
        cudaEventRecord(e0, b->stream);
        if (int rc = record_small(b.get())) { cudaEventDestroy(e0); cudaEventDestroy(e1); return rc; }
        cudaEventRecord(e1, b->stream);
        if (int rc = sync_bounded(b->stream)) { cudaEventDestroy(e0); cudaEventDestroy(e1); return rc; }
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (threads == 512 && !warmed) {  // the first run of all only warms up
          warmed = true;
          cudaEventRecord(e0, b->stream);
          if (int rc = record_small(b.get())) { cudaEventDestroy(e0); cudaEventDestroy(e1); return rc; }
          cudaEventRecord(e1, b->stream);
          if (int rc = sync_bounded(b->stream)) { cudaEventDestroy(e0); cudaEventDestroy(e1); return rc; }
          cudaEventElapsedTime(&ms, e0, e1);
        }
        if (ms < best) { best = ms; best_threads = threads; }
      }
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      b->threads = best_threads;
      b->stats.threads = best_threads;
      b->stats.small_ms = best;
      // The small-instance job as a CUDA graph, replayed by every rbk_batch_run.
      if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        return fail(RBK_ERR_CUDA, "graph capture");
      const int rc = record_small(b.get());
      const cudaError_t ce = cudaStreamEndCapture(b->stream, &b->graph);
      if (rc) return rc;
      if (ce != cudaSuccess || cudaGraphInstantiate(&b->exec, b->graph, 0) != cudaSuccess)
        return fail(RBK_ERR_CUDA, "graph instantiate");
    }
    if (int rc = tune_shapes(b.get())) return rc;
    *out = b.release();
    return RBK_OK;
  } catch (std::bad_alloc const&) {
    return fail(RBK_ERR_OOM, "batch: memory exhausted");
  } catch (std::exception const& e) {
    return fail(RBK_ERR_STATE, e.what());
  }
}

extern "C" int rbk_batch_run(rbk_batch* b, const double* theta, double* energies, double* grads)
{
  try {
    if (!b || !energies || (b->total_params > 0 && (!theta || !grads))) return fail(RBK_ERR_INVALID, "bad batch arguments");
    if (cudaSetDevice(b->device) != cudaSuccess) return fail(RBK_ERR_CUDA, "cudaSetDevice");
    const auto t0 = std::chrono::steady_clock::now();
    const size_t np = static_cast<size_t>(b->total_params);
    if (np) std::memcpy(b->h_theta, theta, sizeof(double) * np);
    if (!b->programs.empty() && cudaGraphLaunch(b->exec, b->stream) != cudaSuccess) return fail(RBK_ERR_CUDA, "graph launch");
    // Large instances meanwhile, through the engine's adjoint sweep: worker
    // threads take them largest first, each on its own streams and reusable
    // state pairs, so that host planning overlaps device work.
    if (!b->large.empty()) {
      if (b->pools.empty()) b->pools.resize(static_cast<size_t>(b->workers));
      std::atomic<size_t> next{0};
      std::atomic<int> first_rc{RBK_OK};
      std::mutex err_mu;
      std::string err;
      auto work = [&](int wid) {
        cudaSetDevice(b->device);
        auto& pool = b->pools[static_cast<size_t>(wid)];
        while (first_rc.load() == RBK_OK) {
          const size_t k = next.fetch_add(1);
          if (k >= b->large.size()) break;
          const int i = b->large[k];
          const int pb = b->param_begin[i];
          const auto& gs = b->large_gates[k];
          const int nt = static_cast<int>(b->large_coeffs[k].size() / 2);
          const int nq = static_cast<int>(b->large_strings[k].size() / static_cast<size_t>(nt));
          int rc = RBK_OK;
          auto it = pool.find(nq);
          if (it == pool.end()) {
            rbk::adjoint_workspace* w = nullptr;
            rc = rbk::adjoint_workspace_create(nq, b->precision, b->device, &w);
            const auto sh = b->shape_of.find(nq);
            if (rc == RBK_OK && sh != b->shape_of.end()) rc = rbk::adjoint_workspace_set_shape(w, sh->second);
            if (rc == RBK_OK) it = pool.emplace(nq, w).first;
            else if (w) rbk::adjoint_workspace_destroy(w);
          }
          if (rc == RBK_OK)
            rc = rbk::adjoint_run(it->second, gs.data(), static_cast<int>(gs.size()), theta + pb, b->num_params[i], nt,
                                  b->large_strings[k].data(), b->large_coeffs[k].data(), &energies[i], grads + pb);
          if (rc != RBK_OK) {
            int expected = RBK_OK;
            if (first_rc.compare_exchange_strong(expected, rc)) {
              std::lock_guard<std::mutex> lk(err_mu);
              err = rbk_last_error();
            }
          }
        }
      };
      std::vector<std::thread> threads;
      for (int t = 1; t < b->workers; ++t) threads.emplace_back(work, t);
      work(0);
      for (auto& t : threads) t.join();
      if (first_rc.load() != RBK_OK) {
        // The launches still read and write the batch's buffers.
        if (!b->programs.empty()) sync_bounded(b->stream);
        return fail(first_rc.load(), "batch: " + err);
      }
    }
    if (!b->programs.empty()) {
      if (int rc = sync_bounded(b->stream)) return rc;
      for (size_t k = 0; k < b->programs.size(); ++k) {
        const int i = b->set_index[k], pb = b->param_begin[i];
        const rbk::sa_program& P = b->programs[k];
        const double* o = b->set.overlaps(static_cast<int>(k));
        energies[i] = b->set.energies()[k];
        for (int p = 0; p < b->num_params[i]; ++p) grads[pb + p] = 0.0;
        for (size_t s = 0; s < P.slot_param.size(); ++s) grads[pb + P.slot_param[s]] += -2.0 * P.slot_scale[s] * o[s];
      }
    }
    b->stats.last_run_ms = 1e3 * std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return RBK_OK;
  } catch (std::bad_alloc const&) {
    return fail(RBK_ERR_OOM, "batch: memory exhausted");
  } catch (std::exception const& e) {
    return fail(RBK_ERR_STATE, e.what());
  }
}

extern "C" int rbk_batch_set_workers(rbk_batch* b, int workers)
{
  if (!b || workers < 1 || workers > 64) return fail(RBK_ERR_INVALID, "workers must be between 1 and 64");
  cudaSetDevice(b->device);
  for (auto& pool : b->pools)
    for (auto& kv : pool) rbk::adjoint_workspace_destroy(kv.second);
  b->pools.clear();
  b->workers = workers;
  return RBK_OK;
}

extern "C" int rbk_batch_get_stats(const rbk_batch* b, rbk_batch_stats* out)
{
  if (!b || !out) return fail(RBK_ERR_INVALID, "null argument");
  *out = b->stats;
  return RBK_OK;
}

extern "C" int rbk_batch_destroy(rbk_batch* b)
{
  if (b) {
    cudaSetDevice(b->device);
    delete b;
  }
  return RBK_OK;
}
