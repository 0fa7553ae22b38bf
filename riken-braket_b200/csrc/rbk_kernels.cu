// rbk_kernels.cu -- sm_100a kernels of the state-vector engine.
//
//   (the fused tile pass lives in rbk_tile.cu)
//   small_circuit_kernel  a whole queue of gates on a state of up to 12 qubits.
//   reductions         norm, probabilities, Z / pair sums for spins and Pauli
//                      strings, inner product: warp-shuffle + block reduction
//                      with FP64 accumulation, per-block partials reduced in a
//                      fixed order (deterministic).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <vector>

#include "rbk_device.cuh"
#include "rbk_internal.h"
#include "rbk_kernels.h"
#include "rbk_sample_scan.h"
#include "rbk_small_core.cuh"

namespace rbk {

// ---------------------------------------------------------------------------
// Whole circuits on states of one CTA
// ---------------------------------------------------------------------------

// A queue of gates on a state of up to kSmallBits qubits, in one CTA: the state
// and the program are read into shared memory once, every phase (small_phase)
// moves 8 amplitudes per thread into registers, applies its gates there and
// writes them back, and the state goes back to HBM at the end.  Arithmetic is
// complex<double> for both precisions (a complex<float> state is rounded once,
// at the end).
//   Bound by latency: a phase costs two shared-memory moves and a barrier, a
// gate its dispatch and its FP64 work on one SM.  One launch per gate (below
// one tile) took 2.7 us of device and 2.9 us of host time a gate; the tile
// passes at 11 and 12 qubits put a pass of 12 gates on 1 or 2 CTAs of 4 warps.
//   8 qubits, 200 random gates: 772 us of device and 468 us of host time with a
// launch per gate, 126 and 31 us here.
template <int CAP>
struct small_params {
  uint32_t num_ops, num_phases;
  alignas(8) small_phase phases[CAP];
  small_op ops[CAP];
};

constexpr int kSmallCircuitThreads = 512;  // 1024 (64 registers) spilled
template <typename Real, int CAP>
__global__ void __launch_bounds__(kSmallCircuitThreads, 1)
small_circuit_kernel(typename ctype<Real>::c* __restrict__ state, int n, const __grid_constant__ small_params<CAP> P)
{
  using C = typename ctype<Real>::c;
  constexpr int NR = 1 << kSmallRegBits;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* s = reinterpret_cast<double2*>(smem_raw);
  const uint32_t size = 1u << n, padded = max(size, uint32_t(NR));
  small_op* ops = reinterpret_cast<small_op*>(s + padded);
  __shared__ small_phase phases[CAP];  // indexed by the phase: a constant-cache miss per line otherwise
  {
    // Through a generic pointer: the threads read the parameter block side by side,
    // where indexing it by the thread would go word by word through the constant cache.
    const uint64_t* src = reinterpret_cast<const uint64_t*>(P.ops);
    asm volatile("" : "+l"(src));
    uint64_t* dst = reinterpret_cast<uint64_t*>(ops);
    for (uint32_t i = threadIdx.x; i < P.num_ops * uint32_t(sizeof(small_op) / 8); i += blockDim.x) dst[i] = src[i];
    const uint64_t* psrc = reinterpret_cast<const uint64_t*>(P.phases);
    asm volatile("" : "+l"(psrc));
    for (uint32_t i = threadIdx.x; i < P.num_phases; i += blockDim.x) reinterpret_cast<uint64_t*>(phases)[i] = psrc[i];
  }
  // Slots are swizzled (smem_slot) so that the lanes of a phase reach distinct banks whichever bits it holds.
  for (uint32_t i = threadIdx.x; i < padded; i += blockDim.x) {
    double2 v{0.0, 0.0};
    if (i < size) {
      const C x = state[i];
      v = double2{double(x.x), double(x.y)};
    }
    s[smem_slot<0>(i)] = v;
  }
  __syncthreads();
  for (uint32_t p = 0; p < P.num_phases; ++p) {
    const small_phase ph = phases[p];
    uint32_t rs[kSmallRegBits];
#pragma unroll
    for (int k = 0; k < kSmallRegBits; ++k) rs[k] = smem_slot<0>(1u << ph.reg[k]);
    for (uint32_t t = threadIdx.x; t < padded / NR; t += blockDim.x) {
      uint32_t base = t;
#pragma unroll
      for (int k = 0; k < kSmallRegBits; ++k) base = uint32_t(insert_zero(base, ph.reg[k]));
      const uint32_t sb = smem_slot<0>(base);
      double2 a[NR];
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        uint32_t x = sb;
#pragma unroll
        for (int k = 0; k < kSmallRegBits; ++k)
          if ((i >> k) & 1) x ^= rs[k];
        a[i] = s[x];
      }
      uint32_t signs = 0;
      small_header h = small_load_header(ops + ph.begin);
      for (uint32_t g = ph.begin; g < ph.end; ++g) {
        const small_header next = small_load_header(ops + min(g + 1, P.num_ops - 1));
        small_gate<false, false>(a, a, h, ops + g, base, signs);
        h = next;
      }
      if (signs) small_signs(a, signs);
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        uint32_t x = sb;
#pragma unroll
        for (int k = 0; k < kSmallRegBits; ++k)
          if ((i >> k) & 1) x ^= rs[k];
        s[x] = a[i];
      }
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < size; i += blockDim.x) {
    const double2 v = s[smem_slot<0>(i)];
    state[i] = C{Real(v.x), Real(v.y)};
  }
}

// A program of one phase and a few gates, 8 amplitudes a thread straight from HBM
// and back: with one phase the state needs no shared memory and no single CTA, and
// what is left is the launch.  50 gates in a launch each, 11 qubits: complex<double>
// 438 us in small_circuit_kernel, 321 here; complex<float> 431 and 324.  At 9 gates
// of one phase both take 23.5 us with the wait.
constexpr int kSmallDirectOps = 8, kSmallDirectThreads = 64;
struct small_direct_params {
  uint32_t num_ops, pad;
  small_phase phase;
  small_op ops[kSmallDirectOps];
};

template <typename Real>
__global__ void __launch_bounds__(kSmallDirectThreads)
small_direct_kernel(typename ctype<Real>::c* __restrict__ state, int n, const __grid_constant__ small_direct_params P)
{
  using C = typename ctype<Real>::c;
  constexpr int NR = 1 << kSmallRegBits;
  const uint32_t size = 1u << n;
  uint32_t base = blockIdx.x * kSmallDirectThreads + threadIdx.x;
  if (base >= (max(size, uint32_t(NR)) >> kSmallRegBits)) return;
#pragma unroll
  for (int k = 0; k < kSmallRegBits; ++k) base = uint32_t(insert_zero(base, P.phase.reg[k]));
  uint32_t idx[NR];
  double2 a[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    idx[i] = base;
#pragma unroll
    for (int k = 0; k < kSmallRegBits; ++k)
      if ((i >> k) & 1) idx[i] |= 1u << P.phase.reg[k];
    const C v = idx[i] < size ? state[idx[i]] : C{Real(0), Real(0)};
    a[i] = double2{double(v.x), double(v.y)};
  }
  uint32_t signs = 0;
  for (uint32_t g = 0; g < P.num_ops; ++g) small_gate<false, false>(a, a, small_load_header(&P.ops[g]), &P.ops[g], base, signs);
  if (signs) small_signs(a, signs);
#pragma unroll
  for (int i = 0; i < NR; ++i)
    if (idx[i] < size) state[idx[i]] = C{Real(a[i].x), Real(a[i].y)};
}

static unsigned grid_for(uint64_t work, int threads)
{
  uint64_t b = (work + threads - 1) / threads;
  const uint64_t cap = 148ull * 16;
  if (b > cap) b = cap;
  return (unsigned)(b == 0 ? 1 : b);
}

template <typename Real, int CAP>
static cudaError_t launch_small_cap(typename ctype<Real>::c* state, int n, const small_op* ops, int num_ops,
                                    const small_phase* phases, int num_phases, cudaStream_t stream)
{
  const uint32_t padded = std::max(1u << n, 1u << kSmallRegBits);
  const size_t smem = sizeof(double2) * padded + sizeof(small_op) * size_t(num_ops);
  constexpr size_t most = sizeof(double2) * (size_t(1) << kSmallBits) + sizeof(small_op) * CAP;
  static std::atomic<bool> configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(small_circuit_kernel<Real, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  small_params<CAP> P;
  P.num_ops = static_cast<uint32_t>(num_ops);
  P.num_phases = static_cast<uint32_t>(num_phases);
  std::copy(ops, ops + num_ops, P.ops);
  std::copy(phases, phases + num_phases, P.phases);
  const int threads = static_cast<int>(std::max(32u, std::min(uint32_t(kSmallCircuitThreads), padded >> kSmallRegBits)));
  small_circuit_kernel<Real, CAP><<<1, threads, smem, stream>>>(state, n, P);
  return cudaGetLastError();
}

// The parameter block is copied at every launch whatever it holds, so short
// programs take a short one (2.8, 11 and 32 KB).
template <typename Real>
cudaError_t launch_small(void* state, int n, const small_op* ops, int num_ops, const small_phase* phases, int num_phases,
                         cudaStream_t stream)
{
  static_assert(sizeof(small_params<kSmallGates>) <= 32640, "parameter block");
  if (n < 1 || n > kSmallBits || num_ops < 1 || num_ops > kSmallGates || num_phases < 1 || num_phases > num_ops)
    return cudaErrorInvalidValue;
  auto* a = static_cast<typename ctype<Real>::c*>(state);
  if (num_phases == 1 && num_ops <= kSmallDirectOps) {
    small_direct_params P{};
    P.num_ops = static_cast<uint32_t>(num_ops);
    P.phase = phases[0];
    std::copy(ops, ops + num_ops, P.ops);
    const unsigned groups = std::max(1u << n, 1u << kSmallRegBits) >> kSmallRegBits;
    small_direct_kernel<Real><<<(groups + kSmallDirectThreads - 1) / kSmallDirectThreads, kSmallDirectThreads, 0, stream>>>(a, n, P);
    return cudaGetLastError();
  }
  if (num_ops <= 32) return launch_small_cap<Real, 32>(a, n, ops, num_ops, phases, num_phases, stream);
  if (num_ops <= 128) return launch_small_cap<Real, 128>(a, n, ops, num_ops, phases, num_phases, stream);
  return launch_small_cap<Real, kSmallGates>(a, n, ops, num_ops, phases, num_phases, stream);
}
template cudaError_t launch_small<double>(void*, int, const small_op*, int, const small_phase*, int, cudaStream_t);
template cudaError_t launch_small<float>(void*, int, const small_op*, int, const small_phase*, int, cudaStream_t);

// ---------------------------------------------------------------------------
// Basis-state initialisation
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void set_basis_kernel(typename ctype<Real>::c* a, uint64_t size, uint64_t index)
{
  using C = typename ctype<Real>::c;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < size; i += stride)
    a[i] = i == index ? C{(Real)1, (Real)0} : C{(Real)0, (Real)0};
}

template <typename Real>
cudaError_t launch_set_basis(void* state, int n, uint64_t index, cudaStream_t stream)
{
  const uint64_t size = 1ull << n;
  set_basis_kernel<Real><<<grid_for(size, 256), 256, 0, stream>>>(static_cast<typename ctype<Real>::c*>(state), size, index);
  return cudaGetLastError();
}
template cudaError_t launch_set_basis<double>(void*, int, uint64_t, cudaStream_t);
template cudaError_t launch_set_basis<float>(void*, int, uint64_t, cudaStream_t);

// ---------------------------------------------------------------------------
// Reductions.  Each block writes `width` doubles of partial sums; one block
// then sums the partials in block order (deterministic for a given grid).
// ---------------------------------------------------------------------------
constexpr int kRedThreads = 256;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums `count` per-thread values over the block; thread 0 writes them to out.
template <int MAXW>
__device__ __forceinline__ void block_sum_store(double* vals, int count, double* out)
{
  __shared__ double red[kRedThreads / 32][MAXW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = 0; k < count; ++k) {
    double v = warp_sum(vals[k]);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < count) {
    double s = 0;
    for (int w = 0; w < kRedThreads / 32; ++w) s += red[w][threadIdx.x];
    out[threadIdx.x] = s;
  }
}

// out[c] = sum over the blocks of partials[b * width + c], one block of
// kFinishThreads threads per column: thread t takes blocks t, t + kFinishThreads,
// ... in order, then a fixed butterfly adds the lanes and the warps follow in
// order, so the sum is the same on every run.  Bound by the latency of its
// loads, which are independent here: 592 partials in 3 us, where one thread
// per column adding them one after the other took 45 to 52 us.
constexpr int kFinishThreads = 128;
__global__ void __launch_bounds__(kFinishThreads)
finish_partials_kernel(const double* __restrict__ partials, int blocks, int width, double* __restrict__ out)
{
  __shared__ double red[kFinishThreads / 32];
  const int c = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s = 0;
  for (int b = threadIdx.x; b < blocks; b += kFinishThreads) s += partials[size_t(b) * width + c];
  s = warp_sum(s);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kFinishThreads / 32; ++w) s += red[w];
    out[c] = s;
  }
}

// Z sums: out[0] = sum |a|^2, out[1 + q] = sum of |a|^2 over the amplitudes
// whose physical bit q is set.  Launched with exactly 2^kZsumLogThreads
// threads in total, so that bits below kZsumLogThreads of every index a thread
// visits are that thread's global id and only the higher bits vary (fewer
// blocks where the state has fewer amplitudes than that).
constexpr int kZsumLogThreads = 17;
static int zsum_blocks(int n) { return 1 << (std::max(8, std::min(n, kZsumLogThreads)) - 8); }
static_assert(kRedThreads == 1 << 8, "zsum_blocks counts 256-thread blocks");
template <typename Real>
__global__ void __launch_bounds__(kRedThreads) zsum_kernel(const typename ctype<Real>::c* __restrict__ a, int n, double* partials)
{
  constexpr int HI = kMaxQubits - kZsumLogThreads;
  const uint64_t size = 1ull << n;
  const uint64_t gid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  double total = 0, hi[HI];
#pragma unroll
  for (int k = 0; k < HI; ++k) hi[k] = 0;
  for (uint64_t k = 0; (k << kZsumLogThreads) + gid < size; ++k) {
    const auto v = a[(k << kZsumLogThreads) | gid];
    const double p = double(v.x) * double(v.x) + double(v.y) * double(v.y);
    total += p;
#pragma unroll
    for (int b = 0; b < HI; ++b) if ((k >> b) & 1) hi[b] += p;
  }
  double vals[1 + kMaxQubits];
  vals[0] = total;
  for (int q = 0; q < n; ++q) {
    if (q < kZsumLogThreads) vals[1 + q] = ((gid >> q) & 1) ? total : 0.0;
    else {
      double h = 0;
#pragma unroll
      for (int b = 0; b < HI; ++b) if (b == q - kZsumLogThreads) h = hi[b];
      vals[1 + q] = h;
    }
  }
  block_sum_store<1 + kMaxQubits>(vals, n + 1, partials + size_t(blockIdx.x) * (n + 1));
}

// Pair sums for Pauli strings sharing one flip mask F:
//   out = sum_i conj(a_i) a_{i^F} W(i),  W(i) = sum_t w_t (-1)^popcount(i & s_t)
// with complex weights w_t (terms given in physical bits).  F == 0 is allowed.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
pauli_kernel(const typename ctype<Real>::c* __restrict__ a, int n, uint64_t flip,
             const pauli_terms T, double* partials)
{
  const uint64_t size = 1ull << n;
  double re = 0, im = 0;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  if (flip == 0) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < size; i += stride) {
      const auto v = a[i];
      const double p = double(v.x) * double(v.x) + double(v.y) * double(v.y);
      double wr = 0, wi = 0;
      for (int t = 0; t < T.count; ++t) {
        const double s = (__popcll(i & T.sign[t]) & 1) ? -1.0 : 1.0;
        wr += s * T.w[t][0]; wi += s * T.w[t][1];
      }
      re += p * wr; im += p * wi;
    }
  } else {
    const int low = __ffsll((long long)flip) - 1;
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < (size >> 1); v += stride) {
      const uint64_t i = insert_zero(v, low), j = i ^ flip;
      const auto ai = a[i], aj = a[j];
      // c = conj(a_i) a_j ;  conj(a_j) a_i = conj(c)
      const double cr = double(ai.x) * double(aj.x) + double(ai.y) * double(aj.y);
      const double ci = double(ai.x) * double(aj.y) - double(ai.y) * double(aj.x);
      for (int t = 0; t < T.count; ++t) {
        const double si = (__popcll(i & T.sign[t]) & 1) ? -1.0 : 1.0;
        const double sj = (__popcll(j & T.sign[t]) & 1) ? -1.0 : 1.0;
        // si * c * w + sj * conj(c) * w
        const double xr = si * cr + sj * cr;
        const double xi = si * ci - sj * ci;
        re += xr * T.w[t][0] - xi * T.w[t][1];
        im += xr * T.w[t][1] + xi * T.w[t][0];
      }
    }
  }
  double vals[2] = {re, im};
  block_sum_store<2>(vals, 2, partials + size_t(blockIdx.x) * 2);
}

// observe_group (rbk_kernels.h).  Persistent CTAs, two per SM; a thread loads
// the 2^RB amplitudes of a tile that vary in the top RB tile bits, so the flips
// of those bits and every sum of |a|^2 come straight from the loaded registers;
// the other flips are read back from shared memory (slots smem_slot, conflict
// free) in register phases of RB bits.  The next tile's loads are issued before
// the phases, so that they are in flight while the phases run.
//   Bounds: HBM (one read) against 2 FP64 multiply-adds per amplitude and flip
// and (phases + 1) shared-memory moves of the tile.  Sums of |a|^2 cost one
// square per amplitude for all bits: the bits above the tile take a warp's
// total once per tile (lane l keeps the sum of bit l of the tile index).
//   27 qubits complex<double> (2 GiB): energy of 27 ZZ and 27 X strings with all
// spins 19.1 -> 3.5 ms; before, 28 reads of 0.45 ms, one per flip mask and each
// waited for, and four spin reads of 0.59 ms.
// A tile is 2^11 amplitudes for both precisions: with 16 amplitudes a thread
// (complex<float>) the sums of 12 bits and the two register copies spilled.
// Phase p's registers and thread bits, one hexadecimal digit per tile bit,
// lowest first (lanes 0-2 of every layout reach distinct bank groups of the
// swizzled slots for complex<double>); own: how many of its registers' flips
// belong to the phase.
struct observe_shape {
  static constexpr int RB = kObserveRegBits, K = 8 + RB, NE = 1 << RB, PHASES = 4;
  static __host__ __device__ constexpr int reg(int p, int k) { return ((p == 0 ? 0xA98 : p == 1 ? 0x210 : p == 2 ? 0x043 : 0x765) >> (4 * k)) & 15; }
  static __host__ __device__ constexpr int own(int p) { return p == 2 ? 2 : 3; }
  static __host__ __device__ constexpr int thr(int p, int b)
  {
    return ((p == 0 ? 0x76543210u : p == 1 ? 0x765A9843u : p == 2 ? 0x765A8921u : 0xA9843210u) >> (4 * b)) & 15;
  }
};

// The flips that belong to phase P from a thread's registers.
template <typename Real, int P>
__device__ __forceinline__ void observe_flips(const typename ctype<Real>::c (&e)[observe_shape::NE], int mask,
                                              double (&xr)[observe_shape::K], double (&xi)[observe_shape::K])
{
  using SH = observe_shape;
#pragma unroll
  for (int k = 0; k < SH::own(P); ++k) {
    const int f = SH::reg(P, k);
    if ((mask >> f) & 1) {
#pragma unroll
      for (int i = 0; i < (1 << SH::RB); ++i) {
        if ((i >> k) & 1) continue;
        const auto u = e[i], w = e[i | (1 << k)];
        xr[f] = __fma_rn(double(u.x), double(w.x), __fma_rn(double(u.y), double(w.y), xr[f]));
        xi[f] = __fma_rn(double(u.x), double(w.y), __fma_rn(-double(u.y), double(w.x), xi[f]));
      }
    }
  }
}

// Phase P and those after it, each reading the tile in its layout.
template <typename Real, int P>
__device__ __forceinline__ void observe_phases(const typename ctype<Real>::c* tile, int mask, double (&xr)[observe_shape::K],
                                               double (&xi)[observe_shape::K])
{
  using SH = observe_shape;
  constexpr int VB = precision_traits<Real>::VB, RB = SH::RB, NE = 1 << RB;
  if constexpr (P < SH::PHASES) {
    int mine = 0;
#pragma unroll
    for (int k = 0; k < SH::own(P); ++k) mine |= 1 << SH::reg(P, k);
    if (mask & mine) {
      uint32_t j = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) j |= ((threadIdx.x >> b) & 1u) << SH::thr(P, b);
      const uint32_t sb = smem_slot<VB>(j);
      typename ctype<Real>::c e[NE];
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        uint32_t sidx = sb;
#pragma unroll
        for (int k = 0; k < RB; ++k)
          if ((i >> k) & 1) sidx ^= smem_slot<VB>(1u << SH::reg(P, k));
        e[i] = tile[sidx];
      }
      observe_flips<Real, P>(e, mask, xr, xi);
    }
    observe_phases<Real, P + 1>(tile, mask, xr, xi);
  }
}

template <typename Real, bool ZSUMS, bool DIAG>
__global__ void __launch_bounds__(kRedThreads, 2)
observe_kernel(const typename ctype<Real>::c* __restrict__ a, int n, const __grid_constant__ observe_group S, uint64_t num_tiles,
               double* partials)
{
  using C = typename ctype<Real>::c;
  using SH = observe_shape;
  constexpr int VB = precision_traits<Real>::VB, RB = SH::RB, NE = 1 << RB, K = 8 + RB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tile = reinterpret_cast<C*>(smem_raw);
  const uint32_t tid = threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t tphys = 0;
  for (int b = 0; b < 8; ++b) tphys |= uint64_t((tid >> b) & 1u) << S.tile_phys[b];
  auto tile_base = [&](uint64_t t) {
    uint64_t base = 0;
    for (int r = 0; r < S.num_runs; ++r) base |= ((t >> S.run_src[r]) & ((1ull << S.run_len[r]) - 1)) << S.run_dst[r];
    return base;
  };
  auto load = [&](uint64_t t, C (&v)[NE]) {
    const uint64_t base = tile_base(t) | tphys;
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      uint64_t p = base;
#pragma unroll
      for (int b = 0; b < RB; ++b)
        if ((i >> b) & 1) p |= 1ull << S.tile_phys[8 + b];
      v[i] = __ldcs(a + p);
    }
  };
  // Parity of every diagonal string on this thread's tile bits, one bit per string.
  uint64_t tpar = 0;
  for (int k = 0; DIAG && k < S.diag_terms; ++k) tpar |= uint64_t(__popcll(tphys & S.sign[k]) & 1) << k;
  const bool flips_any = S.flip_mask != 0;
  double xr[K], xi[K];
#pragma unroll
  for (int f = 0; f < K; ++f) xr[f] = xi[f] = 0.0;
  double total = 0.0, zreg[RB], zout = 0.0, dsum = 0.0;
#pragma unroll
  for (int b = 0; b < RB; ++b) zreg[b] = 0.0;

  C v[NE];
  if (blockIdx.x < num_tiles) load(blockIdx.x, v);
  for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x) {
    if constexpr (ZSUMS || DIAG) {
      double c[NE];
      if constexpr (DIAG) {
        // Parities of the strings on the bits outside the tile, lane k string k (and k + 32), then
        // per register pattern the classes' weights; a Walsh transform turns the patterns into W.
        const uint64_t base = tile_base(t);
        const uint32_t p0 = __ballot_sync(0xffffffffu, lane < S.diag_terms && (__popcll(base & S.sign[lane]) & 1));
        const uint32_t p1 = __ballot_sync(0xffffffffu, lane + 32 < S.diag_terms && (__popcll(base & S.sign[lane + 32]) & 1));
        const uint64_t par = tpar ^ ((uint64_t(p1) << 32) | p0);
#pragma unroll
        for (int p = 0; p < NE; ++p) {
          double w = 0.0;
          for (int k = S.class_begin[p]; k < S.class_begin[p + 1]; ++k)
            w = __fma_rn(S.class_w[k], double(__popcll(S.class_mask[k]) - 2 * __popcll(par & S.class_mask[k])), w);
          c[p] = w;
        }
#pragma unroll
        for (int b = 0; b < RB; ++b)
#pragma unroll
          for (int i = 0; i < NE; ++i) {
            if ((i >> b) & 1) continue;
            const double s0 = c[i], s1 = c[i | (1 << b)];
            c[i] = s0 + s1;
            c[i | (1 << b)] = s0 - s1;
          }
      }
      double tot = 0.0;
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const double p = double(v[i].x) * double(v[i].x) + double(v[i].y) * double(v[i].y);
        if constexpr (DIAG) dsum = __fma_rn(p, c[i], dsum);
        if constexpr (ZSUMS) {
          tot += p;
#pragma unroll
          for (int b = 0; b < RB; ++b)
            if ((i >> b) & 1) zreg[b] += p;
        }
      }
      if constexpr (ZSUMS) {
        total += tot;
        const double w = warp_sum(tot);
        if ((t >> lane) & 1) zout += w;
      }
    }
    observe_flips<Real, 0>(v, S.flip_mask, xr, xi);
    const bool more = t + gridDim.x < num_tiles;
    if (flips_any) {
      __syncthreads();  // the previous tile is no longer read
#pragma unroll
      for (int i = 0; i < NE; ++i) tile[smem_slot<VB>(tid) ^ smem_slot<VB>(uint32_t(i) << 8)] = v[i];
      __syncthreads();
    }
    if (more) load(t + gridDim.x, v);
    observe_phases<Real, 1>(tile, S.flip_mask, xr, xi);
  }
  // Block sums in a fixed order, one output column after the other.
  constexpr int COLS = 2 * K + 1 + kMaxQubits + 1;
  __shared__ double red[kRedThreads / 32][COLS];
  int col = 0;
#pragma unroll
  for (int f = 0; f < K; ++f) {
    if ((S.flip_mask >> f) & 1) {
      const double a0 = warp_sum(xr[f]), a1 = warp_sum(xi[f]);
      if (lane == 0) { red[warp][col] = a0; red[warp][col + 1] = a1; }
      col += 2;
    }
  }
  if constexpr (ZSUMS) {
    // Column 1 + q: the physical bit q of thread bits, register bits, then tile-index bits.
    const double tt = warp_sum(total);
    if (lane == 0) red[warp][col] = tt;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const double z = warp_sum(((tid >> b) & 1u) ? total : 0.0);
      if (lane == 0) red[warp][col + 1 + S.tile_phys[b]] = z;
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const double z = warp_sum(zreg[b]);
      if (lane == 0) red[warp][col + 1 + S.tile_phys[8 + b]] = z;
    }
    for (int r = 0; r < S.num_runs; ++r)
      if (lane >= S.run_src[r] && lane < S.run_src[r] + S.run_len[r])
        red[warp][col + 1 + S.run_dst[r] + (lane - S.run_src[r])] = zout;
    col += 1 + n;
  }
  if constexpr (DIAG) {
    const double d = warp_sum(dsum);
    if (lane == 0) red[warp][col] = d;
    col += 1;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < col; k += blockDim.x) {
    double acc = 0.0;
    for (int w = 0; w < kRedThreads / 32; ++w) acc += red[w][k];
    partials[size_t(blockIdx.x) * col + k] = acc;
  }
}

// launch_observe_small: one block per sum, each reading the state from L2, no
// partial sums and no second launch.  The sums of a state in one CTA's shared
// memory, a warp for each, took two rounds of 16 warps and ended at 11 qubits; with
// two observe_kernel launches spins of 12 qubits in complex<float> took 44.8 us,
// 31 here (35 with one tile of 2^12 amplitudes); energies of 11 and fewer gain too.
constexpr int kSmallThreads = 256;
template <typename Real>
__global__ void __launch_bounds__(kSmallThreads)
observe_small_kernel(const typename ctype<Real>::c* __restrict__ a, int n, const __grid_constant__ pauli_terms T,
                     double* __restrict__ out)
{
  const uint32_t size = 1u << n;
  const int w = blockIdx.x;
  double v[2] = {0.0, 0.0};
  if (w < n) {  // x_b of bit b = w
    for (uint32_t k = threadIdx.x; k < size / 2; k += kSmallThreads) {
      const uint32_t i = uint32_t(insert_zero(k, w));
      const auto x = a[i], y = a[i | (1u << w)];
      v[0] += double(x.x) * double(y.x) + double(x.y) * double(y.y);
      v[1] += double(x.x) * double(y.y) - double(x.y) * double(y.x);
    }
  } else {  // the plain sum (n), the sum over bit b set (n + 1 + b), the diagonal strings (2 n + 1)
    const uint32_t need = w > n && w <= 2 * n ? 1u << (w - n - 1) : 0u;
    for (uint32_t i = threadIdx.x; i < size; i += kSmallThreads) {
      if ((i & need) != need) continue;
      const auto x = a[i];
      const double p = double(x.x) * double(x.x) + double(x.y) * double(x.y);
      double f = 1.0;
      if (w == 2 * n + 1) {
        f = 0.0;
        for (int t = 0; t < T.count; ++t) f += (__popc(i & uint32_t(T.sign[t])) & 1) ? -T.w[t][0] : T.w[t][0];
      }
      v[0] += p * f;
    }
  }
  __shared__ double red[kSmallThreads / 32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double re = warp_sum(v[0]), im = warp_sum(v[1]);
  if (lane == 0) { red[warp][0] = re; red[warp][1] = im; }
  __syncthreads();
  if (threadIdx.x < 2) {
    double s = 0.0;
    for (int k = 0; k < kSmallThreads / 32; ++k) s += red[k][threadIdx.x];
    if (w < n) out[2 * w + threadIdx.x] = s;
    else if (threadIdx.x == 0) out[n + w] = s;
  }
}

// <b| P |a> summed over Pauli strings sharing one flip mask F:
//   out = sum_i conj(b_i) a_{i^F} W(i),  W(i) = sum_t w_t (-1)^popcount(i & s_t)
// ((P a)_i = coeff(i) a_{i^F}, ket/include/ket/gate/utility/pauli_index_coeff.hpp:17-59).
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
pauli2_kernel(const typename ctype<Real>::c* __restrict__ a, const typename ctype<Real>::c* __restrict__ b, int n,
              uint64_t flip, const pauli_terms T, double* partials)
{
  const uint64_t size = 1ull << n;
  double re = 0, im = 0;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < size; i += stride) {
    const auto x = a[i ^ flip], y = b[i];
    // c = conj(b_i) a_{i^F}
    const double cr = double(y.x) * double(x.x) + double(y.y) * double(x.y);
    const double ci = double(y.x) * double(x.y) - double(y.y) * double(x.x);
    double wr = 0, wi = 0;
    for (int t = 0; t < T.count; ++t) {
      const double s = (__popcll(i & T.sign[t]) & 1) ? -1.0 : 1.0;
      wr += s * T.w[t][0];
      wi += s * T.w[t][1];
    }
    re += cr * wr - ci * wi;
    im += cr * wi + ci * wr;
  }
  double vals[2] = {re, im};
  block_sum_store<2>(vals, 2, partials + size_t(blockIdx.x) * 2);
}

// <b|a> = sum conj(b_i) a_i
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
inner_kernel(const typename ctype<Real>::c* __restrict__ a, const typename ctype<Real>::c* __restrict__ b,
             uint64_t size, double* partials)
{
  double re = 0, im = 0;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < size; i += stride) {
    const auto x = a[i], y = b[i];
    re += double(y.x) * double(x.x) + double(y.y) * double(x.y);
    im += double(y.x) * double(x.y) - double(y.y) * double(x.x);
  }
  double vals[2] = {re, im};
  block_sum_store<2>(vals, 2, partials + size_t(blockIdx.x) * 2);
}

// |a_i|^2 for i in [offset, offset + count) (physical order).
template <typename Real>
__global__ void probs_kernel(const typename ctype<Real>::c* __restrict__ a, uint64_t offset, uint64_t count, double* out)
{
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < count; i += stride) {
    const auto v = a[offset + i];
    out[i] = double(v.x) * double(v.x) + double(v.y) * double(v.y);
  }
}

int reduction_blocks() { return 148 * 4; }

// Blocks for a reduction over 2^n items: no more than there are items for.
static int reduction_blocks_for(int n)
{
  return n >= 18 ? reduction_blocks() : std::min(reduction_blocks(), std::max(1, 1 << std::max(0, n - 8)));
}

template <typename Real>
cudaError_t launch_zsum(const void* state, int n, double* partials, double* out, cudaStream_t stream)
{
  const int blocks = zsum_blocks(n);
  zsum_kernel<Real><<<blocks, kRedThreads, 0, stream>>>(static_cast<const typename ctype<Real>::c*>(state), n, partials);
  finish_partials_kernel<<<n + 1, kFinishThreads, 0, stream>>>(partials, blocks, n + 1, out);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_pauli(const void* state, int n, uint64_t flip, const pauli_terms& terms, double* partials, double* out, cudaStream_t stream)
{
  const int blocks = reduction_blocks_for(n);
  pauli_kernel<Real><<<blocks, kRedThreads, 0, stream>>>(static_cast<const typename ctype<Real>::c*>(state), n, flip, terms, partials);
  finish_partials_kernel<<<2, kFinishThreads, 0, stream>>>(partials, blocks, 2, out);
  return cudaGetLastError();
}

int observe_width(const observe_group& g, int n)
{
  return 2 * __builtin_popcount(static_cast<unsigned>(g.flip_mask)) + (g.zsums ? 1 + n : 0) + (g.diag_classes > 0 ? 1 : 0);
}

template <typename Real, bool ZSUMS, bool DIAG>
static cudaError_t launch_observe_form(const typename ctype<Real>::c* state, int n, const observe_group& g, uint64_t tiles,
                                       int blocks, double* partials, cudaStream_t stream)
{
  const size_t smem = sizeof(typename ctype<Real>::c) << g.K;
  static std::atomic<bool> configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(observe_kernel<Real, ZSUMS, DIAG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  observe_kernel<Real, ZSUMS, DIAG><<<blocks, kRedThreads, smem, stream>>>(state, n, g, tiles, partials);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_observe(const void* state, int n, const observe_group& g, double* partials, double* out, cudaStream_t stream)
{
  constexpr int K = 8 + observe_shape::RB;
  const int width = observe_width(g, n);
  if (g.K != K || K > n || n - K > 32 || n > kMaxQubits || (g.flip_mask >> K) != 0 || width < 1 ||
      (g.zsums && g.diag_classes > 0) || g.diag_terms < 0 ||
      g.diag_terms > kObserveTerms || g.diag_classes < 0 || g.diag_classes > kObserveTerms)
    return cudaErrorInvalidValue;
  const uint64_t tiles = 1ull << (n - K);
  const int blocks = static_cast<int>(std::min<uint64_t>(tiles, 148 * 2));
  const auto* a = static_cast<const typename ctype<Real>::c*>(state);
  const cudaError_t e = g.diag_classes > 0 ? launch_observe_form<Real, false, true>(a, n, g, tiles, blocks, partials, stream)
                        : g.zsums          ? launch_observe_form<Real, true, false>(a, n, g, tiles, blocks, partials, stream)
                                           : launch_observe_form<Real, false, false>(a, n, g, tiles, blocks, partials, stream);
  if (e != cudaSuccess) return e;
  finish_partials_kernel<<<width, kFinishThreads, 0, stream>>>(partials, blocks, width, out);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_observe_small(const void* state, int n, const pauli_terms& terms, double* out, cudaStream_t stream)
{
  if (n < 1 || n > kObserveSmallBits || terms.count < 0 || terms.count > kMaxPauliTerms) return cudaErrorInvalidValue;
  observe_small_kernel<Real><<<2 * n + 2, kSmallThreads, 0, stream>>>(
    static_cast<const typename ctype<Real>::c*>(state), n, terms, out);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_pauli2(const void* a, const void* b, int n, uint64_t flip, const pauli_terms& terms, double* partials,
                          double* out, cudaStream_t stream)
{
  const int blocks = reduction_blocks_for(n);
  pauli2_kernel<Real><<<blocks, kRedThreads, 0, stream>>>(static_cast<const typename ctype<Real>::c*>(a),
                                                          static_cast<const typename ctype<Real>::c*>(b), n, flip, terms, partials);
  finish_partials_kernel<<<2, kFinishThreads, 0, stream>>>(partials, blocks, 2, out);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_inner(const void* a, const void* b, int n, double* partials, double* out, cudaStream_t stream)
{
  const int blocks = reduction_blocks_for(n);
  inner_kernel<Real><<<blocks, kRedThreads, 0, stream>>>(static_cast<const typename ctype<Real>::c*>(a),
                                                         static_cast<const typename ctype<Real>::c*>(b), 1ull << n, partials);
  finish_partials_kernel<<<2, kFinishThreads, 0, stream>>>(partials, blocks, 2, out);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_probs(const void* state, uint64_t offset, uint64_t count, double* out, cudaStream_t stream)
{
  probs_kernel<Real><<<grid_for(count, 256), 256, 0, stream>>>(static_cast<const typename ctype<Real>::c*>(state), offset, count, out);
  return cudaGetLastError();
}

template cudaError_t launch_zsum<double>(const void*, int, double*, double*, cudaStream_t);
template cudaError_t launch_zsum<float>(const void*, int, double*, double*, cudaStream_t);
template cudaError_t launch_pauli<double>(const void*, int, uint64_t, const pauli_terms&, double*, double*, cudaStream_t);
template cudaError_t launch_pauli<float>(const void*, int, uint64_t, const pauli_terms&, double*, double*, cudaStream_t);
template cudaError_t launch_observe<double>(const void*, int, const observe_group&, double*, double*, cudaStream_t);
template cudaError_t launch_observe<float>(const void*, int, const observe_group&, double*, double*, cudaStream_t);
template cudaError_t launch_observe_small<double>(const void*, int, const pauli_terms&, double*, cudaStream_t);
template cudaError_t launch_observe_small<float>(const void*, int, const pauli_terms&, double*, cudaStream_t);
template cudaError_t launch_pauli2<double>(const void*, const void*, int, uint64_t, const pauli_terms&, double*, double*, cudaStream_t);
template cudaError_t launch_pauli2<float>(const void*, const void*, int, uint64_t, const pauli_terms&, double*, double*, cudaStream_t);
template cudaError_t launch_inner<double>(const void*, const void*, int, double*, double*, cudaStream_t);
template cudaError_t launch_inner<float>(const void*, const void*, int, double*, double*, cudaStream_t);
template cudaError_t launch_probs<double>(const void*, uint64_t, uint64_t, double*, cudaStream_t);
template cudaError_t launch_probs<float>(const void*, uint64_t, uint64_t, double*, cudaStream_t);

}  // namespace rbk

namespace rbk {

// ---------------------------------------------------------------------------
// Adjoint-gradient helpers
// ---------------------------------------------------------------------------

// dst_i = sum_g sum_{t in g} w_t (-1)^popcount(i & sign_t) src_{i ^ flip_g}
// (a Pauli-string sum applied to a state; pauli_index_coeff.hpp:17-59 form).
template <typename Real>
__global__ void pauli_apply_kernel(const typename ctype<Real>::c* __restrict__ src, typename ctype<Real>::c* __restrict__ dst,
                                   uint64_t size, const pauli_sum P)
{
  using C = typename ctype<Real>::c;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < size; i += stride) {
    double re = 0, im = 0;
    for (int g = 0; g < P.num_groups; ++g) {
      const C v = src[i ^ P.flip[g]];
      double wr = 0, wi = 0;
      for (int t = P.begin[g]; t < P.begin[g + 1]; ++t) {
        const double s = (__popcll(i & P.sign[t]) & 1) ? -1.0 : 1.0;
        wr += s * P.w[t][0];
        wi += s * P.w[t][1];
      }
      re += wr * double(v.x) - wi * double(v.y);
      im += wr * double(v.y) + wi * double(v.x);
    }
    dst[i] = C{(Real)re, (Real)im};
  }
}

template <typename Real>
cudaError_t launch_pauli_apply(const void* src, void* dst, int n, const pauli_sum& P, cudaStream_t stream)
{
  const uint64_t size = 1ull << n;
  pauli_apply_kernel<Real><<<grid_for(size, 256), 256, 0, stream>>>(
    static_cast<const typename ctype<Real>::c*>(src), static_cast<typename ctype<Real>::c*>(dst), size, P);
  return cudaGetLastError();
}

// One pass of launch_pauli_apply_tiled: tile bits tile_phys[0..10] (the block
// index deposited run by run into the other bits), the pass's groups as tile
// masks of their flips and their terms.
constexpr int kTileSumTerms = 96;
constexpr int kTileSumBits = 11;
// pair_group >= 0: that group's terms are all two-bit Z-type strings with one
// real weight pw (ZZ couplings), and its weight at j is
//   pw * (count - 2 * (number of pairs with odd parity at j)),
// the pairs on adjacent bits counted at once as popcount((j ^ j >> 1) & madj)
// and the others one by one from other[].
constexpr int kTilePairOthers = 16;
struct pauli_tile_pass {
  int32_t num_groups, first;
  uint8_t tile_phys[16], num_runs, run_src[16], run_len[16], run_dst[16];
  uint8_t begin[kMaxSumGroups + 1];
  uint16_t flip_local[kMaxSumGroups];
  uint64_t sign[kTileSumTerms];
  double w[kTileSumTerms][2];
  int32_t pair_group, pair_count, num_others, pad;
  double pw;
  uint64_t madj;
  uint8_t other[kTilePairOthers][2];
};

// Persistent CTAs, one tile of src at a time in shared memory; thread t holds
// tile indices t + 256 it (it = 0..7), whose partners j ^ flip it reads from
// the tile.  dst is written (first pass) or accumulated, in place.  The groups
// run in the outer loop, so that a group's constants are fetched once for the
// thread's 8 amplitudes: with the amplitudes outside, indexed constant loads kept
// their pipe 70 % busy: three terms of 23 qubits in complex<float>
// took 176 us each, now 70; of 20 qubits in complex<double> 27 us, now 13.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads, 2)
pauli_apply_tile_kernel(const typename ctype<Real>::c* __restrict__ src, typename ctype<Real>::c* __restrict__ dst,
                        const __grid_constant__ pauli_tile_pass T, uint64_t num_tiles)
{
  using C = typename ctype<Real>::c;
  constexpr int NE = 1 << (kTileSumBits - 8);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tile = reinterpret_cast<C*>(smem_raw);
  const uint32_t tid = threadIdx.x;
  uint64_t tphys = 0;
  for (int b = 0; b < 8; ++b) tphys |= uint64_t((tid >> b) & 1u) << T.tile_phys[b];
  for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x) {
    uint64_t base = tphys;
    for (int r = 0; r < T.num_runs; ++r) base |= ((t >> T.run_src[r]) & ((1ull << T.run_len[r]) - 1)) << T.run_dst[r];
    uint64_t phys[NE];
#pragma unroll
    for (int it = 0; it < NE; ++it) {
      phys[it] = base;
#pragma unroll
      for (int b = 0; b < kTileSumBits - 8; ++b)
        if ((it >> b) & 1) phys[it] |= 1ull << T.tile_phys[8 + b];
    }
    // Both loads of the tile issued together: src, and the dst the pass adds to
    // (read here, before any store to dst, so that the loads stay in flight at once).
    C v[NE], d[NE];
#pragma unroll
    for (int it = 0; it < NE; ++it) v[it] = __ldcs(src + phys[it]);
    if (!T.first) {
#pragma unroll
      for (int it = 0; it < NE; ++it) d[it] = __ldcs(dst + phys[it]);
    }
    __syncthreads();  // the previous tile is no longer read
#pragma unroll
    for (int it = 0; it < NE; ++it) tile[tid | (uint32_t(it) << 8)] = v[it];
    __syncthreads();
    double re[NE], im[NE];
#pragma unroll
    for (int it = 0; it < NE; ++it) {
      re[it] = T.first ? 0.0 : double(d[it].x);
      im[it] = T.first ? 0.0 : double(d[it].y);
    }
    for (int g = 0; g < T.num_groups; ++g) {
      const uint32_t fl = T.flip_local[g];
      const int t0 = T.begin[g], t1 = T.begin[g + 1];
      if (t1 == t0 + 1 && T.sign[t0] == 0) {  // one term, no sign bits: a constant weight
        const double wr = T.w[t0][0], wi = T.w[t0][1];
        if (wi == 0.0) {
#pragma unroll
          for (int it = 0; it < NE; ++it) {
            const C a = tile[(tid | (uint32_t(it) << 8)) ^ fl];
            re[it] = __fma_rn(wr, double(a.x), re[it]);
            im[it] = __fma_rn(wr, double(a.y), im[it]);
          }
          continue;
        }
#pragma unroll
        for (int it = 0; it < NE; ++it) {
          const C a = tile[(tid | (uint32_t(it) << 8)) ^ fl];
          re[it] += wr * double(a.x) - wi * double(a.y);
          im[it] += wr * double(a.y) + wi * double(a.x);
        }
      } else if (g == T.pair_group) {
        const double pw = T.pw;
        int odd[NE];
#pragma unroll
        for (int it = 0; it < NE; ++it) odd[it] = __popcll((phys[it] ^ (phys[it] >> 1)) & T.madj);
        for (int k = 0; k < T.num_others; ++k) {
          const int b0 = T.other[k][0], b1 = T.other[k][1];
#pragma unroll
          for (int it = 0; it < NE; ++it) odd[it] += int(((phys[it] >> b0) ^ (phys[it] >> b1)) & 1);
        }
#pragma unroll
        for (int it = 0; it < NE; ++it) {
          const C a = tile[tid | (uint32_t(it) << 8)];  // the diagonal group: no flip
          const double w = pw * double(T.pair_count - 2 * odd[it]);
          re[it] = __fma_rn(w, double(a.x), re[it]);
          im[it] = __fma_rn(w, double(a.y), im[it]);
        }
      } else {
        double wr[NE], wi[NE];
#pragma unroll
        for (int it = 0; it < NE; ++it) wr[it] = wi[it] = 0.0;
        for (int k = t0; k < t1; ++k) {
          const uint64_t sign = T.sign[k];
          const double w0 = T.w[k][0], w1 = T.w[k][1];
#pragma unroll
          for (int it = 0; it < NE; ++it) {
            const bool neg = __popcll(phys[it] & sign) & 1;
            wr[it] += neg ? -w0 : w0;
            wi[it] += neg ? -w1 : w1;
          }
        }
#pragma unroll
        for (int it = 0; it < NE; ++it) {
          const C a = tile[(tid | (uint32_t(it) << 8)) ^ fl];
          re[it] += wr[it] * double(a.x) - wi[it] * double(a.y);
          im[it] += wr[it] * double(a.y) + wi[it] * double(a.x);
        }
      }
    }
#pragma unroll
    for (int it = 0; it < NE; ++it) v[it] = C{(Real)re[it], (Real)im[it]};
#pragma unroll
    for (int it = 0; it < NE; ++it) __stcs(dst + phys[it], v[it]);
  }
}

template <typename Real>
cudaError_t launch_pauli_apply_tiled(const void* src, void* dst, int n, const pauli_sum& P, cudaStream_t stream)
{
  constexpr int LOWB = 3, FREE = kTileSumBits - LOWB;
  if (n < kTileSumBits || n > 63) return launch_pauli_apply<Real>(src, dst, n, P, stream);
  // Group the flips into layouts: each layout's high bits (>= LOWB) number at most FREE.
  std::vector<std::vector<int>> passes;
  std::vector<uint64_t> highs;
  int diag = -1;
  for (int g = 0; g < P.num_groups; ++g) {
    const uint64_t f = P.flip[g];
    if (f == 0) { diag = g; continue; }
    const uint64_t hb = f & ~((1ull << LOWB) - 1);
    if (__builtin_popcountll(hb) > FREE) return launch_pauli_apply<Real>(src, dst, n, P, stream);
    bool placed = false;
    for (size_t q = 0; q < passes.size() && !placed; ++q) {
      int terms = 0;
      for (int h : passes[q]) terms += P.begin[h + 1] - P.begin[h];
      if (__builtin_popcountll(highs[q] | hb) <= FREE && terms + (P.begin[g + 1] - P.begin[g]) <= kTileSumTerms &&
          static_cast<int>(passes[q].size()) < kMaxSumGroups) {
        passes[q].push_back(g);
        highs[q] |= hb;
        placed = true;
      }
    }
    if (!placed) { passes.push_back({g}); highs.push_back(hb); }
  }
  if (passes.empty()) { passes.push_back({}); highs.push_back(0); }
  if (diag >= 0) {
    int terms = P.begin[diag + 1] - P.begin[diag];
    for (int h : passes[0]) terms += P.begin[h + 1] - P.begin[h];
    if (terms > kTileSumTerms) return launch_pauli_apply<Real>(src, dst, n, P, stream);
    passes[0].insert(passes[0].begin(), diag);
  }
  static std::atomic<bool> configured[64] = {};
  const size_t smem = sizeof(typename ctype<Real>::c) << kTileSumBits;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(pauli_apply_tile_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const uint64_t tiles = 1ull << (n - kTileSumBits);
  const int blocks = static_cast<int>(std::min<uint64_t>(tiles, uint64_t(sms) * 4));
  for (size_t q = 0; q < passes.size(); ++q) {
    pauli_tile_pass T{};
    T.first = q == 0 ? 1 : 0;
    std::vector<int> bits;
    for (int b = 0; b < LOWB; ++b) bits.push_back(b);
    for (int b = LOWB; b < n; ++b)
      if ((highs[q] >> b) & 1) bits.push_back(b);
    for (int b = LOWB; static_cast<int>(bits.size()) < kTileSumBits; ++b)  // fillers
      if (!((highs[q] >> b) & 1)) bits.push_back(b);
    std::sort(bits.begin(), bits.end());
    uint64_t mask = 0;
    for (int b = 0; b < kTileSumBits; ++b) { T.tile_phys[b] = static_cast<uint8_t>(bits[static_cast<size_t>(b)]); mask |= 1ull << bits[static_cast<size_t>(b)]; }
    int runs = 0, srcb = 0;
    for (int b = 0; b < n;) {
      if ((mask >> b) & 1) { ++b; continue; }
      int len = 0;
      while (b + len < n && !((mask >> (b + len)) & 1)) ++len;
      T.run_src[runs] = static_cast<uint8_t>(srcb);
      T.run_len[runs] = static_cast<uint8_t>(len);
      T.run_dst[runs] = static_cast<uint8_t>(b);
      ++runs;
      srcb += len;
      b += len;
    }
    T.num_runs = static_cast<uint8_t>(runs);
    int k = 0;
    T.num_groups = static_cast<int>(passes[q].size());
    for (int gi = 0; gi < T.num_groups; ++gi) {
      const int g = passes[q][static_cast<size_t>(gi)];
      uint32_t fl = 0;
      for (int b = 0; b < kTileSumBits; ++b)
        if ((P.flip[g] >> T.tile_phys[b]) & 1) fl |= 1u << b;
      T.flip_local[gi] = static_cast<uint16_t>(fl);
      T.begin[gi] = static_cast<uint8_t>(k);
      for (int t = P.begin[g]; t < P.begin[g + 1]; ++t, ++k) {
        T.sign[k] = P.sign[t];
        T.w[k][0] = P.w[t][0];
        T.w[k][1] = P.w[t][1];
      }
    }
    T.begin[T.num_groups] = static_cast<uint8_t>(k);
    // The ZZ-coupling form of the diagonal group, where it applies.
    T.pair_group = -1;
    if (q == 0 && diag >= 0 && P.begin[diag + 1] > P.begin[diag]) {
      const int t0 = P.begin[diag], t1 = P.begin[diag + 1];
      bool pairs = true;
      uint64_t madj = 0;
      int others = 0;
      for (int t = t0; t < t1 && pairs; ++t) {
        const uint64_t sg = P.sign[t];
        pairs = __builtin_popcountll(sg) == 2 && P.w[t][1] == 0.0 && P.w[t][0] == P.w[t0][0];
        if (!pairs) break;
        const int a = __builtin_ctzll(sg), b = 63 - __builtin_clzll(sg);
        if (b == a + 1 && !((madj >> a) & 1)) {
          madj |= 1ull << a;
        } else if (others < kTilePairOthers) {
          T.other[others][0] = static_cast<uint8_t>(a);
          T.other[others][1] = static_cast<uint8_t>(b);
          ++others;
        } else {
          pairs = false;
        }
      }
      if (pairs) {
        T.pair_group = 0;  // the diagonal group is the pass's first
        T.pair_count = t1 - t0;
        T.pw = P.w[t0][0];
        T.madj = madj;
        T.num_others = others;
      }
    }
    pauli_apply_tile_kernel<Real><<<blocks, kRedThreads, smem, stream>>>(
      static_cast<const typename ctype<Real>::c*>(src), static_cast<typename ctype<Real>::c*>(dst), T, tiles);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
template cudaError_t launch_pauli_apply_tiled<double>(const void*, void*, int, const pauli_sum&, cudaStream_t);
template cudaError_t launch_pauli_apply_tiled<float>(const void*, void*, int, const pauli_sum&, cudaStream_t);

// Several overlaps in one launch: blockIdx.y selects the Pauli of overlap y;
// partials of overlap y sit at partials[(y * gridDim.x + x) * 2].
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
overlaps_kernel(const typename ctype<Real>::c* __restrict__ lam, const typename ctype<Real>::c* __restrict__ psi,
                uint64_t size, const __grid_constant__ overlap_set S, double* partials)
{
  const overlap_spec P = S.spec[blockIdx.y];
  double re = 0, im = 0;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < size; i += stride) {
    const auto l = lam[i], p = psi[i ^ P.flip];
    const double s = (__popcll(i & P.sign) & 1) ? -1.0 : 1.0;
    const double cr = double(l.x) * double(p.x) + double(l.y) * double(p.y);
    const double ci = double(l.x) * double(p.y) - double(l.y) * double(p.x);
    re += s * (cr * P.wr - ci * P.wi);
    im += s * (cr * P.wi + ci * P.wr);
  }
  double vals[2] = {re, im};
  block_sum_store<2>(vals, 2, partials + (size_t(blockIdx.y) * gridDim.x + blockIdx.x) * 2);
}

// Sum of the (re, im) partials p[0..blocks) by one warp: lane l takes blocks
// l, l + 32, ... in order, then a fixed butterfly adds the lanes.  The order is
// the same on every run; the loads of a lane are independent, so the sum costs
// a few L2 round trips instead of one per block.
__device__ __forceinline__ double2 warp_sum_partials(const double* __restrict__ p, int blocks)
{
  const int lane = threadIdx.x & 31;
  double re = 0, im = 0;
  for (int b = lane; b < blocks; b += 32) {
    re += p[2 * b];
    im += p[2 * b + 1];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
  }
  return make_double2(re, im);
}

// out[2y], out[2y+1] = sum over the partials of overlap y (one warp per overlap).
__global__ void finish_overlaps_kernel(const double* __restrict__ partials, int blocks, double* __restrict__ out)
{
  const double2 v = warp_sum_partials(partials + size_t(blockIdx.x) * blocks * 2, blocks);
  if (threadIdx.x == 0) {
    out[2 * blockIdx.x] = v.x;
    out[2 * blockIdx.x + 1] = v.y;
  }
}

size_t overlaps_partials_doubles() { return size_t(reduction_blocks()) * 2 * kMaxOverlaps; }

template <typename Real>
cudaError_t launch_overlaps(const void* lam, const void* psi, int n, const overlap_set& set, double* partials, double* out,
                            cudaStream_t stream)
{
  if (set.count < 1 || set.count > kMaxOverlaps) return cudaErrorInvalidValue;
  const int blocks = reduction_blocks();
  overlaps_kernel<Real><<<dim3(blocks, set.count), kRedThreads, 0, stream>>>(
    static_cast<const typename ctype<Real>::c*>(lam), static_cast<const typename ctype<Real>::c*>(psi), 1ull << n, set,
    partials);
  finish_overlaps_kernel<<<set.count, 32, 0, stream>>>(partials, blocks, out);
  return cudaGetLastError();
}
// Tiled form: CTA b stages the tile of psi and lambda whose bits outside
// T.tile_phys spell b (as a fused pass does) and evaluates every overlap of
// the set whose flip bit is a tile bit, reading each state once for the whole
// set instead of once per overlap.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
tile_overlaps_kernel(const typename ctype<Real>::c* __restrict__ lam, const typename ctype<Real>::c* __restrict__ psi,
                     const __grid_constant__ tile_overlap_set T, double* partials)
{
  using C = typename ctype<Real>::c;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* ps = reinterpret_cast<C*>(smem_raw);
  C* ls = ps + (1u << T.K);
  __shared__ double red[kMaxOverlaps][kRedThreads / 32][2];
  const uint32_t tile = 1u << T.K;
  uint64_t base = 0;
  {
    const uint64_t b = blockIdx.x;
    for (int r = 0; r < T.num_runs; ++r) base |= ((b >> T.run_src[r]) & ((1ull << T.run_len[r]) - 1)) << T.run_dst[r];
  }
  auto phys_of = [&](uint32_t j) {
    uint64_t p = base;
    for (int b = 0; b < T.K; ++b) p |= uint64_t((j >> b) & 1u) << T.tile_phys[b];
    return p;
  };
  for (uint32_t j = threadIdx.x; j < tile; j += blockDim.x) {
    const uint64_t p = phys_of(j);
    ps[j] = psi[p];
    ls[j] = lam[p];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int y = 0; y < T.count; ++y) {
    const tile_overlap_spec S = T.spec[y];
    const double base_sign = (__popcll(base & S.sign) & 1) ? -1.0 : 1.0;
    double re = 0, im = 0;
    for (uint32_t j = threadIdx.x; j < tile; j += blockDim.x) {
      const C l = ls[j], p = ps[j ^ S.flip_local];
      const double s = (__popc(j & S.sign_local) & 1) ? -base_sign : base_sign;
      const double cr = double(l.x) * double(p.x) + double(l.y) * double(p.y);
      const double ci = double(l.x) * double(p.y) - double(l.y) * double(p.x);
      re += s * (cr * S.wr - ci * S.wi);
      im += s * (cr * S.wi + ci * S.wr);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (lane == 0) { red[y][warp][0] = re; red[y][warp][1] = im; }
  }
  __syncthreads();
  for (int y = threadIdx.x; y < T.count; y += blockDim.x) {
    double re = 0, im = 0;
    for (int w = 0; w < kRedThreads / 32; ++w) { re += red[y][w][0]; im += red[y][w][1]; }
    partials[(size_t(y) * gridDim.x + blockIdx.x) * 2] = re;
    partials[(size_t(y) * gridDim.x + blockIdx.x) * 2 + 1] = im;
  }
}

__global__ void finish_tile_overlaps_kernel(const double* __restrict__ partials, int blocks,
                                            const __grid_constant__ tile_overlap_set T, double* __restrict__ out)
{
  const double2 v = warp_sum_partials(partials + size_t(blockIdx.x) * blocks * 2, blocks);
  if (threadIdx.x == 0) {
    out[2 * T.spec[blockIdx.x].out_slot] = v.x;
    out[2 * T.spec[blockIdx.x].out_slot + 1] = v.y;
  }
}

size_t tile_overlaps_partials_doubles(int n, int K) { return (size_t(1) << (n > K ? n - K : 0)) * 2 * kMaxOverlaps; }

template <typename Real>
cudaError_t launch_tile_overlaps(const void* lam, const void* psi, int n, const tile_overlap_set& set, double* partials,
                                 double* out, cudaStream_t stream)
{
  if (set.count < 1 || set.count > kMaxOverlaps || n < set.K) return cudaErrorInvalidValue;
  const size_t smem = 2 * sizeof(typename ctype<Real>::c) << set.K;
  static std::atomic<bool> configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(tile_overlaps_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (16 << 12));
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  const unsigned tiles = unsigned(1ull << (n - set.K));
  tile_overlaps_kernel<Real><<<tiles, kRedThreads, smem, stream>>>(static_cast<const typename ctype<Real>::c*>(lam),
                                                                  static_cast<const typename ctype<Real>::c*>(psi), set,
                                                                  partials);
  finish_tile_overlaps_kernel<<<set.count, 32, 0, stream>>>(partials, int(tiles), set, out);
  return cudaGetLastError();
}
// zsum2_set (rbk_kernels.h): exactly 2^kZsumLogThreads threads, thread gid
// visiting indices (k << kZsumLogThreads) | gid as in zsum_kernel.  Per block
// the partial sums of c_j = conj(lam_j) psi_j: the total, then for every bit q
// the sum over j with bit q set.  k runs in groups of 8 where it can: the
// group's three low bits of k are known at compile time, and its higher bits
// add the group's sum once instead of once per amplitude.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
zsum2_kernel(const typename ctype<Real>::c* __restrict__ lam, const typename ctype<Real>::c* __restrict__ psi, int n,
             double* partials)
{
  constexpr int HI = kMaxQubits - kZsumLogThreads;
  const uint64_t size = 1ull << n;
  const uint64_t gid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  double tr = 0, ti = 0, hr[HI], hi[HI];
#pragma unroll
  for (int k = 0; k < HI; ++k) hr[k] = hi[k] = 0;
  const uint64_t ks = size >> kZsumLogThreads;  // k values of every thread (n >= kZsumLogThreads)
  if (ks >= 8) {
    for (uint64_t m = 0; m < ks / 8; ++m) {
      double gr = 0, gi = 0, r0 = 0, i0 = 0, r1 = 0, i1 = 0, r2 = 0, i2 = 0;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const uint64_t j = ((m * 8 + r) << kZsumLogThreads) | gid;
        const auto l = __ldcs(lam + j), p = __ldcs(psi + j);
        const double cr = double(l.x) * double(p.x) + double(l.y) * double(p.y);
        const double ci = double(l.x) * double(p.y) - double(l.y) * double(p.x);
        gr += cr;
        gi += ci;
        if (r & 1) { r0 += cr; i0 += ci; }
        if (r & 2) { r1 += cr; i1 += ci; }
        if (r & 4) { r2 += cr; i2 += ci; }
      }
      tr += gr;
      ti += gi;
      hr[0] += r0; hi[0] += i0;
      hr[1] += r1; hi[1] += i1;
      hr[2] += r2; hi[2] += i2;
#pragma unroll
      for (int b = 3; b < HI; ++b)
        if ((m >> (b - 3)) & 1) { hr[b] += gr; hi[b] += gi; }
    }
  } else {
    for (uint64_t k = 0; (k << kZsumLogThreads) + gid < size; ++k) {
      const uint64_t j = (k << kZsumLogThreads) | gid;
      const auto l = __ldcs(lam + j), p = __ldcs(psi + j);
      const double cr = double(l.x) * double(p.x) + double(l.y) * double(p.y);
      const double ci = double(l.x) * double(p.y) - double(l.y) * double(p.x);
      tr += cr;
      ti += ci;
#pragma unroll
      for (int b = 0; b < HI; ++b)
        if ((k >> b) & 1) { hr[b] += cr; hi[b] += ci; }
    }
  }
  double vals[2 * (1 + kMaxQubits)];
  vals[0] = tr;
  vals[1] = ti;
  for (int q = 0; q < n; ++q) {
    double a = 0, c = 0;
    if (q < kZsumLogThreads) {
      if ((gid >> q) & 1) { a = tr; c = ti; }
    } else {
#pragma unroll
      for (int b = 0; b < HI; ++b)
        if (b == q - kZsumLogThreads) { a = hr[b]; c = hi[b]; }
    }
    vals[2 + 2 * q] = a;
    vals[3 + 2 * q] = c;
  }
  block_sum_store<2 * (1 + kMaxQubits)>(vals, 2 * (n + 1), partials + size_t(blockIdx.x) * 2 * (n + 1));
}

// One warp per entry: S_q = total - 2 (sum over bit q set), out = w S_q.
__global__ void finish_zsum2_kernel(const double* __restrict__ partials, int blocks, int n,
                                    const __grid_constant__ zsum2_set set, double* __restrict__ out)
{
  const int lane = threadIdx.x & 31, width = 2 * (n + 1);
  const int q = set.spec[blockIdx.x].bit;
  double tr = 0, ti = 0, or_ = 0, oi = 0;
  for (int b = lane; b < blocks; b += 32) {
    const double* p = partials + size_t(b) * width;
    tr += p[0];
    ti += p[1];
    or_ += p[2 + 2 * q];
    oi += p[3 + 2 * q];
  }
  tr = warp_sum(tr);
  ti = warp_sum(ti);
  or_ = warp_sum(or_);
  oi = warp_sum(oi);
  if (lane == 0) {
    const double sr = tr - 2.0 * or_, si = ti - 2.0 * oi;
    const double wr = set.spec[blockIdx.x].wr, wi = set.spec[blockIdx.x].wi;
    const int slot = set.spec[blockIdx.x].out_slot;
    out[2 * slot] = sr * wr - si * wi;
    out[2 * slot + 1] = sr * wi + si * wr;
  }
}

template <typename Real>
cudaError_t launch_zsum2(const void* lam, const void* psi, int n, const zsum2_set& set, double* partials, double* out,
                         cudaStream_t stream)
{
  if (set.count < 1 || set.count > kMaxOverlaps || n < 1 || n > kMaxQubits) return cudaErrorInvalidValue;
  for (int y = 0; y < set.count; ++y)
    if (set.spec[y].bit < 0 || set.spec[y].bit >= n) return cudaErrorInvalidValue;
  const int blocks = zsum_blocks(n);
  zsum2_kernel<Real><<<blocks, kRedThreads, 0, stream>>>(static_cast<const typename ctype<Real>::c*>(lam),
                                                          static_cast<const typename ctype<Real>::c*>(psi), n, partials);
  finish_zsum2_kernel<<<set.count, 32, 0, stream>>>(partials, blocks, n, set, out);
  return cudaGetLastError();
}

// pair_overlap_set (rbk_kernels.h): persistent CTAs, two per SM, each taking
// tiles blockIdx.x, + gridDim.x, ...; both states' tiles of 2^11 amplitudes
// sit in shared memory at the fused pass's swizzled slots.  In register phase
// p a thread holds the 8 amplitudes of each state whose tile bits
// phase_reg[p][0..2] vary; flip f = 3 p + k is register bit k of phase p.
constexpr int kPairBlocksPerSm = 2;
template <typename Real>
__global__ void __launch_bounds__(kRedThreads, kPairBlocksPerSm)
pair_overlaps_kernel(const typename ctype<Real>::c* __restrict__ lam, const typename ctype<Real>::c* __restrict__ psi,
                     const __grid_constant__ pair_overlap_set PS, uint64_t num_tiles, double* partials)
{
  const spin_group& S = PS.g;
  using C = typename ctype<Real>::c;
  constexpr int VB = precision_traits<Real>::VB;
  constexpr int RB = kPairRegBits, NE = 1 << RB, KT = 8 + RB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tl = reinterpret_cast<C*>(smem_raw);
  C* tp = tl + (1u << KT);
  const uint32_t tid = threadIdx.x;
  uint64_t tphys = 0;
  for (int b = 0; b < 8; ++b) tphys |= uint64_t((tid >> b) & 1u) << S.tile_phys[b];
  const uint32_t st = smem_slot<VB>(tid);
  uint32_t sbase[kSpinPhases];
#pragma unroll
  for (int p = 0; p < kSpinPhases; ++p) {
    uint32_t j = 0;
    if (p < S.nphases)
      for (int b = 0; b < 8; ++b) j |= ((tid >> b) & 1u) << S.phase_thr[p][b];
    sbase[p] = smem_slot<VB>(j);
  }
  // A_f + s_f B_f per flip (s_f = -1 for Y type), which is all the result needs.
  double xr[kMaxPairFlips], xi[kMaxPairFlips];
#pragma unroll
  for (int f = 0; f < kMaxPairFlips; ++f) xr[f] = xi[f] = 0.0;
  for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x) {
    uint64_t base = tphys;
    for (int r = 0; r < S.num_runs; ++r) base |= ((t >> S.run_src[r]) & ((1ull << S.run_len[r]) - 1)) << S.run_dst[r];
    C vl[NE], vp[NE];
#pragma unroll
    for (int it = 0; it < NE; ++it) {
      uint64_t p = base;
#pragma unroll
      for (int b = 0; b < RB; ++b)
        if ((it >> b) & 1) p |= 1ull << S.tile_phys[8 + b];
      vl[it] = __ldcs(lam + p);
      vp[it] = __ldcs(psi + p);
    }
    __syncthreads();  // the previous tile is no longer read
#pragma unroll
    for (int it = 0; it < NE; ++it) {
      const uint32_t s = st ^ smem_slot<VB>(uint32_t(it) << 8);
      tl[s] = vl[it];
      tp[s] = vp[it];
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kSpinPhases; ++p) {
      if (p < S.nphases) {
        uint32_t rs[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) rs[k] = smem_slot<VB>(1u << S.phase_reg[p][k]);
        C el[NE], ep[NE];
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          uint32_t sidx = sbase[p];
#pragma unroll
          for (int k = 0; k < RB; ++k)
            if ((i >> k) & 1) sidx ^= rs[k];
          el[i] = tl[sidx];
          ep[i] = tp[sidx];
        }
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int f = p * RB + k;
          if (f < kMaxPairFlips && f < S.nflips) {
            const double s = PS.flip[f].minus ? -1.0 : 1.0;
#pragma unroll
            for (int i = 0; i < NE; ++i) {
              if ((i >> k) & 1) continue;
              const C l0 = el[i], l1 = el[i | (1 << k)], p0 = ep[i], p1 = ep[i | (1 << k)];
              const double ar = double(l0.x) * double(p1.x) + double(l0.y) * double(p1.y);
              const double ai = double(l0.x) * double(p1.y) - double(l0.y) * double(p1.x);
              const double br = double(l1.x) * double(p0.x) + double(l1.y) * double(p0.y);
              const double bi = double(l1.x) * double(p0.y) - double(l1.y) * double(p0.x);
              xr[f] += __fma_rn(s, br, ar);
              xi[f] += __fma_rn(s, bi, ai);
            }
          }
        }
      }
    }
  }
  // Block sums, in a fixed order: A_f + s_f B_f as 2 doubles per flip.
  __shared__ double red[kRedThreads / 32][2 * kMaxPairFlips];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int f = 0; f < kMaxPairFlips; ++f) {
    if (f < S.nflips) {
      const double a0 = warp_sum(xr[f]), a1 = warp_sum(xi[f]);
      if (lane == 0) { red[warp][2 * f] = a0; red[warp][2 * f + 1] = a1; }
    }
  }
  __syncthreads();
  const int width = 2 * S.nflips;
  for (int k = threadIdx.x; k < width; k += blockDim.x) {
    double acc = 0.0;
    for (int w = 0; w < kRedThreads / 32; ++w) acc += red[w][k];
    partials[size_t(blockIdx.x) * width + k] = acc;
  }
}

// One warp per flip: A + s B over the blocks, then out = w (A + s B).
__global__ void finish_pair_overlaps_kernel(const double* __restrict__ partials, int blocks, int nflips,
                                            const __grid_constant__ pair_overlap_set set, double* __restrict__ out)
{
  const int lane = threadIdx.x & 31, f = blockIdx.x, width = 2 * nflips;
  double xr = 0, xi = 0;
  for (int b = lane; b < blocks; b += 32) {
    xr += partials[size_t(b) * width + 2 * f];
    xi += partials[size_t(b) * width + 2 * f + 1];
  }
  xr = warp_sum(xr);
  xi = warp_sum(xi);
  if (lane == 0) {
    const double wr = set.flip[f].wr, wi = set.flip[f].wi;
    const int slot = set.flip[f].out_slot;
    out[2 * slot] = xr * wr - xi * wi;
    out[2 * slot + 1] = xr * wi + xi * wr;
  }
}

size_t pair_overlaps_partials_doubles() { return size_t(148) * kPairBlocksPerSm * 2 * kMaxPairFlips; }

template <typename Real>
cudaError_t launch_pair_overlaps(const void* lam, const void* psi, int n, const pair_overlap_set& set, double* partials,
                                 double* out, cudaStream_t stream)
{
  const spin_group& g = set.g;
  if (g.K != 8 + kPairRegBits || g.K > n || g.nflips < 1 || g.nflips > kMaxPairFlips || g.nphases < 1 ||
      g.nphases > kSpinPhases || g.nphases * kPairRegBits < g.nflips)
    return cudaErrorInvalidValue;
  const size_t smem = 2 * sizeof(typename ctype<Real>::c) << g.K;
  static std::atomic<bool> configured[64] = {};
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(pair_overlaps_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const uint64_t tiles = 1ull << (n - g.K);
  // Capped at 148 SMs' worth: the partials buffer is sized for that.
  const int blocks = static_cast<int>(std::min<uint64_t>(tiles, uint64_t(std::min(sms, 148)) * kPairBlocksPerSm));
  pair_overlaps_kernel<Real><<<blocks, kRedThreads, smem, stream>>>(static_cast<const typename ctype<Real>::c*>(lam),
                                                                   static_cast<const typename ctype<Real>::c*>(psi), set, tiles,
                                                                   partials);
  finish_pair_overlaps_kernel<<<g.nflips, 32, 0, stream>>>(partials, blocks, g.nflips, set, out);
  return cudaGetLastError();
}
// pair_rotate_set (rbk_kernels.h): the tile traffic of pair_overlaps_kernel
// plus a write-back.  Per tile: both states' tiles into shared memory; in each
// register phase the overlaps of the phase's flips, then their gates on both
// states in registers, written back to the same slots; after the last phase
// the tiles go back to HBM where they came from.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads, kPairBlocksPerSm)
pair_rotate_kernel(typename ctype<Real>::c* __restrict__ lam, typename ctype<Real>::c* __restrict__ psi,
                   const __grid_constant__ pair_rotate_set PS, uint64_t num_tiles, double* partials)
{
  const spin_group& S = PS.g;
  using C = typename ctype<Real>::c;
  constexpr int VB = precision_traits<Real>::VB;
  constexpr int RB = kPairRegBits, NE = 1 << RB, KT = 8 + RB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* tl = reinterpret_cast<C*>(smem_raw);
  C* tp = tl + (1u << KT);
  // Im(w_f (A_f + s_f B_f)) per flip and thread, kept in shared memory between
  // tiles to spare registers.
  __shared__ double acc[kMaxRotFlips][kRedThreads];
  const uint32_t tid = threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int f = 0; f < kMaxRotFlips; ++f) acc[f][tid] = 0.0;
  uint64_t tphys = 0;
  for (int b = 0; b < 8; ++b) tphys |= uint64_t((tid >> b) & 1u) << S.tile_phys[b];
  const uint32_t st = smem_slot<VB>(tid);
  // Pre-step state (PS.pre): the diagonal's factor over this thread's tile bits
  // and over each register slot's bits; Z sums per thread (total and register
  // bits) and per warp (bits outside the tile).
  const pre_diag& D = PS.pre;
  __shared__ double2 fthr[kRedThreads], freg[1 << kPairRegBits];
  __shared__ uint64_t mthr[kRedThreads];  // partner row of this thread's tile bits, XORed; bit 63: their pair parity
  __shared__ double zt[4][kRedThreads];
  __shared__ double zh[kMaxQubits][kRedThreads / 32];
  if (D.active) {
    double2 f{1.0, 0.0};
    for (int b = 0; b < 8; ++b)
      if ((tid >> b) & 1) f = cmul(f, double2{D.u[S.tile_phys[b]][0], D.u[S.tile_phys[b]][1]});
    fthr[tid] = f;
    uint64_t m = 0;
    uint32_t qt = 0;
    for (int b = 0; b < 8; ++b)
      if ((tid >> b) & 1) {
        m ^= D.full[S.tile_phys[b]];
        qt ^= __popcll(tphys & D.adj[S.tile_phys[b]]);
      }
    mthr[tid] = (m & ~(1ull << 63)) | (uint64_t(qt & 1u) << 63);
    if (tid < (1u << kPairRegBits)) {
      double2 r{1.0, 0.0};
      for (int b = 0; b < kPairRegBits; ++b)
        if ((tid >> b) & 1) r = cmul(r, double2{D.u[S.tile_phys[8 + b]][0], D.u[S.tile_phys[8 + b]][1]});
      freg[tid] = r;
    }
    for (int k = 0; k < 4; ++k) zt[k][tid] = 0.0;
    for (int q = tid; q < kMaxQubits * (kRedThreads / 32); q += kRedThreads) zh[q / (kRedThreads / 32)][q % (kRedThreads / 32)] = 0.0;
    __syncthreads();
  }
  auto tile_base = [&](uint64_t t) {
    uint64_t b = tphys;
    for (int r = 0; r < S.num_runs; ++r) b |= ((t >> S.run_src[r]) & ((1ull << S.run_len[r]) - 1)) << S.run_dst[r];
    return b;
  };
  // Phase 0 is the load layout (register bits = tile bits 8..10, thread bits
  // 0..7): a tile goes from HBM straight into its registers.  The next tile's
  // loads are issued before this tile's store, so that they are in flight
  // while the store runs.
  C el[NE], ep[NE];
  auto load_tile = [&](uint64_t b) {
#pragma unroll
    for (int it = 0; it < NE; ++it) {
      uint64_t p = b;
#pragma unroll
      for (int k = 0; k < RB; ++k)
        if ((it >> k) & 1) p |= 1ull << S.tile_phys[8 + k];
      el[it] = __ldcs(lam + p);
      ep[it] = __ldcs(psi + p);
    }
  };
  if (blockIdx.x < num_tiles) load_tile(tile_base(blockIdx.x));
  for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x) {
    const uint64_t base = tile_base(t);
    {
      C* vl = el;
      C* vp = ep;
      if (D.active) {
        if (D.nz > 0) {
          // Im conj(lam_j) psi_j: thread total, register-bit sums, and the warp's
          // total for the bits outside the tile that are set in this tile.
          double tot = 0.0, r0 = 0.0, r1 = 0.0, r2 = 0.0;
#pragma unroll
          for (int it = 0; it < NE; ++it) {
            const double c = double(vl[it].x) * double(vp[it].y) - double(vl[it].y) * double(vp[it].x);
            tot += c;
            if (it & 1) r0 += c;
            if (it & 2) r1 += c;
            if (it & 4) r2 += c;
          }
          zt[0][tid] += tot;
          zt[1][tid] += r0;
          zt[2][tid] += r1;
          zt[3][tid] += r2;
          const double wtot = warp_sum(tot);
          if (lane == 0)
            for (uint64_t hb = base ^ tphys; hb; hb &= hb - 1) zh[__ffsll(static_cast<long long>(hb)) - 1][warp] += wtot;
        }
        // The diagonal: g times u over the set bits, times (-1)^Q.
        double2 f{D.g[0], D.g[1]};
        for (uint64_t hb = base ^ tphys; hb; hb &= hb - 1) {
          const int q = __ffsll(static_cast<long long>(hb)) - 1;
          f = cmul(f, double2{D.u[q][0], D.u[q][1]});
        }
        f = cmul(f, fthr[tid]);
        // Q(base) = Q(bits outside the tile) ^ Q(thread bits) ^ their cross
        // pairs; the first is the same for the whole CTA (uniform loop).
        const uint64_t hbase = base ^ tphys;
        uint32_t qb = 0;
        for (uint64_t hb = hbase; hb; hb &= hb - 1) qb ^= __popcll(hbase & D.adj[__ffsll(static_cast<long long>(hb)) - 1]);
        const uint64_t mt = mthr[tid];
        qb ^= uint32_t(mt >> 63) ^ __popcll(hbase & mt & ~(1ull << 63));
#pragma unroll
        for (int it = 0; it < NE; ++it) {
          double2 fi = cmul(f, freg[it]);
          if ((qb ^ (D.qr >> it) ^ __popcll(base & D.mr[it])) & 1) fi = double2{-fi.x, -fi.y};
          const C fc{Real(fi.x), Real(fi.y)};
          vl[it] = cmul(vl[it], fc);
          vp[it] = cmul(vp[it], fc);
        }
      }
      // The previous tile's last shared-memory reads (its store, in the load
      // layout) were made by this warp on the slots phase 0 writes.
      __syncwarp();
    }
#pragma unroll
    for (int p = 0; p < kSpinPhases; ++p) {
      if (p < S.nphases) {
        uint32_t j = 0;
        for (int b = 0; b < 8; ++b) j |= ((tid >> b) & 1u) << S.phase_thr[p][b];
        const uint32_t sbase = smem_slot<VB>(j);
        uint32_t rs[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) rs[k] = smem_slot<VB>(1u << S.phase_reg[p][k]);
        if (p > 0) {
#pragma unroll
          for (int i = 0; i < NE; ++i) {
            uint32_t sidx = sbase;
#pragma unroll
            for (int k = 0; k < RB; ++k)
              if ((i >> k) & 1) sidx ^= rs[k];
            el[i] = tl[sidx];
            ep[i] = tp[sidx];
          }
        }
        // The phase's overlaps, all before its gates (the gates of a run commute):
        // the amplitudes are widened once for the three flips.  Widened at each use,
        // conversions kept their pipe 48 % busy in complex<float> (gradient of 23
        // qubits 3.83 -> 3.60 ms); complex<double> is the same either way.
        uint32_t okinds = 0;
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int f = p * RB + k;
          if (f < kMaxRotFlips && f < S.nflips) okinds |= uint32_t(PS.flip[f].okind) << (2 * k);
        }
        if (okinds != 0) {
          double2 dl[NE], dp[NE];
#pragma unroll
          for (int i = 0; i < NE; ++i) {
            dl[i] = double2{double(el[i].x), double(el[i].y)};
            dp[i] = double2{double(ep[i].x), double(ep[i].y)};
          }
#pragma unroll
          for (int k = 0; k < RB; ++k) {
            const int f = p * RB + k;
            const uint32_t okind = (okinds >> (2 * k)) & 3u;
            if (f >= kMaxRotFlips || okind == 0) continue;
            // Im(w (A + s B)) = wi Re(A + s B) + wr Im(A + s B); A and B are summed
            // on their own and weighted once per tile.
            double ar = 0.0, br = 0.0, ai = 0.0, bi = 0.0;
#pragma unroll
            for (int i = 0; i < NE; ++i) {
              if ((i >> k) & 1) continue;
              const double2 l0 = dl[i], l1 = dl[i | (1 << k)], p0 = dp[i], p1 = dp[i | (1 << k)];
              if (okind & 1) {
                ar = __fma_rn(l0.x, p1.x, __fma_rn(l0.y, p1.y, ar));
                br = __fma_rn(l1.x, p0.x, __fma_rn(l1.y, p0.y, br));
              }
              if (okind & 2) {
                ai = __fma_rn(l0.x, p1.y, __fma_rn(-l0.y, p1.x, ai));
                bi = __fma_rn(l1.x, p0.y, __fma_rn(-l1.y, p0.x, bi));
              }
            }
            const double s = PS.flip[f].minus ? -1.0 : 1.0;
            acc[f][tid] += PS.flip[f].wi * __fma_rn(s, br, ar) + PS.flip[f].wr * __fma_rn(s, bi, ai);
          }
        }
        // The gates, lambda's registers first and written back before psi's,
        // so that fewer registers are live at once.
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int f = p * RB + k;
          if (f < kMaxRotFlips && f < S.nflips && PS.flip[f].mkind != 2) {
            const double* m = PS.flip[f].m;
            if (PS.flip[f].mkind == 1) {
#pragma unroll
              for (int i = 0; i < NE; ++i) {
                if ((i >> k) & 1) continue;
                const int i1 = i | (1 << k);
                const C l0 = el[i], l1 = el[i1];
                el[i] = rmac2(l0, l1, Real(m[0]), Real(m[2]));
                el[i1] = rmac2(l0, l1, Real(m[4]), Real(m[6]));
              }
            } else {
#pragma unroll
              for (int i = 0; i < NE; ++i) {
                if ((i >> k) & 1) continue;
                const int i1 = i | (1 << k);
                const C l0 = el[i], l1 = el[i1];
                el[i] = cmac2(l0, l1, Real(m[0]), Real(m[1]), Real(m[2]), Real(m[3]));
                el[i1] = cmac2(l0, l1, Real(m[4]), Real(m[5]), Real(m[6]), Real(m[7]));
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          uint32_t sidx = sbase;
#pragma unroll
          for (int k = 0; k < RB; ++k)
            if ((i >> k) & 1) sidx ^= rs[k];
          tl[sidx] = el[i];
        }
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int f = p * RB + k;
          if (f < kMaxRotFlips && f < S.nflips && PS.flip[f].mkind != 2) {
            const double* m = PS.flip[f].m;
            if (PS.flip[f].mkind == 1) {
#pragma unroll
              for (int i = 0; i < NE; ++i) {
                if ((i >> k) & 1) continue;
                const int i1 = i | (1 << k);
                const C p0 = ep[i], p1 = ep[i1];
                ep[i] = rmac2(p0, p1, Real(m[0]), Real(m[2]));
                ep[i1] = rmac2(p0, p1, Real(m[4]), Real(m[6]));
              }
            } else {
#pragma unroll
              for (int i = 0; i < NE; ++i) {
                if ((i >> k) & 1) continue;
                const int i1 = i | (1 << k);
                const C p0 = ep[i], p1 = ep[i1];
                ep[i] = cmac2(p0, p1, Real(m[0]), Real(m[1]), Real(m[2]), Real(m[3]));
                ep[i1] = cmac2(p0, p1, Real(m[4]), Real(m[5]), Real(m[6]), Real(m[7]));
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          uint32_t sidx = sbase;
#pragma unroll
          for (int k = 0; k < RB; ++k)
            if ((i >> k) & 1) sidx ^= rs[k];
          tp[sidx] = ep[i];
        }
        // The next phase (or the store) reads other threads' slots: those of
        // other warps too where the warp index moves to other tile bits.
        if (PS.block_sync[p]) __syncthreads();
        else __syncwarp();
      }
    }
    // The store addresses are recomputed from an opaque copy of the tile base:
    // kept from the loads, the eight of them would hold 16 registers through the phases.
    uint64_t sbase_hbm;
    asm volatile("mov.b64 %0, %1;" : "=l"(sbase_hbm) : "l"(base));
    if (t + gridDim.x < num_tiles) load_tile(tile_base(t + gridDim.x));
#pragma unroll
    for (int it = 0; it < NE; ++it) {
      const uint32_t s = st ^ smem_slot<VB>(uint32_t(it) << 8);
      uint64_t p = sbase_hbm;
#pragma unroll
      for (int b = 0; b < RB; ++b)
        if ((it >> b) & 1) p |= 1ull << S.tile_phys[8 + b];
      __stcs(lam + p, tl[s]);
      __stcs(psi + p, tp[s]);
    }
  }
  // Block sums in a fixed order, one double per flip; then, with Z sums, the
  // total and the sum over j with each physical bit set (tile bits from the
  // per-thread sums, the others from the per-warp sums).
  constexpr int NZ = 1 + 8 + kPairRegBits;
  __shared__ double red[kRedThreads / 32][kMaxRotFlips + NZ];
#pragma unroll
  for (int f = 0; f < kMaxRotFlips; ++f) {
    if (f < S.nflips) {
      const double a = warp_sum(acc[f][tid]);
      if (lane == 0) red[warp][f] = a;
    }
  }
  const bool zs = D.active && D.nz > 0;
  if (zs) {
    double v[NZ];
    v[0] = zt[0][tid];
#pragma unroll
    for (int b = 0; b < 8; ++b) v[1 + b] = ((tid >> b) & 1) ? zt[0][tid] : 0.0;
#pragma unroll
    for (int k = 0; k < kPairRegBits; ++k) v[9 + k] = zt[1 + k][tid];
#pragma unroll
    for (int k = 0; k < NZ; ++k) {
      const double a = warp_sum(v[k]);
      if (lane == 0) red[warp][kMaxRotFlips + k] = a;
    }
  }
  __syncthreads();
  const int nzw = zs ? 1 + kMaxQubits : 0;
  const int width = S.nflips + nzw;
  for (int k = threadIdx.x; k < width; k += blockDim.x) {
    double sum = 0.0;
    if (k < S.nflips) {
      for (int w = 0; w < kRedThreads / 32; ++w) sum += red[w][k];
    } else {
      const int q = k - S.nflips - 1;  // -1: the total
      int col = -1;
      if (q < 0) col = 0;
      for (int b = 0; b < 8 + kPairRegBits; ++b)
        if (q >= 0 && S.tile_phys[b] == q) col = 1 + b;
      if (col >= 0) {
        for (int w = 0; w < kRedThreads / 32; ++w) sum += red[w][kMaxRotFlips + col];
      } else {
        for (int w = 0; w < kRedThreads / 32; ++w) sum += zh[q][w];
      }
    }
    partials[size_t(blockIdx.x) * width + k] = sum;
  }
}

// One warp per overlap of the launches whose partial sums are kept in `partials`:
// out[2 slot] = 0 (the real part is not formed), out[2 slot + 1] = the sum of the
// entry's column over its launch's blocks -- Im(w (A + s B)) -- or, for a Z entry,
// w (total - 2 sum over bit q set).
__global__ void finish_pair_rotate_kernel(const double* __restrict__ partials, const pair_rotate_result* __restrict__ entries,
                                          int count, double* __restrict__ out)
{
  const int lane = threadIdx.x & 31, e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (e >= count) return;
  const pair_rotate_result R = entries[e];
  const double* p = partials + R.begin;
  double x = 0, o = 0;
  for (int b = lane; b < R.blocks; b += 32) {
    x += p[size_t(b) * R.width + R.column];
    if (R.second >= 0) o += p[size_t(b) * R.width + R.second];
  }
  x = warp_sum(x);
  o = warp_sum(o);
  if (lane == 0) {
    out[2 * R.slot] = 0.0;
    out[2 * R.slot + 1] = R.second >= 0 ? R.w * (x - 2.0 * o) : x;
  }
}

cudaError_t launch_finish_pair_rotate(const double* partials, const pair_rotate_result* entries, int count, double* out,
                                      cudaStream_t stream)
{
  if (count < 1) return cudaSuccess;
  finish_pair_rotate_kernel<<<(count + 3) / 4, 128, 0, stream>>>(partials, entries, count, out);
  return cudaGetLastError();
}

size_t pair_rotate_partials_doubles() { return size_t(148) * kPairBlocksPerSm * (kMaxRotFlips + 1 + kMaxQubits); }

template <typename Real>
cudaError_t launch_pair_rotate(void* lam, void* psi, int n, const pair_rotate_set& set, double* partials, size_t begin,
                               std::vector<pair_rotate_result>& results, size_t* used, cudaStream_t stream)
{
  const spin_group& g = set.g;
  if (g.K != 8 + kPairRegBits || g.K > n || n > kMaxQubits || g.nflips < 1 || g.nflips > kMaxRotFlips || g.nphases < 1 ||
      g.nphases > kSpinPhases || g.nphases * kPairRegBits < g.nflips)
    return cudaErrorInvalidValue;
  const int nz = set.pre.active ? set.pre.nz : 0;
  if (nz < 0 || nz > kMaxQubits) return cudaErrorInvalidValue;
  for (int k = 0; k < nz; ++k)
    if (set.pre.z[k].bit < 0 || set.pre.z[k].bit >= n) return cudaErrorInvalidValue;
  const size_t smem = 2 * sizeof(typename ctype<Real>::c) << g.K;
  static std::atomic<bool> configured[64] = {};
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(pair_rotate_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const uint64_t tiles = 1ull << (n - g.K);
  // Capped at 148 SMs' worth: the partials buffer is sized for that.
  const int blocks = static_cast<int>(std::min<uint64_t>(tiles, uint64_t(std::min(sms, 148)) * kPairBlocksPerSm));
  pair_rotate_kernel<Real><<<blocks, kRedThreads, smem, stream>>>(static_cast<typename ctype<Real>::c*>(lam),
                                                                 static_cast<typename ctype<Real>::c*>(psi), set, tiles,
                                                                 partials + begin);
  const int width = g.nflips + (nz > 0 ? 1 + kMaxQubits : 0);
  for (int f = 0; f < g.nflips; ++f)
    if (set.flip[f].out_slot >= 0) results.push_back({begin, blocks, width, f, -1, set.flip[f].out_slot, 0, 1.0});
  for (int k = 0; k < nz; ++k)
    results.push_back({begin, blocks, width, g.nflips, g.nflips + 1 + set.pre.z[k].bit, set.pre.z[k].out_slot, 0, set.pre.z[k].wr});
  *used = size_t(blocks) * size_t(width);
  return cudaGetLastError();
}
template cudaError_t launch_pair_rotate<double>(void*, void*, int, const pair_rotate_set&, double*, size_t,
                                                std::vector<pair_rotate_result>&, size_t*, cudaStream_t);
template cudaError_t launch_pair_rotate<float>(void*, void*, int, const pair_rotate_set&, double*, size_t,
                                               std::vector<pair_rotate_result>&, size_t*, cudaStream_t);

template cudaError_t launch_zsum2<double>(const void*, const void*, int, const zsum2_set&, double*, double*, cudaStream_t);
template cudaError_t launch_zsum2<float>(const void*, const void*, int, const zsum2_set&, double*, double*, cudaStream_t);
template cudaError_t launch_pair_overlaps<double>(const void*, const void*, int, const pair_overlap_set&, double*, double*, cudaStream_t);
template cudaError_t launch_pair_overlaps<float>(const void*, const void*, int, const pair_overlap_set&, double*, double*, cudaStream_t);

template cudaError_t launch_tile_overlaps<double>(const void*, const void*, int, const tile_overlap_set&, double*, double*, cudaStream_t);
template cudaError_t launch_tile_overlaps<float>(const void*, const void*, int, const tile_overlap_set&, double*, double*, cudaStream_t);

template cudaError_t launch_overlaps<double>(const void*, const void*, int, const overlap_set&, double*, double*, cudaStream_t);
template cudaError_t launch_overlaps<float>(const void*, const void*, int, const overlap_set&, double*, double*, cudaStream_t);

template cudaError_t launch_pauli_apply<double>(const void*, void*, int, const pauli_sum&, cudaStream_t);
template cudaError_t launch_pauli_apply<float>(const void*, void*, int, const pauli_sum&, cudaStream_t);

}  // namespace rbk

namespace rbk {

// ---------------------------------------------------------------------------
// Sampling: the device form of ket::generate_events
// (ket/include/ket/generate_events.hpp:18-51), the upper_bound of a random
// value among the inclusive prefix sums of |a_i|^2.
//
// The prefix sums are kept at two levels only: one sum per block of
// 2^kSampleBlockLog amplitudes and the scanned sums of chunks of
// 2^kSampleChunkLog amplitudes.  A sample searches the chunks, then the 32
// block sums of its chunk, then re-reads the 128 amplitudes of its block.  The
// state is read once and 8 bytes are written per 128 amplitudes, so the call
// is bound by that read; a prefix value per amplitude wrote and re-read 24
// bytes for each and needed half the state's size of scratch (26 qubits
// complex<double>: 0.74 ms of scans, 0.4 to 3 ms more for allocating and
// freeing 512 MB; now 0.2 ms).
// ---------------------------------------------------------------------------
constexpr int kSampleBlockLog = 7;   // 32 lanes x 4 amplitudes
constexpr int kSampleChunkLog = 12;  // 32 blocks: one per lane
constexpr int kSampleWarps = 4;

// One warp per chunk: sums[b] = sum of |a|^2 over block b (0 for blocks past the
// end of a state smaller than a chunk), chunk_sums[c] = their sum.
template <typename Real>
__global__ void __launch_bounds__(kSampleWarps * 32)
sample_sums_kernel(const typename ctype<Real>::c* __restrict__ a, uint64_t size, uint64_t chunks, double* __restrict__ sums,
                   double* __restrict__ chunk_sums)
{
  using C = typename ctype<Real>::c;
  constexpr int kGroup = 4;  // blocks whose loads are in flight together
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t c = uint64_t(blockIdx.x) * kSampleWarps + (threadIdx.x >> 5);
  if (c >= chunks) return;
  const uint64_t base = c << kSampleChunkLog;
  double mine = 0.0;  // lane l: the sum of block l
  for (int g = 0; g < 32; g += kGroup) {
    C v[kGroup][4];
#pragma unroll
    for (int b = 0; b < kGroup; ++b)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint64_t i = base + (uint64_t(g + b) << kSampleBlockLog) + uint64_t(k * 32) + lane;
        v[b][k] = i < size ? __ldcs(a + i) : C{Real(0), Real(0)};
      }
#pragma unroll
    for (int b = 0; b < kGroup; ++b) {
      double p = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) p += double(v[b][k].x) * double(v[b][k].x) + double(v[b][k].y) * double(v[b][k].y);
      p = warp_sum(p);
      if (lane == uint32_t(g + b)) mine = p;
    }
  }
  sums[(c << (kSampleChunkLog - kSampleBlockLog)) + lane] = mine;
  // The chunk's sum as the inclusive scan that sample_kernel forms: its last lane.
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, mine, o);
    if (lane >= uint32_t(o)) mine += y;
  }
  if (lane == 31) chunk_sums[c] = mine;
}

// Inclusive scan of v[0..count) in place by one block: thread t sums and then
// rewrites its own run of consecutive values (rbk_sample_scan.h).  At most 2^21
// chunks (33 qubits).
constexpr int kSampleScanThreads = 1024;
__global__ void __launch_bounds__(kSampleScanThreads) sample_scan_kernel(double* __restrict__ v, uint64_t count)
{
  static_assert(kSampleScanThreads == 32 * 32, "a lane for every warp");
  __shared__ double warp_tot[32], warp_end[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t per = (count + kSampleScanThreads - 1) / kSampleScanThreads;
  const uint64_t lo = min(count, threadIdx.x * per), hi = min(count, lo + per);
  uint64_t last;
  double incl = scan_run(v, lo, hi, &last);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  // Every warp scans the warps' sums (and below their ends): lane w has those of warps 0 .. w.
  double sums = warp_tot[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, sums, o);
    if (lane >= o) sums += y;
  }
  const double off = __shfl_sync(0xffffffffu, sums, max(warp - 1, 0));
  double end = last > lo ? (warp > 0 ? off + incl : incl) : 0.0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end = scan_later(y, end);
  }
  if (lane == 31) warp_end[warp] = end;
  __syncthreads();
  double ends = warp_end[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, ends, o);
    if (lane >= o) ends = scan_later(y, ends);
  }
  double prev = __shfl_sync(0xffffffffu, ends, max(warp - 1, 0));
  if (warp == 0) prev = 0.0;
  const double y = __shfl_up_sync(0xffffffffu, end, 1);
  scan_write(v, lo, hi, last, lane > 0 ? scan_later(prev, y) : prev, scan_later(prev, end));
}

// One warp per sample: events[k] = first index whose prefix sum exceeds r[k].
// Where rounding between the levels leaves no such entry inside the chunk or
// block that a search chose, its last entry of non-zero weight is taken, so an
// amplitude of weight zero is never drawn.  r[k] at or above the last prefix
// sum (rounding) gives the last index, as does a state whose sums are NaN.
template <typename Real>
__global__ void __launch_bounds__(kSampleWarps * 32)
sample_kernel(const typename ctype<Real>::c* __restrict__ a, uint64_t size, uint64_t chunks, const double* __restrict__ sums,
              const double* __restrict__ prefix, const double* __restrict__ r, int num, uint64_t* __restrict__ events)
{
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * kSampleWarps + (threadIdx.x >> 5);
  if (k >= num) return;
  const double x = r[k];
  // First chunk whose prefix exceeds x, by a 32-way search: lane l looks at the end of the l-th part.
  uint64_t lo = 0, hi = chunks;
  while (hi - lo > 1) {
    const uint64_t step = (hi - lo + 31) / 32;
    const uint64_t end = min(hi, lo + uint64_t(lane + 1) * step);
    const uint32_t over = __ballot_sync(0xffffffffu, prefix[end - 1] > x);
    const uint64_t part = over ? uint64_t(__ffs(static_cast<int>(over)) - 1) : 31;
    const uint64_t nlo = min(hi - 1, lo + part * step);
    hi = min(hi, nlo + step);
    lo = nlo;
  }
  if (!(prefix[lo] > x)) {
    if (lane == 0) events[k] = size - 1;
    return;
  }
  // The block of the chunk: lane l holds block l.
  double base = lo > 0 ? prefix[lo - 1] : 0.0;
  const double s = sums[(lo << (kSampleChunkLog - kSampleBlockLog)) + uint64_t(lane)];
  double incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  uint32_t over = __ballot_sync(0xffffffffu, base + incl > x && s > 0.0);
  uint32_t some = __ballot_sync(0xffffffffu, s > 0.0);
  const int blk = over ? __ffs(static_cast<int>(over)) - 1 : some ? 31 - __clz(static_cast<int>(some)) : 0;
  const double upto = __shfl_sync(0xffffffffu, incl, blk > 0 ? blk - 1 : 0);
  if (blk > 0) base += upto;
  // The amplitude: lane l holds the four consecutive ones from 4 l.
  const uint64_t first = (lo << kSampleChunkLog) + (uint64_t(blk) << kSampleBlockLog) + uint64_t(4 * lane);
  double p[4], tot = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    p[j] = 0.0;
    if (first + j < size) {
      const auto v = a[first + j];
      p[j] = double(v.x) * double(v.x) + double(v.y) * double(v.y);
    }
    tot += p[j];
  }
  incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  double run = __shfl_up_sync(0xffffffffu, incl, 1);
  run = base + (lane > 0 ? run : 0.0);
  int hit = -1, last = -1;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    run += p[j];
    if (p[j] > 0.0) {
      last = j;
      if (hit < 0 && run > x) hit = j;
    }
  }
  over = __ballot_sync(0xffffffffu, hit >= 0);
  some = __ballot_sync(0xffffffffu, last >= 0);
  const int src = over ? __ffs(static_cast<int>(over)) - 1 : some ? 31 - __clz(static_cast<int>(some)) : 0;
  if (lane == src) events[k] = min(size - 1, first + uint64_t(over ? hit : some ? last : 0));
}

static uint64_t sample_chunks(int n) { return n > kSampleChunkLog ? 1ull << (n - kSampleChunkLog) : 1; }

// Block sums, then chunk prefixes.
size_t sample_scratch_doubles(int n) { return sample_chunks(n) * ((1u << (kSampleChunkLog - kSampleBlockLog)) + 1); }

// scratch: sample_scratch_doubles(n) doubles; *total points at the sum of |a|^2 in it.
template <typename Real>
cudaError_t launch_sample_sums(const void* amps, int n, double* scratch, const double** total, cudaStream_t stream)
{
  const uint64_t chunks = sample_chunks(n);
  double* prefix = scratch + (chunks << (kSampleChunkLog - kSampleBlockLog));
  sample_sums_kernel<Real><<<(unsigned)((chunks + kSampleWarps - 1) / kSampleWarps), kSampleWarps * 32, 0, stream>>>(
    static_cast<const typename ctype<Real>::c*>(amps), 1ull << n, chunks, scratch, prefix);
  if (chunks > 1) sample_scan_kernel<<<1, kSampleScanThreads, 0, stream>>>(prefix, chunks);
  *total = prefix + (chunks - 1);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_sample(const void* amps, int n, const double* scratch, const double* r, int num, uint64_t* events,
                          cudaStream_t stream)
{
  const uint64_t chunks = sample_chunks(n);
  sample_kernel<Real><<<(num + kSampleWarps - 1) / kSampleWarps, kSampleWarps * 32, 0, stream>>>(
    static_cast<const typename ctype<Real>::c*>(amps), 1ull << n, chunks, scratch,
    scratch + (chunks << (kSampleChunkLog - kSampleBlockLog)), r, num, events);
  return cudaGetLastError();
}

template cudaError_t launch_sample_sums<double>(const void*, int, double*, const double**, cudaStream_t);
template cudaError_t launch_sample_sums<float>(const void*, int, double*, const double**, cudaStream_t);
template cudaError_t launch_sample<double>(const void*, int, const double*, const double*, int, uint64_t*, cudaStream_t);
template cudaError_t launch_sample<float>(const void*, int, const double*, const double*, int, uint64_t*, cudaStream_t);

}  // namespace rbk

namespace rbk {

// ---------------------------------------------------------------------------
// SHORBOX: ket::shor_box (ket/include/ket/shor_box.hpp) writes, for every
// exponent e < 2^nx, the amplitude 2^(-nx/2) at the index whose top nx qubits
// hold e bit-reversed and whose low n - nx qubits hold (base^e mod divisor)
// truncated to n - nx bits; e = 0 holds 1 (the running value starts at 1 and
// is reduced only after use).  The reference walks e sequentially; here every
// thread computes its own power by squaring.  With divisor, base < 2^32 every
// product stays below 2^64, so the values are the reference's exactly.
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void shor_box_kernel(typename ctype<Real>::c* __restrict__ a, int n, int nx, uint64_t divisor, uint64_t base,
                                Real coeff)
{
  using C = typename ctype<Real>::c;
  const uint64_t count = 1ull << nx;
  const int low = n - nx;
  const uint64_t low_mask = (1ull << low) - 1;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t e = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; e < count; e += stride) {
    uint64_t v = 1;
    if (e > 0) {
      uint64_t x = base % divisor, r = 1 % divisor;
      for (uint64_t k = e; k; k >>= 1) {
        if (k & 1) r = r * x % divisor;
        x = x * x % divisor;
      }
      v = r;
    }
    const uint64_t rev = nx > 0 ? (__brevll(e) >> (64 - nx)) : 0;
    a[(rev << low) | (v & low_mask)] = C{coeff, (Real)0};
  }
}

template <typename Real>
cudaError_t launch_shor_box(void* state, int n, int nx, uint64_t divisor, uint64_t base, double coeff, cudaStream_t stream)
{
  const uint64_t count = 1ull << nx;
  shor_box_kernel<Real><<<grid_for(count, 256), 256, 0, stream>>>(static_cast<typename ctype<Real>::c*>(state), n, nx,
                                                                divisor, base, static_cast<Real>(coeff));
  return cudaGetLastError();
}
template cudaError_t launch_shor_box<double>(void*, int, int, uint64_t, uint64_t, double, cudaStream_t);
template cudaError_t launch_shor_box<float>(void*, int, int, uint64_t, uint64_t, double, cudaStream_t);

}  // namespace rbk
