// rbk_small_adjoint.cu -- see rbk_small_adjoint.h.
//
// One instance is one CTA (n <= 12) or one cluster of 2^(n - 12) CTAs.  Both
// states stay in shared memory; the CTAs of a cluster hold consecutive ranges
// and reach each other's over distributed shared memory.  A register phase
// (small_phase) moves 8 amplitudes of a state per thread into registers and
// applies its gates there, so that a layer of one-qubit rotations costs n / 3
// exchanges and barriers; a parameter's overlap is taken from the same
// registers before its gate is un-applied.  Arithmetic in registers is
// complex<double> for both precisions, storage is the batch's precision.
//   Bound by FP64 work on the instance's SMs and by the latency of a phase
// (two moves, a barrier, the reductions).  The one-gate sweeps of one CTA per
// instance before took about 1 us a sweep (12 qubits, 16 layers: 2.2 ms) and
// 13 to 15 qubits took 1.05 to 1.15 ms for 10 layers in engine launches.
#include "rbk_small_adjoint.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <complex>
#include <cstring>
#include <string>

#include "rbk_device.cuh"
#include "rbk_kernels.h"
#include "rbk_plan.h"
#include "rbk_small_core.cuh"

namespace rbk {
namespace {

constexpr int kSaThreads = 512;
constexpr int kSaPhaseOps = 48;  // ops of one phase, staged in shared memory twice
constexpr int kSaPhaseSlots = 8;  // overlaps of one phase: a column of partial sums per thread each, staged twice
constexpr int kSaRegs = kSmallSlots;
constexpr int kSaLocalBits = 12;  // amplitudes a CTA holds of each state

struct sa_args {
  const sa_inst* inst;
  const sa_phase* phases;
  const sa_rot* rots;
  const sa_term* terms;
  small_op* ops;
  const double* theta;
  double* partial;
  double* energy;
  double* overlaps;
};

__device__ __forceinline__ double sa_warp_sum(double v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank)
{
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// An amplitude of a state in shared memory (of this CTA, or of the cluster at a mapped address).
template <typename Real, int CS> struct sa_mem;
template <int CS> struct sa_mem<double, CS> {
  static __device__ __forceinline__ double2 get(uint32_t a)
  {
    double2 v;
    if constexpr (CS > 1) asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    else asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
  }
  static __device__ __forceinline__ void put(uint32_t a, double2 v)
  {
    if constexpr (CS > 1) asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" :: "r"(a), "d"(v.x), "d"(v.y) : "memory");
    else asm volatile("st.shared.v2.f64 [%0], {%1, %2};" :: "r"(a), "d"(v.x), "d"(v.y) : "memory");
  }
};
template <int CS> struct sa_mem<float, CS> {
  static __device__ __forceinline__ double2 get(uint32_t a)
  {
    float2 v;
    if constexpr (CS > 1) asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    else asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return double2{double(v.x), double(v.y)};
  }
  static __device__ __forceinline__ void put(uint32_t a, double2 d)
  {
    const float x = float(d.x), y = float(d.y);
    if constexpr (CS > 1) asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" :: "r"(a), "f"(x), "f"(y) : "memory");
    else asm volatile("st.shared.v2.f32 [%0], {%1, %2};" :: "r"(a), "f"(x), "f"(y) : "memory");
  }
};

template <int CS>
__device__ __forceinline__ void sa_sync()
{
  if constexpr (CS > 1) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// Im <lambda| P |psi> over this thread's amplitudes, P = X or Y on register bit B.
template <int B>
__device__ __forceinline__ double sa_overlap(const double2 (&p)[kSaRegs], const double2 (&l)[kSaRegs], bool y)
{
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < kSaRegs; ++i) {
    if (i & (1 << B)) continue;
    const double2 l0 = l[i], l1 = l[i | (1 << B)], p0 = p[i], p1 = p[i | (1 << B)];
    if (y) s += (l1.x * p0.x + l1.y * p0.y) - (l0.x * p1.x + l0.y * p1.y);
    else s += (l0.x * p1.y - l0.y * p1.x) + (l1.x * p0.y - l1.y * p0.x);
  }
  return s;
}

// The shared-memory address of each register slot of a phase.
template <typename Real, int CS>
__device__ __forceinline__ void sa_addresses(uint32_t smem, uint32_t base, const uint8_t (&reg)[kSmallRegBits], int local_bits,
                                             uint32_t (&addr)[kSaRegs])
{
  constexpr uint32_t S = uint32_t(sizeof(typename ctype<Real>::c));
#pragma unroll
  for (int i = 0; i < kSaRegs; ++i) {
    uint32_t x = base;
#pragma unroll
    for (int k = 0; k < kSmallRegBits; ++k)
      if ((i >> k) & 1) x |= 1u << reg[k];
    const uint32_t local = CS > 1 ? x & ((1u << local_bits) - 1) : x;
    addr[i] = smem + smem_slot<0>(local) * S;
    if constexpr (CS > 1) addr[i] = map_rank(addr[i], x >> local_bits);
  }
}

template <typename Real, int CS>
__global__ void __launch_bounds__(kSaThreads, 1) small_adjoint_kernel(const sa_args A, int first)
{
  constexpr int kClusterLog = CS == 8 ? 3 : CS == 4 ? 2 : CS == 2 ? 1 : 0;
  constexpr uint32_t S = uint32_t(sizeof(typename ctype<Real>::c));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) small_op ops[2][kSaPhaseOps];
  const sa_inst I = A.inst[first + blockIdx.x / CS];
  const uint32_t rank = blockIdx.x % CS;  // cluster dimensions (CS, 1, 1): the CTA's rank in its cluster
  const int local_bits = max(I.n, kSmallRegBits) - kClusterLog;
  const uint32_t local = 1u << local_bits, groups = local / kSaRegs;
  const uint32_t psi = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)), lam = psi + local * S;
  // Per-thread overlap sums: columns[buffer][overlap of the phase][thread].
  double* const columns = reinterpret_cast<double*>(smem_raw + 2 * size_t(local) * S);
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  const uint32_t warps = blockDim.x >> 5, all_warps = warps * CS, gwarp = rank * warps + (tid >> 5);
  double* partial = A.partial + I.partial_begin;
  small_op* gops = A.ops + I.op_begin;
  const sa_phase* phases = A.phases + I.phase_begin;
  const double* theta = A.theta + I.theta_begin;

  // Matrices of the parametrised rotations.
  for (int k = int(rank * blockDim.x + tid); k < I.num_rots; k += int(blockDim.x * CS)) {
    const sa_rot r = A.rots[I.rot_begin + k];
    const double phi = (r.param >= 0 ? r.scale * theta[r.param] : 0.0) + r.offset;
    double sn, cs;
    sincos(phi, &sn, &cs);
    small_op& o = gops[r.op];
    if (o.rot == 1) {         // cos I + i sin X
      o.m[0] = cs; o.m[1] = 0; o.m[2] = 0; o.m[3] = sn; o.m[4] = 0; o.m[5] = sn; o.m[6] = cs; o.m[7] = 0;
    } else if (o.rot == 2) {  // cos I + i sin Y
      o.m[0] = cs; o.m[1] = 0; o.m[2] = sn; o.m[3] = 0; o.m[4] = -sn; o.m[5] = 0; o.m[6] = cs; o.m[7] = 0;
    } else {                  // diag(e^{i phi}, e^{-i phi})
      o.m[0] = cs; o.m[1] = sn; o.m[2] = cs; o.m[3] = -sn;
    }
  }
  for (uint32_t i = tid; i < local; i += blockDim.x) {
    const uint32_t a = psi + smem_slot<0>(i) * S;
    sa_mem<Real, 1>::put(a, double2{rank == 0 && i == 0 ? 1.0 : 0.0, 0.0});
  }
  __threadfence();
  sa_sync<CS>();

  // Ops of a phase into staging buffer b, through L2 (the matrices above were written by other CTAs too).
  auto stage = [&](const sa_phase& ph, int b) {
    const char* src = reinterpret_cast<const char*>(gops + ph.begin);
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&ops[b][0]));
    const uint32_t words = uint32_t(ph.end - ph.begin) * uint32_t(sizeof(small_op) / 16);
    for (uint32_t i = tid; i < words; i += blockDim.x)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(dst + 16 * i), "l"(src + 16 * i) : "memory");
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto staged = [&]() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); };
  auto group_base = [&](uint32_t g, const sa_phase& ph) {
    uint32_t base = rank * groups + g;
#pragma unroll
    for (int k = 0; k < kSmallRegBits; ++k) base = uint32_t(insert_zero(base, ph.reg[k]));
    return base;
  };

  // Forward.
  if (I.num_phases > 0) {
    stage(phases[0], 0);
    staged();
    __syncthreads();
  }
  sa_phase next = I.num_phases > 0 ? phases[0] : sa_phase{};
  for (int p = 0; p < I.num_phases; ++p) {
    const sa_phase ph = next;
    const int b = p & 1, count = ph.end - ph.begin;
    if (p + 1 < I.num_phases) {
      next = phases[p + 1];
      stage(next, b ^ 1);
    }
    for (uint32_t g = tid; g < groups; g += blockDim.x) {
      const uint32_t base = group_base(g, ph);
      uint32_t addr[kSaRegs];
      sa_addresses<Real, CS>(psi, base, ph.reg, local_bits, addr);
      double2 a[kSaRegs];
#pragma unroll
      for (int i = 0; i < kSaRegs; ++i) a[i] = sa_mem<Real, CS>::get(addr[i]);
      uint32_t signs = 0;
      small_header h = small_load_header(&ops[b][0]);
      for (int k = 0; k < count; ++k) {
        const small_header next_h = small_load_header(&ops[b][min(k + 1, count - 1)]);
        small_gate<false, false>(a, a, h, &ops[b][k], base, signs);
        h = next_h;
      }
      if (signs) small_signs(a, signs);
#pragma unroll
      for (int i = 0; i < kSaRegs; ++i) sa_mem<Real, CS>::put(addr[i], a[i]);
    }
    staged();
    sa_sync<CS>();
  }

  // lambda = H psi, E = <psi|lambda>.
  {
    const sa_term* terms = A.terms + I.term_begin;
    const uint32_t size = 1u << I.n;
    double er = 0.0;
    for (uint32_t j = tid; j < local; j += blockDim.x) {
      const uint32_t i = rank * local + j;
      double lr = 0.0, li = 0.0;
      double2 v{0.0, 0.0};
      uint32_t have = ~0u;
      for (int t = 0; t < I.num_terms && i < size; ++t) {
        const sa_term T = terms[t];
        if (T.flip != have) {
          have = T.flip;
          const uint32_t x = i ^ T.flip;
          uint32_t a = psi + smem_slot<0>(x & (local - 1)) * S;
          if constexpr (CS > 1) a = map_rank(a, x >> local_bits);
          v = sa_mem<Real, CS>::get(a);
        }
        const bool neg = __popc(i & T.sign) & 1;
        const double wr = neg ? -T.wr : T.wr, wi = neg ? -T.wi : T.wi;
        lr += wr * v.x - wi * v.y;
        li += wr * v.y + wi * v.x;
      }
      const uint32_t off = smem_slot<0>(j) * S;
      sa_mem<Real, 1>::put(lam + off, double2{lr, li});
      const double2 pv = sa_mem<Real, 1>::get(psi + off);
      er += pv.x * lr + pv.y * li;
    }
    er = sa_warp_sum(er);
    if (lane == 0) partial[size_t(I.num_slots) * CS + gwarp] = er;
  }
  if (I.num_phases > 0) {
    next = phases[I.num_phases - 1];
    stage(next, (I.num_phases - 1) & 1);
    staged();
  }
  sa_sync<CS>();

  // Reverse: every op un-applied from both states, a rotation's overlap taken before it.
  const uint32_t rounds = (groups + blockDim.x - 1) / blockDim.x;
  for (int p = I.num_phases - 1; p >= 0; --p) {
    const sa_phase ph = next;
    const int b = p & 1, count = ph.end - ph.begin;
    if (p > 0) {
      next = phases[p - 1];
      stage(next, b ^ 1);
    }
    for (uint32_t r = 0; r < rounds; ++r) {  // whole warps together: the overlaps are warp sums
      const uint32_t g = r * blockDim.x + tid;
      const bool active = g < groups;
      const uint32_t base = group_base(active ? g : 0u, ph);
      uint32_t addr[kSaRegs];
      sa_addresses<Real, CS>(psi, base, ph.reg, local_bits, addr);
      const uint32_t to_lam = lam - psi;
      double2 a[kSaRegs], l[kSaRegs];
#pragma unroll
      for (int i = 0; i < kSaRegs; ++i) {
        a[i] = l[i] = double2{0.0, 0.0};
        if (active) {
          a[i] = sa_mem<Real, CS>::get(addr[i]);
          l[i] = sa_mem<Real, CS>::get(addr[i] + to_lam);
        }
      }
      uint32_t signs = 0;
      small_header h = small_load_header(&ops[b][count - 1]);
      for (int k = count - 1; k >= 0; --k) {
        const small_header next_h = small_load_header(&ops[b][max(k - 1, 0)]);
        if (h.slot() >= 0) {
          double s = 0.0;
          if (h.rot() == 3) {  // sign flips not applied yet are on both states: no matter
            const uint32_t m1 = (base & h.dbase()) ? kAllSlots : h.hi();
#pragma unroll
            for (int i = 0; i < kSaRegs; ++i)
              s += small_flip(l[i].x * a[i].y - l[i].y * a[i].x, (m1 << (31 - i)) & 0x80000000u);
          } else {
            if (signs) {
              small_signs(a, signs);
              small_signs(l, signs);
              signs = 0;
            }
            const uint32_t t = h.code() % 3u;  // target register bit
            s = t == 0 ? sa_overlap<0>(a, l, h.rot() == 2) : t == 1 ? sa_overlap<1>(a, l, h.rot() == 2) : sa_overlap<2>(a, l, h.rot() == 2);
          }
          double* c = columns + (size_t(b) * kSaPhaseSlots + size_t(h.slot() - ph.slot_begin)) * blockDim.x + tid;
          *c = r > 0 ? *c + s : s;
        }
        small_gate<true, true>(a, l, h, &ops[b][k], base, signs);
        h = next_h;
      }
      if (signs) {
        small_signs(a, signs);
        small_signs(l, signs);
      }
      if (active) {
        // Addresses formed again from an opaque copy of the base: kept through the gates they would hold 8 registers.
        uint32_t again = base;
        asm volatile("" : "+r"(again));
        sa_addresses<Real, CS>(psi, again, ph.reg, local_bits, addr);
#pragma unroll
        for (int i = 0; i < kSaRegs; ++i) {
          sa_mem<Real, CS>::put(addr[i], a[i]);
          sa_mem<Real, CS>::put(addr[i] + to_lam, l[i]);
        }
      }
    }
    staged();
    sa_sync<CS>();
    // The phase's overlaps over the CTA, one warp each, while other warps are in the next phase.
    for (int q = int(tid >> 5); q < ph.slots; q += int(warps)) {
      const double* c = columns + (size_t(b) * kSaPhaseSlots + size_t(q)) * blockDim.x;
      double s = 0.0;
      for (uint32_t i = lane; i < blockDim.x; i += 32) s += c[i];
      s = sa_warp_sum(s);
      if (lane == 0) partial[size_t(ph.slot_begin + q) * CS + rank] = s;
    }
  }
  __threadfence();
  sa_sync<CS>();  // the partial sums of every CTA are visible
  for (int s = int(rank * blockDim.x + tid); s <= I.num_slots; s += int(blockDim.x * CS)) {
    double acc = 0.0;
    for (uint32_t w = 0; w < (s == I.num_slots ? all_warps : uint32_t(CS)); ++w) acc += __ldcg(partial + size_t(s) * CS + w);
    if (s == I.num_slots) A.energy[I.out] = acc;
    else A.overlaps[I.slot_begin + s] = acc;
  }
}

// ---- host side ------------------------------------------------------------

using cplx = std::complex<double>;
constexpr double kOneDivRootTwo = 0.707106781186547524400844362104849039284835937688474036588;
constexpr double kTwoPi = 6.28318530717958647692528676655900576839433879875021164195;

void put(double* m, int k, cplx v) { m[2 * k] = v.real(); m[2 * k + 1] = v.imag(); }

// The engine's records of the fixed gates (rbk_hadamard, rbk_phase_shift2/3, ...); a
// rotation gets kind and qubits here and its matrix on the device.
bool lower_gate(int n, const rbk_circuit_gate& g, hgate& h)
{
  h = hgate{};
  h.target2 = -1;
  const bool two = g.kind == RBK_GATE_CNOT || g.kind == RBK_GATE_CZ || g.kind == RBK_GATE_U || g.kind == RBK_GATE_SWAP;
  if (g.qubits[0] < 0 || g.qubits[0] >= n) return false;
  if (two && (g.qubits[1] < 0 || g.qubits[1] >= n || g.qubits[1] == g.qubits[0])) return false;
  const uint64_t b0 = 1ull << g.qubits[0], b1 = two ? 1ull << g.qubits[1] : 0;
  h.target = static_cast<int8_t>(g.qubits[0]);
  auto phase = [&](cplx c) {
    h.kind = OPK_DIAG;
    h.diag_one = 1;
    put(h.m, 0, {1.0, 0.0});
    put(h.m, 1, c);
  };
  switch (g.kind) {
    case RBK_GATE_H:
      h.kind = OPK_MAT;
      put(h.m, 0, {kOneDivRootTwo, 0}); put(h.m, 1, {kOneDivRootTwo, 0});
      put(h.m, 2, {kOneDivRootTwo, 0}); put(h.m, 3, {-kOneDivRootTwo, 0});
      return true;
    case RBK_GATE_X: h.kind = OPK_X; return true;
    case RBK_GATE_Y: h.kind = OPK_Y; return true;
    case RBK_GATE_Z: h.kind = OPK_NEG; h.target = -1; h.cmask = b0; return true;
    case RBK_GATE_U1: phase(std::exp(cplx{0, g.angles[0]})); return true;
    case RBK_GATE_U2: {
      const cplx c1 = std::exp(cplx{0, g.angles[0]}), c2 = std::exp(cplx{0, g.angles[1]});
      const cplx mc1 = kOneDivRootTwo * c1;
      h.kind = OPK_MAT;
      put(h.m, 0, {kOneDivRootTwo, 0}); put(h.m, 1, -(kOneDivRootTwo * c2));
      put(h.m, 2, mc1); put(h.m, 3, mc1 * c2);
      return true;
    }
    case RBK_GATE_U3: {
      const double sine = std::sin(0.5 * g.angles[0]), cosine = std::cos(0.5 * g.angles[0]);
      const cplx c2 = std::exp(cplx{0, g.angles[1]}), c3 = std::exp(cplx{0, g.angles[2]});
      h.kind = OPK_MAT;
      put(h.m, 0, {cosine, 0}); put(h.m, 1, -(sine * c3));
      put(h.m, 2, sine * c2); put(h.m, 3, (cosine * c3) * c2);
      return true;
    }
    case RBK_GATE_CNOT:  // qubits[0] = control, qubits[1] = target
      h.kind = OPK_X;
      h.target = static_cast<int8_t>(g.qubits[1]);
      h.cmask = b0;
      return true;
    case RBK_GATE_CZ: h.kind = OPK_NEG; h.target = -1; h.cmask = b0 | b1; return true;
    case RBK_GATE_U: {
      const int k = static_cast<int>(g.angles[0]), ak = k < 0 ? -k : k;
      cplx c = std::exp(cplx{0, std::ldexp(kTwoPi, -ak)});
      if (k < 0) c = std::conj(c);
      phase(c);
      h.target = static_cast<int8_t>(g.qubits[1]);
      h.cmask = b0;
      return true;
    }
    case RBK_GATE_EX: case RBK_GATE_EY: h.kind = OPK_MAT; return true;
    case RBK_GATE_EZ: h.kind = OPK_DIAG; return true;
    case RBK_GATE_SWAP:
      h.kind = HK_SWAP;
      h.target2 = static_cast<int8_t>(g.qubits[1]);
      return true;
    default: return false;
  }
}

int rot_type(int kind) { return kind == RBK_GATE_EX ? 1 : kind == RBK_GATE_EY ? 2 : kind == RBK_GATE_EZ ? 3 : 0; }

int sa_fail(int code, const std::string& m) { return set_last_error(code, m.c_str()); }

size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

int cluster_of(int n) { return n > kSaLocalBits ? 1 << (n - kSaLocalBits) : 1; }
int threads_of(int n, int most)
{
  const int need = std::max(32, (1 << std::max(0, std::min(n, kSaLocalBits) - kSmallRegBits)));
  return std::min(need, std::min(most, kSaThreads));
}

template <typename Real, int CS>
cudaError_t launch_class(const sa_args& args, int first, int count, int n, int threads, cudaStream_t stream)
{
  const int local_bits = std::max(kSmallRegBits, std::min(n, kSaLocalBits));
  constexpr size_t column = 2 * kSaPhaseSlots * sizeof(double);  // of each thread
  const size_t smem = 2 * (sizeof(typename ctype<Real>::c) << local_bits) + column * size_t(threads);
  static std::atomic<bool> configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(small_adjoint_kernel<Real, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(2 * (sizeof(typename ctype<Real>::c) << kSaLocalBits) + column * kSaThreads));
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(count) * CS);
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = CS;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, small_adjoint_kernel<Real, CS>, args, first);
}

template <typename Real>
cudaError_t launch_class(const sa_args& args, int first, int count, int n, int threads, cudaStream_t stream)
{
  switch (cluster_of(n)) {
    case 1: return launch_class<Real, 1>(args, first, count, n, threads, stream);
    case 2: return launch_class<Real, 2>(args, first, count, n, threads, stream);
    case 4: return launch_class<Real, 4>(args, first, count, n, threads, stream);
    case 8: return launch_class<Real, 8>(args, first, count, n, threads, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

bool sa_plan(int n, const rbk_circuit_gate* gates, int num_gates, int num_terms, const char* strings, const double* coeffs,
             sa_program& out)
{
  if (n < 1 || n > kSmallAdjointBits) return false;
  out = sa_program{};
  out.n = n;
  std::vector<hgate> queue(static_cast<size_t>(num_gates));
  for (int i = 0; i < num_gates; ++i)
    if (!lower_gate(n, gates[i], queue[static_cast<size_t>(i)])) return false;
  std::vector<int> perm(static_cast<size_t>(n)), inv(static_cast<size_t>(n));
  for (int q = 0; q < n; ++q) perm[static_cast<size_t>(q)] = inv[static_cast<size_t>(q)] = q;
  std::vector<char> marked(queue.size(), 0);
  for (size_t i = 0; i < queue.size(); ++i) marked[i] = gates[i].param >= 0 && rot_type(gates[i].kind) ? 1 : 0;
  plan_small_phases(n, queue, perm, inv, static_cast<size_t>(kSaPhaseOps), marked, kSaPhaseSlots,
                    [&](const std::vector<small_op>& ops, const std::vector<size_t>& from, const small_phase& phase) {
                      sa_phase ph{};
                      std::memcpy(ph.reg, phase.reg, sizeof(ph.reg));
                      ph.begin = static_cast<int32_t>(out.ops.size());
                      ph.slot_begin = static_cast<int32_t>(out.slot_param.size());
                      for (size_t k = 0; k < ops.size(); ++k) {
                        const rbk_circuit_gate& g = gates[from[k]];
                        small_op o = ops[k];
                        o.rot = static_cast<uint8_t>(rot_type(g.kind));
                        if (o.rot) {  // the matrix comes on the device
                          if (o.rot < 3) o.code = static_cast<uint8_t>((o.rot == 2 ? SMALL_REAL : SMALL_MAT) + o.treg);
                          else o.code = SMALL_DIAG;
                          out.rots.push_back({static_cast<int32_t>(out.ops.size()), g.param, g.scale, g.angles[0]});
                          if (g.param >= 0) {
                            o.slot = static_cast<int32_t>(out.slot_param.size());
                            out.slot_param.push_back(g.param);
                            out.slot_scale.push_back(g.scale);
                          }
                        }
                        out.ops.push_back(o);
                      }
                      ph.end = static_cast<int32_t>(out.ops.size());
                      ph.slots = static_cast<int32_t>(out.slot_param.size()) - ph.slot_begin;
                      out.phases.push_back(ph);
                    });
  static const cplx pow_mi[4] = {{1, 0}, {0, -1}, {-1, 0}, {0, 1}};
  for (int t = 0; t < num_terms; ++t) {
    uint32_t x = 0, y = 0, z = 0;
    for (int q = 0; q < n; ++q) {
      const char c = strings[static_cast<size_t>(t) * static_cast<size_t>(n) + static_cast<size_t>(q)];
      const uint32_t b = 1u << perm[static_cast<size_t>(q)];
      if (c == 'X') x |= b;
      else if (c == 'Y') y |= b;
      else if (c == 'Z') z |= b;
      else if (c != 'I') return false;
    }
    const cplx w = cplx{coeffs[2 * t], coeffs[2 * t + 1]} * pow_mi[__builtin_popcount(y) & 3];
    out.terms.push_back({x | y, y | z, w.real(), w.imag()});
  }
  std::stable_sort(out.terms.begin(), out.terms.end(), [](const sa_term& a, const sa_term& b) { return a.flip < b.flip; });
  return true;
}

int sa_set::fetch(cudaStream_t stream)
{
  if (cudaMemcpyAsync(h_out_, d_out_, sizeof(double) * (insts_.size() + size_t(slots_)), cudaMemcpyDeviceToHost, stream) != cudaSuccess)
    return sa_fail(RBK_ERR_CUDA, "small adjoint: results");
  return RBK_OK;
}

sa_set::~sa_set()
{
  if (h_out_) cudaFreeHost(h_out_);
  if (d_image_) cudaFree(d_image_);
  if (h_image_) cudaFreeHost(h_image_);
  if (d_partial_) cudaFree(d_partial_);
  if (d_out_) cudaFree(d_out_);
}

int sa_set::assign(int precision, const std::vector<const sa_program*>& programs, const double* theta, int num_theta,
                   cudaStream_t stream)
{
  precision_ = precision;
  std::vector<int> order(programs.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = static_cast<int>(i);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return programs[size_t(a)]->n > programs[size_t(b)]->n; });
  insts_.clear();
  slot_begin_.assign(programs.size(), 0);
  size_t ops = 0, phases = 0, rots = 0, terms = 0, partial = 0;
  slots_ = 0;
  for (int i : order) {
    const sa_program& P = *programs[size_t(i)];
    sa_inst I{};
    I.n = P.n;
    I.num_phases = int32_t(P.phases.size());
    I.num_rots = int32_t(P.rots.size());
    I.num_slots = int32_t(P.slot_param.size());
    I.num_terms = int32_t(P.terms.size());
    I.op_begin = int32_t(ops);
    I.phase_begin = int32_t(phases);
    I.rot_begin = int32_t(rots);
    I.slot_begin = slots_;
    I.term_begin = int32_t(terms);
    I.theta_begin = P.theta_begin;
    I.out = i;
    I.partial_begin = int64_t(partial);
    slot_begin_[size_t(i)] = slots_;
    ops += P.ops.size();
    phases += P.phases.size();
    rots += P.rots.size();
    terms += P.terms.size();
    slots_ += I.num_slots;
    // an overlap per CTA, the energy per warp
    partial += size_t(cluster_of(P.n)) * (size_t(I.num_slots) + size_t(threads_of(size_class(P.n), kSaThreads) / 32));
    insts_.push_back(I);
  }
  if (ops > size_t(INT32_MAX) || terms > size_t(INT32_MAX)) return sa_fail(RBK_ERR_UNSUPPORTED, "batch: too many gates");
  off_phase_ = align16(sizeof(sa_inst) * insts_.size());
  off_rot_ = align16(off_phase_ + sizeof(sa_phase) * phases);
  off_term_ = align16(off_rot_ + sizeof(sa_rot) * rots);
  off_op_ = align16(off_term_ + sizeof(sa_term) * terms);
  off_theta_ = align16(off_op_ + sizeof(small_op) * ops);
  const size_t bytes = off_theta_ + sizeof(double) * size_t(theta ? num_theta : 0);
  auto grow = [&](size_t want, size_t& cap, auto&& alloc) {
    if (want <= cap) return true;
    cap = 0;
    if (!alloc(want + want / 4 + 256)) return false;
    cap = want + want / 4 + 256;
    return true;
  };
  const bool ok =
    grow(bytes, image_cap_, [&](size_t n) {
      if (d_image_) cudaFree(d_image_);
      if (h_image_) cudaFreeHost(h_image_);
      d_image_ = h_image_ = nullptr;
      return cudaMalloc(reinterpret_cast<void**>(&d_image_), n) == cudaSuccess &&
             cudaMallocHost(reinterpret_cast<void**>(&h_image_), n) == cudaSuccess;
    }) &&
    grow(partial, partial_cap_, [&](size_t n) {
      if (d_partial_) cudaFree(d_partial_);
      d_partial_ = nullptr;
      return cudaMalloc(reinterpret_cast<void**>(&d_partial_), sizeof(double) * n) == cudaSuccess;
    }) &&
    grow(programs.size() + size_t(slots_), out_cap_, [&](size_t n) {
      if (d_out_) cudaFree(d_out_);
      if (h_out_) cudaFreeHost(h_out_);
      d_out_ = h_out_ = nullptr;
      return cudaMalloc(reinterpret_cast<void**>(&d_out_), sizeof(double) * n) == cudaSuccess &&
             cudaMallocHost(reinterpret_cast<void**>(&h_out_), sizeof(double) * n) == cudaSuccess;
    });
  if (!ok) {
    cudaGetLastError();
    return sa_fail(RBK_ERR_OOM, "small adjoint: memory exhausted");
  }
  std::memcpy(h_image_, insts_.data(), sizeof(sa_inst) * insts_.size());
  for (const sa_inst& I : insts_) {
    const sa_program& P = *programs[size_t(I.out)];
    std::memcpy(h_image_ + off_phase_ + sizeof(sa_phase) * size_t(I.phase_begin), P.phases.data(), sizeof(sa_phase) * P.phases.size());
    std::memcpy(h_image_ + off_rot_ + sizeof(sa_rot) * size_t(I.rot_begin), P.rots.data(), sizeof(sa_rot) * P.rots.size());
    std::memcpy(h_image_ + off_term_ + sizeof(sa_term) * size_t(I.term_begin), P.terms.data(), sizeof(sa_term) * P.terms.size());
    std::memcpy(h_image_ + off_op_ + sizeof(small_op) * size_t(I.op_begin), P.ops.data(), sizeof(small_op) * P.ops.size());
  }
  if (theta && num_theta > 0) std::memcpy(h_image_ + off_theta_, theta, sizeof(double) * size_t(num_theta));
  if (cudaMemcpyAsync(d_image_, h_image_, bytes, cudaMemcpyHostToDevice, stream) != cudaSuccess)
    return sa_fail(RBK_ERR_CUDA, "small adjoint: upload");
  return RBK_OK;
}

int sa_set::launch(const double* d_theta, int max_threads, cudaStream_t stream, const std::vector<cudaStream_t>& side,
                   const std::vector<cudaEvent_t>& events)
{
  sa_args A{};
  A.inst = reinterpret_cast<const sa_inst*>(d_image_);
  A.phases = reinterpret_cast<const sa_phase*>(d_image_ + off_phase_);
  A.rots = reinterpret_cast<const sa_rot*>(d_image_ + off_rot_);
  A.terms = reinterpret_cast<const sa_term*>(d_image_ + off_term_);
  A.ops = reinterpret_cast<small_op*>(d_image_ + off_op_);
  A.theta = d_theta ? d_theta : reinterpret_cast<const double*>(d_image_ + off_theta_);
  A.partial = d_partial_;
  A.energy = d_out_;
  A.overlaps = d_out_ + insts_.size();
  size_t used = 0;
  for (size_t i = 0; i < insts_.size();) {
    const int cls = size_class(insts_[i].n), n = insts_[i].n;  // the first is the largest of its class
    size_t j = i;
    while (j < insts_.size() && size_class(insts_[j].n) == cls) ++j;
    cudaStream_t on = stream;
    if (i > 0 && used < side.size()) {
      on = side[used];
      if (used == 0 && cudaEventRecord(events[0], stream) != cudaSuccess) return sa_fail(RBK_ERR_CUDA, "small adjoint: fork");
      if (cudaStreamWaitEvent(on, events[0], 0) != cudaSuccess) return sa_fail(RBK_ERR_CUDA, "small adjoint: fork");
      ++used;
    }
    const int threads = threads_of(n, max_threads);
    const cudaError_t e = precision_ == RBK_C128 ? launch_class<double>(A, int(i), int(j - i), n, threads, on)
                                                 : launch_class<float>(A, int(i), int(j - i), n, threads, on);
    if (e != cudaSuccess) return sa_fail(RBK_ERR_CUDA, std::string("small adjoint: ") + cudaGetErrorString(e));
    i = j;
  }
  for (size_t k = 0; k < used; ++k)
    if (cudaEventRecord(events[1 + k], side[k]) != cudaSuccess || cudaStreamWaitEvent(stream, events[1 + k], 0) != cudaSuccess)
      return sa_fail(RBK_ERR_CUDA, "small adjoint: join");
  return RBK_OK;
}

}  // namespace rbk
