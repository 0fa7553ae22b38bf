// rbk_small_adjoint.h -- energies and adjoint gradients of circuits whose two
// state vectors fit the shared memory of one CTA or of one cluster of CTAs.
// The host plans a circuit (its register phases do not depend on the parameters:
// a batch plans when it is created, a single gradient at every call); a launch then
// does the whole job of every instance.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "rbk.h"
#include "rbk_internal.h"

namespace rbk {

// Up to here an instance is one cluster of at most 8 CTAs (the portable
// limit) with 2^12 amplitudes of both states each.
constexpr int kSmallAdjointBits = 15;

struct sa_term { uint32_t flip, sign; double wr, wi; };  // (P psi)_i = w (-1)^popcount(i & sign) psi_{i ^ flip}
struct sa_rot { int32_t op, param; double scale, offset; };  // ops[op].m from phi = scale * theta[param] + offset
// Ops [begin, end) and their overlaps [slot_begin, slot_begin + slots), numbered in op order.
struct sa_phase { uint8_t reg[kSmallRegBits], pad; int32_t begin, end, slot_begin, slots; };

// One planned circuit, in physical bits.
struct sa_program {
  int n = 0;
  std::vector<small_op> ops;
  std::vector<sa_phase> phases;
  std::vector<sa_rot> rots;
  std::vector<sa_term> terms;      // sorted by flip
  std::vector<int> slot_param;     // parameter and scale of overlap s
  std::vector<double> slot_scale;
  int theta_begin = 0;             // the instance's first parameter in the launch's parameter vector
};

// false: not a circuit that these launches take (size, an invalid qubit, an
// unknown gate or Pauli character); the caller's general path judges it.
bool sa_plan(int n, const rbk_circuit_gate* gates, int num_gates, int num_terms, const char* strings, const double* coeffs,
             sa_program& out);

struct sa_inst {
  int32_t n, num_phases, num_rots, num_slots, num_terms, op_begin, phase_begin, rot_begin, slot_begin, term_begin, theta_begin, out;
  int64_t partial_begin;
};

// Planned instances on one device, used from one thread at a time.
class sa_set {
public:
  ~sa_set();
  // Lays the programs out and copies them to the device on `stream`, with the
  // parameter vector when theta is given (else launch gets a device pointer).
  // Buffers grow as needed and are kept.  Returns an rbk_status.  The pinned
  // image may be rewritten only after the stream has finished with the last one.
  int assign(int precision, const std::vector<const sa_program*>& programs, const double* theta, int num_theta,
             cudaStream_t stream);
  // Every instance on `stream` (further streams join it for the size classes
  // when side streams are given); CTAs of at most max_threads threads.
  int launch(const double* d_theta, int max_threads, cudaStream_t stream, const std::vector<cudaStream_t>& side,
             const std::vector<cudaEvent_t>& events);
  int count() const { return static_cast<int>(insts_.size()); }
  // Copies the results to pinned host memory on `stream`: energies[count()] in
  // program order, then the overlaps Im <lambda|P|psi> of every slot.
  int fetch(cudaStream_t stream);
  const double* energies() const { return h_out_; }
  const double* overlaps(int program) const { return h_out_ + insts_.size() + slot_begin_[static_cast<size_t>(program)]; }
  // Instances of one size class share a launch: 15, 14, 13, 12, 11 and at most 10 qubits.
  static int size_class(int n) { return n > 10 ? n : 10; }

private:
  int precision_ = 0, slots_ = 0;
  std::vector<sa_inst> insts_;  // largest first
  std::vector<int> slot_begin_;
  char* d_image_ = nullptr;
  char* h_image_ = nullptr;  // pinned
  size_t image_cap_ = 0, partial_cap_ = 0, out_cap_ = 0;
  size_t off_phase_ = 0, off_rot_ = 0, off_term_ = 0, off_op_ = 0, off_theta_ = 0;
  double* d_partial_ = nullptr;
  double* d_out_ = nullptr;
  double* h_out_ = nullptr;  // pinned
};

}  // namespace rbk
