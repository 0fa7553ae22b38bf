// rbk_plan.h -- host-side fusion planner: queued gates -> fused tile passes.
#pragma once

#include <cstdint>
#include <functional>
#include <vector>

#include "rbk_internal.h"

namespace rbk {

// A queued gate in LOGICAL qubits.  kind is an op_kind, or HK_SWAP for an
// uncontrolled SWAP, which only relabels the layout map.
constexpr uint8_t HK_SWAP = 100;

struct hgate {
  uint8_t kind;
  int8_t target;     // MAT/X/Y/DIAG target; SWAP: first qubit; -1 for NEG
  int8_t target2;    // SWAP: second qubit
  uint8_t diag_one;  // DIAG with d0 == 1 exactly
  uint64_t cmask;    // controls (NEG: every qubit of the phase flip)
  double m[8];
};

inline bool is_dense(const hgate& g) { return g.kind == OPK_MAT; }

struct plan_params {
  int n;         // state qubits
  int K;         // tile bits
  int R;         // register bits
  int LOW;       // low physical bits that are always tile bits (coalescing)
  int vbits;     // log2 amplitudes per 16-byte vector
  int dense_budget;  // max dense 2x2 gates per pass
  bool fold_x = true;  // fold CNOT / X gates at the end of a phase into its write layout
  bool merge_1q = true;  // merge consecutive uncontrolled single-qubit gates on one qubit
  bool defer_x = true;   // register phases take CNOT / X gates last (so that they fold)
  bool phase_runs = true;  // runs of phase gates behind one PHASES header
  bool layers = true;      // uncontrolled 2x2 gates on distinct register bits behind one LAYER header
  bool straight = false;   // passes that allow it in straight form (dev_pass::straight)
  int factored_min = 3;    // layers of at least this many gates take the factored form (0: never)
};

// The same circuit with fewer and cheaper gates for the fused passes.  An
// uncontrolled diagonal, X or Y gate is multiplied into the matrix before it on
// its qubit where the gates between commute with it.  A matrix gives its right
// factor to the matrix before it where the gates between commute with that
// factor: a diagonal through controls and phases, an X rotation through CNOT
// targets.  What is left of it is (diagonal) x (real rotation), which a factored
// layer runs without pre factors (3/4 of its FP64 work).
std::vector<hgate> simplify_queue(int n, const std::vector<hgate>& gates);

// Plans `gates` (in order) into passes, updating the layout map
// perm (logical -> physical) and inv (physical -> logical).
void plan_passes(const plan_params& p, const std::vector<hgate>& gates, std::vector<int>& perm,
                 std::vector<int>& inv, std::vector<dev_pass>& out);
// The same, each pass handed to emit as soon as it is planned (perm and inv are
// those after it); emit returning false ends the planning, as does the result.
bool plan_passes(const plan_params& p, const std::vector<hgate>& gates, std::vector<int>& perm, std::vector<int>& inv,
                 const std::function<bool(const dev_pass&)>& emit);

// Passes that only move data so that perm becomes `target` (a permutation of
// 0..n-1: logical qubit q on physical bit target[q]); the multi-qubit form of
// ket::mpi's swap_permutated_local_qubits
// (ket/include/ket/mpi/utility/detail/swap_permutated_local_qubits.hpp:26-81).
void plan_layout(const plan_params& p, std::vector<int>& perm, std::vector<int>& inv, const std::vector<int>& target,
                 std::vector<dev_pass>& out);
// plan_layout to the identity.
void plan_canonicalize(const plan_params& p, std::vector<int>& perm, std::vector<int>& inv,
                       std::vector<dev_pass>& out);

// A small state's launch: at most kSmallGates gates in register phases.
struct small_program {
  std::vector<small_op> ops;
  std::vector<small_phase> phases;
};

// The queue in register phases of a small state: emit(ops, indices, phase) for
// each, with the ops in physical bits, the gates they come from, and the phase's
// register bits.  A phase takes, in order, every gate that commutes with those
// it leaves behind (it looks past a few hundred of them) and whose target is, or
// can still join, its register bits, at most max_ops of them and max_marked of
// the marked ones (marked: one entry per gate, or empty); SWAPs only update the
// layout map.  The time is linear in the number of gates.
void plan_small_phases(int n, const std::vector<hgate>& gates, std::vector<int>& perm, std::vector<int>& inv, size_t max_ops,
                       const std::vector<char>& marked, int max_marked,
                       const std::function<void(const std::vector<small_op>&, const std::vector<size_t>&, const small_phase&)>& emit);

// The queue as launches of the small-state kernel (n <= kSmallBits).
void plan_small(int n, const std::vector<hgate>& gates, std::vector<int>& perm, std::vector<int>& inv,
                std::vector<small_program>& out);

}  // namespace rbk
