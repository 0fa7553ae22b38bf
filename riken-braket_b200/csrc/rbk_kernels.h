// rbk_kernels.h -- host-side launchers of the kernels in rbk_kernels.cu.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "rbk_internal.h"

namespace rbk {

constexpr int kMaxPauliTerms = 64;

// Pauli strings that share one flip mask, as weights of sign patterns:
//   W(i) = sum_t w_t * (-1)^popcount(i & sign_t)     (physical bits)
struct pauli_terms {
  int count;
  uint64_t sign[kMaxPauliTerms];
  double w[kMaxPauliTerms][2];
};

// One fused pass with tile shape `shape` (see tile_shape in rbk_internal.h).
template <typename Real> cudaError_t launch_tile_pass(void* state, int n, const dev_pass& pass, int shape, cudaStream_t stream);
// One small-state program (plan_small) on a state of n <= kSmallBits qubits.
template <typename Real> cudaError_t launch_small(void* state, int n, const small_op* ops, int num_ops, const small_phase* phases,
                                                  int num_phases, cudaStream_t stream);
template <typename Real> cudaError_t launch_set_basis(void* state, int n, uint64_t index, cudaStream_t stream);
// ket::shor_box on a zeroed state: 2^nx amplitudes of value coeff (divisor, base < 2^32).
template <typename Real>
cudaError_t launch_shor_box(void* state, int n, int nx, uint64_t divisor, uint64_t base, double coeff, cudaStream_t stream);

int reduction_blocks();

// Records msg as the calling thread's rbk_last_error() and returns code.
int set_last_error(int code, const char* msg);
// Scratch needed by the reductions below, in doubles.
// The most is the Z sums' 512 blocks of 1 + n sums (1.3 MB of slack on top made
// creating a state map fresh device memory more often than not).
inline size_t reduction_scratch_doubles() { return size_t(1 << 9) * (1 + kMaxQubits) + 64; }

template <typename Real> cudaError_t launch_zsum(const void* state, int n, double* partials, double* out, cudaStream_t stream);
template <typename Real> cudaError_t launch_pauli(const void* state, int n, uint64_t flip, const pauli_terms& terms,
                                                  double* partials, double* out, cudaStream_t stream);
// <b| sum_t w_t P_t |a> for strings sharing the flip mask `flip`.
template <typename Real> cudaError_t launch_pauli2(const void* a, const void* b, int n, uint64_t flip, const pauli_terms& terms,
                                                   double* partials, double* out, cudaStream_t stream);
template <typename Real> cudaError_t launch_inner(const void* a, const void* b, int n, double* partials, double* out,
                                                  cudaStream_t stream);
template <typename Real> cudaError_t launch_probs(const void* state, uint64_t offset, uint64_t count, double* out,
                                                  cudaStream_t stream);

// A sum of Pauli strings grouped by flip mask, for applying H to a state:
// group g holds terms [begin[g], begin[g+1]).
constexpr int kMaxSumGroups = 64;
constexpr int kMaxSumTerms = 128;
struct pauli_sum {
  int num_groups;
  int pad;
  uint64_t flip[kMaxSumGroups];
  int begin[kMaxSumGroups + 1];
  int pad2;
  uint64_t sign[kMaxSumTerms];
  double w[kMaxSumTerms][2];
};

template <typename Real> cudaError_t launch_pauli_apply(const void* src, void* dst, int n, const pauli_sum& P, cudaStream_t stream);
// The same sum in tiled passes: each pass takes the groups whose flip bits lie
// in one tile layout (the low 3 bits plus up to 8 more), reads src once and
// writes (first pass) or adds to dst; the diagonal group rides in the first
// pass.  Falls back to launch_pauli_apply below 11 qubits or when a group's
// flip does not fit one layout.
template <typename Real> cudaError_t launch_pauli_apply_tiled(const void* src, void* dst, int n, const pauli_sum& P,
                                                              cudaStream_t stream);
// Up to kMaxOverlaps overlaps <lam| P_y |psi> in one launch; out[2y], out[2y+1] = (re, im) of overlap y.
constexpr int kMaxOverlaps = 64;
struct overlap_spec { uint64_t flip, sign; double wr, wi; };
struct overlap_set { int count; int pad; overlap_spec spec[kMaxOverlaps]; };
size_t overlaps_partials_doubles();
template <typename Real> cudaError_t launch_overlaps(const void* lam, const void* psi, int n, const overlap_set& set,
                                                     double* partials, double* out, cudaStream_t stream);
// The same for overlaps whose flip bits are all tile bits of one tile layout:
// each state is read once per launch.  flip_local / sign_local are tile-index
// masks; sign bits outside the tile go in sign (physical); the result of spec y
// goes to out[2 out_slot], out[2 out_slot + 1].  K <= 12.
struct tile_overlap_spec { uint32_t flip_local, sign_local; uint64_t sign; double wr, wi; int32_t out_slot, pad; };
struct tile_overlap_set {
  int count, K;
  uint8_t tile_phys[16];
  uint8_t num_runs, run_src[16], run_len[16], run_dst[16];
  tile_overlap_spec spec[kMaxOverlaps];
};
size_t tile_overlaps_partials_doubles(int n, int K);

template <typename Real> cudaError_t launch_tile_overlaps(const void* lam, const void* psi, int n, const tile_overlap_set& set,
                                                          double* partials, double* out, cudaStream_t stream);

// The register phases of a tile of 2^(8 + RB) amplitudes held by 256 threads, and
// where its other bits lie: tile t's bits outside tile_phys spell t, deposited
// run by run; in phase p a thread holds the 2^RB amplitudes whose tile bits
// phase_reg[p][0..RB-1] vary, at the tile bits phase_thr[p][0..7] that its
// index gives; flip f = p * RB + k is register bit k of phase p (entries past
// nflips are fillers).
constexpr int kSpinPhases = 4;
struct spin_group {
  int K, num_runs, nflips, nphases;
  uint8_t tile_phys[16], run_src[16], run_len[16], run_dst[16];
  uint8_t phase_reg[kSpinPhases][4];
  uint8_t phase_thr[kSpinPhases][8];
};

// One-qubit sums of one tile layout in one read of the state.  Tile bits
// tile_phys[0..K-1] (K = kObserveTileBits), the tile index deposited run by run
// into the others.  For every tile bit b in flip_mask
//   x_b = sum over j with tile bit b clear of conj(a_j) a_{j | b}   (complex);
// with `zsums`, sum |a_j|^2 in all and over j with each physical bit set; with
// diag_classes > 0, sum |a_j|^2 W(j), W(j) = sum_t w_t (-1)^popcount(j & sign_t)
// over diag_terms real-weighted Z-type strings.  The strings come in classes of
// one weight and one pattern on the thread's register bits (the top RB tile
// bits), sorted by pattern: class c has the strings of bit mask class_mask[c].
// out: (x_b re, im) for the bits of flip_mask in ascending order, then 1 + n
// sums (zsums), then the diagonal sum (diag_classes > 0).
constexpr int kObserveTerms = 64;
constexpr int kObserveRegBits = 3;
constexpr int kObserveTileBits = 8 + kObserveRegBits;
struct observe_group {
  int32_t K, num_runs, flip_mask, zsums, diag_terms, diag_classes;  // zsums or diag_classes > 0, not both
  uint8_t tile_phys[16], run_src[16], run_len[16], run_dst[16];
  uint64_t sign[kObserveTerms];
  uint64_t class_mask[kObserveTerms];
  double class_w[kObserveTerms];
  uint8_t class_begin[(1 << kObserveRegBits) + 1];  // classes of register pattern p: [begin[p], begin[p + 1])
};
int observe_width(const observe_group& g, int n);
template <typename Real> cudaError_t launch_observe(const void* state, int n, const observe_group& g, double* partials, double* out,
                                                    cudaStream_t stream);
// The same for a small state (n <= kObserveSmallBits), in one launch: every x_b, the
// 1 + n sums of |a_j|^2, and the diagonal sum of `terms` (real weights), in that order.
constexpr int kObserveSmallBits = 12;
template <typename Real> cudaError_t launch_observe_small(const void* state, int n, const pauli_terms& terms, double* out,
                                                          cudaStream_t stream);

// Overlaps of one-qubit Paulis in one read of both states (the adjoint sweep's
// rotation runs).  Z type: S_q = sum_j (-1)^{j_q} conj(lam_j) psi_j for
// physical bit q; out[2 slot] = w * S_q for each entry.
struct zsum2_set {
  int count, pad;
  struct { int32_t bit, out_slot; double wr, wi; } spec[kMaxOverlaps];
};
// X / Y type, for the flips of one tile layout (spin_group with K = 11: three
// register bits and eight thread bits, both states' tiles in shared memory):
//   A_f = sum over j with tile bit b_f clear of conj(lam_j) psi_{j | b_f},
//   B_f = the same with lam and psi exchanged in position (conj(lam_{j | b_f}) psi_j),
// out[2 slot_f] = w_f (A_f + B_f) (X, minus 0) or w_f (A_f - B_f) (Y: minus 1,
// the sign bit is the flip).
constexpr int kMaxPairFlips = 8;
constexpr int kPairRegBits = 3;
struct pair_overlap_set {
  spin_group g;
  struct { int32_t out_slot, minus; double wr, wi; } flip[kMaxPairFlips];
};
size_t pair_overlaps_partials_doubles();
// The one-qubit gates of an adjoint run applied to both states in the same
// read and write, with the X / Y-type overlaps of the run's rotations taken
// from that read.  Same tile layout as pair_overlap_set, up to kMaxRotFlips
// register-phase bits (every tile bit).  Flip f: the overlap (as in
// pair_overlap_set; out_slot < 0 for none) from the amplitudes before its
// gate, then m (m00 m01 m10 m11 as (re, im)) on lam and psi.  The gates act on
// distinct bits and commute, so an overlap is the same whichever of the other
// gates are already applied.  Only the imaginary part of w (A + s B), which the
// gradient takes, is summed: out[2 slot] = 0, out[2 slot + 1] = Im.
// okind picks the arithmetic of the overlap: 1 when wr = 0 (only the real parts
// of A and B enter, as for Y types), 2 when wi = 0 (only the imaginary parts, X
// types), 3 otherwise (0: no overlap); mkind 1 marks a real matrix (EY, H),
// 2 a filler position without a gate.  Phase 0 must be the load layout:
// register bits 8, 9, 10 and thread bits 0..7 of the tile, in order.
// block_sync[p] = 1: the layout after phase p (the next phase's, or the load
// layout for the store) puts other tile bits on the warp index, so the
// exchange waits for the whole CTA; 0: every warp reads back only slots it
// wrote itself, and a warp barrier suffices.
constexpr int kMaxRotFlips = 12;
// Optional first step of a launch: a diagonal that both states still owe,
// applied at load time, and Z-type overlaps taken there (a diagonal with
// |d| = 1 leaves conj(lam_j) psi_j unchanged, so before or after is the same).
//   factor(j) = g * prod over the physical bits b set in j of u[b] * (-1)^Q(j),
//   Q(j) = sum over the bits b set in j of popcount(j & adj[b])   (mod 2),
// adj[b] holding b's controlled-Z partners above b.  For register slot it
// (tile bits 8..10), mr[it] is the XOR of the full partner rows of its set
// bits and bit it of qr the parity of its pairs among themselves.  Z entries:
// out[2 slot + 1] = wr Im(S_q), S_q = sum_j (-1)^{j_q} conj(lam_j) psi_j, out[2 slot] = 0.
struct pre_diag {
  int32_t active, nz;
  double g[2];
  double u[kMaxQubits][2];
  uint64_t adj[kMaxQubits];
  uint64_t full[kMaxQubits];  // all partners of each bit (both directions)
  uint64_t mr[8];
  uint32_t qr, pad;
  struct { int32_t bit, out_slot; double wr; } z[kMaxQubits];
};
struct pair_rotate_set {
  spin_group g;
  struct { int32_t out_slot, minus, okind, mkind; double wr, wi; double m[8]; } flip[kMaxRotFlips];
  uint8_t block_sync[kSpinPhases];
  uint8_t pad[4];
  pre_diag pre;
};
size_t pair_rotate_partials_doubles();  // per block: nflips overlap sums, then 1 + n Z sums when pre.nz > 0
// A launch leaves its partial sums at partials[begin ..] (*used doubles of them)
// and adds what they mean to `results`; launch_finish_pair_rotate forms the
// overlaps of many launches at once (a finish after each took 5 us and a launch,
// 48 times in a 20-qubit gradient of 16 layers).
struct pair_rotate_result {
  uint64_t begin;
  int32_t blocks, width, column, second, slot, pad;
  double w;
};
template <typename Real> cudaError_t launch_pair_rotate(void* lam, void* psi, int n, const pair_rotate_set& set, double* partials,
                                                        size_t begin, std::vector<pair_rotate_result>& results, size_t* used,
                                                        cudaStream_t stream);
cudaError_t launch_finish_pair_rotate(const double* partials, const pair_rotate_result* entries, int count, double* out,
                                      cudaStream_t stream);
template <typename Real> cudaError_t launch_zsum2(const void* lam, const void* psi, int n, const zsum2_set& set,
                                                  double* partials, double* out, cudaStream_t stream);
template <typename Real> cudaError_t launch_pair_overlaps(const void* lam, const void* psi, int n, const pair_overlap_set& set,
                                                          double* partials, double* out, cudaStream_t stream);

// Sampling: block sums and chunk prefixes of |a_i|^2 in scratch
// (sample_scratch_doubles(n) doubles; *total: device address of the sum over the
// state), then events[k] = upper_bound of r[k] among the prefix sums.
size_t sample_scratch_doubles(int n);
template <typename Real> cudaError_t launch_sample_sums(const void* amps, int n, double* scratch, const double** total,
                                                        cudaStream_t stream);
template <typename Real> cudaError_t launch_sample(const void* amps, int n, const double* scratch, const double* r, int num,
                                                   uint64_t* events, cudaStream_t stream);

// Dense k-qubit unitaries.
// Tensor cores (complex<float>, k = 5 or 6, n >= k + 7): w_split holds W_hi then
// W_lo (tc_w_split_floats(k) floats) in the kernel's operand layout; the kernel
// needs tc_shared_bytes(k) of shared memory and sets *error_flag on a timeout.
// Physical bits of the tensor-core kernel's rows: target_bit[i] is target i, row_bit[j]
// row-index bit j of a 128-row tile, and the tile index is deposited run by run
// into the remaining bits (n >= k + 7).
struct tc_layout {
  uint8_t target_bit[6];
  uint8_t row_bit[7];
  uint8_t num_runs;
  uint8_t run_src[16], run_len[16], run_dst[16];
};
size_t tc_w_split_floats(int k);
size_t tc_shared_bytes(int k);
cudaError_t launch_unitary_tf32x3(void* state, int n, int k, const float* w_split, int* error_flag, int grid,
                                  const tc_layout& layout, cudaStream_t stream);
// CUDA cores, any precision.  U is 2^k x 2^k complex (re, im) in row-major order
// on the device.  k <= kBlockMaxBits: tiles of 2^kBlockTileBits amplitudes (the
// whole state where n is smaller; elems amplitudes) over tile_phys, ascending;
// tile_local[b] is 1 << (kBlockTileBits - k + i) where tile bit b is target i,
// and 1 << r where it is row bit r.
constexpr int kBlockMaxBits = 6;
constexpr int kBlockTileBits = 11;
struct block_layout {
  uint32_t elems;
  uint16_t tile_local[kBlockTileBits];
  uint8_t tile_phys[kBlockTileBits];
  uint8_t num_runs, run_src[16], run_len[16], run_dst[16];
};
template <typename Real> cudaError_t launch_block_unitary(void* state, int n, int k, const double* U, const block_layout& layout,
                                                          cudaStream_t stream);
// k <= 10, targets on the low k physical bits.
template <typename Real> cudaError_t launch_dense_rows(void* state, int n, int k, const double* U, cudaStream_t stream);

}  // namespace rbk
