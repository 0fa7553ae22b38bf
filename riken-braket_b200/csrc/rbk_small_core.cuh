// rbk_small_core.cuh -- the gates of a small-state phase on a thread's registers
// (small_op in rbk_internal.h), shared by the one-CTA circuits and the one-launch
// gradients.
//
// These kernels run one to four warps per scheduler, so what a gate costs is its
// chain of dependent steps.  The record's header comes as one 16-byte load and
// its matrix as four more, issued together; one jump picks straight-line code for
// the target bit; and sign flips (Z, CZ) are only noted, in a mask of register
// slots, and applied before the next gate that mixes slots.  With fields loaded
// one by one and branches per pair a gate took about 0.5 us (8 qubits, one warp,
// 200 random gates: 106 us, now 90; 8-qubit
// brick with spins 112 -> 101 us, batch of 96 gradients of 10 to 15 qubits 3.69 -> 2.37 ms).
#pragma once

#include "rbk_device.cuh"
#include "rbk_internal.h"

namespace rbk {

constexpr int kSmallSlots = 1 << kSmallRegBits;
constexpr uint32_t kAllSlots = (1u << kSmallSlots) - 1;

// A record's first 16 bytes, unpacked where they are used.
struct small_header {
  uint4 v;
  __device__ __forceinline__ uint32_t code() const { return v.x & 0xff; }
  __device__ __forceinline__ uint32_t act() const { return (v.x >> 8) & 0xff; }
  __device__ __forceinline__ uint32_t hi() const { return (v.x >> 16) & 0xff; }
  __device__ __forceinline__ uint32_t rot() const { return v.x >> 24; }
  __device__ __forceinline__ uint32_t cbase() const { return v.y & 0xffff; }
  __device__ __forceinline__ uint32_t dbase() const { return v.y >> 16; }
  __device__ __forceinline__ int32_t slot() const { return int32_t(v.z); }
};

__device__ __forceinline__ small_header small_load_header(const small_op* op)
{
  return {*reinterpret_cast<const uint4*>(op)};
}

// The matrix (a diagonal gate's factors in m00 and m01), or its inverse: the
// conjugate transpose.
struct small_matrix { double2 m00, m01, m10, m11; };
template <bool INV>
__device__ __forceinline__ small_matrix small_load_matrix(const small_op* op, uint32_t code)
{
  const double2* m = reinterpret_cast<const double2*>(op->m);
  small_matrix r{m[0], m[1], m[2], m[3]};
  if (INV) {
    const double2 t = r.m01, u = code >= SMALL_DIAG ? r.m01 : r.m10;
    r = {double2{r.m00.x, -r.m00.y}, double2{u.x, -u.y}, double2{t.x, -t.y}, double2{r.m11.x, -r.m11.y}};
  }
  return r;
}

__device__ __forceinline__ double small_flip(double v, uint32_t sign)  // sign: 0 or 1 << 31
{
  return __hiloint2double(__double2hiint(v) ^ int(sign), __double2loint(v));
}

// Applies the noted sign flips.
__device__ __forceinline__ void small_signs(double2 (&a)[kSmallSlots], uint32_t signs)
{
#pragma unroll
  for (int i = 0; i < kSmallSlots; ++i) {
    const uint32_t s = (signs << (31 - i)) & 0x80000000u;
    a[i].x = small_flip(a[i].x, s);
    a[i].y = small_flip(a[i].y, s);
  }
}

__device__ __forceinline__ double small_select(bool p, double a, double b)
{
  return __hiloint2double(p ? __double2hiint(a) : __double2hiint(b), p ? __double2loint(a) : __double2loint(b));
}

// KIND 0: any matrix, 1: real, 2: X, 3: Y, on register bit B of the slots in act.
// X and Y move values through selects on act, also where all slots are in it: as
// plain swaps in one arm of the dispatch they made the arms' register
// assignments disagree, and the copies where they rejoin spilled.
template <int B, int KIND, bool ALL>
__device__ __forceinline__ void small_pairs(double2 (&a)[kSmallSlots], uint32_t act, const small_matrix& m)
{
#pragma unroll
  for (int i = 0; i < kSmallSlots; ++i) {
    if (i & (1 << B)) continue;
    double2 &x = a[i], &y = a[i | (1 << B)];
    const double2 a0 = x, a1 = y;
    const bool in = (act >> i) & 1u;
    if constexpr (KIND == 2) {
      x = double2{small_select(in, a1.x, a0.x), small_select(in, a1.y, a0.y)};
      y = double2{small_select(in, a0.x, a1.x), small_select(in, a0.y, a1.y)};
    } else if constexpr (KIND == 3) {
      x = double2{small_select(in, a1.y, a0.x), small_select(in, -a1.x, a0.y)};
      y = double2{small_select(in, -a0.y, a1.x), small_select(in, a0.x, a1.y)};
    } else {
      if (!ALL && !in) continue;
      if constexpr (KIND == 0) {
        x = cmac2(a0, a1, m.m00.x, m.m00.y, m.m01.x, m.m01.y);
        y = cmac2(a0, a1, m.m10.x, m.m10.y, m.m11.x, m.m11.y);
      } else {
        x = rmac2(a0, a1, m.m00.x, m.m01.x);
        y = rmac2(a0, a1, m.m10.x, m.m11.x);
      }
    }
  }
}

// One target gate on one state or on both (the adjoint sweep's).
template <int B, int KIND, bool TWO>
__device__ __forceinline__ void small_target(double2 (&a)[kSmallSlots], double2 (&l)[kSmallSlots], uint32_t act, const small_matrix& m)
{
  if (KIND >= 2 || act == kAllSlots) {
    small_pairs<B, KIND, true>(a, act, m);
    if (TWO) small_pairs<B, KIND, true>(l, act, m);
  } else {
    small_pairs<B, KIND, false>(a, act, m);
    if (TWO) small_pairs<B, KIND, false>(l, act, m);
  }
}

// a[i] *= the slot's factor: f1 on the slots of m1, f0 on those of m0.
__device__ __forceinline__ void small_factors(double2 (&a)[kSmallSlots], uint32_t m0, uint32_t m1, double2 f0, double2 f1)
{
#pragma unroll
  for (int i = 0; i < kSmallSlots; ++i) {
    const bool one = (m1 >> i) & 1u;
    const double2 f{one ? f1.x : f0.x, one ? f1.y : f0.y};
    if (((m0 | m1) >> i) & 1u) a[i] = cmul(a[i], f);
  }
}

// The gate `op` (its header h) or its inverse on the registers of a thread with
// base index `base`, on one state or on both; `signs` holds the sign flips not
// applied yet.
template <bool TWO, bool INV>
__device__ __forceinline__ void small_gate(double2 (&a)[kSmallSlots], double2 (&l)[kSmallSlots], const small_header& h,
                                           const small_op* op, uint32_t base, uint32_t& signs)
{
  const uint32_t code = h.code(), act = h.act();
  const bool on = (base & h.cbase()) == h.cbase();
  if (code == SMALL_NEG) {
    if (on) signs ^= act;
    return;
  }
  const small_matrix m = small_load_matrix<INV>(op, code);
  if (code >= SMALL_DIAG) {
    if (!on) return;
    const uint32_t m1 = act & ((base & h.dbase()) ? kAllSlots : h.hi());
    const uint32_t m0 = code == SMALL_DIAG ? act & ~m1 : 0u;
    small_factors(a, m0, m1, m.m00, m.m01);
    if (TWO) small_factors(l, m0, m1, m.m00, m.m01);
    return;
  }
  if (signs) {
    small_signs(a, signs);
    if (TWO) small_signs(l, signs);
    signs = 0;
  }
  if (!on) return;
  switch (code) {
    case SMALL_MAT + 0: small_target<0, 0, TWO>(a, l, act, m); break;
    case SMALL_MAT + 1: small_target<1, 0, TWO>(a, l, act, m); break;
    case SMALL_MAT + 2: small_target<2, 0, TWO>(a, l, act, m); break;
    case SMALL_REAL + 0: small_target<0, 1, TWO>(a, l, act, m); break;
    case SMALL_REAL + 1: small_target<1, 1, TWO>(a, l, act, m); break;
    case SMALL_REAL + 2: small_target<2, 1, TWO>(a, l, act, m); break;
    case SMALL_X + 0: small_target<0, 2, TWO>(a, l, act, m); break;
    case SMALL_X + 1: small_target<1, 2, TWO>(a, l, act, m); break;
    case SMALL_X + 2: small_target<2, 2, TWO>(a, l, act, m); break;
    case SMALL_Y + 0: small_target<0, 3, TWO>(a, l, act, m); break;
    case SMALL_Y + 1: small_target<1, 3, TWO>(a, l, act, m); break;
    default: small_target<2, 3, TWO>(a, l, act, m); break;
  }
}

}  // namespace rbk
