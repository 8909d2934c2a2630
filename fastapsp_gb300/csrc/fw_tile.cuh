// fw_tile.cuh -- arithmetic shared by the (min,+) and Floyd-Warshall kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.cuh"

namespace fapk {

constexpr int kBlk = 64;  // 64-row / 64-column blocks (the Floyd-Warshall pivot block)

// Packed int32 form.  Keys are (min(d, kPackH) << 7) | idx: idx 0 marks the
// value the output held before the product, idx = k+1 the candidate k.  One
// DPX __viaddmin_u32 per add-min then yields the minimum and, on equal
// distances, the smallest idx -- the current value first, then the first k
// -- which is the strict-improvement, ascending-k rule of the reference.  Two
// keys sum to at most (2 * kPackH) << 7 | 127 < 2^32, so nothing wraps, and
// saturation at kPackH commutes with + and min, so the results are exact when
// every finite result stays below kPackH (checked by the caller).  With
// predecessors K <= 127, so the final idx names k* directly and the
// predecessor is read once, in the epilogue, from B's predecessor row k*.
constexpr unsigned kPackH = (1u << 24) - 1;
constexpr unsigned kIdxBits = 7;
constexpr unsigned kIdxMask = (1u << kIdxBits) - 1;
constexpr int kMaxPackedK = 127;

// Layout of the FP32 strip kernels' operands in shared memory: entry (k, m)
// of A^T and entry (k, col) of B sit at row k, position m ^ swz(k) and
// col ^ swz(k) -- the 4-entry chunks of step group k / 4 permuted by XOR with
// its low three bits.  Within a group the permutation is the same, so a
// thread's four consecutive rows or columns stay one aligned 16-byte chunk;
// after the add-mins, threads that look up entries of different step groups
// of the same rows or columns hit different banks.  The packed form keeps
// the plain layout (SWZ false).
template <bool SWZ>
__device__ __forceinline__ int swz(int k) {
  return SWZ ? ((k >> 2) & 7) << 2 : 0;
}

// Four add-mins of the FP32 kernels, steps k0 .. k0 + 3: the current value
// replaced by the minimum of the four sums when that is below it (a strict
// improvement), and then the group tag (k0 + 1) too.  That leaves the step of
// the last strict improvement in the tagged group: its first step whose sum
// equals the final value, since every earlier step's sum is above it
// (strip_resolve_f32 finds it after the loop).  Four FP32 adds, two 3-input
// minimums with the current value as an input, a compare and one select.
__device__ __forceinline__ void strip_addmin4_f32(unsigned &acc, int &tag, const unsigned a[4],
                                                  const unsigned b[4], int grp) {
  const unsigned v0 = __float_as_uint(__fadd_rn(__uint_as_float(a[0]), __uint_as_float(b[0])));
  const unsigned v1 = __float_as_uint(__fadd_rn(__uint_as_float(a[1]), __uint_as_float(b[1])));
  const unsigned v2 = __float_as_uint(__fadd_rn(__uint_as_float(a[2]), __uint_as_float(b[2])));
  const unsigned v3 = __float_as_uint(__fadd_rn(__uint_as_float(a[3]), __uint_as_float(b[3])));
  const unsigned nacc = __vimin3_u32(acc, __vimin3_u32(v0, v1, v2), v3);
  tag = nacc != acc ? grp : tag;
  acc = nacc;
}

// Two FP32 sums (steps k and k + 1) of operands held as pairs; their bits.
__device__ __forceinline__ uint2 add2_f32(unsigned long long a, unsigned long long b) {
  unsigned long long z;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(z) : "l"(a), "l"(b));
  return make_uint2((unsigned)z, (unsigned)(z >> 32));
}

// strip_addmin4_f32 on units of four steps: two paired adds instead of four.
__device__ __forceinline__ void unit_addmin_f32(unsigned &acc, int &tag, const ulonglong2 &a, const ulonglong2 &b,
                                                int grp) {
  const uint2 v = add2_f32(a.x, b.x), w = add2_f32(a.y, b.y);
  const unsigned nacc = __vimin3_u32(acc, __vimin3_u32(v.x, v.y, w.x), w.y);
  tag = nacc != acc ? grp : tag;
  acc = nacc;
}

// strip_resolve_f32 on the units of the tagged group.
__device__ __forceinline__ int unit_resolve_f32(unsigned acc, int tag, const ulonglong2 &a, const ulonglong2 &b) {
  const uint2 v = add2_f32(a.x, b.x), w = add2_f32(a.y, b.y);
  const int j = v.x == acc ? 0 : v.y == acc ? 1 : w.x == acc ? 2 : 3;
  return tag > 0 ? tag + j : 0;
}

// The step idx (k + 1) of an output whose last strict improvement fell in the
// group tagged `tag` (0: none): the group's first step whose sum has the
// final value's bits.  ap / bp point at the output's A and B entries of the
// group's first step (strides sa, sb between steps).
__device__ __forceinline__ int strip_resolve_f32(unsigned acc, int tag, const unsigned *ap, int sa,
                                                 const unsigned *bp, int sb) {
  const unsigned v0 = __float_as_uint(__fadd_rn(__uint_as_float(ap[0]), __uint_as_float(bp[0])));
  const unsigned v1 = __float_as_uint(__fadd_rn(__uint_as_float(ap[sa]), __uint_as_float(bp[sb])));
  const unsigned v2 = __float_as_uint(__fadd_rn(__uint_as_float(ap[2 * sa]), __uint_as_float(bp[2 * sb])));
  const int j = v0 == acc ? 0 : v1 == acc ? 1 : v2 == acc ? 2 : 3;
  return tag > 0 ? tag + j : 0;
}

}  // namespace fapk
