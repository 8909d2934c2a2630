// mp_common.cuh -- copies, segment lookup and row stores shared by the min-plus kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.cuh"

namespace fapk {

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::); }
__device__ __forceinline__ void cp_async_wait_0() { asm volatile("cp.async.wait_group 0;\n" ::); }

__device__ __forceinline__ const MpSegment &find_segment(const MpSegment *__restrict__ segs,
                                                         int nseg, int tile) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (segs[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
  }
  return segs[lo];
}

// In-part columns of the inner rows take the part's Floyd-Warshall values
// (the decode of MysubMatDecode_path, util_Myalgorithm.h:236-247, for these
// rows), so the min-plus epilogue writes every column once.
__device__ __forceinline__ bool fw_column(const MpSegment &s, int col, int64_t &off) {
  if (s.col_part == nullptr || s.col_part[col] != s.part) return false;
  off = (int64_t)(s.col_local[col] - s.local0);
  return true;
}

// Stores the values of a 64-column row segment held by 16 lanes (4
// consecutive columns a lane; p = this lane's first column) where the row is
// not 16-byte aligned: each lane stores the aligned 16-byte chunk that starts
// inside its quad, completed with the next lane's first values; the ragged
// ends of the segment (lane 0's values before the first boundary, lane 15's
// after the last) go as single stores.  All 32 lanes call it (the values
// move by shuffles within each half-warp); `ok` drops the stores of a row
// outside the matrix.  (A case split on the misalignment, which is the same
// for the whole warp, measured slower than these selects.)
template <typename V>
__device__ __forceinline__ void store_quad_unaligned(V *p, const V v[4], int tx, bool ok) {
  V nx[4];
#pragma unroll
  for (int q = 0; q < 4; q++) nx[q] = __shfl_down_sync(0xffffffffu, v[q], 1, 16);
  if (!ok) return;
  const int o = (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3);  // the same for the whole segment
  if (o == 0) {
    __stcs(reinterpret_cast<uint4 *>(p), make_uint4((unsigned)v[0], (unsigned)v[1], (unsigned)v[2], (unsigned)v[3]));
    return;
  }
  if (tx < 15) {  // chunk [p + 4 - o, p + 8 - o): v[4 - o .. 3], then nx[0 .. 3 - o]
    const V w0 = o == 1 ? v[3] : o == 2 ? v[2] : v[1];
    const V w1 = o == 1 ? nx[0] : o == 2 ? v[3] : v[2];
    const V w2 = o == 1 ? nx[1] : o == 2 ? nx[0] : v[3];
    const V w3 = o == 1 ? nx[2] : o == 2 ? nx[1] : nx[0];
    __stcs(reinterpret_cast<uint4 *>(p + 4 - o), make_uint4((unsigned)w0, (unsigned)w1, (unsigned)w2, (unsigned)w3));
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q >= 4 - o) p[q] = v[q];
  }
  if (tx == 0) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q < 4 - o) p[q] = v[q];
  }
}

// Whether the output rows allow 16-byte stores of 4 consecutive columns.
template <bool PRED>
__device__ __forceinline__ bool vec_stores_ok(const MpSegment &s) {
  bool ok = (s.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(s.C) & 15) == 0;
  if (PRED) ok = ok && (s.ldcp & 3) == 0 && (reinterpret_cast<uintptr_t>(s.Cp) & 15) == 0;
  return ok;
}

// Stores the 4 outputs of columns col0..col0+3 of `row` (those < N), after
// the part-column override; one 16-byte store per array when all 4 are in
// range and the rows are aligned.
template <typename T, bool PRED>
__device__ __forceinline__ void store_quad(const MpSegment &s, int row, int col0, T d[4],
                                           int32_t p[4], bool vec) {
#pragma unroll
  for (int q = 0; q < 4; q++) {
    int64_t j;
    if (col0 + q < s.N && fw_column(s, col0 + q, j)) {
      d[q] = static_cast<const T *>(s.F)[(int64_t)row * s.ldf + j];
      if (PRED) p[q] = s.Fp[(int64_t)row * s.ldf + j];
    }
  }
  T *crow = static_cast<T *>(s.C) + (int64_t)row * s.ldc;
  int32_t *prow = PRED ? s.Cp + (int64_t)row * s.ldcp : nullptr;
  if (vec && col0 + 3 < s.N) {
    uint4 dv;
    dv.x = Dist<T>::bits(d[0]);
    dv.y = Dist<T>::bits(d[1]);
    dv.z = Dist<T>::bits(d[2]);
    dv.w = Dist<T>::bits(d[3]);
    *reinterpret_cast<uint4 *>(crow + col0) = dv;
    if (PRED) *reinterpret_cast<int4 *>(prow + col0) = make_int4(p[0], p[1], p[2], p[3]);
    return;
  }
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (col0 + q < s.N) {
      crow[col0 + q] = d[q];
      if (PRED) prow[col0 + q] = p[q];
    }
}

// Numbers the strips of a launch and chooses their length in 128-column units.
// CTAs of an SM share its issue slots, so the launch ends with the SM that got
// the most strips: their number rounded up, times a strip's 64-column tiles and
// two more for its start (the staging of A), is made least over the lengths that
// give nearly every slot of the GPU (`per_sm` CTAs an SM) a strip; the shortest
// where none does.  Against the longest power of two with three strips an SM:
// 877 x 114,599 x 19 FP32 475 -> 439 us, 2,000 x 20,000 x 19 FP32 204 -> 181 us;
// counting turns of the slots instead takes 384 strips for 4,000 x 9,000 x 36
// packed, 203 us instead of 189 (576 strips).
// `strips` gives a segment's strips of a length.
template <typename Strips>
inline int number_strips(MpSegment *segs, int nseg, int sm_count, int per_sm, int *per, Strips strips) {
  auto count = [&](int units) {
    long long n = 0;
    for (int i = 0; i < nseg; i++) n += strips(segs[i], units);
    return n;
  };
  long long best = -1;
  *per = 1;
  for (int units = 1; units <= 16; units++) {
    const long long n = count(units), cost = (n + sm_count - 1) / sm_count * (2 * units + 2);
    if (n * 20 >= 17LL * per_sm * sm_count && (best < 0 || cost <= best)) best = cost, *per = units;
  }
  int n = 0;
  for (int i = 0; i < nseg; i++) {
    segs[i].strip_begin = n;
    n += strips(segs[i], *per);
  }
  return n;
}

}  // namespace fapk
