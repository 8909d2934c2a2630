// fw_pivot.cu -- the pivot chain of the blocked Floyd-Warshall.
//
// Reference counterparts: floyd_CPU_path (fap/kernel/floyd.h:38-49) and the
// first two phases of the GPU form (fw_kernel1, FW_kernel1A2,
// fap/kernel/cuda/floyd.cu:26-267).
//
// Round r of the blocked form closes the pivot block (r, r) and updates block
// row and column r with it (the panels); the remaining tiles follow in
// fw_rest.cu, except block row and column r + 1, which get
// round r's update here, at the start of round r + 1, so that they need not
// wait for the other tiles (lookahead).  Two launches a round over all the
// matrices of a batch:
//
//   fw_close_kernel  one CTA per matrix: round r - 1's update of the pivot
//                    block, then its closure;
//   fw_panel_kernel  one CTA per 64 x 64 block of block row and column r:
//                    round r - 1's update, then the product with the closed
//                    pivot block, the block staying in registers and shared
//                    memory between the two.
//
// The panel kernel rewrites blocks (r, r - 1) and (r - 1, r) while its other
// CTAs use their earlier values; the closing kernel leaves those values in a
// copy of its own.
//
// The chain is what a few matrices' rounds cost, and it is latency: a CTA per
// block spreads it over the GPU, and no tile is half empty.  One 910-vertex
// FP32 matrix took 82 us a round (update, closure and panels in three strip
// launches of 128-row tiles) and takes 44; 256 FP32 matrices of 256 to 1,024
// vertices 23.9 -> 18.9 ms; 512 int32 matrices of 32 to 2,048 (a cluster of
// four CTAs a matrix, walking its panel blocks) 58.2 -> 51.3 ms.  Of the chain
// of one FP32 matrix (39 us at 2.07 GHz): loads 3, each 64^3 product 4 (32
// add-mins a cycle on its one SM), the closure 9, its steps 2.6.  At two CTAs an
// SM the kernels have 64 registers a thread, and the FP32 ones with predecessors
// spill (stores / loads: closing 56 / 80 bytes, panels 184 / 108).

#include <cuda_runtime.h>
#include <stdint.h>

#include "fw_tile.cuh"
#include "kernels.cuh"
#include "launch.h"

namespace fapk {

namespace {

// A 64 x 64 block, 4 rows x 2 columns a thread, a warp all columns of its rows.
// (256 threads of 4 x 4 entries issued 0.39 instructions a cycle and scheduler,
// two warps each waiting on their own chains.)
constexpr int kPivThreads = 512;
constexpr int kPivC = 2;

// Words of a matrix's copies of blocks (r + 1, r) and (r, r + 1), and of the
// latter's predecessors.
constexpr int64_t kLookWords = 3 * kBlk * kBlk;

// Operands of a 64^3 product in shared memory.  A by step: entry (k, row) at
// k * 64 + (row ^ swz(k)); B the same with columns (the packed form's B
// unswizzled): a thread's four rows or two columns of a step are one chunk, and
// A's transposing stores and the FP32 resolve hit different banks.

// A block as a thread holds it: rows 4 ty + i, columns 2 tx + c.
template <typename V>
__device__ __forceinline__ void block_load(V (&out)[4][kPivC], const V *base, int64_t ld, int rb, int cb, int size,
                                           V fill, bool vec) {
  const int r0 = rb * kBlk + (threadIdx.x >> 5) * 4, c0 = cb * kBlk + (threadIdx.x & 31) * kPivC;
  const V *p = base + (int64_t)r0 * ld + c0;
  // the whole block inside (uniform over the CTA): loads without a test between them
  if (rb * kBlk + kBlk <= size && cb * kBlk + kBlk <= size) {
    if (vec) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint2 v = *reinterpret_cast<const uint2 *>(p + i * ld);
        out[i][0] = (V)v.x, out[i][1] = (V)v.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < kPivC; c++) out[i][c] = p[i * ld + c];
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < kPivC; c++) out[i][c] = r0 + i < size && c0 + c < size ? p[i * ld + c] : fill;
}

// FP32: entries above "unreached" (infinities) are unreached.  Every block is a
// panel once or twice, or the pivot block, and these write unreached entries too,
// so a closed matrix holds one value for them.
template <bool F32>
__device__ __forceinline__ void cap_unreached(unsigned (&v)[4][kPivC]) {
  if (!F32) return;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < kPivC; c++) v[i][c] = min(v[i][c], __float_as_uint(Dist<float>::inf()));
}

// A thread's part of an operand into shared memory, and the step groups (of
// four) that it has a finite entry in: as A (transposed; its columns are the
// steps) or as B (its rows are).
template <bool F32>
__device__ __forceinline__ unsigned store_a(unsigned *A, const unsigned (&v)[4][kPivC]) {
  const int ty = threadIdx.x >> 5, tx = threadIdx.x & 31;
  const unsigned INF = F32 ? __float_as_uint(Dist<float>::inf()) : kPackH;
  unsigned low = ~0u;
#pragma unroll
  for (int c = 0; c < kPivC; c++) {
    const int k = tx * kPivC + c;
    uint4 x = make_uint4(v[0][c], v[1][c], v[2][c], v[3][c]);
    low = min(low, min(min(x.x, x.y), min(x.z, x.w)));
    if (!F32)
      x = make_uint4(min(x.x, kPackH) << kIdxBits, min(x.y, kPackH) << kIdxBits, min(x.z, kPackH) << kIdxBits,
                     min(x.w, kPackH) << kIdxBits);
    *reinterpret_cast<uint4 *>(A + k * kBlk + ((ty * 4) ^ swz<true>(k))) = x;
  }
  return low < INF ? 1u << (tx * kPivC >> 2) : 0u;
}
template <bool F32>
__device__ __forceinline__ unsigned store_b(unsigned *B, const unsigned (&v)[4][kPivC]) {
  const int ty = threadIdx.x >> 5, tx = threadIdx.x & 31;
  const unsigned INF = F32 ? __float_as_uint(Dist<float>::inf()) : kPackH;
  unsigned low = ~0u;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint2 x = make_uint2(v[i][0], v[i][1]);
    low = min(low, min(x.x, x.y));
    const unsigned id = (unsigned)(ty * 4 + i + 1);
    if (!F32) x = make_uint2((min(x.x, kPackH) << kIdxBits) | id, (min(x.y, kPackH) << kIdxBits) | id);
    *reinterpret_cast<uint2 *>(B + (ty * 4 + i) * kBlk + ((tx * kPivC) ^ swz<F32>(ty * 4))) = x;
  }
  return low < INF ? 1u << ty : 0u;
}

// c = min(c, A (x) B) over the step groups of `groups`, ties keeping c; step
// (k + 1, 0: kept) says which k an entry took.
template <bool F32, bool PRED>
__device__ __forceinline__ void block_product(unsigned (&c)[4][kPivC], int (&step)[4][kPivC], const unsigned *A,
                                              const unsigned *B, unsigned groups) {
  const int ty = threadIdx.x >> 5, tx = threadIdx.x & 31;
  unsigned acc[4][kPivC];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < kPivC; j++) {
      acc[i][j] = F32 ? __float_as_uint(Dist<float>::inf()) : kPackH << kIdxBits;
      step[i][j] = 0;
    }
  auto four = [&](int k0) {  // steps k0 .. k0 + 3
    const unsigned *ap = A + k0 * kBlk + ((ty * 4) ^ swz<true>(k0));
    const unsigned *bp = B + k0 * kBlk + ((tx * kPivC) ^ swz<F32>(k0));
    unsigned a[4][4], b[kPivC][4];  // [row or column][step]
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint4 x = *reinterpret_cast<const uint4 *>(ap + q * kBlk);
      const uint2 y = *reinterpret_cast<const uint2 *>(bp + q * kBlk);
      a[0][q] = x.x, a[1][q] = x.y, a[2][q] = x.z, a[3][q] = x.w;
      b[0][q] = y.x, b[1][q] = y.y;
    }
    if constexpr (F32) {
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < kPivC; j++) strip_addmin4_f32(acc[i][j], step[i][j], a[i], b[j], k0 + 1);
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < kPivC; j++) acc[i][j] = __viaddmin_u32(a[i][q], b[j][q], acc[i][j]);
    }
  };
  if (groups == 0xffffu) {
#pragma unroll 2
    for (int k0 = 0; k0 < kBlk; k0 += 4) four(k0);
  } else {
    for (unsigned left = groups; left; left &= left - 1) four((__ffs(left) - 1) * 4);
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < kPivC; j++) {
      if constexpr (F32) {
        int s = 0;
        if (acc[i][j] < c[i][j]) {
          c[i][j] = acc[i][j];
          s = 1;
          if (PRED) {
            const int k0 = max(step[i][j] - 1, 0), sw = swz<true>(k0);
            s = strip_resolve_f32(acc[i][j], step[i][j], A + k0 * kBlk + ((ty * 4) ^ sw) + i, kBlk,
                                  B + k0 * kBlk + ((tx * kPivC) ^ sw) + j, kBlk);
          }
        }
        step[i][j] = s;
      } else {
        const unsigned key = min(min(c[i][j], kPackH) << kIdxBits, acc[i][j]);
        step[i][j] = (int)(key & kIdxMask);
        if (step[i][j]) c[i][j] = key >> kIdxBits;
      }
    }
}

// The OR of every thread's mask (a barrier on either side of the caller's
// writes to the operands is the caller's).
__device__ __forceinline__ void mask_or(unsigned *dst, unsigned mine) {
  mine = __reduce_or_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicOr(dst, mine);
}

struct CloseSmem {
  // Round prev's operands; then, row k: column k (A, as an operand) and row k
  // (B) of the block as they stood at step k.
  unsigned A[kBlk * kBlk], B[kBlk * kBlk];
  int32_t P[kBlk][kBlk];        // predecessors: round prev's, then the block's own
  unsigned S[kBlk][kBlk];       // row k's last steps as they stood at step k (packed: in its keys)
  unsigned vr[4][kBlk], vt[4][kBlk], vc[4][kBlk];  // the next four rows, their steps, and columns
};

// The step after `base` (k + 1; 0: none) of a value whose last improvement was
// tagged with its group of four: the group's first sum equal to the value.
__device__ __forceinline__ unsigned close_resolve(const CloseSmem &sm, unsigned value, unsigned tag, int i, int j) {
  const int k0 = max((int)tag - 1, 0), sw = swz<true>(k0);
  return (unsigned)strip_resolve_f32(value, (int)tag, sm.A + k0 * kBlk + (i ^ sw), kBlk, sm.B + k0 * kBlk + j, kBlk);
}

// Round job.prev's update of the pivot block, and its closure: sequential k
// as the reference's floyd_CPU_path (fap/kernel/floyd.h:37-48), strict
// improvements only -- four steps at a time.  Step k needs row and column k
// as they stand at step k, and those of steps k0 .. k0 + 3 follow from rows
// and columns k0 .. k0 + 3 as they stand at step k0 alone: 128 threads work
// them out (one column or row each, the 4 x 4 corner each for itself), then
// every entry takes its four candidates at once.  That is two barriers for
// four steps, and in FP32 two instructions an add-min (a group of four keeps
// only the group of its last improvement) instead of four.
// An entry's predecessor is that of (its last step, column) as it stood at
// that step; the rows' steps are kept as they pass and followed afterwards.
template <bool F32, bool PRED>
__global__ void __launch_bounds__(kPivThreads, 2)
    fw_close_kernel(const FwDiagJob *__restrict__ jobs, unsigned *looks) {
  extern __shared__ __align__(16) unsigned char piv_smem[];
  CloseSmem &sm = *reinterpret_cast<CloseSmem *>(piv_smem);
  __shared__ unsigned s_groups[2];
  const FwDiagJob job = jobs[blockIdx.x];
  const int ty = threadIdx.x >> 5, tx = threadIdx.x & 31;
  const int q = job.block, r = job.prev;
  const unsigned INF = F32 ? __float_as_uint(Dist<float>::inf()) : Dist<uint32_t>::inf();
  unsigned *const D = static_cast<unsigned *>(job.D);
  const bool vec = (job.ld & 1) == 0 && (reinterpret_cast<uintptr_t>(D) & 7) == 0;
  const bool vecp = PRED && (job.ld & 1) == 0 && (reinterpret_cast<uintptr_t>(job.P) & 7) == 0;
  unsigned d[4][kPivC];
  int32_t p[4][kPivC];
  int step[4][kPivC];
  block_load(d, const_cast<const unsigned *>(D), job.ld, q, q, job.size, INF, vec);
  cap_unreached<F32>(d);
  if (PRED) block_load(p, const_cast<const int32_t *>(job.P), job.ld, q, q, job.size, -1, vecp);
  if (r >= 0) {
    unsigned a[4][kPivC], b[4][kPivC];
    int32_t bp[4][kPivC];
    block_load(a, const_cast<const unsigned *>(D), job.ld, q, r, job.size, INF, vec);
    block_load(b, const_cast<const unsigned *>(D), job.ld, r, q, job.size, INF, vec);
    if (PRED) block_load(bp, const_cast<const int32_t *>(job.P), job.ld, r, q, job.size, -1, vecp);
    if (threadIdx.x < 2) s_groups[threadIdx.x] = 0u;
    __syncthreads();
    mask_or(&s_groups[0], store_a<F32>(sm.A, a));
    mask_or(&s_groups[1], store_b<F32>(sm.B, b));
#pragma unroll
    for (int i = 0; i < 4; i++) {  // the copies that the panel kernel reads
      uint2 *look = reinterpret_cast<uint2 *>(looks + job.look * kLookWords) + (ty * 4 + i) * (kBlk / 2) + tx;
      look[0] = make_uint2(a[i][0], a[i][1]);
      look[kBlk * kBlk / 2] = make_uint2(b[i][0], b[i][1]);
      if (PRED) {
        look[kBlk * kBlk] = make_uint2((unsigned)bp[i][0], (unsigned)bp[i][1]);
        *reinterpret_cast<int2 *>(&sm.P[ty * 4 + i][tx * kPivC]) = make_int2(bp[i][0], bp[i][1]);
      }
    }
    __syncthreads();
    block_product<F32, PRED>(d, step, sm.A, sm.B, s_groups[0] & s_groups[1]);
    if (PRED) {
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < kPivC; c++)
          if (step[i][c]) p[i][c] = sm.P[step[i][c] - 1][tx * kPivC + c];
      __syncthreads();  // every read of B's predecessors is done
    }
  }
  // Closure.  Entries outside the matrix are unreached with a zero diagonal.
#pragma unroll
  for (int i = 0; i < 4; i++) {
#pragma unroll
    for (int c = 0; c < kPivC; c++)
      if (q * kBlk + ty * 4 + i >= job.size && tx * kPivC + c == ty * 4 + i) d[i][c] = 0u;
    if (PRED) *reinterpret_cast<int2 *>(&sm.P[ty * 4 + i][tx * kPivC]) = make_int2(p[i][0], p[i][1]);
  }
  unsigned acc[4][kPivC];  // packed: keys; FP32: values, with the steps beside them
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < kPivC; c++) {
      acc[i][c] = F32 ? d[i][c] : min(d[i][c], kPackH) << kIdxBits;
      step[i][c] = 0;
    }
  auto publish = [&](int g) {  // rows and columns 4 g .. 4 g + 3
    if (ty == g) {             // (this warp's rows)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        *reinterpret_cast<uint2 *>(&sm.vr[i][tx * kPivC]) = make_uint2(acc[i][0], acc[i][1]);
        if (F32 && PRED)
          *reinterpret_cast<uint2 *>(&sm.vt[i][tx * kPivC]) = make_uint2((unsigned)step[i][0], (unsigned)step[i][1]);
      }
    }
    if ((tx >> 1) == g) {
#pragma unroll
      for (int c = 0; c < kPivC; c++)
        *reinterpret_cast<uint4 *>(&sm.vc[(tx & 1) * kPivC + c][ty * 4]) =
            make_uint4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
    }
  };
  // Values of the packed form without their steps, sums and minimums of either.
  auto bare = [](unsigned v) { return F32 ? v : v & ~kIdxMask; };
  auto relax = [](unsigned x, unsigned a, unsigned b) {
    return F32 ? min(x, __float_as_uint(__uint_as_float(a) + __uint_as_float(b))) : __viaddmin_u32(a, b, x);
  };
  publish(0);
  __syncthreads();
  for (int g = 0; g < kBlk / 4; g++) {
    const int k0 = g * 4;
    if (threadIdx.x < 2 * kBlk) {
      unsigned m[4][4];  // the corner: rows and columns k0 .. k0 + 3
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint4 v = *reinterpret_cast<const uint4 *>(&sm.vr[i][k0]);
        m[i][0] = bare(v.x), m[i][1] = bare(v.y), m[i][2] = bare(v.z), m[i][3] = bare(v.w);
      }
      // entry (i, j) of the corner at step k0 + min(i, j)
#pragma unroll
      for (int k = 0; k < 3; k++)
#pragma unroll
        for (int i = k + 1; i < 4; i++)
#pragma unroll
          for (int j = k + 1; j < 4; j++) m[i][j] = relax(m[i][j], m[i][k], m[k][j]);
      const bool is_row = threadIdx.x < kBlk;  // uniform over the warp
      const int x = threadIdx.x & (kBlk - 1);
      unsigned v[4], s[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        v[i] = is_row ? sm.vr[i][x] : bare(sm.vc[i][x]);
        s[i] = F32 && PRED && is_row ? sm.vt[i][x] : 0u;
      }
      if (is_row) {
        unsigned b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
          for (int k = 0; k < i; k++) {
            const unsigned was = v[i];
            v[i] = relax(v[i], m[i][k], b[k]);
            if (F32 && PRED && v[i] != was) s[i] = kBlk + 1 + (unsigned)(k0 + k + 1);  // a step, not a group
          }
          b[i] = F32 ? v[i] : bare(v[i]) | (unsigned)(k0 + i + 1);
          sm.B[(k0 + i) * kBlk + x] = b[i];
          if (PRED) sm.S[k0 + i][x] = F32 ? s[i] : v[i] & kIdxMask;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
          for (int k = 0; k < i; k++) v[i] = relax(v[i], v[k], m[k][i]);
          sm.A[(k0 + i) * kBlk + (x ^ swz<true>(k0))] = v[i];
        }
      }
    }
    __syncthreads();
    unsigned a[4][4], b[kPivC][4];  // [row or column][step]
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 av = *reinterpret_cast<const uint4 *>(sm.A + (k0 + k) * kBlk + ((ty * 4) ^ swz<true>(k0)));
      const uint2 bv = *reinterpret_cast<const uint2 *>(sm.B + (k0 + k) * kBlk + tx * kPivC);
      a[0][k] = av.x, a[1][k] = av.y, a[2][k] = av.z, a[3][k] = av.w;
      b[0][k] = bv.x, b[1][k] = bv.y;
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int c = 0; c < kPivC; c++) {
        if constexpr (F32) {
          strip_addmin4_f32(acc[i][c], step[i][c], a[i], b[c], k0 + 1);
        } else {
#pragma unroll
          for (int k = 0; k < 4; k++) acc[i][c] = __viaddmin_u32(a[i][k], b[c][k], acc[i][c]);
        }
      }
    if (g + 1 < kBlk / 4) publish(g + 1);
    __syncthreads();
  }
  if (PRED) {
    if (F32) {  // the groups of the rows' steps, and of the entries', to steps
      for (int x = threadIdx.x; x < kBlk * kBlk; x += kPivThreads) {
        const int k = x / kBlk, j = x % kBlk;
        const unsigned t = sm.S[k][j];
        sm.S[k][j] = t > kBlk ? t - (kBlk + 1) : close_resolve(sm, sm.B[k * kBlk + j], t, k, j);
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < kPivC; c++)
          step[i][c] = (int)close_resolve(sm, acc[i][c], (unsigned)step[i][c], ty * 4 + i, tx * kPivC + c);
      __syncthreads();
    }
    if (threadIdx.x < kBlk) {
      const int j = threadIdx.x;
#pragma unroll 8
      for (int k = 0; k < kBlk; k++) {
        const int s = (int)sm.S[k][j];
        if (s) sm.P[k][j] = sm.P[s - 1][j];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int row = q * kBlk + ty * 4 + i;
#pragma unroll
    for (int c = 0; c < kPivC; c++) {
      const int col = q * kBlk + tx * kPivC + c;
      if (row >= job.size || col >= job.size) continue;
      const int s = F32 ? step[i][c] : (int)(acc[i][c] & kIdxMask);
      D[(int64_t)row * job.ld + col] = s ? (F32 ? acc[i][c] : acc[i][c] >> kIdxBits) : d[i][c];
      if (PRED) job.P[(int64_t)row * job.ld + col] = s ? sm.P[s - 1][tx * kPivC + c] : p[i][c];
    }
  }
}

// The job whose panel blocks include block `x` of the launch: a warp probes 32
// jobs at a time.
__device__ __forceinline__ int find_job(const FwDiagJob *jobs, int njobs, int x) {
  const int lane = threadIdx.x & 31;
  int lo = 0, len = njobs;
  while (len > 1) {
    const int each = (len + 31) / 32, i = lane * each;
    const unsigned below = __ballot_sync(0xffffffffu, i < len && jobs[lo + i].panel_begin <= x);
    const int at = (__popc(below) - 1) * each;
    lo += at;
    len = min(each, len - at);
  }
  return lo;
}

struct PanelSmem {
  unsigned A[kBlk * kBlk], B[kBlk * kBlk];  // round prev's operands; then the block itself as one of them
  unsigned Q[kBlk * kBlk];    // the closed pivot block: A of the row panel, B of the column panel
  int32_t X[kBlk][kBlk];      // row panel: the block's predecessors
};

// Block row and column job.block: round job.prev's update, then the product
// with the closed pivot block (row panel: pivot (x) block; column panel:
// block (x) pivot).
template <bool F32, bool PRED>
__global__ void __launch_bounds__(kPivThreads, 2)
    fw_panel_kernel(const FwDiagJob *__restrict__ jobs, int njobs, const unsigned *looks) {
  extern __shared__ __align__(16) unsigned char piv_smem[];
  PanelSmem &sm = *reinterpret_cast<PanelSmem *>(piv_smem);
  __shared__ unsigned s_groups[4];
  const FwDiagJob &job = jobs[find_job(jobs, njobs, blockIdx.x)];
  const int ty = threadIdx.x >> 5, tx = threadIdx.x & 31;
  const int q = job.block, r = job.prev, size = job.size;
  const int64_t ld = job.ld;
  const int others = (size + kBlk - 1) / kBlk - 1;
  const int local = blockIdx.x - job.panel_begin;
  const bool rowp = local < others;  // uniform over the CTA
  const int b0 = rowp ? local : local - others, b = b0 < q ? b0 : b0 + 1;
  const int rb = rowp ? q : b, cb = rowp ? b : q;
  const unsigned INF = F32 ? __float_as_uint(Dist<float>::inf()) : Dist<uint32_t>::inf();
  unsigned *const D = static_cast<unsigned *>(job.D);
  int32_t *const P = job.P;
  const bool vec = (ld & 1) == 0 && (reinterpret_cast<uintptr_t>(D) & 7) == 0;
  const bool vecp = PRED && (ld & 1) == 0 && (reinterpret_cast<uintptr_t>(P) & 7) == 0;
  if (threadIdx.x < 4) s_groups[threadIdx.x] = 0u;
  unsigned x[4][kPivC], t[4][kPivC];
  int step1[4][kPivC], step[4][kPivC];
  block_load(x, const_cast<const unsigned *>(D), ld, rb, cb, size, INF, vec);
  cap_unreached<F32>(x);
  block_load(t, const_cast<const unsigned *>(D), ld, q, q, size, INF, vec);
  __syncthreads();
  if (rowp) mask_or(&s_groups[0], store_a<F32>(sm.Q, t));
  else mask_or(&s_groups[0], store_b<F32>(sm.Q, t));
  if (PRED && rowp) {
    int32_t p[4][kPivC];
    block_load(p, const_cast<const int32_t *>(P), ld, rb, cb, size, -1, vecp);
#pragma unroll
    for (int i = 0; i < 4; i++)
      *reinterpret_cast<int2 *>(&sm.X[ty * 4 + i][tx * kPivC]) = make_int2(p[i][0], p[i][1]);
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < kPivC; c++) step1[i][c] = 0;
  int32_t p1[4][kPivC];  // predecessors that round prev's update brought
  if (r >= 0 && b != r) {
    const unsigned *look = looks + job.look * kLookWords;
    if (rowp) {  // A: block (q, r) as it was, B: block (r, b)
      block_load(t, look, kBlk, 0, 0, kBlk, INF, true);
      mask_or(&s_groups[1], store_a<F32>(sm.A, t));
      block_load(t, const_cast<const unsigned *>(D), ld, r, b, size, INF, vec);
      mask_or(&s_groups[2], store_b<F32>(sm.B, t));
    } else {  // A: block (b, r), B: block (r, q) as it was
      block_load(t, const_cast<const unsigned *>(D), ld, b, r, size, INF, vec);
      mask_or(&s_groups[1], store_a<F32>(sm.A, t));
      block_load(t, look + kBlk * kBlk, kBlk, 0, 0, kBlk, INF, true);
      mask_or(&s_groups[2], store_b<F32>(sm.B, t));
    }
    __syncthreads();
    block_product<F32, PRED>(x, step1, sm.A, sm.B, s_groups[1] & s_groups[2]);
    if (PRED) {
      const int32_t *lp = reinterpret_cast<const int32_t *>(look) + 2 * kBlk * kBlk;
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < kPivC; c++) {
          const int s = step1[i][c], j = tx * kPivC + c;
          p1[i][c] = -1;
          if (s) p1[i][c] = rowp ? P[(int64_t)(r * kBlk + s - 1) * ld + b * kBlk + j] : lp[(s - 1) * kBlk + j];
          if (s && rowp) sm.X[ty * 4 + i][j] = p1[i][c];
        }
    }
    __syncthreads();  // the operands may be replaced
  }
  // The block itself joins the pivot block as the other operand.
  unsigned mine;
  if (rowp) mine = store_b<F32>(sm.B, x);
  else mine = store_a<F32>(sm.A, x);
  mask_or(&s_groups[3], mine);
  __syncthreads();
  block_product<F32, PRED>(x, step, rowp ? sm.Q : sm.A, rowp ? sm.B : sm.Q, s_groups[0] & s_groups[3]);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int row = rb * kBlk + ty * 4 + i;
#pragma unroll
    for (int c = 0; c < kPivC; c++) {
      const int j = tx * kPivC + c, col = cb * kBlk + j, s = step[i][c];
      const bool kept = !s && !step1[i][c];
      if ((kept && !(F32 && x[i][c] == INF)) || row >= size || col >= size) continue;
      D[(int64_t)row * ld + col] = x[i][c];
      if (PRED && !kept)
        P[(int64_t)row * ld + col] = !s ? p1[i][c]
                                     : rowp ? sm.X[s - 1][j]
                                            : P[(int64_t)(q * kBlk + s - 1) * ld + q * kBlk + j];
    }
  }
}

template <bool F32, bool PRED>
cudaError_t launch_close(const FwDiagJob *d_jobs, int njobs, unsigned *looks, cudaStream_t st) {
  ++launch_count();
  fw_close_kernel<F32, PRED><<<njobs, kPivThreads, sizeof(CloseSmem), st>>>(d_jobs, looks);
  return cudaGetLastError();
}

template <bool F32, bool PRED>
cudaError_t launch_panel(const FwDiagJob *d_jobs, int njobs, int blocks, const unsigned *looks, cudaStream_t st) {
  ++launch_count();
  fw_panel_kernel<F32, PRED><<<blocks, kPivThreads, sizeof(PanelSmem), st>>>(d_jobs, njobs, looks);
  return cudaGetLastError();
}

template <bool F32, bool PRED>
cudaError_t set_attrs() {
  cudaError_t e = cudaFuncSetAttribute(fw_close_kernel<F32, PRED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(CloseSmem));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(fw_panel_kernel<F32, PRED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(PanelSmem));
}

}  // namespace

size_t fw_look_bytes() { return (size_t)kLookWords * 4; }

cudaError_t init_fw_pivot_kernels() {
  cudaError_t e;
  if ((e = set_attrs<true, true>()) != cudaSuccess || (e = set_attrs<true, false>()) != cudaSuccess ||
      (e = set_attrs<false, true>()) != cudaSuccess || (e = set_attrs<false, false>()) != cudaSuccess)
    return e;
  return cudaSuccess;
}

cudaError_t launch_fw_chain(bool f32, bool pred, const FwDiagJob *d_jobs, int njobs, int blocks, void *look,
                            cudaStream_t st) {
  if (njobs <= 0) return cudaSuccess;
  unsigned *const at = static_cast<unsigned *>(look);
  cudaError_t e;
  if (f32) e = pred ? launch_close<true, true>(d_jobs, njobs, at, st) : launch_close<true, false>(d_jobs, njobs, at, st);
  else e = pred ? launch_close<false, true>(d_jobs, njobs, at, st) : launch_close<false, false>(d_jobs, njobs, at, st);
  if (e != cudaSuccess || blocks <= 0) return e;
  if (f32)
    return pred ? launch_panel<true, true>(d_jobs, njobs, blocks, at, st)
                : launch_panel<true, false>(d_jobs, njobs, blocks, at, st);
  return pred ? launch_panel<false, true>(d_jobs, njobs, blocks, at, st)
              : launch_panel<false, false>(d_jobs, njobs, blocks, at, st);
}

}  // namespace fapk
