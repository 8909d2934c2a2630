// minplus.cu -- (min,+) tile products and the blocked Floyd-Warshall phases.
//
// Reference counterparts: the min-plus product with predecessors
// (min_plus_path_CPU_advanced, fap/kernel/minplus.h:51-65; GPU kernel
// MatrixMulCUDA6_path, fap/kernel/cuda/minplus.cu:32-189) and the blocked
// Floyd-Warshall (floyd_CPU_path, fap/kernel/floyd.h:38-49; GPU kernels
// fw_kernel1 / FW_kernel1A2 / fw_kernel3, fap/kernel/cuda/floyd.cu:26-267).
//
// Kernels of this file:
//  - mp_strip_kernel (FP32, and int32 whose finite results stay below 2^24 - 1;
//    at most 48 steps): packed keys (d << 7) | idx, one DPX __viaddmin_u32 per
//    add-min, which gives the minimum and, on ties, the smallest idx -- the
//    current value (idx 0) first, then the first k.  A stays resident for a
//    strip of column tiles, and the steps k whose A column or B row has no
//    finite entry in the tile are skipped (such a candidate never wins).
//    Other products: mp_deep.cu.
//  - mp_tile_kernel (Floyd-Warshall panels and remaining tiles of wide int32).
//    One CTA computes C = min(C, A (x) B) for a 128x128 output tile with 256
//    threads, 8x8 outputs per thread in registers, k staged in chunks of 32
//    by cp.async with a two-stage pipeline; the argmin is the chunk-local k
//    of the last strict improvement, resolved against the staged
//    B-predecessor tile after each chunk.  A batch of segments (one per FW
//    panel) is one launch; each CTA finds its segment by binary search over
//    the segments' first tile.
//
// Floyd-Warshall over 64-wide pivot blocks: once the pivot block is closed
// (shortest paths through its own vertices, zero diagonal), the row panel is
// D_rr (x) D_rj, the column panel D_ir (x) D_rr and every other tile
// min(D_ij, D_ir (x) D_rj).  Ties keep the current value, so predecessors
// follow P[i][j] = P[k][j] on strict improvement as in the reference.

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "fw_tile.cuh"
#include "kernels.cuh"
#include "launch.h"
#include "mp_common.cuh"

namespace fapk {

namespace {

constexpr int kTile = 128;   // CTA tile (rows and columns)
constexpr int kBK = 32;      // k chunk staged in shared memory
constexpr int kThreads = 256;
constexpr int kApad = kBK + 1;  // A rows padded against bank conflicts

struct MpSmem {
  unsigned A[2][kTile][kApad];
  unsigned B[2][kBK][kTile];
  int32_t Bp[2][kBK][kTile];
};

// Block index of list entry g of 0..nblocks-1 without block `skip`, or of the
// one-block list `fix`; -1 past the list.
__device__ __forceinline__ int list_block(int g, int skip, int fix, int nblocks) {
  if (fix >= 0) return g == 0 ? fix : -1;
  const int b = skip >= 0 && g >= skip ? g + 1 : g;
  return b < nblocks ? b : -1;
}

// Stages k-chunk [k0, k0+32) of A (128 rows, 4-byte cp.async into the padded
// rows) and B (128 columns), and of B's predecessors when WITH_BP (16-byte
// cp.async of 4 columns where aligned); entries outside the matrices are
// written directly as "unreached" / -1.
template <bool WITH_BP>
__device__ __forceinline__ void load_chunk(MpSmem &sm, int buf, const MpSegment &s, const int rbase[2],
                                           const int cbase[2], int k0) {
  const int t = threadIdx.x;
  const unsigned INF = Dist<uint32_t>::inf();
  // A: 128 rows x 32 k; consecutive threads take consecutive k of one row.
  {
    const int kk = t & 31;
    const int kg = k0 + kk;
#pragma unroll 4
    for (int it = 0; it < kTile / 8; it++) {
      const int m = (t >> 5) + 8 * it;
      const int rb = rbase[m >> 6];
      const int row = rb + (m & 63);
      unsigned *dst = &sm.A[buf][m][kk];
      if (rb >= 0 && row < s.M && kg < s.K) {
        cp_async4(dst, static_cast<const unsigned *>(s.A) + (int64_t)row * s.lda + kg);
      } else {
        *dst = INF;
      }
    }
  }
  // B (and its predecessors): 32 k x 128 columns; a warp takes one row k,
  // 4 consecutive columns a lane.
  {
    const int j4 = (t & 31) * 4;
    const int cb = cbase[j4 >> 6];
    const int col = cb + (j4 & 63);
    const bool full = cb >= 0 && col + 3 < s.N;
    const bool vec = full && (s.ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(s.B) & 15) == 0;
    const bool vecp = WITH_BP && full && (s.ldbp & 3) == 0 && (reinterpret_cast<uintptr_t>(s.Bp) & 15) == 0;
#pragma unroll 4
    for (int it = 0; it < kBK / 8; it++) {
      const int kk = (t >> 5) + 8 * it;
      const int kg = k0 + kk;
      unsigned *dst = &sm.B[buf][kk][j4];
      const unsigned *src = static_cast<const unsigned *>(s.B) + (int64_t)kg * s.ldb + col;
      if (kg < s.K && vec) {
        cp_async16(dst, src);
      } else {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (cb >= 0 && col + q < s.N && kg < s.K) cp_async4(dst + q, src + q);
          else dst[q] = INF;
        }
      }
      if constexpr (WITH_BP) {
        int32_t *dp = &sm.Bp[buf][kk][j4];
        const int32_t *sp = s.Bp + (int64_t)kg * s.ldbp + col;
        if (kg < s.K && vecp) {
          cp_async16(dp, sp);
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (cb >= 0 && col + q < s.N && kg < s.K) cp_async4(dp + q, sp + q);
            else dp[q] = -1;
          }
        }
      }
    }
  }
}

// Output tile geometry of one CTA, resolved from its segment.
struct TileGeom {
  int rbase[2], cbase[2];
  int ty, tx;
};

__device__ __forceinline__ TileGeom tile_geom(const MpSegment &s, int tile) {
  TileGeom g;
  const int local = tile - s.tile_begin;
  const int tyt = local / s.tiles_x, txt = local - tyt * s.tiles_x;
  const int nbr = (s.M + kBlk - 1) / kBlk, nbc = (s.N + kBlk - 1) / kBlk;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    int rb = list_block(2 * tyt + i, s.row_skip, s.row_fix, nbr);
    int cb = list_block(2 * txt + i, s.col_skip, s.col_fix, nbc);
    g.rbase[i] = rb >= 0 ? rb * kBlk : -1;
    g.cbase[i] = cb >= 0 ? cb * kBlk : -1;
  }
  g.ty = threadIdx.x >> 4;
  g.tx = threadIdx.x & 15;
  return g;
}

__device__ __forceinline__ int out_row(const TileGeom &g, int r) {
  return g.rbase[r >> 2] < 0 ? -1 : g.rbase[r >> 2] + g.ty * 4 + (r & 3);
}
__device__ __forceinline__ int out_col(const TileGeom &g, int c) {
  return g.cbase[c >> 2] < 0 ? -1 : g.cbase[c >> 2] + g.tx * 4 + (c & 3);
}
__device__ __forceinline__ int smem_row(const TileGeom &g, int r) { return (r >> 2) * kBlk + g.ty * 4 + (r & 3); }
__device__ __forceinline__ int smem_col(const TileGeom &g, int c) { return (c >> 2) * kBlk + g.tx * 4 + (c & 3); }

// Floyd-Warshall tiles of int32 matrices outside the packed range.  One
// __vibmin_u32 gives both the new minimum and whether the current value was
// kept (ties keep it: strict improvement).  An add-min is then add + vibmin +
// select; the argmin is the chunk-local k of
// the last strict improvement, resolved against the staged predecessor tile
// after each chunk.
template <bool PRED>
__device__ __forceinline__ void tile_wide(MpSmem &sm, const MpSegment &s, const TileGeom &g) {
  const unsigned INF = Dist<uint32_t>::inf();
  unsigned acc[8][8];
  int32_t pred[8][8];
  int arg[8][8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int row = out_row(g, r);
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int col = out_col(g, c);
      acc[r][c] = INF;
      pred[r][c] = -1;
      arg[r][c] = -1;
      if (s.init_from_c && row >= 0 && row < s.M && col >= 0 && col < s.N) {
        acc[r][c] = static_cast<const unsigned *>(s.C)[(int64_t)row * s.ldc + col];
        if (PRED) pred[r][c] = s.Cp[(int64_t)row * s.ldcp + col];
      }
    }
  }
  const int nchunks = (s.K + kBK - 1) / kBK;
  if (nchunks > 0) load_chunk<PRED>(sm, 0, s, g.rbase, g.cbase, 0);
  cp_async_commit();
  for (int ch = 0; ch < nchunks; ch++) {
    const int buf = ch & 1;
    if (ch + 1 < nchunks) load_chunk<PRED>(sm, buf ^ 1, s, g.rbase, g.cbase, (ch + 1) * kBK);
    cp_async_commit();
    cp_async_wait_1();
    __syncthreads();
    const int kn = min(kBK, s.K - ch * kBK);  // steps of this chunk (the rest is fill)
#pragma unroll 2
    for (int kk = 0; kk < kn; kk++) {
      unsigned a[8], b[8];
#pragma unroll
      for (int r = 0; r < 8; r++) a[r] = sm.A[buf][smem_row(g, r)][kk];
#pragma unroll
      for (int c = 0; c < 8; c++) b[c] = sm.B[buf][kk][smem_col(g, c)];
#pragma unroll
      for (int r = 0; r < 8; r++)
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const unsigned v = a[r] + b[c];
          if (PRED) {
            bool keep;
            acc[r][c] = __vibmin_u32(acc[r][c], v, &keep);
            arg[r][c] = keep ? arg[r][c] : kk;
          } else {
            acc[r][c] = min(acc[r][c], v);
          }
        }
    }
    if (PRED) {
#pragma unroll
      for (int r = 0; r < 8; r++)
#pragma unroll
        for (int c = 0; c < 8; c++)
          if (arg[r][c] >= 0) {
            pred[r][c] = sm.Bp[buf][arg[r][c]][smem_col(g, c)];
            arg[r][c] = -1;
          }
    }
    __syncthreads();
  }
  cp_async_wait_0();
  const bool vec = vec_stores_ok<PRED>(s);
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int row = out_row(g, r);
    if (row < 0 || row >= s.M) continue;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (g.cbase[h] < 0) continue;
      const int col0 = g.cbase[h] + g.tx * 4;
      if (col0 >= s.N) continue;
      unsigned d[4];
      int32_t p[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        d[q] = acc[r][h * 4 + q];
        p[q] = pred[r][h * 4 + q];
      }
      store_quad<uint32_t, PRED>(s, row, col0, d, p, vec);
    }
  }
}

// Strip form of the packed min-plus for products that do not accumulate into
// C (the inner rows of every part) with K <= kStripMaxK.  One CTA owns a
// strip: one 128-row tile of a segment and the 64-column tiles of up to
// 16 x 128 consecutive columns.  A's 128 x K block is staged once
// per strip (transposed, so that a thread's 8 row operands of one k are two
// 16-byte loads); B's K x TN tiles are double-buffered, so the next tile's
// copy is in flight while the current one is multiplied; B's predecessor
// rows of the tile's active steps, its own-part FW values and the next
// tile's column flags are copied behind the DPX loop.  The part's own
// columns of a tile (the Floyd-Warshall values replace the product there)
// are listed when the tile's column flags land, and the FW values of up to
// kOwnCap of them are staged; further own columns are read from global
// memory in the epilogue.  The descriptor search, the staging of A and the
// pipeline fill of the tile kernel are paid once per strip instead of once
// per tile.  Shared memory (ks = K rounded up to 4):
//   B[2][ks][TN] | Bp[1 + ks][TN] | colp[2][TN] | coll[2][TN] | ownidx[2][TN] |
//   Fst[kOwnCap][128] | Fpst[kOwnCap][128] | A^T[ks][128]
// and, FP32 only, Ar[128][strip_ar_stride(kseg)] (A row-major) |
// Bq[ks / 4][64] (the current tile's B by step group: 16-byte unit (g, col)
// holds steps 4g .. 4g + 3 of column col).
// Row 0 of Bp holds -1, so the predecessor of every output is Bp[idx][col]
// with the key's idx as it is (0 when unreached).
// Work counters of the strip min-plus (diagnostics): [tiles, tiles with no
// active step, add-mins executed (active steps x the tile's 128 x TN
// outputs, summed over tiles)], summed per CTA.
__device__ unsigned long long g_strip_counters[3];

constexpr int kStripCols = 64;   // columns of a tile
// Largest K of the strip form.  128 x 64 tiles with 8 x 4 outputs a thread,
// three CTAs per SM: on sparse products most of a tile's time is its fixed work
// (B keys, masks, epilogue), whose latencies only more resident warps hide
// (against 128 x 128 tiles at two CTAs per SM 16 % faster on a 65,536-vertex
// geometric graph; four CTAs per SM for K <= 32, at 64 registers a thread, no
// faster).  Above, mp_deep.cu's tiles, which share the staging of A among fewer
// columns but keep three CTAs per SM at any K, are faster: products of 2,000 x
// 20,000 at K = 36 / 48 / 72 / 100, packed 223 / 272 / 381 / 482 us here and 237 /
// 260 / 334 / 412 us there, FP32 285 / 400 / 521 / 667 and 277 / 305 / 439 / 560 us;
// the min-plus of a 128 x 128 grid in 16 parts (K from 41 to 92) 2.07 ms with
// every part here (128 x 128 tiles above 48), 1.79 ms with those above 48 there.
// (FP32, whose tiles take more shared memory: 40.)
constexpr int kStripMaxK = 48, kStripMaxKF32 = 40;
constexpr int kOwnCap = 12;

// Row stride of the FP32 strip kernel's row-major copy of A for kseg
// steps: kseg, or kseg + 4 when kseg / 4 is even, so that the stride in
// 16-byte units is odd.
__host__ __device__ constexpr int strip_ar_stride(int kseg) { return ((kseg >> 2) & 1) ? kseg : kseg + 4; }

// Shared memory of the strip kernel, in bytes; F32 adds
// the row-major copy of A ([128][ks + 4] at most) and the step-group copy
// of B ([ks / 4][64] 16-byte units, within [64][ks + 4] words).
template <bool F32>
__host__ __device__ constexpr size_t strip_smem_bytes(int ks) {
  constexpr int TN = kStripCols;
  return ((size_t)2 * ks * TN + (size_t)(ks + 1) * TN + 6 * TN + (size_t)2 * kOwnCap * kTile +
          (size_t)ks * kTile + (F32 ? (size_t)(kTile + TN) * (ks + 4) : 0)) * 4;
}

__device__ __forceinline__ const MpSegment &find_strip_segment(const MpSegment *__restrict__ segs,
                                                               int nseg, int strip) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (segs[mid].strip_begin <= strip) lo = mid; else hi = mid - 1;
  }
  return segs[lo];
}

// Copies a ks x TN tile of a row-major 4-byte matrix (rows < K, columns
// [col0, col0 + TN) < N) into dst[ks][TN] (SWZ: chunks permuted by swz);
// each thread moves 4 consecutive columns of a row per pass (one 16-byte
// copy when `vec`), and writes `fill` where the source is outside the matrix.
template <int TN, bool SWZ = false>
__device__ __forceinline__ void strip_load_rows(unsigned *dst, const unsigned *src, int64_t ld,
                                                int K, int N, int ks, int col0, bool vec,
                                                unsigned fill) {
  constexpr int TPR = TN / 4;  // threads per row
  const int t = threadIdx.x;
  const int j = (t % TPR) * 4;
  const int col = col0 + j;
  for (int kk = t / TPR; kk < ks; kk += kThreads / TPR) {
    unsigned *d = dst + kk * TN + (j ^ swz<SWZ>(kk));
    const unsigned *g = src + (int64_t)kk * ld + col;
    if (kk < K && vec && col + 3 < N) {
      cp_async16(d, g);
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (kk < K && col + q < N) cp_async4(d + q, g + q);
        else d[q] = fill;
      }
    }
  }
}

// Sets the bits of kmask for the warp's rows of a B tile (two rows of 16
// lanes, starting at lane 0's row kk, which is even) that have a finite entry:
// one ballot and one atomic per warp.
__device__ __forceinline__ void strip_mark_rows(unsigned *kmask, int kk, bool fin) {
  const unsigned bal = __ballot_sync(0xffffffffu, fin);
  if ((threadIdx.x & 31) == 0) {  // lane 0 holds the warp's first (even) row
    const unsigned bits = ((bal & 0xffffu) ? 1u : 0u) | ((bal >> 16) ? 2u : 0u);
    if (bits) atomicOr(&kmask[kk >> 5], bits << (kk & 31));
  }
}

// Turns the B values this thread copied (same mapping as strip_load_rows)
// into keys (d << 7) | (k + 1), and sets bit k of kmask (a 128-bit mask in
// shared memory) for every row k that has a finite entry in the tile.
// F32: the values stay (FP32 bits, "unreached" = the bits of 1e8);
// the row bits are set and the values are also written to Bq, the tile's
// copy by step group (word 4 (g TN + col) + q is step 4g + q of column col).
// ks is a multiple of 4, so a warp's rows are all below ks or all at or past
// it, and the warp's lanes run the loop together.
template <bool F32>
__device__ __forceinline__ void strip_keys_b(unsigned *Bs, int ks, unsigned *kmask,
                                             unsigned *Bq) {
  constexpr int TN = kStripCols, TPR = TN / 4;
  static_assert(TPR == 16, "row marks assume 16 lanes a row");
  const int t = threadIdx.x;
  const int j = (t % TPR) * 4;
  for (int kk = t / TPR; kk < ks; kk += kThreads / TPR) {
    uint4 *p = reinterpret_cast<uint4 *>(Bs + kk * TN + j);
    const unsigned idx = (unsigned)(kk & kMaxPackedK) + 1u;
    uint4 v = *p;
    if (F32) {
      strip_mark_rows(kmask, kk, min(min(v.x, v.y), min(v.z, v.w)) < __float_as_uint(Dist<float>::inf()));
      unsigned *q = Bq + ((kk >> 2) * TN + j) * 4 + (kk & 3);
      q[0] = v.x;
      q[4] = v.y;
      q[8] = v.z;
      q[12] = v.w;
      continue;
    }
    const bool fin = min(min(v.x, v.y), min(v.z, v.w)) < kPackH;
    v.x = (min(v.x, kPackH) << kIdxBits) | idx;
    v.y = (min(v.y, kPackH) << kIdxBits) | idx;
    v.z = (min(v.z, kPackH) << kIdxBits) | idx;
    v.w = (min(v.w, kPackH) << kIdxBits) | idx;
    *p = v;
    strip_mark_rows(kmask, kk, fin);
  }
}

// One add-min of the strip kernel: packed keys (one DPX instruction), or
// FP32 bits with the step idx of the last strict improvement kept in `arg`.
template <bool F32>
__device__ __forceinline__ void strip_addmin(unsigned &acc, int &arg, unsigned a, unsigned b, int idx) {
  if constexpr (F32) {
    const unsigned v = __float_as_uint(__uint_as_float(a) + __uint_as_float(b));
    bool keep;
    acc = __vibmin_u32(acc, v, &keep);
    arg = keep ? arg : idx;
  } else {
    acc = __viaddmin_u32(a, b, acc);
  }
}

// The same for the strip min-plus, from row-major copies of the operands:
// Ar[128][ars] (row m's steps contiguous, ars = strip_ar_stride(kseg)) and
// Bq, the tile's B by step group (16-byte unit g * 64 + col: steps 4g ..
// 4g + 3 of column col).
// One 16-byte load gives a row's or a column's four steps of a group, so the
// resolve takes two loads per output.  Eight consecutive columns of one step
// group are eight consecutive units of Bq, in eight different bank groups,
// and so they stay when the lanes' step groups differ (the resolve); Ar's
// stride is odd in 16-byte units, so the two rows (four apart) that a warp
// reads in the loop lie in different bank groups, and one row's different
// step groups (the resolve) too, up to eight groups apart.  The thread's
// rows are r0 .. r0 + 3 and r0 + 64 .. r0 + 67, its columns tx, tx + 16,
// tx + 32 and tx + 48.  B operands load two columns at a time (24 operands
// live).
template <bool PRED>
__device__ __forceinline__ void addmin_groups_rows_f32(unsigned (&acc)[8][4], int (&arg)[8][4],
                                                       const unsigned *Ar, int ars, int kseg, int r0,
                                                       const unsigned *Bq, int tx) {
  const unsigned *arow = Ar + r0 * ars;  // row r0 + m at arow + m * ars
  const uint4 *bq = reinterpret_cast<const uint4 *>(Bq) + tx;  // (g, tx + 16 c) at bq[g * 64 + 16 c]
  for (int kk = 0; kk < kseg; kk += 4) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      unsigned a[4][4];  // [row of the half][step]
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const uint4 v = *reinterpret_cast<const uint4 *>(arow + (h * kBlk + r) * ars + kk);
        a[r][0] = v.x, a[r][1] = v.y, a[r][2] = v.z, a[r][3] = v.w;
      }
#pragma unroll
      for (int ch = 0; ch < 2; ch++) {
        unsigned b[2][4];  // [column of the pair][step]
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const uint4 v = bq[(kk >> 2) * 64 + (ch * 2 + c) * 16];
          b[c][0] = v.x, b[c][1] = v.y, b[c][2] = v.z, b[c][3] = v.w;
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
          for (int c = 0; c < 2; c++)
            strip_addmin4_f32(acc[h * 4 + r][ch * 2 + c], arg[h * 4 + r][ch * 2 + c], a[r], b[c], kk + 1);
      }
    }
  }
  if (PRED) {
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const int tag = arg[r][c];
        const int k0 = tag > 0 ? tag - 1 : 0;
        const uint4 av = *reinterpret_cast<const uint4 *>(arow + ((r >> 2) * kBlk + (r & 3)) * ars + k0);
        const uint4 bv = bq[(k0 >> 2) * 64 + c * 16];
        const unsigned v0 = __float_as_uint(__fadd_rn(__uint_as_float(av.x), __uint_as_float(bv.x)));
        const unsigned v1 = __float_as_uint(__fadd_rn(__uint_as_float(av.y), __uint_as_float(bv.y)));
        const unsigned v2 = __float_as_uint(__fadd_rn(__uint_as_float(av.z), __uint_as_float(bv.z)));
        const unsigned m = acc[r][c];
        const int j = v0 == m ? 0 : v1 == m ? 1 : v2 == m ? 2 : 3;
        arg[r][c] = tag > 0 ? tag + j : 0;
      }
  }
}

// 128x64 tiles, 8x4 outputs per thread; packed keys three CTAs per SM.
// F32: FP32 distances (any range), two CTAs per SM.  The product keeps each
// output's value bits (non-negative floats order like them) and which step
// made its last strict improvement: in groups of four steps
// (addmin_groups_rows_f32) where at least half of the tile's steps are active,
// else step by step (fl(a + b), then __vibmin_u32 for the minimum and whether
// the current value was kept).  Either is the reference's strict-<,
// ascending-k rule, as the packed form's.
template <bool PRED, bool F32>
__global__ void __launch_bounds__(kThreads, F32 ? 2 : 3)
    mp_strip_kernel(const MpSegment *__restrict__ segs, int nseg, int ks, int per) {
  constexpr int TN = kStripCols;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned *Bs = reinterpret_cast<unsigned *>(smem_raw);  // [2][ks][TN]
  int32_t *Bps = reinterpret_cast<int32_t *>(Bs + 2 * ks * TN);  // [1 + ks][TN]
  int32_t *colp = Bps + (ks + 1) * TN;  // [2][TN] col_part of the tile's columns (per tile parity)
  int32_t *coll = colp + 2 * TN;        // [2][TN] col_local of the tile's columns
  int32_t *ownidx = coll + 2 * TN;      // [2][TN] own column: staging slot, or -2 (not staged); else -1
  unsigned *Fst = reinterpret_cast<unsigned *>(ownidx + 2 * TN);  // [kOwnCap][128 rows]
  int32_t *Fpst = reinterpret_cast<int32_t *>(Fst + kOwnCap * kTile);  // [kOwnCap][128 rows]
  unsigned *As = reinterpret_cast<unsigned *>(Fpst + kOwnCap * kTile);  // A^T [ks][128]
  unsigned *Ar = As + ks * kTile;        // F32: A row-major [128][ars]
  unsigned *Bq = Ar + kTile * (ks + 4);  // F32: the tile's B by step group [ks / 4][64][4]
  __shared__ MpSegment seg;
  __shared__ int s_own[2];                   // own columns of the tile (per tile parity)
  __shared__ int16_t s_ownlist[2][kOwnCap];  // their tile columns, by slot
  __shared__ unsigned s_kmask[2][4];         // rows k of B with a finite entry (per tile parity)
  __shared__ unsigned s_amask[4];            // columns k of A with a finite entry (per strip)
  if (threadIdx.x == 0) {
    seg = find_strip_segment(segs, nseg, blockIdx.x);
    s_own[0] = s_own[1] = 0;
  }
  if (threadIdx.x < 8) (&s_kmask[0][0])[threadIdx.x] = 0u;
  if (threadIdx.x < 4) s_amask[threadIdx.x] = 0u;
  if (threadIdx.x < TN) Bps[threadIdx.x] = -1;  // predecessor of idx 0
  __syncthreads();
  const MpSegment &s = seg;
  const int strips_x = (s.tiles_x + per - 1) / per;
  const int local = blockIdx.x - s.strip_begin;
  const int rt = local / strips_x;
  // column tiles of TN: this strip's 128-column tiles (`per` of them), split
  const int jt0 = (local - rt * strips_x) * per * (128 / TN);
  const int jt1 = min(jt0 + per * (128 / TN), (s.N + TN - 1) / TN);
  const int row0 = rt * kTile;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const unsigned INF = F32 ? __float_as_uint(Dist<float>::inf()) : Dist<uint32_t>::inf();
  const int kseg = (s.K + 3) & ~3;  // this segment's K rounded up to 4 (<= ks)
  const int ars = strip_ar_stride(kseg);  // F32: Ar's row stride
  const bool vec_b = (s.ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(s.B) & 15) == 0;
  const bool vec_bp = PRED && (s.ldbp & 3) == 0 && (reinterpret_cast<uintptr_t>(s.Bp) & 15) == 0;
  const bool vec_c = vec_stores_ok<PRED>(s);
  // The epilogue's view of C in registers (the descriptor is in shared memory,
  // which the compiler reads again after every barrier): this thread's rows
  // are the same for every tile of the strip.
  // (Row offsets within a strip are below 2^31 elements: callers send no
  // leading dimension of 2^24 or more here.)
  const int m_rows = s.M, n_cols = s.N;
  const int ldc = (int)s.ldc, ldcp = (int)s.ldcp;
  unsigned *const c_thr = static_cast<unsigned *>(s.C) + (int64_t)(row0 + ty * 4) * s.ldc;
  int32_t *const p_thr = PRED ? s.Cp + (int64_t)(row0 + ty * 4) * s.ldcp : nullptr;

  auto load_flags = [&](int col0, int fb) {  // column flags of a tile, into parity fb
    if (threadIdx.x < TN) {
      const int j = threadIdx.x, col = col0 + j;
      if (s.col_part != nullptr && col < s.N) {
        cp_async4(&colp[fb * TN + j], s.col_part + col);
        cp_async4(&coll[fb * TN + j], s.col_local + col);
      } else {
        colp[fb * TN + j] = -1;
      }
    }
  };
  // B's predecessor rows of the steps k in (lo, hi) only (row k goes to Bps
  // row k + 1); warp w copies every eighth of them, 4 columns a lane.
  auto load_bp_rows = [&](int col0, unsigned long long lo, unsigned long long hi) {
    const int warp = threadIdx.x >> 5;
    const int j = (threadIdx.x & 31) * 4, col = col0 + j;
    int i = 0;
    while (lo | hi) {
      int k;
      if (lo) {
        k = __ffsll(lo) - 1;
        lo &= lo - 1ull;
      } else {
        k = 64 + __ffsll(hi) - 1;
        hi &= hi - 1ull;
      }
      if ((i++ & 7) == warp && j < TN) {
        int32_t *d = Bps + (k + 1) * TN + j;
        const int32_t *g = s.Bp + (int64_t)k * s.ldbp + col;
        if (vec_bp && col + 3 < s.N) {
          cp_async16(d, g);
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (col + q < s.N) cp_async4(d + q, g + q);
            else d[q] = -1;
          }
        }
      }
    }
  };

  // Prologue: A, B and the column flags of the first tile.  A^T is copied
  // with consecutive threads on consecutive rows (its shared-memory rows are
  // contiguous), the FP32 row-major copy with consecutive threads on
  // consecutive steps of a row (contiguous in both memories).
  for (int idx = threadIdx.x; idx < kTile * kseg; idx += kThreads) {
    const int kk = idx >> 7, m = idx & (kTile - 1);
    unsigned *d = &As[idx];
    if (row0 + m < s.M && kk < s.K)
      cp_async4(d, static_cast<const unsigned *>(s.A) + (int64_t)(row0 + m) * s.lda + kk);
    else
      *d = INF;
    if (F32) {
      const int mr = idx / kseg, kr = idx - mr * kseg;
      unsigned *dr = &Ar[mr * ars + kr];
      if (row0 + mr < s.M && kr < s.K)
        cp_async4(dr, static_cast<const unsigned *>(s.A) + (int64_t)(row0 + mr) * s.lda + kr);
      else
        *dr = INF;
    }
  }
  strip_load_rows<TN>(Bs, static_cast<const unsigned *>(s.B), s.ldb, s.K, s.N, kseg, jt0 * TN, vec_b, INF);
  load_flags(jt0 * TN, 0);
  cp_async_commit();

  // Per tile: two barriers.  (A) after the B keys, masks and own-column list;
  // then the tile's predecessor rows (active steps only), its staged FW
  // values and the next tile's flags are copied (one group), then the next
  // tile's B (a second group), while the add-mins issue; (B) once the first
  // group has landed, before the epilogue.  The next B is waited for at the
  // top of the next tile, so it also has the epilogue to land.  Every buffer
  // written between (A) and (B) was last read before (A); the flags and
  // own-column slots are double-buffered by tile parity because the epilogue
  // of one tile runs into the next tile's list without a barrier.
  unsigned long long n_tiles = 0, n_empty = 0, n_steps = 0;  // work counters (thread 0)
  for (int jt = jt0; jt < jt1; jt++) {
    const int buf = (jt - jt0) & 1;
    unsigned *Bcur = Bs + buf * ks * TN;
    cp_async_wait_0();  // this tile's B (and, first tile, A and the flags)
    if (jt == jt0)  // A keys; a warp converts 32 entries of one step k and marks finite ones
      for (int idx = threadIdx.x; idx < kTile * kseg; idx += kThreads) {
        const unsigned v = As[idx];
        if (!F32) As[idx] = min(v, kPackH) << kIdxBits;
        const int kk = idx >> 7;
        if (__any_sync(0xffffffffu, F32 ? v < INF : v < kPackH) && (threadIdx.x & 31) == 0)
          atomicOr(&s_amask[kk >> 5], 1u << (kk & 31));
      }
    strip_keys_b<F32>(Bcur, kseg, s_kmask[buf], Bq);
    // List the tile's own columns (threads 0..TN-1 copied their column's
    // flags; slots are taken in any order through a counter).
    if (threadIdx.x == 0) s_own[buf ^ 1] = 0;  // used by the next tile
    if (threadIdx.x < 4) s_kmask[buf ^ 1][threadIdx.x] = 0u;
    if (threadIdx.x < TN) {
      const int j = threadIdx.x;
      const bool own = colp[buf * TN + j] == s.part;
      const unsigned bal = __ballot_sync(0xffffffffu, own);
      int base = 0;
      if ((threadIdx.x & 31) == 0 && bal) base = atomicAdd(&s_own[buf], __popc(bal));
      base = __shfl_sync(0xffffffffu, base, 0);
      int slot = -1;
      if (own) {
        slot = base + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u));
        if (slot < kOwnCap) s_ownlist[buf][slot] = (int16_t)j;
        else slot = -2;
      }
      ownidx[buf * TN + j] = slot;
    }
    __syncthreads();  // (A)
    if (jt + 1 < jt1) load_flags((jt + 1) * TN, buf ^ 1);
    const int nown = min(s_own[buf], kOwnCap);
    if (nown > 0) {  // stage the FW values of the own columns (rows of this tile)
      for (int it = threadIdx.x; it < nown * kTile; it += kThreads) {
        const int sl = it / kTile, m = it - sl * kTile;
        if (row0 + m < s.M) {
          const int64_t off =
              (int64_t)(row0 + m) * s.ldf + (coll[buf * TN + s_ownlist[buf][sl]] - s.local0);
          cp_async4(&Fst[sl * kTile + m], static_cast<const unsigned *>(s.F) + off);
          if (PRED) cp_async4(&Fpst[sl * kTile + m], s.Fp + off);
        }
      }
    }
    // Only the steps k whose B row has a finite entry in this tile and whose
    // A column has one in this strip can change an output (any other
    // candidate is at least "unreached", which never wins).
    unsigned long long mlo = (unsigned long long)(s_kmask[buf][0] & s_amask[0]) |
                             ((unsigned long long)(s_kmask[buf][1] & s_amask[1]) << 32);
    unsigned long long mhi = (unsigned long long)(s_kmask[buf][2] & s_amask[2]) |
                             ((unsigned long long)(s_kmask[buf][3] & s_amask[3]) << 32);
    const int nact = __popcll(mlo) + __popcll(mhi);
    n_tiles++;
    n_empty += nact == 0;
    // (FP32 with at least half of the steps active runs all of them)
    n_steps += (unsigned long long)(F32 && nact > 0 && 2 * nact >= kseg ? kseg : nact) * kTile * TN;
    if (PRED && nact == s.K && s.K > 0)  // every step active: all rows, 16-byte copies spread over the CTA
      strip_load_rows<TN>(reinterpret_cast<unsigned *>(Bps + TN), reinterpret_cast<const unsigned *>(s.Bp),
                          s.ldbp, s.K, s.N, kseg, jt * TN, vec_bp, 0xffffffffu);
    else if (PRED && nact > 0)
      load_bp_rows(jt * TN, mlo, mhi);
    cp_async_commit();
    if (jt + 1 < jt1)  // B[buf ^ 1] was last read by the previous tile's add-mins, before (B)
      strip_load_rows<TN>(Bs + (buf ^ 1) * ks * TN, static_cast<const unsigned *>(s.B), s.ldb, s.K,
                          s.N, kseg, (jt + 1) * TN, vec_b, INF);
    cp_async_commit();

    unsigned acc[8][4];
    int arg[8][4];  // F32: step idx of the last strict improvement (0: none)
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        acc[r][c] = F32 ? INF : kPackH << kIdxBits;
        arg[r][c] = 0;
      }
    // When every step is active the loop runs over all k (unrolled);
    // otherwise it walks the set bits of the mask -- on graphs with limited
    // reachability most steps are skipped.  Either way the next step's
    // operands load while the current step's add-mins issue.
    {
      // the thread's operands of step k
      auto a_at = [&](int k) { return As + k * kTile + ty * 4; };
      auto b_at = [&](int k) { return Bcur + k * TN + tx * 4; };
      // B operands of step k: four consecutive columns (packed keys), or
      // the FP32 thread's columns tx + 16 c (lanes of a row read
      // consecutive words)
      auto load_b = [&](int k) {
        if (F32) {
          const unsigned *q = Bcur + k * TN + tx;
          return make_uint4(q[0], q[16], q[32], q[48]);
        }
        return *reinterpret_cast<const uint4 *>(b_at(k));
      };
      // FP32 with at least half of the steps active: all steps in groups
      // of four (steps that are not active, or at or past K, hold
      // "unreached" on one side and never win).
      const bool grouped = F32 && nact > 0 && 2 * nact >= kseg;
      if (grouped) {
        if constexpr (F32) addmin_groups_rows_f32<PRED>(acc, arg, Ar, ars, kseg, ty * 4, Bq, tx);
      } else if (nact == s.K && s.K > 0) {
        uint4 na0 = *reinterpret_cast<const uint4 *>(a_at(0));
        uint4 na1 = *reinterpret_cast<const uint4 *>(a_at(0) + kBlk);
        uint4 nb = load_b(0);
#pragma unroll 2
        for (int kk = 0; kk < kseg; kk++) {
          const unsigned a[8] = {na0.x, na0.y, na0.z, na0.w, na1.x, na1.y, na1.z, na1.w};
          const unsigned b[4] = {nb.x, nb.y, nb.z, nb.w};
          const int kn = kk + 1 < kseg ? kk + 1 : kk;
          na0 = *reinterpret_cast<const uint4 *>(a_at(kn));
          na1 = *reinterpret_cast<const uint4 *>(a_at(kn) + kBlk);
          nb = load_b(kn);
#pragma unroll
          for (int r = 0; r < 8; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) strip_addmin<F32>(acc[r][c], arg[r][c], a[r], b[c], kk + 1);
        }
      } else if (nact > 0) {
        auto next_k = [&]() {  // lowest remaining step, or -1
          if (mlo) {
            const int b = __ffsll(mlo) - 1;
            mlo &= mlo - 1ull;
            return b;
          }
          if (mhi) {
            const int b = __ffsll(mhi) - 1;
            mhi &= mhi - 1ull;
            return 64 + b;
          }
          return -1;
        };
        int kk = next_k();
        uint4 na0 = *reinterpret_cast<const uint4 *>(a_at(kk));
        uint4 na1 = *reinterpret_cast<const uint4 *>(a_at(kk) + kBlk);
        uint4 nb = load_b(kk);
        while (kk >= 0) {
          const unsigned a[8] = {na0.x, na0.y, na0.z, na0.w, na1.x, na1.y, na1.z, na1.w};
          const unsigned b[4] = {nb.x, nb.y, nb.z, nb.w};
          const int cur = kk;
          kk = next_k();
          const int kn = kk >= 0 ? kk : 0;
          na0 = *reinterpret_cast<const uint4 *>(a_at(kn));
          na1 = *reinterpret_cast<const uint4 *>(a_at(kn) + kBlk);
          nb = load_b(kn);
#pragma unroll
          for (int r = 0; r < 8; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) strip_addmin<F32>(acc[r][c], arg[r][c], a[r], b[c], cur + 1);
        }
      }
    }

    cp_async_wait_1();
    __syncthreads();  // (B)
    // Epilogue: distances, predecessors from the staged rows, own-part
    // columns from the part's Floyd-Warshall matrix (only when the tile has
    // any; the test is uniform over the CTA).
    const int colbase = jt * TN;
    if constexpr (F32) {
      // FP32: the thread's columns are tx + 16 c, so each of the four
      // 4-byte streaming stores of a row writes 64 consecutive bytes per
      // half-warp, whatever the alignment of the row.  The value is at most
      // "unreached"; step idx 0 reads predecessor -1.
      if (nown == 0 && colbase + TN <= n_cols) {  // (uniform) no own column, every column inside
#pragma unroll
        for (int r = 0; r < 8; r++) {
          const int rr = (r >> 2) * kBlk + (r & 3);
          if (row0 + ty * 4 + rr >= m_rows) continue;
          unsigned *cq = c_thr + rr * ldc + colbase + tx;
          int32_t *pq = PRED ? p_thr + rr * ldcp + colbase + tx : nullptr;
#pragma unroll
          for (int c = 0; c < 4; c++) {
            __stcs(cq + 16 * c, acc[r][c]);
            if (PRED) __stcs(pq + 16 * c, Bps[arg[r][c] * TN + tx + 16 * c]);
          }
        }
        continue;
      }
      unsigned ownm = 0;  // bit c: column tx + 16 c is the part's own
      if (nown > 0) {
#pragma unroll
        for (int c = 0; c < 4; c++)
          if (ownidx[buf * TN + tx + 16 * c] != -1) ownm |= 1u << c;
      }
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int rr = (r >> 2) * kBlk + (r & 3);  // row offset from this thread's first row
        const int row = row0 + ty * 4 + rr;
        if (row >= m_rows) continue;
        unsigned *crow = c_thr + rr * ldc;
        int32_t *prow = PRED ? p_thr + rr * ldcp : nullptr;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int sc = tx + 16 * c, col = colbase + sc;
          unsigned d = acc[r][c];
          int32_t pv = PRED ? Bps[arg[r][c] * TN + sc] : -1;
          if ((ownm >> c) & 1u) {
            const int oi = ownidx[buf * TN + sc];
            if (oi >= 0) {  // own-part column: the FW value, staged
              d = Fst[oi * kTile + row - row0];
              if (PRED) pv = Fpst[oi * kTile + row - row0];
            } else if (oi == -2 && col < n_cols) {  // own-part column beyond the staging slots
              const int64_t fj = coll[buf * TN + sc] - s.local0;
              d = static_cast<const unsigned *>(s.F)[(int64_t)row * s.ldf + fj];
              if (PRED) pv = s.Fp[(int64_t)row * s.ldf + fj];
            }
          }
          if (col < n_cols) {  // streaming stores: the rows are not read again here
            __stcs(crow + col, d);
            if (PRED) __stcs(prow + col, pv);
          }
        }
      }
      continue;
    }
    const int sc0 = tx * 4, col0 = colbase + sc0;
    unsigned ownmask = 0;  // bit q: this thread's column sc0 + q is the part's own
    if (nown > 0) {
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (ownidx[buf * TN + sc0 + q] != -1) ownmask |= 1u << q;
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int rr = (r >> 2) * kBlk + (r & 3);  // row offset from this thread's first row
      const int row = row0 + ty * 4 + rr;
      if (row >= m_rows || col0 >= n_cols) continue;
      unsigned *crow = c_thr + rr * ldc;
      int32_t *prow = PRED ? p_thr + rr * ldcp : nullptr;
      unsigned d[4] = {INF, INF, INF, INF};
      int32_t p[4] = {-1, -1, -1, -1};
      // a quad of unreached outputs (the common case on sparse graphs)
      // needs no decode and no predecessor gathers
      const unsigned qmin = min(min(acc[r][0], acc[r][1]), min(acc[r][2], acc[r][3]));
      if (qmin < (kPackH << kIdxBits)) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const unsigned key = acc[r][q];
          const unsigned dist = key >> kIdxBits;
          d[q] = dist >= kPackH ? INF : dist;
          if (PRED) p[q] = Bps[(key & kIdxMask) * TN + sc0 + q];
        }
      }
      if (ownmask) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (!((ownmask >> q) & 1u)) continue;
          const int oi = ownidx[buf * TN + sc0 + q];
          if (oi >= 0) {  // own-part column: the FW value, staged
            d[q] = Fst[oi * kTile + row - row0];
            if (PRED) p[q] = Fpst[oi * kTile + row - row0];
          } else if (oi == -2) {  // own-part column beyond the staging slots
            const int64_t fj = coll[buf * TN + sc0 + q] - s.local0;
            d[q] = static_cast<const unsigned *>(s.F)[(int64_t)row * s.ldf + fj];
            if (PRED) p[q] = s.Fp[(int64_t)row * s.ldf + fj];
          }
        }
      }
      if (vec_c && col0 + 3 < n_cols) {  // streaming stores: the rows are not read again here
        __stcs(reinterpret_cast<uint4 *>(crow + col0), make_uint4(d[0], d[1], d[2], d[3]));
        if (PRED) __stcs(reinterpret_cast<int4 *>(prow + col0), make_int4(p[0], p[1], p[2], p[3]));
      } else {
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (col0 + q < n_cols) {
            crow[col0 + q] = d[q];
            if (PRED) prow[col0 + q] = p[q];
          }
      }
    }
  }
  cp_async_wait_0();
  if (threadIdx.x == 0 && n_tiles > 0) {
    atomicAdd(&g_strip_counters[0], n_tiles);
    atomicAdd(&g_strip_counters[1], n_empty);
    atomicAdd(&g_strip_counters[2], n_steps);
  }
}

template <bool PRED>
__global__ void __launch_bounds__(kThreads, 1)
    mp_tile_kernel(const MpSegment *__restrict__ segs, int nseg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MpSmem &sm = *reinterpret_cast<MpSmem *>(smem_raw);
  // The segment descriptor stays in shared memory (read where needed) so that
  // the accumulators, argmins and predecessors keep the registers.
  __shared__ MpSegment seg;
  const int tile = blockIdx.x;
  if (threadIdx.x == 0) seg = find_segment(segs, nseg, tile);
  __syncthreads();
  const MpSegment &s = seg;
  const TileGeom g = tile_geom(s, tile);
  tile_wide<PRED>(sm, s, g);
}

// Largest finite int32 value (< 2^30) of the strided matrix blockIdx.y,
// atomicMax-ed into out[blockIdx.y * step] once a CTA.  The CTAs (blockIdx.x)
// stride over pieces of kMaxCols columns of a row, so that few long rows keep
// as many loads in flight as many short ones.
constexpr int kMaxCols = 1024;
__global__ void __launch_bounds__(256)
    max_finite_kernel(const MatRef *__restrict__ mats, unsigned *out, int step) {
  __shared__ unsigned s_max;
  const MatRef mr = mats[blockIdx.y];
  const unsigned *D = static_cast<const unsigned *>(mr.p);
  if (threadIdx.x == 0) s_max = 0u;
  __syncthreads();
  const int per_row = (mr.cols + kMaxCols - 1) / kMaxCols;
  const int64_t pieces = (int64_t)mr.rows * per_row;
  unsigned m = 0;
  for (int64_t p = blockIdx.x; p < pieces; p += gridDim.x) {
    const int64_t r = p / per_row;
    const int c0 = (int)(p - r * per_row) * kMaxCols + threadIdx.x;
    const unsigned *row = D + r * mr.ld;
#pragma unroll
    for (int i = 0; i < kMaxCols / 256; i++) {
      const int c = c0 + 256 * i;
      const unsigned v = c < mr.cols ? row[c] : 0u;
      if (v < Dist<uint32_t>::inf()) m = max(m, v);
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(&s_max, m);
  __syncthreads();
  if (threadIdx.x == 0 && s_max) atomicMax(out + blockIdx.y * step, s_max);
}

// Closes a 64x64 block held in shared memory (D values, P predecessors, row
// pitch 65): sequential k as the reference's floyd_CPU_path
// (fap/kernel/floyd.h:37-48), strict improvements only, P[i][j] = P[k][j].
// Each thread keeps its 4x4 entries in registers; row k and column k do not
// change at step k (zero diagonal), so their owners publish them for the
// next step into a double-buffered row/column copy and one barrier per step
// suffices.  Ends with the closed block back in D/P and a barrier.
template <typename T, bool PRED>
__device__ __forceinline__ void close_block(T (*D)[kBlk + 1], int32_t (*P)[kBlk + 1]) {
  __shared__ T rowk[2][kBlk], colk[2][kBlk];
  __shared__ int32_t prowk[2][kBlk];
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  T d[4][4];
  int32_t p[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      d[i][c] = D[ty * 4 + i][tx * 4 + c];
      p[i][c] = PRED ? P[ty * 4 + i][tx * 4 + c] : -1;
    }
  // publish row 0 / column 0
  if (ty == 0)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      rowk[0][tx * 4 + c] = d[0][c];
      if (PRED) prowk[0][tx * 4 + c] = p[0][c];
    }
  if (tx == 0)
#pragma unroll
    for (int i = 0; i < 4; i++) colk[0][ty * 4 + i] = d[i][0];
  __syncthreads();
  for (int k = 0; k < kBlk; k++) {
    const int buf = k & 1;
    T a[4], b[4];
    int32_t bp[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      a[q] = colk[buf][ty * 4 + q];
      b[q] = rowk[buf][tx * 4 + q];
      if (PRED) bp[q] = prowk[buf][tx * 4 + q];
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const T v = Dist<T>::add(a[i], b[c]);
        if (v < d[i][c]) {
          d[i][c] = v;
          if (PRED) p[i][c] = bp[c];
        }
      }
    const int kn = k + 1;
    if (kn < kBlk) {
      const int kq = kn & 3;
      if (ty == (kn >> 2))
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (i == kq)
#pragma unroll
            for (int c = 0; c < 4; c++) {
              rowk[buf ^ 1][tx * 4 + c] = d[i][c];
              if (PRED) prowk[buf ^ 1][tx * 4 + c] = p[i][c];
            }
      if (tx == (kn >> 2))
#pragma unroll
        for (int c = 0; c < 4; c++)
          if (c == kq)
#pragma unroll
            for (int i = 0; i < 4; i++) colk[buf ^ 1][ty * 4 + i] = d[i][c];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      D[ty * 4 + i][tx * 4 + c] = d[i][c];
      if (PRED) P[ty * 4 + i][tx * 4 + c] = p[i][c];
    }
  __syncthreads();
}

// Closes the 64x64 pivot block of one matrix per CTA (close_block).
template <typename T, bool PRED>
__global__ void __launch_bounds__(256)
    fw_diag_kernel(const FwDiagJob *__restrict__ jobs) {
  __shared__ T D[kBlk][kBlk + 1];
  __shared__ int32_t P[kBlk][kBlk + 1];
  const FwDiagJob job = jobs[blockIdx.x];
  const int base = job.block * kBlk;
  const T INF = Dist<T>::inf();
  T *Dg = static_cast<T *>(job.D);
  for (int idx = threadIdx.x; idx < kBlk * kBlk; idx += blockDim.x) {
    const int i = idx >> 6, j = idx & 63;
    const int gi = base + i, gj = base + j;
    const bool ok = gi < job.size && gj < job.size;
    D[i][j] = ok ? Dg[(int64_t)gi * job.ld + gj] : (i == j ? (T)0 : INF);
    if (PRED) P[i][j] = ok ? job.P[(int64_t)gi * job.ld + gj] : -1;
  }
  __syncthreads();
  close_block<T, PRED>(D, P);
  for (int idx = threadIdx.x; idx < kBlk * kBlk; idx += blockDim.x) {
    const int i = idx >> 6, j = idx & 63;
    const int gi = base + i, gj = base + j;
    if (gi < job.size && gj < job.size) {
      Dg[(int64_t)gi * job.ld + gj] = D[i][j];
      if (PRED) job.P[(int64_t)gi * job.ld + gj] = P[i][j];
    }
  }
}

template <bool PRED>
cudaError_t launch_mp_t(const MpSegment *d_segs, int nseg, int tiles, cudaStream_t st) {
  if (tiles <= 0 || nseg <= 0) return cudaSuccess;
  ++launch_count();
  mp_tile_kernel<PRED><<<tiles, kThreads, sizeof(MpSmem), st>>>(d_segs, nseg);
  return cudaGetLastError();
}

template <bool PRED, bool F32>
cudaError_t launch_strip_t(const MpSegment *d_segs, int nseg, int strips, int ks, int per, cudaStream_t st) {
  if (strips <= 0 || nseg <= 0) return cudaSuccess;
  ++launch_count();
  mp_strip_kernel<PRED, F32><<<strips, kThreads, strip_smem_bytes<F32>(ks), st>>>(d_segs, nseg, ks, per);
  return cudaGetLastError();
}

template <bool PRED, bool F32>
cudaError_t set_strip_attr() {
  return cudaFuncSetAttribute(mp_strip_kernel<PRED, F32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)strip_smem_bytes<F32>((minplus_strip_max_k(F32) + 3) & ~3));
}

template <bool PRED>
cudaError_t set_mp_attr() {
  return cudaFuncSetAttribute(mp_tile_kernel<PRED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MpSmem));
}

}  // namespace

cudaError_t launch_minplus_tiles(bool pred, const MpSegment *d_segs, int nseg, int tiles, cudaStream_t st) {
  return pred ? launch_mp_t<true>(d_segs, nseg, tiles, st) : launch_mp_t<false>(d_segs, nseg, tiles, st);
}

cudaError_t launch_minplus_strips(bool f32, bool pred, const MpSegment *d_segs, int nseg, int strips, int max_k,
                                  int per, cudaStream_t st) {
  if (max_k < 0 || max_k > minplus_strip_max_k(f32) || per < 1) return cudaErrorInvalidValue;
  const int ks = (max_k + 3) & ~3;
  if (f32)
    return pred ? launch_strip_t<true, true>(d_segs, nseg, strips, ks, per, st)
                : launch_strip_t<false, true>(d_segs, nseg, strips, ks, per, st);
  return pred ? launch_strip_t<true, false>(d_segs, nseg, strips, ks, per, st)
              : launch_strip_t<false, false>(d_segs, nseg, strips, ks, per, st);
}

namespace {
int strips_of(const MpSegment &s, int per) { return (s.M + kTile - 1) / kTile * ((s.tiles_x + per - 1) / per); }
}  // namespace

int number_minplus_strips(bool f32, MpSegment *segs, int nseg, int sm_count, int *per) {
  return number_strips(segs, nseg, sm_count, f32 ? 2 : 3, per, strips_of);
}

int minplus_strip_max_k(bool f32) { return f32 ? kStripMaxKF32 : kStripMaxK; }

cudaError_t launch_max_finite(const MatRef *d_mats, int nmats, unsigned *out, int step, cudaStream_t st) {
  if (nmats <= 0) return cudaSuccess;
  ++launch_count();
  // (CTAs for every SM whatever the number of matrices)
  max_finite_kernel<<<dim3(max(32, 1216 / nmats), nmats), 256, 0, st>>>(d_mats, out, step);
  return cudaGetLastError();
}

unsigned pack_limit() { return kPackH; }

cudaError_t strip_counters(unsigned long long out[3], bool reset) {
  cudaError_t e = rows_counters(out, reset);
  unsigned long long strip[3], deep[3];
  if (e == cudaSuccess) e = deep_counters(deep, reset);
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(strip, g_strip_counters, sizeof(strip));
  if (e != cudaSuccess) return e;
  for (int i = 0; i < 3; i++) out[i] += strip[i] + deep[i];
  if (!reset) return e;
  const unsigned long long zero[3] = {0, 0, 0};
  return cudaMemcpyToSymbol(g_strip_counters, zero, sizeof(zero));
}

cudaError_t launch_fw_diag(bool f32, bool pred, const FwDiagJob *d_jobs, int njobs, cudaStream_t st) {
  if (njobs <= 0) return cudaSuccess;
  ++launch_count();
  if (f32 && pred) fw_diag_kernel<float, true><<<njobs, 256, 0, st>>>(d_jobs);
  else if (f32) fw_diag_kernel<float, false><<<njobs, 256, 0, st>>>(d_jobs);
  else if (pred) fw_diag_kernel<uint32_t, true><<<njobs, 256, 0, st>>>(d_jobs);
  else fw_diag_kernel<uint32_t, false><<<njobs, 256, 0, st>>>(d_jobs);
  return cudaGetLastError();
}

cudaError_t init_minplus_kernels() {
  cudaError_t e;
  if ((e = set_mp_attr<true>()) != cudaSuccess) return e;
  if ((e = set_mp_attr<false>()) != cudaSuccess) return e;
  if ((e = set_strip_attr<true, false>()) != cudaSuccess) return e;
  if ((e = set_strip_attr<false, false>()) != cudaSuccess) return e;
  if ((e = set_strip_attr<true, true>()) != cudaSuccess) return e;
  if ((e = set_strip_attr<false, true>()) != cudaSuccess) return e;
  return cudaSuccess;
}

int minplus_tile_rows() { return kTile; }
int fw_block() { return kBlk; }

}  // namespace fapk
