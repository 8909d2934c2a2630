// fw_rest.cu -- the remaining tiles of a Floyd-Warshall round.
//
// Reference counterparts: floyd_CPU_path (fap/kernel/floyd.h:38-49) and the
// third phase of the GPU form (fw_kernel3, fap/kernel/cuda/floyd.cu:26-267).
//
// D_ij = min(D_ij, D_ir (x) D_rj) for every block row i and block column j but
// r's own, and, with the lookahead (fw_pivot.cu), but r + 1's; ties keep D_ij.
// Nearly all of a round's add-mins are here, so the kernel is made for the ALU
// that runs them: per 128 x 64 tile the add-mins of 64 steps and as little
// else as possible.
//
//  - A CTA owns a strip: one 128-row tile of the row list with A = D_ir
//    resident, and `per` consecutive 64-column tiles.  A is read along its
//    rows (coalesced at any alignment) and stored transposed.
//  - B = D_rj: the next tile's values arrive by cp.async behind the add-mins,
//    then become keys in an order of columns that gives a thread's one 16-byte
//    load columns tx, tx + 16, tx + 32 and tx + 48: what the half-warps read
//    and write of a row of C is then 64 consecutive bytes at any alignment
//    (four consecutive columns a thread touch four times the sectors, and
//    stores of improved entries are a large part of the memory pipe's work).
//  - C is not staged: the epilogue reads it from global memory, from lines that
//    a prefetch brought to L2 during the add-mins, and the predecessor of an
//    improved entry is looked up where it is.  What that leaves in shared
//    memory is 64 KB, three CTAs an SM for the packed form, so that one CTA's
//    loads and epilogue run under the others' add-mins.
//  - An entry that does not improve costs a compare.  In FP32 the step inside
//    the group of the last improvement is worked out for improved entries only.
//    What improves in a row is stored together, with its predecessors in flight
//    at once: one entry after the other, each waited for its own.
//
// Measured against the strips before (C and B's predecessors staged by bulk
// tensor copies, two CTAs an SM): a launch of 1.49e10 int32 add-mins (128
// matrices of 576 to 2,048) 1.8 -> 1.23 ms = 12.1 T/s, 61 % of the DPX rate,
// the ALU pipe at 79 %; FP32, 256 matrices of 256 to 1,024: 1.14 -> 0.84 ms.
// Four columns a thread side by side: 1.60 ms; one entry's predecessor after
// the other: 1.35; all sixteen of a half tile at once: 1.45 (and 28 % slower
// on sparse matrices, where few improve).

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "fw_tile.cuh"
#include "kernels.cuh"
#include "launch.h"

namespace fapk {

namespace {

constexpr int kRestThreads = 256;
constexpr int kRows = 128;  // tile rows: two blocks of the row list

// FP32: A and B in 16-byte units of the four steps of a group of a row or a
// column, unit (g, m) of A at g * kAUnits + m, (g, j) of B at g * kBlk + j: the
// adds go in pairs (six instructions a group instead of eight), and the look-up
// of an improved entry's step is two loads instead of six.  256 matrices of 256 to
// 1,024: 15.45 -> 15.21 ms; a road-like graph's 64 matrices of 895: 5.83 -> 5.67.
// (A's extra row is FP32's alone: with it the packed form's three CTAs ask for
// the next larger shared memory, and the smaller L1 costs 8 %.)
constexpr int kAUnits = kRows + 1;  // (odd: the stores of a row's groups hit different banks)

template <bool F32>
struct RestSmem {
  unsigned A[F32 ? kBlk + 1 : kBlk][kRows];  // step k: keys of the strip's rows, row m at m ^ swz(k)
  unsigned B[kBlk][kBlk];     // step k: of the tile's columns, column j at 4 (j % 16) + j / 16
  unsigned next[kBlk][kBlk];  // the next tile's values as they are in memory
};

// Add-mins executed (steps run x the tile's outputs), summed per CTA
// (diagnostics).
__device__ unsigned long long g_fw_counters[1];

__device__ __forceinline__ void copy4(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void copy16(void *smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}

// i-th block of a round's row or column list.
__host__ __device__ __forceinline__ int rest_block(int i, int r, int look) { return i < r ? i : i + 1 + look; }
__host__ __device__ __forceinline__ int rest_blocks(int nb, int look) { return nb - 1 - look; }

// The job that strip x of the launch belongs to: a warp probes 32 at a time.
__device__ __forceinline__ int find_rest(const FwRestJob *jobs, int njobs, int x) {
  const int lane = threadIdx.x & 31;
  int lo = 0, len = njobs;
  while (len > 1) {
    const int each = (len + 31) / 32, i = lane * each;
    const unsigned below = __ballot_sync(0xffffffffu, i < len && jobs[lo + i].strip_begin <= x);
    const int at = (__popc(below) - 1) * each;
    lo += at;
    len = min(each, len - at);
  }
  return lo;
}

template <bool F32, bool PRED>
__global__ void __launch_bounds__(kRestThreads, F32 ? 2 : 3)
    fw_rest_kernel(const FwRestJob *__restrict__ jobs, int njobs, int per) {
  extern __shared__ __align__(16) unsigned char rest_smem[];
  RestSmem<F32> &sm = *reinterpret_cast<RestSmem<F32> *>(rest_smem);
  __shared__ FwRestJob s;
  __shared__ unsigned s_amask[2];     // steps with a finite entry in the strip's rows
  __shared__ unsigned s_bmask[2][2];  // ... and in the tile's columns (per tile parity)
  const int t = threadIdx.x;
  {
    const int j = find_rest(jobs, njobs, blockIdx.x);
    if (t == 0) s = jobs[j];
    if (t < 2) s_amask[t] = 0u;
    if (t < 4) (&s_bmask[0][0])[t] = 0u;
  }
  __syncthreads();
  const int r = s.block, look = s.look, size = s.size;
  const int nct = rest_blocks((size + kBlk - 1) / kBlk, look), sx = (nct + per - 1) / per;
  const int local = blockIdx.x - s.strip_begin, rt = local / sx;
  const int jt0 = (local - rt * sx) * per, jt1 = min(jt0 + per, nct);
  const int row0 = rest_block(2 * rt, r, look) * kBlk;
  const bool two = 2 * rt + 1 < nct;  // the tile's second row block exists (as many rows as columns are listed)
  const int row1 = two ? rest_block(2 * rt + 1, r, look) * kBlk : size;
  const bool vec = (s.ld & 3) == 0 && (reinterpret_cast<uintptr_t>(s.D) & 15) == 0;
  const unsigned INF = F32 ? __float_as_uint(Dist<float>::inf()) : Dist<uint32_t>::inf();
  const unsigned FIN = F32 ? INF : kPackH;  // entries below are finite
  const int ty = t >> 4, tx = t & 15;

  const int ld = (int)s.ld;
  const unsigned *const prow = static_cast<const unsigned *>(s.D) + (int64_t)r * kBlk * s.ld;  // pivot row 0
  const int krows = min(kBlk, size - r * kBlk);
  auto load_b = [&](int jt) {
    const int col0 = rest_block(jt, r, look) * kBlk;
    if (krows == kBlk && col0 + kBlk <= size) {
      if (vec) {
#pragma unroll
        for (int i = 0; i < 4; i++) copy16(&sm.next[ty + 16 * i][tx * 4], prow + (int64_t)(ty + 16 * i) * ld + col0 + tx * 4);
      } else {
#pragma unroll
        for (int i = 0; i < 16; i++)
          copy4(&sm.next[(t >> 6) + 4 * i][t & 63], prow + (int64_t)((t >> 6) + 4 * i) * ld + col0 + (t & 63));
      }
    } else {
      for (int i = 0; i < 16; i++) {
        const int kk = (t >> 6) + 4 * i, j = t & 63;
        if (kk < krows && col0 + j < size) copy4(&sm.next[kk][j], prow + (int64_t)kk * ld + col0 + j);
        else sm.next[kk][j] = INF;
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  load_b(jt0);
  {  // A: 16 threads a row, 4 steps each, transposed into shared memory
    unsigned nib = 0;  // which of the thread's steps have a finite entry
    const int k = tx * 4, col = r * kBlk + k;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      unsigned v[4][4];  // [row][step]
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int m = ty + 16 * (h * 4 + i), row = (h ? row1 : row0) + (m & 63);
        const unsigned *g = static_cast<const unsigned *>(s.D) + (int64_t)row * s.ld + col;
        const bool in = row < size && (h == 0 || two);
        if (in && vec && col + 3 < size) {
          const uint4 x = *reinterpret_cast<const uint4 *>(g);
          v[i][0] = x.x, v[i][1] = x.y, v[i][2] = x.z, v[i][3] = x.w;
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) v[i][q] = in && col + q < size ? g[q] : INF;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int m = ty + 16 * (h * 4 + i);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          nib |= v[i][q] < FIN ? 1u << q : 0u;
          if (!F32) sm.A[k + q][m ^ swz<true>(k)] = min(v[i][q], kPackH) << kIdxBits;
        }
        if (F32)
          reinterpret_cast<uint4 *>(&sm.A[0][0])[tx * kAUnits + m] = make_uint4(v[i][0], v[i][1], v[i][2], v[i][3]);
      }
    }
    const unsigned lo = __reduce_or_sync(0xffffffffu, tx < 8 ? nib << (4 * tx) : 0u);
    const unsigned hi = __reduce_or_sync(0xffffffffu, tx < 8 ? 0u : nib << (4 * tx - 32));
    if ((t & 31) == 0) {
      if (lo) atomicOr(&s_amask[0], lo);
      if (hi) atomicOr(&s_amask[1], hi);
    }
  }
  unsigned long long n_work = 0;
  for (int jt = jt0; jt < jt1; jt++) {
    const int par = (jt - jt0) & 1;
    const int col0 = rest_block(jt, r, look) * kBlk;
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();  // the tile's values are here; every thread is done with the last tile's keys and mask
    if (t < 2) s_bmask[par ^ 1][t] = 0u;
    if constexpr (F32) {  // values to units; the groups with a finite entry
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int g = (t >> 6) + 4 * i, j = t & 63;
        const uint4 v = make_uint4(sm.next[4 * g][j], sm.next[4 * g + 1][j], sm.next[4 * g + 2][j], sm.next[4 * g + 3][j]);
        reinterpret_cast<uint4 *>(&sm.B[0][0])[g * kBlk + j] = v;
        if (__any_sync(0xffffffffu, min(min(v.x, v.y), min(v.z, v.w)) < FIN) && (t & 31) == 0)
          atomicOr(&s_bmask[par][g >> 3], 15u << (4 * (g & 7)));
      }
    } else {  // values to keys; the rows with a finite entry
#pragma unroll
      for (int h = 0; h < 2; h++) {
        unsigned bits = 0;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int kk = ty + 16 * (2 * h + i);
          uint4 v = make_uint4(sm.next[kk][tx], sm.next[kk][tx + 16], sm.next[kk][tx + 32], sm.next[kk][tx + 48]);
          const bool fin = min(min(v.x, v.y), min(v.z, v.w)) < FIN;
          const unsigned id = (unsigned)kk + 1u;
          v.x = (min(v.x, kPackH) << kIdxBits) | id;
          v.y = (min(v.y, kPackH) << kIdxBits) | id;
          v.z = (min(v.z, kPackH) << kIdxBits) | id;
          v.w = (min(v.w, kPackH) << kIdxBits) | id;
          *reinterpret_cast<uint4 *>(&sm.B[kk][tx * 4]) = v;
          const unsigned bal = __ballot_sync(0xffffffffu, fin);  // rows kk of the warp's two ty
          bits |= (((bal & 0xffffu) ? 1u : 0u) | ((bal >> 16) ? 2u : 0u)) << (16 * i);
        }
        if ((t & 31) == 0 && bits) atomicOr(&s_bmask[par][h], bits << ty);
      }
    }
    __syncthreads();  // keys and mask
    if (jt + 1 < jt1) load_b(jt + 1);
    unsigned long long msk = (unsigned long long)(s_bmask[par][0] & s_amask[0]) |
                             ((unsigned long long)(s_bmask[par][1] & s_amask[1]) << 32);
    if (!msk) continue;  // no step can improve an entry
    {  // C's lines to L2 behind the add-mins
      const int m = t >> 1, row = (m < kBlk ? row0 : row1) + (m & 63);
      const int64_t off = (int64_t)row * ld + col0 + (t & 1) * 32;
      if (row < size && col0 + (t & 1) * 32 < size)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(static_cast<const unsigned *>(s.D) + off));
    }
    unsigned acc[8][4];
    int arg[8][4];  // FP32: the group (first step + 1) of the last strict improvement, 0: none
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        acc[i][c] = F32 ? INF : kPackH << kIdxBits;
        arg[i][c] = 0;
      }
    if constexpr (F32) {
      // groups of four steps with an active one (the others hold "unreached"
      // on one side); without a second row block only the first one's rows
      for (int k = 0; k < kBlk; k += 4) {
        if (!((unsigned)(msk >> k) & 15u)) continue;
        n_work += (two ? kRows : kBlk) * kBlk * 4;
        const ulonglong2 *ap = reinterpret_cast<const ulonglong2 *>(&sm.A[0][0]) + (k >> 2) * kAUnits + ty * 4;
        const ulonglong2 *bp = reinterpret_cast<const ulonglong2 *>(&sm.B[0][0]) + (k >> 2) * kBlk + tx;
        ulonglong2 b[4];
#pragma unroll
        for (int c = 0; c < 4; c++) b[c] = bp[16 * c];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          if (h == 1 && !two) break;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const ulonglong2 a = ap[h * kBlk + i];
#pragma unroll
            for (int c = 0; c < 4; c++) unit_addmin_f32(acc[h * 4 + i][c], arg[h * 4 + i][c], a, b[c], k + 1);
          }
        }
      }
    } else {
      const int nact = __popcll(msk);
      n_work += (unsigned long long)nact * (kRows * kBlk);
      auto operands = [&](int k, uint4 &a0, uint4 &a1, uint4 &b) {
        const unsigned *ap = &sm.A[k][(ty * 4) ^ swz<true>(k)];
        a0 = *reinterpret_cast<const uint4 *>(ap);
        a1 = *reinterpret_cast<const uint4 *>(ap + kBlk);
        b = *reinterpret_cast<const uint4 *>(&sm.B[k][tx * 4]);
      };
      auto step = [&](const uint4 &a0, const uint4 &a1, const uint4 &b4) {
        const unsigned a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const unsigned b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int c = 0; c < 4; c++) acc[i][c] = __viaddmin_u32(a[i], b[c], acc[i][c]);
      };
      uint4 a0, a1, b;
      if (nact == kBlk) {  // the next step's operands load under this step's add-mins
        operands(0, a0, a1, b);
        for (int k = 0; k < kBlk; k += 4) {  // (one address a group: the swizzle is the same within it)
          const unsigned *ap = &sm.A[k][(ty * 4) ^ swz<true>(k)];
          const unsigned *bp = &sm.B[k][tx * 4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const uint4 x0 = a0, x1 = a1, y = b;
            if (q < 3) {
              a0 = *reinterpret_cast<const uint4 *>(ap + (q + 1) * kRows);
              a1 = *reinterpret_cast<const uint4 *>(ap + (q + 1) * kRows + kBlk);
              b = *reinterpret_cast<const uint4 *>(bp + (q + 1) * kBlk);
            } else {
              operands((k + 4) & (kBlk - 1), a0, a1, b);
            }
            step(x0, x1, y);
          }
        }
      } else if (msk) {
        int k = __ffsll(msk) - 1;
        operands(k, a0, a1, b);
        do {
          msk &= msk - 1ull;
          const uint4 x0 = a0, x1 = a1, y = b;
          if (msk) operands(__ffsll(msk) - 1, a0, a1, b);
          step(x0, x1, y);
        } while (msk);
      }
    }
    // Entries below the current ones are stored, with the predecessor in
    // pivot row k*.
    const int col = col0 + tx;
    const int32_t *const pred1 = PRED ? s.P + (int64_t)(r * kBlk - 1) * s.ld + col : nullptr;  // step k + 1 at + (k + 1) ld
    auto finish = [&](int h, auto edge) {  // edge: rows or columns of the half tile past the matrix
      const int rowh = (h ? row1 : row0) + ty * 4;
      unsigned *crow = static_cast<unsigned *>(s.D) + (int64_t)rowh * ld + col;
      int32_t *qrow = PRED ? s.P + (int64_t)rowh * ld + col : nullptr;
      unsigned c[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int q = 0; q < 4; q++)
          c[i][q] = !decltype(edge)::value || (rowh + i < size && col + 16 * q < size) ? crow[(int64_t)i * ld + 16 * q] : 0u;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        // a row's entries together: the steps of those that improve (0: kept),
        // their predecessors in flight at once, the stores
        unsigned k[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const unsigned v = acc[h * 4 + i][q];
          k[q] = 0;
          if constexpr (F32) {
            if (v < c[i][q]) {
              const int g = max(arg[h * 4 + i][q] - 1, 0) >> 2;
              // (no step: a value above "unreached" that none reaches)
              k[q] = PRED ? (unsigned)unit_resolve_f32(
                                v, arg[h * 4 + i][q],
                                reinterpret_cast<const ulonglong2 *>(&sm.A[0][0])[g * kAUnits + ty * 4 + h * kBlk + i],
                                reinterpret_cast<const ulonglong2 *>(&sm.B[0][0])[g * kBlk + tx + 16 * q])
                          : (unsigned)arg[h * 4 + i][q];
            }
          } else {
            k[q] = v < min(c[i][q], kPackH) << kIdxBits ? v & kIdxMask : 0u;
          }
        }
        if (k[0] | k[1] | k[2] | k[3]) {
          int32_t pv[4];
#pragma unroll
          for (int q = 0; q < 4; q++) pv[q] = PRED && k[q] ? pred1[(int64_t)(int)k[q] * ld + 16 * q] : 0;
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (k[q]) {
              crow[16 * q] = F32 ? acc[h * 4 + i][q] : acc[h * 4 + i][q] >> kIdxBits;
              if (PRED) qrow[16 * q] = pv[q];
            }
        }
        crow += ld;
        if (PRED) qrow += ld;
      }
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (h == 1 && !two) break;
      if (col0 + kBlk <= size && (h ? row1 : row0) + kBlk <= size) finish(h, std::false_type{});
      else finish(h, std::true_type{});
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (t == 0 && n_work > 0) atomicAdd(&g_fw_counters[0], n_work);
}

template <bool F32, bool PRED>
cudaError_t launch_rest(const FwRestJob *d_jobs, int njobs, int strips, int per, cudaStream_t st) {
  ++launch_count();
  fw_rest_kernel<F32, PRED><<<strips, kRestThreads, sizeof(RestSmem<F32>), st>>>(d_jobs, njobs, per);
  return cudaGetLastError();
}

int strips_of(const FwRestJob &j, int per) {
  const int n = rest_blocks((j.size + kBlk - 1) / kBlk, j.look);
  return (n + 1) / 2 * ((n + per - 1) / per);
}

}  // namespace

int number_fw_rest(FwRestJob *jobs, int njobs, int sm_count, int *per) {
  // The column tiles a CTA takes: the most (up to 8, which amortise the
  // staging of A) that still give the launch one CTA for every slot of the
  // GPU (two per SM).  A single 910-vertex matrix then runs its remaining
  // tiles in 98 CTAs of one tile instead of 14 of eight (its 14 rounds took
  // 2.33 ms in strips of 8, 1.15 ms in single tiles).
  auto count = [&](int tiles) {
    long long strips = 0;
    for (int i = 0; i < njobs; i++) strips += strips_of(jobs[i], tiles);
    return strips;
  };
  *per = 1;
  long long longest = 0;
  for (int tiles = 8; tiles > 1; tiles /= 2) {
    const long long strips = count(tiles);
    if (tiles == 8) longest = strips;
    if (strips >= 2LL * sm_count) {
      *per = tiles;
      break;
    }
  }
  // Of 8 to 4 tiles, where a few strips an SM are all there is, the length that
  // gives the busiest SM the least (a strip's start counted as a tile and a
  // half): the twelve listed block columns of a 64-matrix road-like graph go in
  // three strips of four instead of eight and four (whole solve 22.75 -> 22.45
  // ms), a geometric graph's fifteen in fives (14.81 -> 14.61).  Shorter ones, or
  // those of launches that take less than 8 anyway, measured the same or slower.
  if (*per == 8 && longest < 8LL * sm_count) {
    long long best = 0;
    for (int tiles = 8; tiles >= 4; tiles--) {
      const long long cost = (count(tiles) + sm_count - 1) / sm_count * (2 * tiles + 3);
      if (tiles == 8 || cost < best) best = cost, *per = tiles;
    }
  }
  int strips = 0;
  for (int i = 0; i < njobs; i++) {
    jobs[i].strip_begin = strips;
    strips += strips_of(jobs[i], *per);
  }
  return strips;
}

cudaError_t launch_fw_rest(bool f32, bool pred, const FwRestJob *d_jobs, int njobs, int strips, int per,
                           cudaStream_t st) {
  if (njobs <= 0 || strips <= 0) return cudaSuccess;
  if (f32)
    return pred ? launch_rest<true, true>(d_jobs, njobs, strips, per, st)
                : launch_rest<true, false>(d_jobs, njobs, strips, per, st);
  return pred ? launch_rest<false, true>(d_jobs, njobs, strips, per, st)
              : launch_rest<false, false>(d_jobs, njobs, strips, per, st);
}

cudaError_t fw_rest_counter(unsigned long long *out, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_fw_counters, sizeof(unsigned long long));
  if (e != cudaSuccess || !reset) return e;
  const unsigned long long zero = 0;
  return cudaMemcpyToSymbol(g_fw_counters, &zero, sizeof(zero));
}

cudaError_t init_fw_rest_kernels() {
  cudaError_t e;
#define FAP_REST_ATTR(F, P)                                                                           \
  if ((e = cudaFuncSetAttribute(fw_rest_kernel<F, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                (int)sizeof(RestSmem<F>))) != cudaSuccess)                            \
    return e;
  FAP_REST_ATTR(true, true)
  FAP_REST_ATTR(true, false)
  FAP_REST_ATTR(false, true)
  FAP_REST_ATTR(false, false)
#undef FAP_REST_ATTR
  return cudaSuccess;
}

}  // namespace fapk
