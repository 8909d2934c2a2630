// mp_rows.cu -- the packed int32 min-plus of inner rows that do not start on
// 16-byte boundaries.
//
// Reference counterparts: min_plus_path_CPU_advanced (fap/kernel/minplus.h:
// 51-65) and MatrixMulCUDA6_path (fap/kernel/cuda/minplus.cu:32-189), with the
// decode of the inner rows (MysubMatDecode_path, fap/utils/util_Myalgorithm.h:
// 236-247) in its epilogue.
//
// The product of mp_strip_kernel (minplus.cu) for rows of a length that is no
// multiple of 4 words.  A tile's 64 columns then start anywhere in a 32-byte
// sector, and a sector that two tiles write in turn costs more than twice: 8
// bytes an output to rows of 57,301 words go at 2.7-3.4 TB/s when a warp stores
// 16 or 32 consecutive words of a row wherever they lie, and at 7.5 TB/s when
// each sector is written by one store (rows of 57,344 words: 7.5 TB/s).
//
//  - So every row moves its tiles back to the sector boundary.  A warp takes the
//    rows of one residue modulo 8, whose addresses modulo 32 are the same
//    whatever the leading dimension: its shift is uniform, its columns of the
//    tile are 64 of the 72 that are staged, and nothing is exchanged or kept
//    between tiles.
//  - A CTA owns a strip: 128 rows with A resident in shared memory, and `per`
//    x 128 consecutive columns in tiles of 64.  256 threads, 8 x 4 outputs
//    each; a thread's columns are 16 apart, so that a half-warp stores two whole
//    sectors of a row at once.
//  - The next tile's B arrives by cp.async behind the current tile, and every
//    thread prepares the entries that it copied itself (keys, marks), so that a
//    tile has one barrier.
//  - Steps k without a finite entry in the tile's B row or the strip's A
//    column cannot change an output and are skipped.
//  - The part's own columns take the Floyd-Warshall values, copied to shared
//    memory a tile ahead.
//
// Bound by the instructions of an output that are not add-mins (64 in all, five
// of them add-mins on a geometric graph; 51 % of the issue slots).  Min-plus phase of geometric graphs, against the strip kernel
// with its stores realigned to 16 bytes: 57,301 vertices in 55 parts 12.5 -> 8.4
// ms (3.1 TB/s of results), 24,575 in 23 parts 2.92 -> 2.14 ms, 9,001 in 8 parts
// 0.61 -> 0.53 ms.  Rows on 16-byte boundaries stay with the strips (57,300
// vertices: 8.2 ms there, 9.0 ms here).

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "fw_tile.cuh"
#include "launch.h"
#include "mp_common.cuh"

namespace fapk {

namespace {

constexpr int kMpThreads = 256;
constexpr int kMpRows = 128;
constexpr int kMpCols = 64;       // columns of a tile that a row stores
constexpr int kMpHalo = 8;        // ... and those before them, of which rows take up to 7 in place of the last
constexpr int kMpWide = kMpCols + kMpHalo;
constexpr int kMpOwn = 4;         // own columns of a tile whose values are staged

// Shared memory for segments of up to ks steps (a multiple of 4): keys of A
// [ks][128], of B [2][ks][72].
constexpr size_t mp_rows_smem(int ks) { return (size_t)ks * (kMpRows + 2 * kMpWide) * 4; }

// Words by which a row's tiles move back at most.
__host__ __device__ __forceinline__ int max_shift(const MpSegment &s) {
  return (s.ldc & 7) == 0 ? (int)(reinterpret_cast<uintptr_t>(s.C) >> 2 & 7) : 7;
}
__host__ __device__ __forceinline__ int row_tiles(const MpSegment &s) {
  return (s.N + max_shift(s) + kMpCols - 1) / kMpCols;
}

// Work counters as mp_strip_kernel's (minplus.cu), summed per CTA.
__device__ unsigned long long g_rows_counters[3];

// The segment that strip x of the launch belongs to: a warp probes 32 at a time.
__device__ __forceinline__ int find_strip(const MpSegment *segs, int nseg, int x) {
  const int lane = threadIdx.x & 31;
  int lo = 0, len = nseg;
  while (len > 1) {
    const int each = (len + 31) / 32, i = lane * each;
    const unsigned below = __ballot_sync(0xffffffffu, i < len && segs[lo + i].strip_begin <= x);
    const int at = (__popc(below) - 1) * each;
    lo += at;
    len = min(each, len - at);
  }
  return lo;
}

template <bool PRED>
__global__ void __launch_bounds__(kMpThreads, 3)
    mp_rows_kernel(const MpSegment *__restrict__ segs, int nseg, int ks, int per) {
  extern __shared__ __align__(16) unsigned char mp_smem_raw[];
  unsigned *const A = reinterpret_cast<unsigned *>(mp_smem_raw);
  unsigned *const B = A + ks * kMpRows;
  __shared__ MpSegment s;
  __shared__ unsigned s_amask[4];     // steps with a finite entry in the strip's rows
  // ... and in the tile's columns: in turn of three (being marked, read, cleared
  // for the tile after next), so that one barrier a tile orders them
  __shared__ unsigned s_bmask[3][4];
  // A tile's columns that are the part's own, and their columns of the FW matrix
  // (in turn of three: marked a tile ahead); the values of the first kMpOwn of
  // them, in order: distances, predecessors (per tile parity).
  __shared__ unsigned s_ownmask[3][3];
  __shared__ int32_t s_ownf[3][kMpWide];
  __shared__ unsigned s_f[2][kMpOwn][2][kMpRows];
  __shared__ int32_t s_col[2][2][kMpWide];  // col_part and col_local of the columns, on the way (per tile parity)
  const int t = threadIdx.x;
  {
    const int j = find_strip(segs, nseg, blockIdx.x);
    if (t == 0) s = segs[j];
    if (t < 4) s_amask[t] = 0u;
    if (t < 12) (&s_bmask[0][0])[t] = 0u;
  }
  __syncthreads();
  const int tiles = row_tiles(s), sx = (tiles + per * 2 - 1) / (per * 2);
  const int local = blockIdx.x - s.strip_begin, rt = local / sx;
  const int jt0 = (local - rt * sx) * per * 2, jt1 = min(jt0 + per * 2, tiles);
  const int row0 = rt * kMpRows;
  const int K = s.K, kseg = (K + 3) & ~3;
  const int M = s.M, N = s.N;
  const unsigned INF = Dist<uint32_t>::inf(), NONE = kPackH << kIdxBits;
  const int ty = t >> 4, tx = t & 15, warp = t >> 5;
  // the warp's shift; pos: the place of the thread's first column in the tile
  const int shift = (int)(((reinterpret_cast<uintptr_t>(s.C) >> 2) + (uint64_t)warp * (uint64_t)s.ldc) & 7);
  const int pos = kMpHalo - shift + tx;
  const int64_t ldb = s.ldb;

  // The K x 72 entries of B's columns from 64 jt - 8 on: a thread copies column t
  // % 64 of rows t / 64 + 4 i, then 64 + t % 8 of rows t / 8 + 32 i (outside the
  // matrix: unreached).
  auto load_tile = [&](int jt, int par) {
    const int col0 = jt * kMpCols - kMpHalo;
    auto column = [&](int j, int k0, int step) {
      unsigned *d = B + (par * ks + k0) * kMpWide + j;
      const unsigned *g = static_cast<const unsigned *>(s.B) + k0 * ldb + col0 + j;
      const bool in = (unsigned)(col0 + j) < (unsigned)N;
      for (int k = k0; k < K; k += step, d += step * kMpWide, g += step * ldb)
        if (in) cp_async4(d, g);
        else *d = INF;
    };
    column(t & 63, t >> 6, kMpThreads / 64);
    column(64 + (t & 7), t >> 3, kMpThreads / 8);
  };
  auto in_tile = [&](int jt) {  // the tile has a column t, inside the matrix
    return t < kMpWide && jt < jt1 && (unsigned)(jt * kMpCols - kMpHalo + t) < (unsigned)N;
  };
  auto load_own = [&](int jt, int par) {  // part and position of a tile's columns, a thread's own one
    if (s.col_part != nullptr && in_tile(jt)) {
      cp_async4(&s_col[par][0][t], s.col_part + jt * kMpCols - kMpHalo + t);
      cp_async4(&s_col[par][1][t], s.col_local + jt * kMpCols - kMpHalo + t);
    }
  };
  auto mark_own = [&](int jt, int turn, int par) {  // (behind the wait for load_own's copies)
    if (t < 96) {
      const bool mine = s.col_part != nullptr && in_tile(jt) && s_col[par][0][t] == s.part;
      const unsigned own = __ballot_sync(0xffffffffu, mine);
      if ((t & 31) == 0) s_ownmask[turn][t >> 5] = own;
      if (mine) s_ownf[turn][t] = s_col[par][1][t] - s.local0;
    }
  };
  auto copy_own = [&](int turn, int par) {  // a thread: row t % 128 of the strip, distances or predecessors
    const int m = t & (kMpRows - 1), arr = t >> 7;
    if (row0 + m >= M || (!PRED && arr)) return;
    const unsigned *f = (arr ? reinterpret_cast<const unsigned *>(s.Fp) : static_cast<const unsigned *>(s.F)) +
                        (row0 + m) * s.ldf;
    int q = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
      for (unsigned left = s_ownmask[turn][i]; left && q < kMpOwn; left &= left - 1u, q++)
        cp_async4(&s_f[par][q][arr][m], f + s_ownf[turn][32 * i + __ffs(left) - 1]);
  };
  load_own(jt0, 0);
  load_own(jt0 + 1, 1);
  for (int i = K * kMpWide + t; i < kseg * kMpWide; i += kMpThreads)  // the steps from K to kseg: unreached
    B[i] = B[ks * kMpWide + i] = NONE;
  load_tile(jt0, 0);
  cp_async_commit();
  for (int i = t; i < kMpRows * kseg; i += kMpThreads) {  // A: consecutive threads on consecutive steps of a row
    const int m = i / kseg, k = i - m * kseg;
    const unsigned v = row0 + m < M && k < K
                           ? static_cast<const unsigned *>(s.A)[(row0 + m) * s.lda + k] : INF;
    const int at = (m & 7) * 16 + (m >> 3);  // the rows of a warp side by side
    A[k * kMpRows + (at ^ swz<true>(k))] = min(v, kPackH) << kIdxBits;
  }
  cp_async_wait_0();
  mark_own(jt0, 0, 0);
  __syncthreads();
  copy_own(0, 0);
  cp_async_commit();
  for (int k = t >> 5; k < kseg; k += kMpThreads / 32) {
    bool fin = false;
#pragma unroll
    for (int h = 0; h < kMpRows; h += 32) fin |= A[k * kMpRows + h + (t & 31)] < NONE;
    if (__any_sync(0xffffffffu, fin) && (t & 31) == 0) atomicOr(&s_amask[k >> 5], 1u << (k & 31));
  }

  unsigned long long n_tiles = 0, n_empty = 0, n_work = 0;
  int mi = 0;  // (jt - jt0) % 3
  for (int jt = jt0; jt < jt1; jt++, mi = mi == 2 ? 0 : mi + 1) {
    const int par = (jt - jt0) & 1;
    unsigned *const Bt = B + par * ks * kMpWide;
    cp_async_wait_0();
    const int mn = mi == 2 ? 0 : mi + 1;
    mark_own(jt + 1, mn, par ^ 1);
    // this thread's entries: keys, and which rows have a finite one
    auto entry = [&](unsigned *p, int k) {
      const unsigned v = *p;
      *p = min(v, kPackH) * (1u << kIdxBits) + (unsigned)(k + 1);
      return v < kPackH;
    };
    {
      unsigned *p = Bt + (t >> 6) * kMpWide + (t & 63);
      for (int k = t >> 6; k < K; k += kMpThreads / 64, p += kMpThreads / 64 * kMpWide)
        if (__any_sync(0xffffffffu, entry(p, k)) && (t & 31) == 0) atomicOr(&s_bmask[mi][k >> 5], 1u << (k & 31));
      p = Bt + (t >> 3) * kMpWide + 64 + (t & 7);
      for (int k = t >> 3; k < K; k += kMpThreads / 8, p += kMpThreads / 8 * kMpWide)
        if (entry(p, k)) atomicOr(&s_bmask[mi][k >> 5], 1u << (k & 31));
    }
    __syncthreads();  // keys and marks; every thread is done with the last tile
    if (t < 4) s_bmask[mi == 0 ? 2 : mi - 1][t] = 0u;
    if (jt + 1 < jt1) {
      load_tile(jt + 1, par ^ 1);
      copy_own(mn, par ^ 1);
      load_own(jt + 2, par);
      cp_async_commit();
    }
    const unsigned own0 = s_ownmask[mi][0], own1 = s_ownmask[mi][1], own2 = s_ownmask[mi][2];
    unsigned long long mlo = (unsigned long long)(s_bmask[mi][0] & s_amask[0]) |
                             ((unsigned long long)(s_bmask[mi][1] & s_amask[1]) << 32);
    unsigned long long mhi = (unsigned long long)(s_bmask[mi][2] & s_amask[2]) |
                             ((unsigned long long)(s_bmask[mi][3] & s_amask[3]) << 32);
    const bool empty = (mlo | mhi) == 0;
    const int nact = __popcll(mlo) + __popcll(mhi);
    n_tiles++;
    n_empty += empty;
    n_work += (unsigned long long)nact * (kMpRows * kMpCols);

    unsigned acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) acc[i][c] = NONE;
    auto step = [&](int k) {
      const unsigned *ap = A + k * kMpRows;
      const uint4 a0 = *reinterpret_cast<const uint4 *>(ap + ((ty * 8) ^ swz<true>(k)));
      const uint4 a1 = *reinterpret_cast<const uint4 *>(ap + ((ty * 8 + 4) ^ swz<true>(k)));
      const unsigned *bp = Bt + k * kMpWide + pos;
      const unsigned a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const unsigned b[4] = {bp[0], bp[16], bp[32], bp[48]};
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[i][c] = __viaddmin_u32(a[i], b[c], acc[i][c]);
    };
    if (nact == K) {  // every step, in groups of four
      for (int k = 0; k < kseg; k += 4) {
#pragma unroll
        for (int q = 0; q < 4; q++) step(k + q);
      }
    } else {
      for (; mlo; mlo &= mlo - 1ull) step(__ffsll(mlo) - 1);
      for (; mhi; mhi &= mhi - 1ull) step(63 + __ffsll(mhi));
    }

    const int col = jt * kMpCols - shift + tx;
    const int m0 = warp + 8 * ((ty & 1) * 8);  // the thread's first row of the strip, and every eighth from it
    // step k at + (k + 1) ldbp (in bytes, 32 bits: one multiply-add an address)
    const char *const pred1 = PRED ? reinterpret_cast<const char *>(s.Bp - s.ldbp + col) : nullptr;
    const unsigned ldbp4 = (unsigned)(s.ldbp * 4);
    const int64_t ldc8 = 8 * s.ldc, ldcp8 = 8 * s.ldcp;
    unsigned *crow = static_cast<unsigned *>(s.C) + (row0 + m0) * s.ldc + col;
    int32_t *qrow = PRED ? s.Cp + (row0 + m0) * s.ldcp + col : nullptr;
    auto finish = [&](auto masked) {  // masked: rows or columns past the matrix, or own columns
      constexpr bool kMasked = decltype(masked)::value;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int32_t p[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          unsigned *row = acc[h * 4 + i];
          const bool some = min(min(row[0], row[1]), min(row[2], row[3])) < NONE;
#pragma unroll
          for (int c = 0; c < 4; c++) {
            p[i][c] = -1;
            const unsigned k = some ? row[c] & kIdxMask : 0u;  // 0: unreached (columns past the matrix are)
            if (PRED && k) p[i][c] = *reinterpret_cast<const int32_t *>(pred1 + (uint64_t)k * ldbp4 + 64 * c);
            row[c] = k ? row[c] >> kIdxBits : INF;
          }
        }
        if (kMasked) {
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const int j = pos + 16 * c;
            const unsigned mask = j < 32 ? own0 : j < 64 ? own1 : own2;
            if (!(mask >> (j & 31) & 1u)) continue;
            const int q = (j < 32 ? 0 : j < 64 ? __popc(own0) : __popc(own0) + __popc(own1)) +
                          __popc(mask & ((1u << (j & 31)) - 1u));
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int m = m0 + 8 * (h * 4 + i);
              if (row0 + m >= M) break;
              const int64_t f = (row0 + m) * s.ldf + s_ownf[mi][j];
              acc[h * 4 + i][c] = q < kMpOwn ? s_f[par][q][0][m] : static_cast<const unsigned *>(s.F)[f];
              if (PRED) p[i][c] = q < kMpOwn ? (int32_t)s_f[par][q][1][m] : s.Fp[f];
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
          if (!kMasked || row0 + m0 + 8 * (h * 4 + i) < M) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
              if (kMasked && (unsigned)(col + 16 * c) >= (unsigned)N) continue;
              __stcs(crow + 16 * c, acc[h * 4 + i][c]);  // (the rows are not read again here)
              if (PRED) __stcs(qrow + 16 * c, p[i][c]);
            }
          }
          crow += ldc8;
          if (PRED) qrow += ldcp8;
        }
      }
    };
    if ((own0 | own1 | own2) != 0 || jt == 0 || (jt + 1) * kMpCols > N || row0 + kMpRows > M) {
      finish(std::true_type{});
    } else if (!empty) {
      finish(std::false_type{});
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
          __stcs(crow + 16 * c, INF);
          if (PRED) __stcs(qrow + 16 * c, -1);
        }
        crow += ldc8;
        if (PRED) qrow += ldcp8;
      }
    }
  }
  cp_async_wait_0();
  if (t == 0 && n_tiles > 0) {
    atomicAdd(&g_rows_counters[0], n_tiles);
    atomicAdd(&g_rows_counters[1], n_empty);
    atomicAdd(&g_rows_counters[2], n_work);
  }
}

int strips_of(const MpSegment &s, int per) {
  return (s.M + kMpRows - 1) / kMpRows * ((row_tiles(s) + per * 2 - 1) / (per * 2));
}

}  // namespace

int number_minplus_rows(MpSegment *segs, int nseg, int sm_count, int *per) {
  return number_strips(segs, nseg, sm_count, 3, per, strips_of);
}

cudaError_t launch_minplus_rows(bool pred, const MpSegment *d_segs, int nseg, int strips, int max_k, int per,
                                cudaStream_t st) {
  if (strips <= 0 || nseg <= 0) return cudaSuccess;
  if (max_k < 0 || max_k > minplus_strip_max_k(false) || per < 1) return cudaErrorInvalidValue;
  const int ks = std::max((max_k + 3) & ~3, 4);
  ++launch_count();
  if (pred) mp_rows_kernel<true><<<strips, kMpThreads, mp_rows_smem(ks), st>>>(d_segs, nseg, ks, per);
  else mp_rows_kernel<false><<<strips, kMpThreads, mp_rows_smem(ks), st>>>(d_segs, nseg, ks, per);
  return cudaGetLastError();
}

cudaError_t rows_counters(unsigned long long out[3], bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_rows_counters, sizeof(unsigned long long) * 3);
  if (e != cudaSuccess || !reset) return e;
  const unsigned long long zero[3] = {0, 0, 0};
  return cudaMemcpyToSymbol(g_rows_counters, zero, sizeof(zero));
}

cudaError_t init_mp_rows_kernels() {
  const int smem = (int)mp_rows_smem((minplus_strip_max_k(false) + 3) & ~3);
  cudaError_t e = cudaFuncSetAttribute(mp_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(mp_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

}  // namespace fapk
