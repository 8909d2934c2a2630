// path_walk.cuh -- following a predecessor row from t back to s.
//
// A walk is a chain of dependent loads, about 0.7 us each from device memory:
// 100 to 200 hops of a 4,096-vertex road graph took 280 us however many walks ran
// beside it.  So a walk that is not done after kWalkHops hops gets a CTA: it
// reads the whole row (coalesced, 16 KB there, 2 us), narrowed to 16 bits, and
// one thread walks it in shared memory, 20 ns a hop.  What is done with the
// vertices then runs over all of them at once.
//
// A row costs what it is long, and the chain does not care how many walk beside
// it, so rows are for few walks and short rows (walks_by_row).  A query with its
// path walks twice in device memory, without it once and without the look-up of an
// edge.  By rows / in device memory, us, queries with paths | without | pairs of
// road graphs (hops on average):
//   500 vertices (35)      10,000 walks  65 / 85 | 63 / 43 | 82 / 76,   100,000  268 / 162 | 257 / 46 | 371 / 315
//   1,000 (54)              3,000  58 / 185 | 55 / 52 | 69 / 95,   30,000  156 / 243 | 147 / 52 | 177 / 139
//   4,096 (102)             1,000  51 / 527 | 50 / 70 | 59 / 187,   10,000  115 / 530 | 111 / 74 | 133 / 188
//                          30,000  249 / 604 | 240 / 84 | 275 / 198,   100,000  665 / 660 | 643 / 97 | 749 / 337
//   8,000 (132)             3,000  100 / 755 | 99 / 89 | 113 / 309,   30,000  474 / 1,429 | 463 / 193 | 558 / 438
//   14,000 (177)            1,000  87 / 980 | 86 / 109 | 104 / 437,   10,000  426 / 1,932 | 423 / 261 | 520 / 715
//   28,000 (242)            1,000  149 / 1,278 | 148 / 142 | 185 / 638,   10,000  864 / 3,161 | 856 / 361 | 1,117 / 1,008
// and of grids, whose walks are shorter:
//   1,024 (23)             10,000  59 / 70 | 57 / 40 | 76 / 65,   100,000  209 / 107 | 201 / 41 | 262 / 153
//   10,000 (69)             3,000  89 / 244 | 87 / 61 | 107 / 203,   30,000  444 / 387 | 436 / 112 | 541 / 270
//   22,500 (103)            3,000  191 / 394 | 190 / 75 | 248 / 318,   10,000  509 / 378 | 497 / 100 | 669 / 347
// (The line for queries with paths is the roads': grids lose up to a third near it.)
// Short walks (dense graphs) are finished by the thread that started them and never
// read a row: 8 hops at most left half of a random graph's walks of 8 hops on
// average to rows of 25,000 vertices (10,000 walks 190 us, 46 us without).  Rows of
// more than kWalkMaxN vertices (two CTAs an SM) are walked in device memory.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fapk {

constexpr int kWalkThreads = 256;
constexpr int kWalkHops = 16;
constexpr int kWalkMaxN = 28000;

// Whether `walks` walks go by row: at most `most` of them, and walks x vertices.
inline bool walks_by_row(int n, int64_t walks, int64_t most, int64_t cells) {
  return n <= kWalkMaxN && walks <= most && walks * n <= cells;
}

// Entries of a row in shared memory that are no vertex.
constexpr unsigned kWalkNone = 0xffffu, kWalkBad = 0xfffeu;  // (negative; n or above)

// Dynamic shared memory: the row [n] | the walk's vertices [n + 2].
constexpr size_t walk_smem(int n) { return ((size_t)2 * n + 2) * sizeof(uint16_t); }

// All threads of the CTA: the walk's vertices t, ..., s in `path` and, in every
// thread, their number; `end` is s, or kWalkNone / kWalkBad where the chain
// breaks (a chain longer than the row is bad).
__device__ __forceinline__ int walk_row(const int32_t *prow, int n, int s, int t, uint16_t *row, uint16_t *path,
                                        unsigned &end) {
  __shared__ int s_len;
  __shared__ unsigned s_end;
#pragma unroll 8
  for (int i = threadIdx.x; i < n; i += kWalkThreads) {
    const int v = prow[i];
    row[i] = (uint16_t)(v < 0 ? kWalkNone : v >= n ? kWalkBad : (unsigned)v);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned v = (unsigned)t;
    int len = 1;
    path[0] = (uint16_t)v;
    while (v != (unsigned)s) {
      v = row[v];
      if (v >= (unsigned)n) break;
      if (len > n) {
        v = kWalkBad;
        break;
      }
      path[len++] = (uint16_t)v;
    }
    s_len = len;
    s_end = v;
  }
  __syncthreads();
  end = s_end;
  return s_len;
}

// CTAs of the launch over the walks that got one.
inline int walk_ctas(int n, int walks, int sm_count) {
  const size_t each = walk_smem(n) + 2048;
  const int per_sm = (int)(224u * 1024u / each < 8 ? 224u * 1024u / each : 8);
  return walks < per_sm * sm_count ? walks : per_sm * sm_count;
}

}  // namespace fapk
