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
// it, so rows are for few walks or short rows: walks x vertices up to
// kWalkQueries (a query in device memory walks twice) or kWalkPairs.  Walks of 100
// to 222 hops on road graphs, by rows / in device memory, queries and pairs: 4,096
// vertices 10,000 walks 111 / 529 us and 129 / 191 us, 200,000 walks 1,256 / 711 and
// 1,419 / 491; 8,000 vertices 10,000 walks 191 / 960 and 240 / 415, 200,000 walks
// 2,717 / 1,684 and 3,267 / 799; 24,575 vertices 200 walks 58 / 1,200 and 60 / 544,
// 10,000 walks 753 / 2,778 and 937 / 1,014, 200,000 walks 13,219 / 4,252 us.  Short
// walks (dense graphs) are finished by the thread that started them and never
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
constexpr int64_t kWalkQueries = 400000000, kWalkPairs = 100000000;

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
