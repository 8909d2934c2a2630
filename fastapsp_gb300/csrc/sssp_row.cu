// sssp_row.cu -- shortest paths with one CTA per source.
//
// Reference counterparts: dijkstra_path / batched_sssp_path
// (fap/kernel/batch_sssp.h:79-114, 232-303) and multi_source_Nvidia_sssp
// (fap/kernel/cuda/batch_sssp.cu:177-288).
//
// The batched search (sssp.cu) relaxes a frontier vertex for 8 to 32 sources
// at once, which pays when their frontiers coincide.  Sources of a road
// network or a grid have frontiers of their own, so its CTA walks their union
// and most lanes of a sweep have nothing to do; and few sources make few
// CTAs.  Here a CTA searches for one source, with the frontiers in shared
// memory (and an overflow area in device memory) and one barrier a step.  The
// predecessors follow in a launch of their own over all rows.
//
// The search is the near-far delta-stepping of sssp.cu with the same fixpoint
// dist[v] = min_u fl(dist[u] + w(u, v)), unique for positive weights whatever
// the order of relaxations, and the same predecessor rule: the tight
// in-neighbour u first in (dist[u], u) order.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "launch.h"

namespace fapk {

namespace {

// Which form a search takes, and its threads.  Few sources (one CTA each, one
// per SM): a step is its chain of dependent accesses, so four lanes share a
// vertex, the graph is read as edge records, and the distances are in shared
// memory where n allows.  More: what counts is how many CTAs an SM holds, so
// small ones with the distances in the output rows and one thread a vertex.
// Measured (ms, road graphs; the batched search first): 19 sources of 24,575
// vertices 6.69 -> 0.58 in shared memory (1.43 in the rows); 64 of 114,599
// 27.6 -> 2.49; 470 of 24,575 7.0 -> 1.46 in the rows (2.77 in shared memory,
// a CTA an SM); 2,448 of 114,599 104 -> 27.8 (38 with the edge records).
// Four lanes a vertex instead of one: 0.72 -> 0.58 and 3.1 -> 2.5 for few
// sources, 6.0 -> 9.4 for 1,200 of 57,301.
// Small CTAs hold many rows at once, and frontiers that hop over a large graph read
// them from device memory: 1,500 sources of random graphs of 100,000 vertices (608
// CTAs, 243 MB of rows) with 24 edges a vertex took 232 ms, the batched search 220; wide
// CTAs, one an SM, one source after the other, 70.  12 edges 131 / 134 / 44, 6 edges
// 90 / 83 / 36; 200,000 vertices with 20 edges 244 / 415 / 174; nearest-neighbour graphs
// of 200,000 with 8 edges 100 / 90 (small / wide).  So past four edges a vertex and 220 MB
// of rows the wide ones go on.  Below, it is the graph that decides: nearest-neighbour ones of 52,000 with 8 edges (190 MB)
// 18.7 / 25.7, 65,536 with 5 and 8 (199 MB) 25.3 / 28.1 and 35.1 / 30.4, 114,000 with 5 (208
// MB) 39.9 / 45.1; random ones of 64,000 with 12 (195 MB) 37.5 / 27.0.  With fewer edges
// frontiers are narrow (roads; 114,599 vertices 18.7 / 24.4; a full grid of 202,500 with
// 608 sources 9.4 / 10.0) or little is reached.
enum RowForm { kRowMany, kRowFew, kRowFewSmem };
template <bool SMEM, bool WIDE>
constexpr int kRowThreadsOf = SMEM ? 512 : WIDE ? 1024 : 256;
constexpr int kRowCap = 1024;            // frontier entries kept in shared memory, per list
constexpr size_t kRowSmem = 226 * 1024;  // dynamic; the per-block limit also holds the static part
constexpr int kRowLanes = 4;             // lanes that share a frontier vertex
constexpr int kRowPerWarp = 32 / kRowLanes;
constexpr int kRowEdges = 4;             // in-edges of a vertex in flight together
constexpr int kRowMaxDegree = 64;        // few lanes walk a vertex's edges; 127 fit in a record

// Device scratch of a CTA: overflow of the frontiers [2][n] (8 bytes at most)
// and the far lists [2][n].
__host__ __device__ inline size_t row_scratch(int32_t n) { return (size_t)n * 24; }
__host__ __device__ inline int row_words(int32_t n) { return (n + 31) / 32; }
// The graph as this search reads it: an edge holds its target with the
// target's out-degree above it, where the target's edges start, and the
// weight, and a frontier entry is the first two.  So a vertex's edges are
// addressed by its frontier entry alone, and a step's chain has one access to
// the graph (19 sources of a 24,575-vertex road graph, one thread a vertex:
// 0.92 ms with the row offsets looked up at the vertex, 0.72 ms with records).
constexpr int kRowVBits = 25;
__device__ __forceinline__ int row_vertex(uint2 x) { return (int)(x.x & ((1u << kRowVBits) - 1u)); }
__device__ __forceinline__ int row_degree(uint2 x) { return (int)(x.x >> kRowVBits); }
__device__ __forceinline__ uint2 row_entry(const int32_t *ro, int v) {
  const int e0 = ro[v];
  return make_uint2((unsigned)v | (unsigned)(ro[v + 1] - e0) << kRowVBits, (unsigned)e0);
}

__global__ void __launch_bounds__(256) row_edges_kernel(int64_t m, const int32_t *ro, const int32_t *col,
                                                        const unsigned *w, uint4 *edges) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  const uint2 x = row_entry(ro, col[e]);
  edges[e] = make_uint4(x.x, x.y, w[e], 0u);
}

// lists[2][kRowCap] | bitmaps near[2], far | distances (when they fit)
template <bool SMEM>
__host__ __device__ inline size_t row_smem_bytes(int32_t n) {
  return (size_t)2 * kRowCap * sizeof(uint2) + (size_t)3 * row_words(n) * 4 + (SMEM ? (size_t)n * 4 : 0);
}
constexpr int64_t kRowManyBytes = (int64_t)220 << 20;  // of the rows that small CTAs hold
// CTAs of the form for many sources.
inline int64_t many_ctas(int32_t n, int64_t sources, int sm_count) {
  const size_t smem = row_smem_bytes<false>(n) + 1024;
  return std::min<int64_t>(sources, (int64_t)std::min<size_t>(8, std::max<size_t>(1, (size_t)228 * 1024 / smem)) * sm_count);
}
inline RowForm row_form(int32_t n, int64_t m, int64_t sources, int sm_count) {
  if (sources > sm_count && (m <= 4 * (int64_t)n || many_ctas(n, sources, sm_count) * n * 4 <= kRowManyBytes))
    return kRowMany;
  return row_smem_bytes<true>(n) <= kRowSmem ? kRowFewSmem : kRowFew;
}

__device__ __forceinline__ bool row_set_bit(unsigned *bits, int v) {
  const unsigned m = 1u << (v & 31);
  return (atomicOr(&bits[v >> 5], m) & m) == 0u;
}

// Distances of one source: shared memory, or the output row (read past L1,
// where the atomics land).
template <bool SMEM>
__device__ __forceinline__ unsigned row_dist(const unsigned *d, int v) {
  return SMEM ? d[v] : __ldcg(d + v);
}

// The batch of a search's source number `job`: batches hold at most a.lanes, so
// it is no earlier than job / a.lanes (and there where they are full); a warp
// probes 32 at a time.
__device__ __forceinline__ int row_batch(const SsspArgs &a, int64_t job) {
  const int lane = threadIdx.x & 31;
  for (int b = (int)(job / a.lanes);; b += 31) {
    const unsigned from = __ballot_sync(0xffffffffu, b + lane < a.nbatches && a.batches[b + lane].first <= job);
    if (from != 0xffffffffu) return b + __popc(from) - 1;
  }
}

// Predecessor of v at distance bits dk (below "unreached").
template <typename T>
__device__ __forceinline__ int32_t row_pred(const SsspArgs &a, const unsigned *d, int v, unsigned dk) {
  const unsigned *iwb = static_cast<const unsigned *>(a.iw);
  unsigned bd = ~0u;
  int bu = -1;
  const int e1 = a.iro[v + 1];
  for (int e = a.iro[v]; e < e1; e += kRowEdges) {
    int u[kRowEdges];
    unsigned w[kRowEdges], du[kRowEdges];
#pragma unroll
    for (int q = 0; q < kRowEdges; q++) {
      u[q] = e + q < e1 ? a.icol[e + q] : -1;
      w[q] = e + q < e1 ? iwb[e + q] : 0u;
    }
#pragma unroll
    for (int q = 0; q < kRowEdges; q++) du[q] = u[q] >= 0 ? row_dist<false>(d, u[q]) : Dist<T>::bits(Dist<T>::inf());
#pragma unroll
    for (int q = 0; q < kRowEdges; q++) {
      const unsigned sum = Dist<T>::bits(Dist<T>::add(Dist<T>::from_bits(du[q]), Dist<T>::from_bits(w[q])));
      if (du[q] < Dist<T>::bits(Dist<T>::inf()) && sum == dk && (du[q] < bd || (du[q] == bd && u[q] < bu))) {
        bd = du[q];
        bu = u[q];
      }
    }
  }
  return bu;
}

// WIDE: kRowLanes lanes a frontier vertex, edge records; else one thread a
// vertex, the CSR.
template <typename T, bool PRED, bool SMEM, bool WIDE>
__global__ void __launch_bounds__(kRowThreadsOf<SMEM, WIDE>, WIDE ? 1 : 4)
    sssp_row_kernel(SsspArgs a) {
  extern __shared__ __align__(16) unsigned char row_smem[];
  const int32_t n = a.n;
  const int words = row_words(n);
  uint2 *const s_list = reinterpret_cast<uint2 *>(row_smem);  // [2][kRowCap]
  unsigned *const bits = reinterpret_cast<unsigned *>(s_list + 2 * kRowCap);
  unsigned *const farbits = bits + 2 * words;
  unsigned *const s_dist = farbits + words;
  __shared__ int s_near[3], s_far[2];
  __shared__ unsigned s_minfar;
  __shared__ int s_src;
  __shared__ int64_t s_row;
  uint2 *const over =
      reinterpret_cast<uint2 *>(static_cast<unsigned char *>(a.scratch) + (size_t)blockIdx.x * row_scratch(n));
  int32_t *const farq = reinterpret_cast<int32_t *>(over + 2 * (size_t)n);
  const unsigned INF = Dist<T>::bits(Dist<T>::inf());
  const uint4 *edges = static_cast<const uint4 *>(a.row_edges);
  const unsigned *wb = static_cast<const unsigned *>(a.w);
  const T delta = (T)a.delta;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nthr >> 5;
  auto entry = [&](int par, int i) { return i < kRowCap ? s_list[par * kRowCap + i] : __ldcg(&over[(size_t)par * n + i]); };
  auto put = [&](int par, int i, uint2 x) {
    if (i < kRowCap) s_list[par * kRowCap + i] = x;
    else over[(size_t)par * n + i] = x;
  };
  unsigned long long st_steps = 0, st_splits = 0, st_relaxed = 0, st_scanned = 0, st_batches = 0;
  for (int64_t job = blockIdx.x; job < a.sources; job += gridDim.x) {
    if (warp == 0) {
      const SsspBatch &sb = a.batches[row_batch(a, job)];
      if (lane == 0) s_src = sb.src[job - sb.first], s_row = sb.row_off[job - sb.first];
    }
    __syncthreads();
    const int src = s_src;
    unsigned *const row = static_cast<unsigned *>(a.dist) + s_row;
    unsigned *const d = SMEM ? s_dist : row;
    if (src < 0 || src >= n) {
      if (tid == 0) atomicOr(a.status, kErrBadInput);
      __syncthreads();
      continue;
    }
    for (int i = tid; i < n; i += nthr) d[i] = INF;
    for (int i = tid; i < 3 * words; i += nthr) bits[i] = 0u;
    if (tid < 3) s_near[tid] = 0;
    if (tid < 2) s_far[tid] = 0;
    __syncthreads();
    if (tid == 0) {
      d[src] = 0u;
      bits[src >> 5] = 1u << (src & 31);
      put(0, 0, row_entry(a.ro, src));
      s_near[0] = 1;
    }
    __syncthreads();
    T thr = delta;
    // step counters in turn of three (read, being filled, cleared for the
    // next step), lists in turn of two: one barrier a step
    int at = 0, par = 0, fcur = 0, steps = 0;
    bool capped = false;
    for (;;) {
      for (;;) {
        const int f = s_near[at];
        if (f == 0) break;
        if (++steps > a.iter_cap) {
          capped = true;
          break;
        }
        st_steps++;
        st_relaxed += (unsigned long long)f;
        const int nxt = at == 2 ? 0 : at + 1;
        if (tid == 0) s_near[nxt == 2 ? 0 : nxt + 1] = 0;
        unsigned *const cbits = bits + par * words, *const nbits = bits + (par ^ 1) * words;
        if constexpr (WIDE) {
          // kRowLanes lanes take a vertex, one edge each; a warp runs its trips
          // together, so its pushes take their places with one atomic a list
          for (int base = warp * kRowPerWarp; base < f; base += nwarps * kRowPerWarp) {
            const int i = base + lane / kRowLanes;
            uint2 x = make_uint2(0u, 0u);
            int deg = 0;
            if (i < f) {
              x = entry(par, i);
              deg = row_degree(x);
            }
            const int u = row_vertex(x);
            if (i < f && lane % kRowLanes == 0) atomicAnd(&cbits[u >> 5], ~(1u << (u & 31)));
            const T du = Dist<T>::from_bits(i < f ? row_dist<SMEM>(d, u) : INF);
            for (int e = lane % kRowLanes; __any_sync(0xffffffffu, e < deg); e += kRowLanes) {
              uint2 to = make_uint2(0u, 0u);
              unsigned c = ~0u, old = 0u;
              if (e < deg) {
                const uint4 r = edges[x.y + e];
                to = make_uint2(r.x, r.y);
                c = Dist<T>::bits(Dist<T>::add(du, Dist<T>::from_bits(r.z)));
                old = row_dist<SMEM>(d, row_vertex(to));
                if (c < old) old = atomicMin(&d[row_vertex(to)], c);
              }
              const int v = row_vertex(to);
              const unsigned bit = 1u << (v & 31);
              const bool near = Dist<T>::from_bits(c) < thr;
              const bool push = c < old && (atomicOr(&(near ? nbits : farbits)[v >> 5], bit) & bit) == 0u;
              const unsigned mn = __ballot_sync(0xffffffffu, push && near), mf = __ballot_sync(0xffffffffu, push && !near);
              int bn = 0, bf = 0;
              if (lane == 0 && mn) bn = atomicAdd(&s_near[nxt], __popc(mn));
              if (lane == 0 && mf) bf = atomicAdd(&s_far[fcur], __popc(mf));
              bn = __shfl_sync(0xffffffffu, bn, 0);
              bf = __shfl_sync(0xffffffffu, bf, 0);
              const unsigned below = (1u << lane) - 1u;
              if (push && near) put(par ^ 1, bn + __popc(mn & below), to);
              else if (push) farq[(size_t)fcur * n + bf + __popc(mf & below)] = v;
            }
          }
        } else {
          for (int i = tid; i < f; i += nthr) {
            const int u = row_vertex(entry(par, i));
            atomicAnd(&cbits[u >> 5], ~(1u << (u & 31)));
            const T du = Dist<T>::from_bits(row_dist<SMEM>(d, u));
            const int e1 = a.ro[u + 1];
            for (int e = a.ro[u]; e < e1; e += kRowEdges) {
              int v[kRowEdges];
              unsigned c[kRowEdges], old[kRowEdges];
#pragma unroll
              for (int q = 0; q < kRowEdges; q++) {
                const bool in = e + q < e1;
                v[q] = in ? a.col[e + q] : -1;
                c[q] = in ? Dist<T>::bits(Dist<T>::add(du, Dist<T>::from_bits(wb[e + q]))) : ~0u;
              }
#pragma unroll
              for (int q = 0; q < kRowEdges; q++) old[q] = v[q] >= 0 ? row_dist<SMEM>(d, v[q]) : 0u;
#pragma unroll
              for (int q = 0; q < kRowEdges; q++)
                old[q] = c[q] < old[q] ? atomicMin(&d[v[q]], c[q]) : 0u;
#pragma unroll
              for (int q = 0; q < kRowEdges; q++) {
                if (!(c[q] < old[q])) continue;
                if (Dist<T>::from_bits(c[q]) < thr) {
                  if (row_set_bit(nbits, v[q])) put(par ^ 1, atomicAdd(&s_near[nxt], 1), make_uint2((unsigned)v[q], 0u));
                } else if (row_set_bit(farbits, v[q])) {
                  farq[(size_t)fcur * n + atomicAdd(&s_far[fcur], 1)] = v[q];
                }
              }
            }
          }
        }
        __syncthreads();
        at = nxt;
        par ^= 1;
      }
      if (capped) break;
      const int nf = s_far[fcur];
      if (nf == 0) break;
      if (++steps > a.iter_cap) {
        capped = true;
        break;
      }
      st_splits++;
      st_scanned += (unsigned long long)nf;
      thr += delta;
      __syncthreads();  // every thread has read the counters
      if (tid == 0) s_minfar = INF;
      __syncthreads();
      for (int i = tid; i < nf; i += nthr) {
        const int v = __ldcg(&farq[(size_t)fcur * n + i]);
        const unsigned m = row_dist<SMEM>(d, v);
        if (Dist<T>::from_bits(m) < thr) {
          atomicAnd(&farbits[v >> 5], ~(1u << (v & 31)));
          if (row_set_bit(bits + par * words, v)) put(par, atomicAdd(&s_near[at], 1), row_entry(a.ro, v));
        } else {  // stays, bit kept
          farq[(size_t)(fcur ^ 1) * n + atomicAdd(&s_far[fcur ^ 1], 1)] = v;
          atomicMin(&s_minfar, m);
        }
      }
      __syncthreads();
      // nothing below the new threshold: move it to the far minimum
      if (s_near[at] == 0 && s_minfar < INF) thr = Dist<T>::from_bits(s_minfar) + delta;
      if (tid == 0) s_far[fcur] = 0;
      fcur ^= 1;
      __syncthreads();
    }
    if (capped) {
      if (tid == 0) atomicOr(a.status, kErrSsspCap);
      break;
    }
    if (SMEM)
      for (int v = tid; v < n; v += nthr) row[v] = d[v];
    st_batches++;
    __syncthreads();
  }
  if (tid == 0 && a.stats != nullptr) {
    atomicAdd(&a.stats[0], st_steps);
    atomicAdd(&a.stats[1], st_splits);
    atomicAdd(&a.stats[2], st_relaxed);
    atomicAdd(&a.stats[3], st_scanned);
    atomicAdd(&a.stats[4], st_batches);
  }
}

// Predecessors (and the largest int32 distance) of finished rows: one thread
// per vertex and source, over the whole GPU at once.
template <typename T, bool PRED>
__global__ void __launch_bounds__(256) sssp_row_output_kernel(SsspArgs a) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned INF = Dist<T>::bits(Dist<T>::inf());
  unsigned local_max = 0;
  for (int64_t job = blockIdx.y; job < (int64_t)a.nbatches * a.lanes; job += gridDim.y) {
    const SsspBatch &sb = a.batches[job / a.lanes];
    const int slot = (int)(job % a.lanes);
    if (slot >= sb.count || v >= a.n) continue;
    const unsigned *d = static_cast<const unsigned *>(a.dist) + sb.row_off[slot];
    const unsigned dk = __ldcg(d + v);
    if (dk < INF) local_max = max(local_max, dk);
    if (PRED) a.pred[sb.row_off[slot] + v] = dk < INF ? (v == sb.src[slot] ? v : row_pred<T>(a, d, v, dk)) : -1;
  }
  if (a.maxd != nullptr) {
    local_max = __reduce_max_sync(0xffffffffu, local_max);
    if ((threadIdx.x & 31) == 0 && local_max) atomicMax(a.maxd, local_max);
  }
}

template <typename T, bool PRED, bool SMEM, bool WIDE>
cudaError_t launch_rows(const SsspArgs &a, cudaStream_t st) {
  ++launch_count();
  sssp_row_kernel<T, PRED, SMEM, WIDE>
      <<<a.slots, kRowThreadsOf<SMEM, WIDE>, row_smem_bytes<SMEM>(a.n), st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || (!PRED && a.maxd == nullptr)) return e;
  const dim3 grid((unsigned)((a.n + 255) / 256), (unsigned)std::min<int64_t>((int64_t)a.nbatches * a.lanes, 65535));
  ++launch_count();
  sssp_row_output_kernel<T, PRED><<<grid, 256, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename T, bool PRED>
cudaError_t launch_rows_t(const SsspArgs &a, RowForm form, cudaStream_t st) {
  if (form == kRowMany) return launch_rows<T, PRED, false, false>(a, st);
  return form == kRowFewSmem ? launch_rows<T, PRED, true, true>(a, st) : launch_rows<T, PRED, false, true>(a, st);
}

}  // namespace

size_t sssp_row_scratch_bytes(int32_t n) { return row_scratch(n); }

int sssp_row_ctas(int32_t n, int64_t m, int64_t sources, int sm_count) {
  if (row_form(n, m, sources, sm_count) == kRowMany) return (int)many_ctas(n, sources, sm_count);
  return (int)std::min<int64_t>(sources, sm_count);
}

int sssp_row_ctas_up_to(int32_t n, int64_t m, int64_t sources, int sm_count) {
  const int ctas = sssp_row_ctas(n, m, sources, sm_count);
  if (sources <= sm_count || row_form(n, m, sources, sm_count) == kRowMany) return ctas;
  return std::max(ctas, (int)(kRowManyBytes / 4 / n));  // fewer sources take small CTAs up to the line
}

cudaError_t launch_row_edges(int64_t m, const int32_t *ro, const int32_t *col, const void *w, void *edges,
                             cudaStream_t st) {
  if (m <= 0) return cudaSuccess;
  ++launch_count();
  row_edges_kernel<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(m, ro, col, static_cast<const unsigned *>(w),
                                                                static_cast<uint4 *>(edges));
  return cudaGetLastError();
}

bool sssp_row_fits(int32_t n, int32_t max_deg) {
  return row_smem_bytes<false>(n) <= kRowSmem && n < (1 << kRowVBits) && max_deg <= kRowMaxDegree;
}

cudaError_t init_sssp_row_kernels() {
  cudaError_t e;
#define FAP_ROW_ATTR(T, P)                                                                                           \
  if ((e = cudaFuncSetAttribute(sssp_row_kernel<T, P, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                                (int)kRowSmem)) != cudaSuccess ||                                                    \
      (e = cudaFuncSetAttribute(sssp_row_kernel<T, P, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,     \
                                (int)kRowSmem)) != cudaSuccess ||                                                    \
      (e = cudaFuncSetAttribute(sssp_row_kernel<T, P, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                (int)kRowSmem)) != cudaSuccess)                                                      \
    return e;
  FAP_ROW_ATTR(float, true)
  FAP_ROW_ATTR(float, false)
  FAP_ROW_ATTR(uint32_t, true)
  FAP_ROW_ATTR(uint32_t, false)
#undef FAP_ROW_ATTR
  return cudaSuccess;
}

cudaError_t launch_sssp_rows(bool f32, const SsspArgs &a, int sm_count, cudaStream_t st) {
  if (a.sources <= 0 || a.slots <= 0) return cudaSuccess;
  if (!sssp_row_fits(a.n, 0) || !(a.delta > 0.0) || a.row_edges == nullptr) return cudaErrorInvalidValue;
  const RowForm form = row_form(a.n, a.m, a.sources, sm_count);
  const bool pred = a.pred != nullptr;
  if (f32) return pred ? launch_rows_t<float, true>(a, form, st) : launch_rows_t<float, false>(a, form, st);
  return pred ? launch_rows_t<uint32_t, true>(a, form, st) : launch_rows_t<uint32_t, false>(a, form, st);
}

}  // namespace fapk
