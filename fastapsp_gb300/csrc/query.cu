// query.cu -- point-to-point queries on solve() results kept in device
// memory: the distance of (s, t) and the path from s to t rebuilt from the
// predecessor rows.
//
// Reference counterpart: getDistanceP2P / getPathP2P (fap/fap.h:144-145),
// which the reference declares without bodies (fap/fap.cpp:674-680); its
// results live in host vectors.  Here a caller that solved into device rows
// (fap_solve with device buffers) reads single entries and paths without
// copying the n x n rows to the host.  One thread per query follows the
// predecessors of row s from t back to s (at most n steps: a chain that does
// not reach s is reported as bad input), then, when the path fits the
// caller's slots, walks it again writing the vertices from the end; walks of
// more than a few hops get a CTA each (path_walk.cuh).  10,000 queries with
// paths of 101 vertices on average on a 4,096-vertex road graph: kernels 94 us, 557 us
// with every walk in device memory.

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.cuh"
#include "launch.h"
#include "path_walk.cuh"

namespace fapk {

namespace {

// Query q in device memory, one thread; false: not done after max_hops hops.
__device__ __forceinline__ bool walk_query(const QueryArgs &a, int q, int max_hops) {
  const int32_t s = a.src[q], t = a.dst[q];
  const int32_t *prow = a.pred + (int64_t)a.ed2st[s] * a.n;
  int32_t len = 1, v = t;
  while (v != s) {
    if (len > max_hops && max_hops < a.n) return false;
    v = prow[v];
    if (v < 0 || v >= a.n || len > a.n) {  // broken chain: not predecessors of a solve
      atomicOr(a.status, kErrBadInput);
      a.out_len[q] = 0;
      return true;
    }
    len++;
  }
  a.out_len[q] = len;
  if (a.out_path == nullptr || len > a.max_len) return true;
  int32_t *path = a.out_path + (int64_t)q * a.max_len;
  v = t;
  for (int32_t i = len - 1; i >= 0; i--) {
    path[i] = v;
    v = prow[v];
  }
  return true;
}

// ROWS: walks of more than kWalkHops hops are left to query_rows_kernel.
template <typename T, bool ROWS>
__global__ void __launch_bounds__(128) query_kernel(QueryArgs a) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.nq) return;
  const int32_t s = a.src[q], t = a.dst[q];
  if (s < 0 || s >= a.n || t < 0 || t >= a.n) {
    atomicOr(a.status, kErrBadInput);
    a.out_len[q] = 0;
    return;
  }
  const int64_t row = (int64_t)a.ed2st[s] * a.n;  // row of s in the solve() layout
  const T d = static_cast<const T *>(a.dist)[row + t];
  static_cast<T *>(a.out_dist)[q] = d;
  if (!(d < Dist<T>::inf())) {
    a.out_len[q] = 0;
    return;
  }
  if (!walk_query(a, q, ROWS ? kWalkHops : a.n)) a.rest[atomicAdd(a.nrest, 1)] = q;
}

// The queries that query_kernel left, a CTA each.
__global__ void __launch_bounds__(kWalkThreads) query_rows_kernel(QueryArgs a) {
  extern __shared__ uint16_t walk_smem_raw[];
  uint16_t *const row = walk_smem_raw, *const verts = row + a.n;
  const int nrest = *a.nrest;
  for (int j = blockIdx.x; j < nrest; j += gridDim.x) {
    const int q = a.rest[j], s = a.src[q], t = a.dst[q];
    unsigned end;
    const int len = walk_row(a.pred + (int64_t)a.ed2st[s] * a.n, a.n, s, t, row, verts, end);
    const bool ok = end == (unsigned)s;
    if (threadIdx.x == 0) {
      if (!ok) atomicOr(a.status, kErrBadInput);  // broken chain: not predecessors of a solve
      a.out_len[q] = ok ? len : 0;
    }
    if (ok && a.out_path != nullptr && len <= a.max_len)
      for (int i = threadIdx.x; i < len; i += kWalkThreads)
        a.out_path[(int64_t)q * a.max_len + i] = verts[len - 1 - i];
    __syncthreads();  // (the row and the vertices are overwritten)
  }
}

}  // namespace

cudaError_t init_query_kernels() {
  return cudaFuncSetAttribute(query_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)walk_smem(kWalkMaxN));
}

bool queries_by_row(int32_t n, int32_t walks, bool paths) {
  return paths ? walks_by_row(n, walks, 30000, 400000000) : walks_by_row(n, walks, 2000, 15000000);
}

cudaError_t launch_query(bool f32, const QueryArgs &a, int sm_count, cudaStream_t st) {
  if (a.nq <= 0) return cudaSuccess;
  const unsigned blocks = (unsigned)((a.nq + 127) / 128);
  ++launch_count();
  if (a.nrest == nullptr) {
    if (f32) query_kernel<float, false><<<blocks, 128, 0, st>>>(a);
    else query_kernel<uint32_t, false><<<blocks, 128, 0, st>>>(a);
    return cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(a.nrest, 0, sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  if (f32) query_kernel<float, true><<<blocks, 128, 0, st>>>(a);
  else query_kernel<uint32_t, true><<<blocks, 128, 0, st>>>(a);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  ++launch_count();
  query_rows_kernel<<<walk_ctas(a.n, a.nq, sm_count), kWalkThreads, walk_smem(a.n), st>>>(a);
  return cudaGetLastError();
}

}  // namespace fapk
