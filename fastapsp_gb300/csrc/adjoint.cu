// adjoint.cu -- reverse-mode derivative of shortest-path distances with
// respect to edge weights (no counterpart in the reference).
//
// A shortest-path distance is the sum of the weights along the chosen path,
// so dD[s][t]/dw_e is 1 for every edge on that path and 0 elsewhere (away from
// ties).  Given upstream gradients g for a list of (s, t) pairs, the adjoint
// walks the predecessor path t <- pred[s][t] <- ... <- s recorded by the
// forward pass and adds g to the gradient of each edge it crosses.  One thread
// walks one pair; the walk is capped at the vertex count and flags an error
// instead of looping if the predecessors do not lead back to s.  In the graph
// form, walks of more than a few hops get a CTA each (path_walk.cuh), whose
// threads look up the edges of all hops at once: 10,000 pairs with paths of 101
// vertices on average on a 4,096-vertex road graph, kernels 112 us, 238 us with
// every hop's edge looked up on the way.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "kernels.cuh"
#include "launch.h"
#include "path_walk.cuh"

namespace fapk {

namespace {

// Graph form: pred rows in solve() layout (row of vertex s = ed2st[s]).  Adds gi
// to the gradient of the edge u -> v, the lightest CSR entry u -> v (the one a
// shortest path uses), first in CSR order on equal weights; false: there is none.
__device__ __forceinline__ bool add_edge(const BackwardArgs &a, int u, int v, float gi) {
  int best = -1;
  float bw = 0.0f;
  for (int e = a.ro[u]; e < a.ro[u + 1]; e++)
    if (a.col[e] == v && (best < 0 || a.w[e] < bw)) {
      best = e;
      bw = a.w[e];
    }
  if (best < 0) {
    atomicOr(a.status, kErrBadInput);
    return false;
  }
  atomicAdd(&a.dw[best], gi);
  return true;
}

__global__ void backward_graph_kernel(BackwardArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.npairs) return;
  const int src = a.s[i], dst = a.t[i];
  if (src < 0 || src >= a.n || dst < 0 || dst >= a.n) {
    atomicOr(a.status, kErrBadInput);
    return;
  }
  const int32_t *prow = a.pred + (int64_t)a.ed2st[src] * a.n;
  if (a.nrest != nullptr) {  // longer walks: backward_rows_kernel
    int v = dst, hops = 0;
    while (v != src && hops <= kWalkHops) {
      v = prow[v];
      if (v < 0 || v >= a.n) break;
      hops++;
    }
    if (hops > kWalkHops) {
      a.rest[atomicAdd(a.nrest, 1)] = i;
      return;
    }
  }
  const float gi = a.g[i];
  int v = dst;
  for (int steps = 0; v != src; steps++) {
    const int u = prow[v];
    if (u < 0) return;  // unreached: zero gradient
    if (u >= a.n || steps >= a.n) {
      atomicOr(a.status, kErrBadInput);
      return;
    }
    if (!add_edge(a, u, v, gi)) return;
    v = u;
  }
}

// The pairs that backward_graph_kernel left, a CTA each.
__global__ void __launch_bounds__(kWalkThreads) backward_rows_kernel(BackwardArgs a) {
  extern __shared__ uint16_t walk_smem_raw[];
  uint16_t *const row = walk_smem_raw, *const verts = row + a.n;
  const int nrest = *a.nrest;
  for (int j = blockIdx.x; j < nrest; j += gridDim.x) {
    const int i = a.rest[j], src = a.s[i];
    const float gi = a.g[i];
    unsigned end;
    const int len = walk_row(a.pred + (int64_t)a.ed2st[src] * a.n, a.n, src, a.t[i], row, verts, end);
    if (threadIdx.x == 0 && end == kWalkBad) atomicOr(a.status, kErrBadInput);
    for (int h = threadIdx.x; h + 1 < len; h += kWalkThreads) add_edge(a, verts[h + 1], verts[h], gi);
    __syncthreads();  // (the row and the vertices are overwritten)
  }
}

// Dense form: instance b's predecessor matrix P_b (size_b x size_b, leading
// dimension ld_b); the gradient is the dense matrix dW_b (same shape).
struct DenseInst {
  const int32_t *P;
  float *dW;
  int64_t ld;
  int32_t size;
};

__global__ void backward_dense_kernel(const DenseInst *__restrict__ inst, int32_t ninst,
                                      int32_t npairs, const int32_t *__restrict__ b,
                                      const int32_t *__restrict__ s, const int32_t *__restrict__ t,
                                      const float *__restrict__ g, unsigned *status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npairs) return;
  const int bi = b[i];
  if (bi < 0 || bi >= ninst) {
    atomicOr(status, kErrBadInput);
    return;
  }
  const DenseInst I = inst[bi];
  const int src = s[i], dst = t[i];
  if (src < 0 || src >= I.size || dst < 0 || dst >= I.size) {
    atomicOr(status, kErrBadInput);
    return;
  }
  const float gi = g[i];
  const int32_t *prow = I.P + (int64_t)src * I.ld;
  int v = dst;
  for (int steps = 0; v != src; steps++) {
    const int u = prow[v];
    if (u < 0) return;
    if (u >= I.size || steps >= I.size) {
      atomicOr(status, kErrBadInput);
      return;
    }
    atomicAdd(&I.dW[(int64_t)u * I.ld + v], gi);
    v = u;
  }
}

}  // namespace

bool pairs_by_row(int32_t n, int32_t walks) {
  return walks_by_row(n, walks, std::min<int64_t>(12500, 8 * (int64_t)n), 100000000);
}

cudaError_t init_backward_kernels() {
  return cudaFuncSetAttribute(backward_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)walk_smem(kWalkMaxN));
}

cudaError_t launch_backward_graph(const BackwardArgs &a, int sm_count, cudaStream_t st) {
  if (a.npairs <= 0) return cudaSuccess;
  if (a.nrest != nullptr) {
    cudaError_t e = cudaMemsetAsync(a.nrest, 0, sizeof(int32_t), st);
    if (e != cudaSuccess) return e;
  }
  backward_graph_kernel<<<(a.npairs + 255) / 256, 256, 0, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || a.nrest == nullptr) return e;
  backward_rows_kernel<<<walk_ctas(a.n, a.npairs, sm_count), kWalkThreads, walk_smem(a.n), st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_backward_dense(const void *inst, int32_t ninst, int32_t npairs,
                                  const int32_t *b, const int32_t *s, const int32_t *t,
                                  const float *g, unsigned *status, cudaStream_t st) {
  if (npairs <= 0) return cudaSuccess;
  backward_dense_kernel<<<(npairs + 255) / 256, 256, 0, st>>>(
      static_cast<const DenseInst *>(inst), ninst, npairs, b, s, t, g, status);
  return cudaGetLastError();
}

size_t dense_inst_bytes() { return sizeof(DenseInst); }

void fill_dense_inst(void *dst, const int32_t *P, float *dW, int64_t ld, int32_t size) {
  DenseInst *d = static_cast<DenseInst *>(dst);
  d->P = P;
  d->dW = dW;
  d->ld = ld;
  d->size = size;
}

}  // namespace fapk
