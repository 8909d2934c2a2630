// mp_deep.cu -- min-plus products with any number of steps.
//
// Reference counterpart: the min-plus product with predecessors
// (min_plus_path_CPU_advanced, fap/kernel/minplus.h:51-65; GPU kernel
// MatrixMulCUDA6_path, fap/kernel/cuda/minplus.cu:32-189).
//
// C = A (x) B for the products that the strip kernel (minplus.cu) does not
// take: in a solve, parts of more than 48 boundary vertices (FP32 40); called
// directly, more than 40 steps or fewer than 6 million outputs; and leading
// dimensions of 2^24 and above, and int32 values outside the packed range.  Every
// add-min is an instruction on the integer pipe, so that pipe bounds the kernel,
// and what counts is how few other instructions it sees:
//
//  - Packed int32 (finite results below 2^24 - 1): one __viaddmin_u32 an
//    add-min on keys (d << 7) | idx, where idx counts within a chunk of 64
//    steps; after each chunk an output that improved notes its step and the
//    index is cleared, so that the value it holds wins ties again.
//  - FP32 and wide int32: steps in groups of four that keep the group of the
//    last strict improvement (fw_tile.cuh); after each chunk, while its
//    operands are still in shared memory, an improved output finds the step in
//    its group.  Only the step is kept; the predecessor is read once at the end.
//
// A CTA computes 64 x 64 outputs, 4 x 4 a thread, three CTAs an SM: small
// tiles leave few SMs idle in the last wave (1,000 x 4,000 outputs are 1,008
// tiles, 6.6 an SM).  A and B come in chunks of 64 steps, double-buffered with
// one barrier a chunk; both are read in 16-byte units, A along the steps and B
// along the columns, so no operand is transposed.  Row tiles of a column tile
// are neighbours, so B is read from memory once.  Keeping the predecessors'
// rows in shared memory for the last lookup measured the same as reading them
// from L2, and two or more groups of steps a turn as well.
//
// Measured against 128 x 128 tiles with 8 x 8 outputs a thread (one CTA an SM,
// one step at a time), a whole call with predecessors, its check and its copies
// included: 1,000 x 4,000 x 500 int32 (small values) 625 -> 219 us (the kernel
// 175 us: 11.4 T add-min/s of the 19.9 that the pipe does), FP32 550 -> 276 us;
// 2,000 x 20,000 x 110 int32 600 -> 476 us, FP32 1,096 -> 639 us, wide int32
// 1,220 -> 639 us; 877 x 57,301 x 19 wide int32 630 -> 406 us.  The integer pipe
// is 74 % busy in the packed form (with the add-mins alone 56 %), issue slots
// 74 % in FP32.

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "fw_tile.cuh"
#include "launch.h"
#include "mp_common.cuh"

namespace fapk {

namespace {

constexpr int kDeepTile = 64;     // rows and columns of a CTA
constexpr int kDeepK = 64;        // steps of a chunk (at most kMaxPackedK)
constexpr int kDeepThreads = 256;
constexpr int kDeepPitch = kDeepK + 4;  // of A's rows: 16-byte units, the rows of a warp in different banks

enum DeepForm { kDeepPacked, kDeepF32, kDeepWide };

struct DeepChunk {
  unsigned A[kDeepTile][kDeepPitch];
  unsigned B[kDeepK][kDeepTile];  // columns permuted by swz: lookups of different steps hit different banks
};

// Work counters as mp_strip_kernel's (minplus.cu).
__device__ unsigned long long g_deep_counters[3];

template <DeepForm FORM>
__device__ __forceinline__ unsigned deep_add(unsigned a, unsigned b) {
  return FORM == kDeepF32 ? __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b))) : a + b;
}

__device__ __forceinline__ unsigned word(const uint4 &v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }

// R rows of a matrix from `g` on (nrow of them inside), 64 columns (ncol inside),
// into shared memory, entry (r, c) at dst[r * PITCH + (c ^ SWZ(r))]; the rest is
// `fill`.  vec (all columns inside, 16-byte rows): a thread copies the unit t % 16
// of rows t / 16 + 16 i; else word t % 64 of rows t / 64 + 4 i.
template <int R, int PITCH, bool SWZ>
__device__ __forceinline__ void load_rows(unsigned *dst, const unsigned *g, int64_t ld, bool vec, int nrow, int ncol,
                                          unsigned fill) {
  const int t = threadIdx.x;
  if (vec) {
    const int r0 = t >> 4, c = (t & 15) * 4;
    g += r0 * ld + c;
    dst += r0 * PITCH;
#pragma unroll
    for (int i = 0; i < R / 16; i++, g += 16 * ld) {
      unsigned *d = dst + 16 * i * PITCH + (c ^ swz<SWZ>(r0 + 16 * i));
      if (r0 + 16 * i < nrow) cp_async16(d, g);
      else *reinterpret_cast<uint4 *>(d) = make_uint4(fill, fill, fill, fill);
    }
    return;
  }
  const int r0 = t >> 6, c = t & 63;
  if (c >= ncol) nrow = 0;
  g += r0 * ld + c;
  dst += r0 * PITCH;
#pragma unroll
  for (int i = 0; i < R / 4; i++, g += 4 * ld) {
    unsigned *d = dst + 4 * i * PITCH + (c ^ swz<SWZ>(4 * i));  // (the row's group of four is i)
    if (r0 + 4 * i < nrow) cp_async4(d, g);
    else *d = fill;
  }
}

template <DeepForm FORM, bool PRED>
__global__ void __launch_bounds__(kDeepThreads, 3)
    mp_deep_kernel(const MpSegment *__restrict__ segs, int nseg, int tile0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DeepChunk *const sm = reinterpret_cast<DeepChunk *>(smem_raw);
  __shared__ MpSegment s;
  using T = std::conditional_t<FORM == kDeepF32, float, uint32_t>;
  const int t = threadIdx.x, ty = t >> 4, tx = t & 15;
  const int tile = tile0 + blockIdx.x;
  if (t == 0) s = find_segment(segs, nseg, tile);
  __syncthreads();
  const unsigned INF = Dist<T>::bits(Dist<T>::inf());
  const int M = s.M, N = s.N, K = s.K;
  const int tiles_y = (M + kDeepTile - 1) / kDeepTile, local = tile - s.tile_begin;
  const int row0 = local % tiles_y * kDeepTile, col0 = local / tiles_y * kDeepTile;
  const unsigned *const Ag = static_cast<const unsigned *>(s.A) + (int64_t)row0 * s.lda;
  const unsigned *const Bg = static_cast<const unsigned *>(s.B) + col0;
  const int64_t lda = s.lda, ldb = s.ldb;
  const bool vec_a = (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(Ag) & 15) == 0;
  const bool vec_b = (ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(Bg) & 15) == 0 && col0 + kDeepTile <= N;

  // A chunk of A and B (outside the matrices: unreached).
  auto load = [&](int ch, int buf) {
    const int k0 = ch * kDeepK, kn = K - k0;
    load_rows<kDeepTile, kDeepPitch, false>(&sm[buf].A[0][0], Ag + k0, lda, vec_a && kn >= kDeepK, M - row0, kn, INF);
    load_rows<kDeepK, kDeepTile, true>(&sm[buf].B[0][0], Bg + k0 * ldb, ldb, vec_b, kn, N - col0, INF);
  };
  // Packed: the entries this thread copied become keys; whether it saw a finite one in B.
  auto to_keys = [&](int buf, int kn) {
    unsigned least = INF;
    auto key = [](unsigned v, unsigned idx) { return min(v, kPackH) * (1u << kIdxBits) + idx; };
    if (vec_a && kn >= kDeepK) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint4 *p = reinterpret_cast<uint4 *>(&sm[buf].A[ty + 16 * i][tx * 4]);
        const uint4 v = *p;
        *p = make_uint4(key(v.x, 0), key(v.y, 0), key(v.z, 0), key(v.w, 0));
      }
    } else {
#pragma unroll 4
      for (int r = t >> 6; r < kDeepTile; r += 4) sm[buf].A[r][t & 63] = key(sm[buf].A[r][t & 63], 0);
    }
    if (vec_b) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int k = ty + 16 * i;
        const unsigned idx = PRED ? k + 1 : 0;
        uint4 *p = reinterpret_cast<uint4 *>(&sm[buf].B[k][(tx * 4) ^ swz<true>(k)]);
        const uint4 v = *p;
        least = min(least, min(min(v.x, v.y), min(v.z, v.w)));
        *p = make_uint4(key(v.x, idx), key(v.y, idx), key(v.z, idx), key(v.w, idx));
      }
    } else {
#pragma unroll 4
      for (int k = t >> 6; k < kDeepK; k += 4) {
        unsigned *p = &sm[buf].B[k][(t & 63) ^ swz<true>(k)];
        least = min(least, *p);
        *p = key(*p, PRED ? k + 1 : 0);
      }
    }
    return least < kPackH;
  };

  unsigned acc[4][4];
  int arg[4][4];  // step + 1 of the last strict improvement, 0: none
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      acc[i][c] = FORM == kDeepPacked ? kPackH << kIdxBits : INF;
      arg[i][c] = 0;
    }
  const int nchunks = (K + kDeepK - 1) / kDeepK;
  int n_groups = 0;  // groups of four steps run
  if (nchunks > 0) load(0, 0);
  cp_async_commit();
  for (int ch = 0; ch < nchunks; ch++) {
    const int buf = ch & 1, k0 = ch * kDeepK;
    cp_async_wait_0();
    // the chunk is there; every thread is done with the last one
    bool work = true;
    if (FORM == kDeepPacked) work = __syncthreads_or(to_keys(buf, K - k0));
    else __syncthreads();
    if (ch + 1 < nchunks) load(ch + 1, buf ^ 1);
    cp_async_commit();
    if (!work) continue;  // columns that nothing reaches (unconnected parts)
    const int ng = (min(kDeepK, K - k0) + 3) >> 2;
    n_groups += ng;
#pragma unroll 1
    for (int g = 0; g < ng; g++) {
      uint4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const uint4 *>(&sm[buf].A[ty * 4 + i][g * 4]);
#pragma unroll
      for (int q = 0; q < 4; q++) b[q] = *reinterpret_cast<const uint4 *>(&sm[buf].B[g * 4 + q][(tx * 4) ^ swz<true>(g * 4)]);
      const int tag = k0 + g * 4 + 1;
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          if (FORM == kDeepPacked) {
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][c] = __viaddmin_u32(word(a[i], q), word(b[q], c), acc[i][c]);
          } else {
            const unsigned v0 = deep_add<FORM>(a[i].x, word(b[0], c)), v1 = deep_add<FORM>(a[i].y, word(b[1], c));
            const unsigned v2 = deep_add<FORM>(a[i].z, word(b[2], c)), v3 = deep_add<FORM>(a[i].w, word(b[3], c));
            const unsigned least = __vimin3_u32(acc[i][c], __vimin3_u32(v0, v1, v2), v3);
            if (PRED) arg[i][c] = least != acc[i][c] ? tag : arg[i][c];
            acc[i][c] = least;
          }
        }
    }
    if (PRED) {  // the steps of this chunk's improvements
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          if (FORM == kDeepPacked) {
            const int idx = acc[i][c] & kIdxMask;
            arg[i][c] = idx ? k0 + idx : arg[i][c];
            acc[i][c] -= idx;
          } else if (arg[i][c] > k0) {
            const int g = arg[i][c] - 1 - k0;
            const uint4 a = *reinterpret_cast<const uint4 *>(&sm[buf].A[ty * 4 + i][g]);
            const unsigned *b = &sm[buf].B[g][(tx * 4 + c) ^ swz<true>(g)];
            const unsigned v = acc[i][c];
            arg[i][c] += deep_add<FORM>(a.x, b[0]) == v              ? 0
                         : deep_add<FORM>(a.y, b[kDeepTile]) == v     ? 1
                         : deep_add<FORM>(a.z, b[2 * kDeepTile]) == v ? 2
                                                                      : 3;
          }
        }
    }
  }

  if (PRED) {  // steps -> predecessors
    const int32_t *const bp = s.Bp + col0 + tx * 4;
    const int64_t ldbp = s.ldbp;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int c = 0; c < 4; c++)
        arg[i][c] = arg[i][c] && col0 + tx * 4 + c < N ? bp[(arg[i][c] - 1) * ldbp + c] : -1;
  }

  if (t == 0) {
    atomicAdd(&g_deep_counters[0], 1ull);
    if (n_groups == 0) atomicAdd(&g_deep_counters[1], 1ull);
    atomicAdd(&g_deep_counters[2], (unsigned long long)n_groups * 4 * kDeepTile * kDeepTile);
  }

  const bool own = s.col_part != nullptr, full = col0 + kDeepTile <= N;  // (uniform over the CTA)
  const bool vec = vec_stores_ok<PRED>(s);
  const int col = col0 + tx * 4;
  unsigned *crow = static_cast<unsigned *>(s.C) + (int64_t)(row0 + ty * 4) * s.ldc + col;
  int32_t *prow = PRED ? s.Cp + (int64_t)(row0 + ty * 4) * s.ldcp + col : nullptr;
  const int64_t ldc = s.ldc, ldcp = s.ldcp;
#pragma unroll
  for (int i = 0; i < 4; i++, crow += ldc, prow += PRED ? ldcp : 0) {
    const int row = row0 + ty * 4 + i;
    unsigned d[4];
    int32_t p[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const unsigned v = FORM == kDeepPacked ? acc[i][c] >> kIdxBits : acc[i][c];
      d[c] = FORM == kDeepPacked && v >= kPackH ? INF : v;
      p[c] = arg[i][c];
    }
    if (own) {  // the part's own columns take the Floyd-Warshall values
#pragma unroll
      for (int c = 0; c < 4; c++) {
        int64_t j;
        if (row < M && col + c < N && fw_column(s, col + c, j)) {
          d[c] = static_cast<const unsigned *>(s.F)[(int64_t)row * s.ldf + j];
          if (PRED) p[c] = s.Fp[(int64_t)row * s.ldf + j];
        }
      }
    }
    if (full && vec) {  // streaming stores: the rows are not read again here
      if (row < M) {
        __stcs(reinterpret_cast<uint4 *>(crow), make_uint4(d[0], d[1], d[2], d[3]));
        if (PRED) __stcs(reinterpret_cast<int4 *>(prow), make_int4(p[0], p[1], p[2], p[3]));
      }
    } else if (full) {
      store_quad_unaligned(crow, d, tx, row < M);
      if (PRED) store_quad_unaligned(prow, p, tx, row < M);
    } else if (row < M) {
#pragma unroll
      for (int c = 0; c < 4; c++)
        if (col + c < N) {
          crow[c] = d[c];
          if (PRED) prow[c] = p[c];
        }
    }
  }
}

template <DeepForm FORM, bool PRED>
cudaError_t launch_deep_t(const MpSegment *d_segs, int nseg, int tiles, int tile0, cudaStream_t st) {
  mp_deep_kernel<FORM, PRED><<<tiles, kDeepThreads, 2 * sizeof(DeepChunk), st>>>(d_segs, nseg, tile0);
  return cudaGetLastError();
}

template <DeepForm FORM>
cudaError_t set_deep_attr() {
  cudaError_t e = cudaFuncSetAttribute(mp_deep_kernel<FORM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(2 * sizeof(DeepChunk)));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(mp_deep_kernel<FORM, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(2 * sizeof(DeepChunk)));
}

}  // namespace

int number_minplus_deep(MpSegment *segs, int nseg, int first) {
  for (int i = 0; i < nseg; i++) {
    segs[i].tile_begin = first;
    first += (segs[i].M + kDeepTile - 1) / kDeepTile * ((segs[i].N + kDeepTile - 1) / kDeepTile);
  }
  return first;
}

cudaError_t launch_minplus_deep(bool f32, bool packed, bool pred, const MpSegment *d_segs, int nseg, int tiles,
                                int tile0, cudaStream_t st) {
  if (tiles <= 0 || nseg <= 0) return cudaSuccess;
  ++launch_count();
  if (f32) return pred ? launch_deep_t<kDeepF32, true>(d_segs, nseg, tiles, tile0, st)
                       : launch_deep_t<kDeepF32, false>(d_segs, nseg, tiles, tile0, st);
  if (packed) return pred ? launch_deep_t<kDeepPacked, true>(d_segs, nseg, tiles, tile0, st)
                          : launch_deep_t<kDeepPacked, false>(d_segs, nseg, tiles, tile0, st);
  return pred ? launch_deep_t<kDeepWide, true>(d_segs, nseg, tiles, tile0, st)
              : launch_deep_t<kDeepWide, false>(d_segs, nseg, tiles, tile0, st);
}

cudaError_t deep_counters(unsigned long long out[3], bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_deep_counters, sizeof(unsigned long long) * 3);
  if (e != cudaSuccess || !reset) return e;
  const unsigned long long zero[3] = {0, 0, 0};
  return cudaMemcpyToSymbol(g_deep_counters, zero, sizeof(zero));
}

cudaError_t init_mp_deep_kernels() {
  static_assert(kDeepK <= kMaxPackedK, "a chunk's steps fit the packed index");
  cudaError_t e;
  if ((e = set_deep_attr<kDeepPacked>()) != cudaSuccess) return e;
  if ((e = set_deep_attr<kDeepF32>()) != cudaSuccess) return e;
  return set_deep_attr<kDeepWide>();
}

}  // namespace fapk
