// dgemm_frag.cuh — the FP64 MMA and the shared-memory fragment orders of the
// TMA-staged FP64 kernels (dev_dgemm.cu, dev_kbuild.cu; the layouts are
// described in dev_dgemm.cu), and the tensor maps of their operands.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "tma_util.cuh"

namespace ecg {
namespace dev {
namespace dfrag {

constexpr int DK = 16;  // k depth of a stage: 16 doubles, one 128-byte swizzle row

__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Row (within a 16-row block) that lane group g reads in MMA s of an i-fast
// operand.
__device__ __forceinline__ int jmap(int g, int s) {
  return (g & 1) + 8 * ((g >> 1) & 1) + 2 * (g >> 2) + 4 * s;
}
// Row (within an 8-row block) that lane group g reads of a k-fast operand.
__device__ __forceinline__ int pmap(int g) { return 2 * (g & 3) + (g >> 2); }

// Per-lane fragment offsets (doubles, within one stage's tile) of an operand
// whose warp sub-tile starts at row w0 and has NB 8-row blocks.  k-fast:
// o[q] for k-step kb = 4q, block rb at o[q] + 128 rb.  i-fast:
// o[2 (rb & 1) + (q & 1)] + 256 (rb >> 1) + 64 q.
template <bool KF, int NB>
struct FragOff {
  static constexpr int N = 4;
  uint32_t o[N];
  __device__ __forceinline__ FragOff(int w0, int g, int t) {
    if constexpr (KF) {
      const int p = pmap(g);
      const uint32_t rowbase = (uint32_t)((w0 + p) * 16 + (t & 1));
      const int y = (t >> 1) ^ p;
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = rowbase + (uint32_t)((4 * q) ^ (y << 1));
    } else {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int j = jmap(g, s);
        const uint32_t base =
            (uint32_t)((w0 >> 4) * 256 + t * 16 + (j & 1) + (((j >> 1) ^ t) << 1));
        o[2 * s] = base;
        o[2 * s + 1] = base ^ 8u;
      }
    }
  }
  __device__ __forceinline__ uint32_t at(int rb, int q) const {
    if constexpr (KF)
      return o[q] + 128u * rb;
    else
      return o[2 * (rb & 1) + (q & 1)] + 256u * (rb >> 1) + 64u * q;
  }
};

// Row (or column) of the tile that accumulator row g of block rb stands for.
template <bool KF>
__device__ __forceinline__ int frag_row(int w0, int rb, int g) {
  if constexpr (KF)
    return w0 + 8 * rb + pmap(g);
  else
    return w0 + 16 * (rb >> 1) + jmap(g, rb & 1);
}

// 3-D map over a double operand: inner extent d0 (unit stride), d1 rows
// s1 doubles apart, d2 batch items s2 doubles apart; box (16, b1, 1),
// 128-byte swizzle, out-of-range elements read as zero.
inline int dmap(CUtensorMap* m, const double* base, int64_t d0, int64_t d1, int64_t s1,
                int64_t d2, int64_t s2, int b1) {
  EncodeFn enc = nullptr;
  if (int e = encode_fn(&enc)) return e;
  cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
  cuuint64_t strides[2] = {(cuuint64_t)(s1 * 8), (cuuint64_t)(s2 * 8)};
  cuuint32_t box[3] = {(cuuint32_t)DK, (cuuint32_t)b1, 1};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(base), dims,
                   strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

// a stride (doubles) TMA accepts: a positive multiple of 16 bytes below 2^40 bytes
inline bool stride_ok(int64_t s) { return s > 0 && s % 2 == 0 && s < ((int64_t)1 << 37); }

}  // namespace dfrag
}  // namespace dev
}  // namespace ecg
