// umma.cuh — tcgen05 helpers shared by the split-BF16 kernels (dev_tc.cu,
// dev_tckbuild.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "tma_util.cuh"

namespace ecg {
namespace dev {
namespace umma_ops {

using tma::smem_u32;

// slice pairs (a, b): hi*hi, hi*mid, mid*hi, mid*mid, hi*lo, lo*hi (the first
// three for two slices)
__host__ __device__ constexpr int pair_a(int p) { return p == 2 || p == 3 ? 1 : p == 5 ? 2 : 0; }
__host__ __device__ constexpr int pair_b(int p) { return p == 1 || p == 3 ? 1 : p == 4 ? 2 : 0; }

// UMMA shared-memory descriptor, K-major operand in the 128-byte-swizzled
// canonical layout: 128-byte rows, 8-row (1024-byte) groups.
__device__ __forceinline__ uint64_t umma_desc(const void* p) {
  const uint32_t a = smem_u32(p);
  uint64_t d = (uint64_t)((a & 0x3FFFF) >> 4);  // start address
  d |= (uint64_t)1 << 16;                        // leading byte offset (unused for SW128 K-major)
  d |= (uint64_t)(1024 >> 4) << 32;              // stride byte offset: 8-row group
  d |= (uint64_t)1 << 46;                        // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                        // layout: SWIZZLE_128B
  return d;
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                     uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
          smem_u32(bar)));
}

// 16 columns of this lane's tensor-memory row, from column address `addr`.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
      "%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::);
}

}  // namespace umma_ops
}  // namespace dev
}  // namespace ecg
