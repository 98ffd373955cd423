// dev_tckbuild.cu — the (T) K builds in mixed precision on the sm_100a tensor
// cores (tcgen05 + TMA): for each item z of a batch of occupied triplets
//
//   C_z(r, c) = beta C_z(r, c) + sum_s sum_k A_s[r, k; a_s(z)] B_s[c, k; b_s(z)]
//
// in FP32, with operands split into two BF16 slices (products hi*hi, hi*lo,
// lo*hi accumulated in FP32, ~2^-16 relative), four K segments (the vvvo and
// ovoo products that share an index map into K).  Rows run over the v^2 side.
//
// Persistent, one CTA per SM, 128 x tn tiles: a TMA warp fills a ring of
// stages, one thread issues the MMAs into one of two tensor-memory
// accumulators, eight warps drain the other and update K.
//
// What bounds it: the MMAs and what their one issuing thread does between them
// (a k-block is 12 MMAs of some 100 cycles), then the K traffic (five passes of
// 4 v^3 bytes a triplet).  Hence:
//  * One launch takes all triplets of a batch and all four K segments.
//  * tn covers v in whole tiles of any multiple of 16 columns (kt_width): one of
//    224 at v = 209, where 128-column tiles pad by 22%.
//  * The segment of a k-block is found by selects (seg_at).
//  * The epilogue is a rolled loop over 16-column chunks that fetches the next
//    chunk of K ahead: unrolled over a tile, with all of K's values fetched
//    before the accumulator was waited for, it was slower (v = 129 6.2 against
//    5.4 ms), the issuing thread sharing the instruction cache with it.
//  * One lane a warp polls the accumulator's barrier.
// Measured, the three launches of the largest batch (seven batched GEMMs of fixed
// tiles took 9.0, 13.7 and 14.1 ms): v = 129 5.4 ms, v = 209 12.0, v = 318 12.9 (33
// triplets, 1000 TFLOP/s; at v = 200 the tensor pipe is 39 to 45% active, L2 42 to
// 49%, DRAM 23 to 40%).  Not kept: 32-deep k-blocks in five stages
// and stages of one slice (more loads of less; 3 to 13% slower), L2 prefetch of
// the next tile's rows (10 to 30% slower), 256-row tiles on CTA pairs
// (cta_group::2; v = 318 15.3 ms, v = 129 6.7).
//
// Every mbarrier wait is bounded; on time-out the kernel records a code, lets
// its own loads and MMAs in flight finish (bounded), frees its tensor memory
// and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "ecg_dev.h"
#include "tma_util.cuh"
#include "umma.cuh"

namespace ecg {
namespace dev {

namespace {

using namespace tma;
using namespace umma_ops;

constexpr int TM = 128, TK = 64, NSL = 2, NPAIR = 3;
constexpr int A_BYTES = TM * TK * 2;  // one slice
constexpr int RING_BYTES = 216 * 1024;
constexpr int KT_SMEM = RING_BYTES + 1024 /*barriers*/ + 1024 /*align*/;
constexpr int MAX_STAGES = 8;
constexpr int EPI_WARPS = 8;  // two per lane quarter, alternate 16-column chunks
constexpr int KT_THREADS = 32 * (2 + EPI_WARPS);
constexpr uint32_t TMEM_COLS = 512, ACC_STRIDE = 256;

struct KtMaps {
  CUtensorMap a[KB_MAX_SEG], b[KB_MAX_SEG];
};
// Segment s covers the k-blocks [end[s-1], end[s]); its last k-block issues
// kk_last[s] of the TK/16 MMA steps (the rest of it is zero padding).
struct KtSegs {
  int end[KB_MAX_SEG], kk_last[KB_MAX_SEG];
};
struct KtOut {
  float* C;
  int m, n;
  int64_t scm, scm2, scn;
  int dm, beta, vec;  // vec: scn == 1 and rows on 16 bytes: float4 columns
};
struct KtTiles {
  int mt, nt, items, chunk, tn;
};

struct KtPos {
  int mt, nt, z;
};
__device__ __forceinline__ KtPos kt_pos(const KtTiles& t, uint32_t it) {
  const uint32_t per = (uint32_t)t.mt * t.nt;
  const uint32_t c = it / (per * t.chunk);
  const uint32_t zn = min((uint32_t)t.chunk, (uint32_t)t.items - c * t.chunk);
  const uint32_t r = it - c * per * t.chunk, row = r / (zn * t.nt), q = r - row * zn * t.nt;
  const uint32_t zi = q / t.nt;
  return KtPos{(int)row, (int)(q - zi * t.nt), (int)(c * t.chunk + zi)};
}

// Segment of k-block kb: index, first k-block, MMA steps to issue.  Selects only:
// an indexed read of a parameter goes through local memory, whose lines the
// epilogue's traffic evicts, and had cost the issuing thread a third of its time
// (650 cycles a k-block; v = 318 15.4 -> 12.9 ms).
struct SegPos {
  int s, start, steps;
};
__device__ __forceinline__ SegPos seg_at(const KtSegs& g, int kb) {
  SegPos p{0, 0, kb == g.end[0] - 1 ? g.kk_last[0] : TK / 16};
#pragma unroll
  for (int t = 1; t < KB_MAX_SEG; ++t)
    if (kb >= g.end[t - 1])
      p = SegPos{t, g.end[t - 1], kb == g.end[t] - 1 ? g.kk_last[t] : TK / 16};
  return p;
}

__global__ void __launch_bounds__(KT_THREADS, 1)
    tc_kbuild_kernel(const __grid_constant__ KtMaps maps, const KtOut out, const KtSegs segs,
                     const KtTiles tiles, const KbItem* __restrict__ items,
                     unsigned long long wait_ns, int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tn = tiles.tn, b_bytes = tn * TK * 2, stage_bytes = NSL * (A_BYTES + b_bytes);
  const int stages = min(RING_BYTES / stage_bytes, MAX_STAGES);
  uint64_t* full = (uint64_t*)(smem + RING_BYTES);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;  // [2] accumulator ready
  uint64_t* tempty = tfull + 2;          // [2] accumulator drained
  uint32_t* tmem_slot = (uint32_t*)(tempty + 2);
  int* abort_flag = (int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t total = (uint32_t)tiles.mt * tiles.nt * tiles.items;
  const int nk = segs.end[KB_MAX_SEG - 1];

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    asm volatile("fence.proxy.async.shared::cta;\n" ::);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0, issued = 0;
      uint32_t ph = 0;  // phase of the ring's current round
      for (uint32_t it = blockIdx.x; it < total && !*(volatile int*)abort_flag;
           it += gridDim.x) {
        const KtPos p = kt_pos(tiles, it);
        const KbItem item = items[p.z];
        for (int kb = 0; kb < nk; ++kb) {
          const SegPos sp = seg_at(segs, kb);
          if (issued >= stages && !mbar_wait(&empty[s], ph ^ 1u, wait_ns)) {
            *(volatile int*)err = 65;
            atomicExch(abort_flag, 1);
            break;
          }
          int ia = item.a[0], ib = item.b[0];
#pragma unroll
          for (int t = 1; t < KB_MAX_SEG; ++t)
            if (sp.s == t) {
              ia = item.a[t];
              ib = item.b[t];
            }
          uint8_t* st = smem + s * stage_bytes;
          const int kx = (kb - sp.start) * TK;
          mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
#pragma unroll
          for (int t = 0; t < NSL; ++t) {
            tma_load_4d(st + t * A_BYTES, &maps.a[sp.s], &full[s], kx, p.mt * TM, t, ia);
            tma_load_4d(st + NSL * A_BYTES + t * b_bytes, &maps.b[sp.s], &full[s], kx, p.nt * tn, t,
                        ib);
          }
          if (issued < stages) ++issued;
          if (++s == stages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      // drain: every issued load must land before the CTA can exit
      for (int q = 0; q < issued; ++q) {
        if (--s < 0) {
          s = stages - 1;
          ph ^= 1u;
        }
        mbar_wait(&full[s], ph);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // kind::f16, A/B BF16, D F32, both K-major, M = 128, N = tn
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tn >> 3) << 17) |
                             ((uint32_t)(TM >> 4) << 24);
      int s = 0, last = -1;
      uint32_t ph = 0;
      int lt = 0;
      for (uint32_t it = blockIdx.x; it < total && !*(volatile int*)abort_flag;
           it += gridDim.x, ++lt) {
        const int acc = lt & 1, ua = lt >> 1;
        if (ua > 0 && !mbar_wait(&tempty[acc], (uint32_t)((ua - 1) & 1), wait_ns)) {
          *(volatile int*)err = 68;
          atomicExch(abort_flag, 1);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
        const uint32_t dcol = tmem + (uint32_t)acc * ACC_STRIDE;
        bool ok = true;
        for (int kb = 0; kb < nk; ++kb) {
          if (!mbar_wait(&full[s], ph, wait_ns)) {
            *(volatile int*)err = 66;
            atomicExch(abort_flag, 1);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
          const uint8_t* As = smem + s * stage_bytes;
          const uint8_t* Bs = As + NSL * A_BYTES;
          const int nkk = seg_at(segs, kb).steps;
#pragma unroll
          for (int p = 0; p < NPAIR; ++p) {
            const uint64_t da = umma_desc(As + pair_a(p) * A_BYTES);
            const uint64_t db = umma_desc(Bs + pair_b(p) * b_bytes);
#pragma unroll
            for (int kk = 0; kk < TK / 16; ++kk)
              if (kk < nkk)
                umma(dcol, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), idesc,
                     (kb > 0 || p > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(&empty[s]);
          if (++s == stages) {
            s = 0;
            ph ^= 1u;
          }
        }
        umma_commit(&tfull[acc]);
        last = lt;
        if (!ok) break;
      }
      // the MMAs in flight must finish before the accumulators are freed
      if (last >= 0) mbar_wait(&tfull[last & 1], (uint32_t)((last >> 1) & 1));
    }
  } else {
    const int q = warp & 3, hw = (warp - 2) >> 2;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const int nch = tn / 16;
    int lt = 0;
    for (uint32_t it = blockIdx.x; it < total; it += gridDim.x, ++lt) {
      const KtPos p = kt_pos(tiles, it);
      const int acc = lt & 1;
      const int row = p.mt * TM + q * 32 + lane;
      float* C = out.C + items[p.z].c;
      if (out.dm > 0) {
        const int rq = row / out.dm;
        C += (row - rq * out.dm) * out.scm + rq * out.scm2;
      } else {
        C += row * out.scm;
      }
      const int c0 = p.nt * tn + hw * 16;  // first column of this warp's first chunk
      const bool row_ok = row < out.m;
      // chunk c of the tile: columns 16 c ..; this warp takes every other one and
      // fetches the next chunk's values of K before it updates the current one's
      float old[16], nxt[16];
      auto fetch = [&](int c, float (&x)[16]) {
        const int col = p.nt * tn + c * 16, left = (row_ok && c < nch) ? out.n - col : 0;
        const float* Cc = C + col * out.scn;
        if (out.vec) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (j < left) {
              const float4 y = *reinterpret_cast<const float4*>(Cc + j);
              x[j] = y.x;
              x[j + 1] = y.y;
              x[j + 2] = y.z;
              x[j + 3] = y.w;
            }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < left) x[j] = Cc[j * out.scn];
        }
      };
      if (out.beta) fetch(hw, nxt);
      // one lane polls; the warp goes on only if it saw the accumulator ready and no
      // time-out was recorded, so the warp-wide tcgen05.ld below always runs converged
      const bool ready =
          lane != 0 || mbar_wait(&tfull[acc], (uint32_t)((lt >> 1) & 1), wait_ns);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) {
          *(volatile int*)err = 67;
          atomicExch(abort_flag, 1);
        }
        break;
      }
      if (__any_sync(0xffffffffu, *(volatile int*)abort_flag != 0)) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
#pragma unroll 1
      for (int c = hw; c < nch; c += 2) {
#pragma unroll
        for (int j = 0; j < 16; ++j) old[j] = out.beta ? nxt[j] : 0.f;
        if (out.beta) fetch(c + 2, nxt);
        uint32_t r[16];
        tmem_ld16(tmem + lane_base + (uint32_t)acc * ACC_STRIDE + (uint32_t)(c * 16), r);
        const int col = p.nt * tn + c * 16, left = row_ok ? out.n - col : 0;
        float* Cc = C + col * out.scn;
        if (out.vec) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (j < left)
              *reinterpret_cast<float4*>(Cc + j) = make_float4(
                  __uint_as_float(r[j]) + old[j], __uint_as_float(r[j + 1]) + old[j + 1],
                  __uint_as_float(r[j + 2]) + old[j + 2], __uint_as_float(r[j + 3]) + old[j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < left) Cc[j * out.scn] = __uint_as_float(r[j]) + old[j];
        }
        __syncwarp();  // the next tcgen05.ld wants the whole warp
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "r"(TMEM_COLS));
  }
}

// 4-D map over a stack of split operands: k, row, slice, item; boxes of 64 k and
// box_rows rows, 128-byte swizzle, rows past the operand's read as zero.
int kt_map(EncodeFn enc, CUtensorMap* m, const TcStack& o, int box_rows) {
  const int64_t rp = tc_pad_rows(o.rows), kp = tc_pad_k(o.k);
  cuuint64_t dims[4] = {(cuuint64_t)kp, (cuuint64_t)rp, (cuuint64_t)NSL, (cuuint64_t)o.items};
  cuuint64_t strides[3] = {(cuuint64_t)(kp * 2), (cuuint64_t)(rp * kp * 2),
                           (cuuint64_t)(NSL * rp * kp * 2)};
  cuuint32_t box[4] = {(cuuint32_t)TK, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(o.base), dims,
                   strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

// Tile width for n columns: the fewest tiles of at most 256 columns, each the
// smallest multiple of 16 that covers its share.
int kt_width(int64_t n) {
  const int64_t nt = (n + 255) / 256;
  return (int)(((n + nt - 1) / nt + 15) / 16 * 16);
}

}  // namespace

int tc_kbuild(stream_t s, const TcKbuild& g, int nitems, const KbItem* items, int chunk) {
  if (nitems <= 0) return 0;
  const int64_t lim = (int64_t)1 << 30;
  if (g.nseg < 1 || g.nseg > KB_MAX_SEG || g.m <= 0 || g.n <= 0 || g.m >= lim || g.n >= lim ||
      !g.C || !items || chunk < 1)
    return (int)cudaErrorInvalidValue;
  EncodeFn enc = nullptr;
  if (int e = encode_fn(&enc)) return e;
  const int tn = kt_width(g.n);
  const KtTiles tiles{(int)((g.m + TM - 1) / TM), (int)((g.n + tn - 1) / tn), nitems, chunk, tn};
  const int64_t total = (int64_t)tiles.mt * tiles.nt * nitems;
  if (total >= ((int64_t)1 << 31) || (int64_t)tiles.mt * tiles.nt * chunk >= ((int64_t)1 << 31))
    return (int)cudaErrorInvalidConfiguration;
  KtMaps maps;
  KtSegs segs;
  int end = 0;
  double depth = 0.0;
  for (int q = 0; q < KB_MAX_SEG; ++q) {
    const int u = q < g.nseg ? q : 0;
    if (g.A[u].rows < g.m || g.B[u].rows < g.n || g.A[u].k != g.B[u].k || g.A[u].k <= 0 ||
        ((uintptr_t)g.A[u].base & 15) || ((uintptr_t)g.B[u].base & 15))
      return (int)cudaErrorInvalidValue;
    if (int e = kt_map(enc, &maps.a[q], g.A[u], TM)) return e;
    if (int e = kt_map(enc, &maps.b[q], g.B[u], tn)) return e;
    segs.kk_last[q] = TK / 16;
    if (q < g.nseg) {
      const int64_t k = g.A[q].k, kp = (k + TK - 1) / TK * TK;
      end += (int)(kp / TK);
      segs.kk_last[q] = (int)((k - (kp - TK) + 15) / 16);
      depth += (double)(kp - TK) + 16.0 * segs.kk_last[q];
    }
    segs.end[q] = end;
  }
  // whole float4 columns may run into the pitch's padding
  const bool vec = g.scn == 1 && g.pad4 && g.scm % 4 == 0 && g.scm2 % 4 == 0 &&
                   ((uintptr_t)g.C & 15) == 0;
  const KtOut out{g.C, (int)g.m, (int)g.n, g.scm, g.scm2, g.scn, (int)g.dm, g.beta ? 1 : 0,
                  vec ? 1 : 0};
  // cudaFuncSetAttribute acts on the current device only: one flag per device
  static std::atomic<bool> done[128] = {};
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess) cudaGetLastError();
  if (d < 0 || d >= 128 || !done[d].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(
        tc_kbuild_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KT_SMEM);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return (int)e;
    }
    if (d >= 0 && d < 128) done[d].store(true, std::memory_order_release);
  }
  cudaStream_t st = (cudaStream_t)s;
  const uint64_t w = tc_wait(s);
  int* err = wait_error(s, WAIT_TCKBUILD);
  if (!err) return (int)cudaErrorMemoryAllocation;
  const int slot = ktime_begin(s, KT_TCGEMM);
  tc_kbuild_kernel<<<(unsigned)std::min<int64_t>(total, 148), KT_THREADS, KT_SMEM, st>>>(
      maps, out, segs, tiles, items, w ? (unsigned long long)w : WAIT_NS, err);
  note_launches(1);
  ktime_end(s, KT_TCGEMM, slot, 2.0 * (double)g.m * (double)g.n * depth * NPAIR * nitems);
  return (int)cudaGetLastError();
}

}  // namespace dev
}  // namespace ecg
