// dev_dgemm.cu — FP64 GEMM with TMA-staged operands (sm_100a).
//
// C(m,n) = alpha * A(m,k) B(k,n) + beta * C with unit row stride in C,
// batched (3-D tensor maps, one batch item per grid z) or split over
// K (grid z = K slice, partial products into the stream's split-K buffer,
// summed in a fixed order by splitk_reduce).  tcgen05 has no FP64 kind, so the
// products run on the FP64 MMA pipe (mma.sync m8n8k4 f64).  What the Tensor
// Memory Accelerator takes over is the operand staging: a producer warp issues
// the TMA copies of a 16-deep k-slab of the A and B tiles into a ring of STAGES
// shared-memory stages (128-byte swizzle, mbarrier completion), so the MMA
// warps spend no instructions on address arithmetic or copies, and each warp
// releases a stage through an `empty` mbarrier instead of a block barrier
// (once the MMAs that read it have been issued: see the main loop).
//
// Shared layouts (doubles; rows of 128 bytes whose 16-byte chunks are XOR-
// swizzled with the row index mod 8, as TMA's 128-byte swizzle writes them):
//  * operand contiguous along k ("k-fast"): [row][k 0..15], one box per stage
//  * operand contiguous along its row index ("i-fast"): [row/16][k 0..15]
//    [row%16], one 16 x 16 box per 16 rows
// An MMA may take its 8 rows (columns) and its 4 k in any order, provided the
// epilogue writes each accumulator to the row and column it stands for.  The
// orders below make every half-warp's fragment reads hit 16 distinct 8-byte
// bank pairs under the swizzle (lane group g = lane/4, t = lane%4, k = kb + t):
//  * k-fast: row 2(g%4) + g/4 of an 8-row block
//  * i-fast: MMA s in {0,1} of a 16-row block reads row
//            (g&1) + 8((g>>1)&1) + 2(g>>2) + 4s
//
// Every mbarrier wait is bounded (the stream's tensor-core bound, default
// 1 s): on time-out the kernel records an error code (read by tc_error),
// waits (bounded) for its own copies in flight and returns without writing C.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>

#include "ecg_dev.h"
#include "dgemm_frag.cuh"
#include "tma_util.cuh"

namespace ecg {
namespace dev {

namespace {

using namespace tma;
using namespace dfrag;

template <int BM, int BN, int WM, int WN, int STAGES>
struct DCfg {
  static constexpr int WARPS_M = BM / WM;
  static constexpr int WARPS = (BM / WM) * (BN / WN);
  static constexpr int THREADS = WARPS * 32 + 32;  // and the producer warp
  static constexpr int A_BYTES = BM * DK * 8;
  static constexpr int B_BYTES = BN * DK * 8;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 2 * STAGES * 8;
  static_assert(BM % WM == 0 && BN % WN == 0 && WM % 16 == 0 && WN % 16 == 0, "tile shape");
  static_assert(A_BYTES % 1024 == 0 && B_BYTES % 1024 == 0, "swizzled tiles start on 1024 bytes");
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

struct DOut {
  // element (i, j) of grid-z item z at C + z*scb + i + j*scn
  double* C;
  int64_t m, n, scn, scb;
  double alpha, beta;
  int tri = 0;  // > 0: blocks whose elements all have j / tri < i / tri do nothing
};

template <int BM, int BN, int WM, int WN, int STAGES, int MINB, bool AKF, bool BKF>
__global__ void __launch_bounds__(DCfg<BM, BN, WM, WN, STAGES>::THREADS, MINB)
    dgemm_tma_kernel(const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                     DOut out, int64_t k, int64_t kslice, int split,
                     unsigned long long wait_ns, int* err) {
  using Cfg = DCfg<BM, BN, WM, WN, STAGES>;
  constexpr int MT = WM / 8, NTL = WN / 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + STAGES;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int z = blockIdx.z;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  if (out.tri > 0 && (n0 + BN - 1) / out.tri < m0 / out.tri) return;
  const int64_t kbeg = split ? (int64_t)z * kslice : 0;
  const int64_t kend = split ? (kbeg + kslice < k ? kbeg + kslice : k) : k;
  const int KT = kend > kbeg ? (int)((kend - kbeg + DK - 1) / DK) : 0;
  const int bz = split ? 0 : z;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], Cfg::WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    asm volatile("fence.proxy.async.shared::cta;\n" ::);
  }
  __syncthreads();

  auto issue = [&](int t) {
    const int s = t % STAGES;
    uint8_t* a = smem + s * Cfg::STAGE_BYTES;
    uint8_t* b = a + Cfg::A_BYTES;
    const int kk = (int)(kbeg + (int64_t)t * DK);
    mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
    if constexpr (AKF) {
      tma_load_3d(a, &ma, &full[s], kk, m0, bz);
    } else {
#pragma unroll
      for (int q = 0; q < BM / 16; ++q) tma_load_3d(a + q * 2048, &ma, &full[s], m0 + 16 * q, kk, bz);
    }
    if constexpr (BKF) {
      tma_load_3d(b, &mb, &full[s], kk, n0, bz);
    } else {
#pragma unroll
      for (int q = 0; q < BN / 16; ++q) tma_load_3d(b + q * 2048, &mb, &full[s], n0 + 16 * q, kk, bz);
    }
  };

  if (warp == Cfg::WARPS) {
    // The producer warp: a warp of its own keeps the copies' address
    // arithmetic, waits and issue off the MMA warps, which at one block an SM
    // had been what the others waited for (684^3, 64x64 tiles of four warps:
    // 51 us with thread 0 of an MMA warp issuing, 37 us with this warp).
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)&ma) : "memory");
      asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)&mb) : "memory");
      int t = 0;
      for (; t < KT; ++t) {
        if (t >= STAGES &&
            !mbar_wait(&empty[t % STAGES], (uint32_t)((t / STAGES - 1) & 1), wait_ns)) {
          *(volatile int*)err = 17;
          break;
        }
        issue(t);
      }
      // nothing of this CTA's may be in flight when it exits
      for (int u = t > STAGES ? t - STAGES : 0; u < t; ++u)
        mbar_wait(&full[u % STAGES], (uint32_t)((u / STAGES) & 1), WAIT_NS);
    }
    return;
  }

  const int g = lane >> 2, t4 = lane & 3;
  const int wm0 = (warp % Cfg::WARPS_M) * WM, wn0 = (warp / Cfg::WARPS_M) * WN;
  const FragOff<AKF, MT> fa(wm0, g, t4);
  const FragOff<BKF, NTL> fb(wn0, g, t4);

  double acc[MT][NTL][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  for (int t = 0; t < KT; ++t) {
    const int s = t % STAGES;
    const bool ready = mbar_wait(&full[s], (uint32_t)((t / STAGES) & 1), wait_ns);
    if (!__all_sync(~0u, ready)) {
      if (lane == 0) *(volatile int*)err = 17;
      return;
    }
    // Release the stage of tile t-1 only now, past the wait on tile t: the
    // MMAs of tile t-1 stand before that wait in program order and take its
    // fragments as register operands, so every shared-memory read of that
    // stage has returned.  Releasing it right behind the loads, before the
    // MMAs that wait for them, let the refill overwrite rows that a load still
    // queued behind a neighbouring CTA's epilogue had yet to read (10-15% of
    // the beta = 1 K builds at v = 318 came out with wrong elements).
    if (t >= 1 && lane == 0) mbar_arrive(&empty[(t - 1) % STAGES]);
    const double* As = (const double*)(smem + s * Cfg::STAGE_BYTES);
    const double* Bs = (const double*)(smem + s * Cfg::STAGE_BYTES + Cfg::A_BYTES);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double af[MT], bf[NTL];
#pragma unroll
      for (int i = 0; i < MT; ++i) af[i] = As[fa.at(i, q)];
#pragma unroll
      for (int j = 0; j < NTL; ++j) bf[j] = Bs[fb.at(j, q)];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j) dmma884(acc[i][j], af[i], bf[j]);
    }
  }

  double* C = out.C + (int64_t)z * out.scb;
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int64_t row = m0 + frag_row<AKF>(wm0, i, g);
    if (row >= out.m) continue;
    double* Cr = C + row;
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t col = n0 + frag_row<BKF>(wn0, j, 2 * t4 + h);
        if (col < out.n) {
          double* cp = Cr + col * out.scn;
          double v = out.alpha * acc[i][j][h];
          if (out.beta != 0.0) v += out.beta * *cp;
          *cp = v;
        }
      }
  }
}

// Operand X(i, k) = X[i*si + k*sk + z*sz] (i < ni, k < nk, z < nz) as TMA would
// address it: k-fast when sk == 1 (rows of k, s1 apart), else i-fast (si == 1).
// ok is false when it cannot.  A single item's map still needs a valid third
// stride: the item's extent.
struct DOperand {
  bool ok = false, kfast = false;
  int64_t s1 = 0, sz = 0;
};
DOperand operand(const double* X, int64_t ni, int64_t nk, int64_t si, int64_t sk, int64_t nz,
                 int64_t sz) {
  DOperand d;
  if (((uintptr_t)X & 15) != 0 || (nz > 1 && !stride_ok(sz))) return d;
  int64_t rows;
  if (sk == 1 && (nk > 1 || si != 1)) {
    d.kfast = true;
    rows = ni;
    d.s1 = ni > 1 ? si : (nk + 1) / 2 * 2;
  } else if (si == 1) {
    rows = nk;
    d.s1 = nk > 1 ? sk : (ni + 1) / 2 * 2;
  } else {
    return d;
  }
  d.sz = nz > 1 ? sz : (d.s1 * rows + 1) / 2 * 2;
  d.ok = stride_ok(d.s1) && stride_ok(d.sz);
  return d;
}

// Its map (box 16 k x box_rows rows, or 16 i x 16 k); false when TMA cannot
// address it.
bool operand_map(CUtensorMap* m, bool* kfast, const double* X, int64_t ni, int64_t nk,
                 int64_t si, int64_t sk, int64_t nz, int64_t sz, int box_rows) {
  const DOperand d = operand(X, ni, nk, si, sk, nz, sz);
  if (!d.ok) return false;
  *kfast = d.kfast;
  return d.kfast ? dmap(m, X, nk, ni, d.s1, nz, d.sz, box_rows) == 0
                 : dmap(m, X, ni, nk, d.s1, nz, d.sz, 16) == 0;
}

template <int BM, int BN, int WM, int WN, int STAGES, int MINB, bool AKF, bool BKF>
int launch_dtma(cudaStream_t st, const CUtensorMap& ma, const CUtensorMap& mb, const DOut& out,
                int64_t k, int64_t kslice, int nz, int split) {
  using Cfg = DCfg<BM, BN, WM, WN, STAGES>;
  auto kern = dgemm_tma_kernel<BM, BN, WM, WN, STAGES, MINB, AKF, BKF>;
  // cudaFuncSetAttribute acts on the current device only: one flag per device
  static std::atomic<bool> done[128] = {};
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) {
    cudaGetLastError();
    d = -1;
  }
  if (d < 0 || d >= 128 || !done[d].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM) ==
        cudaSuccess) {
      if (d >= 0 && d < 128) done[d].store(true, std::memory_order_release);
    } else {
      cudaGetLastError();
    }
  }
  const int64_t gx = (out.m + BM - 1) / BM, gy = (out.n + BN - 1) / BN;
  if (gy > 65535 || nz > 65535) return (int)cudaErrorInvalidConfiguration;
  dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)nz);
  unsigned long long w = tc_wait((stream_t)st);
  int* err = wait_error((stream_t)st, WAIT_DGEMM);
  if (!err) return (int)cudaErrorMemoryAllocation;
  kern<<<grid, Cfg::THREADS, Cfg::SMEM, st>>>(ma, mb, out, k, kslice, split, w ? w : WAIT_NS,
                                              err);
  note_launches(1);
  return (int)cudaGetLastError();
}

typedef int (*DtmaLaunch)(cudaStream_t, const CUtensorMap&, const CUtensorMap&, const DOut&,
                          int64_t, int64_t, int, int);

// Tile configurations (blocks an SM, MMA warps): 0: 64x64 (3, four of 32x32);
// 1: 32x32 (4, four of 16x16); 2: 64x32 (3, four of 32x16); 3: 64x64 (2, eight
// of 32x16).  Measured us, configurations 0..3 (4224^3 is 35.0, 32.6, 34.8 and
// 34.3 TF/s; a 128x128 tile of eight warps took 5461 us, 128x64 of four 4622):
//   4224^3           4318  4633  4337  4399
//   1216^3            139   122   115   135
//   684^3              37    33    31    29
//   400^3              23    12    16    18
//   256x256x5776      270   104   163   207
// Large outputs want few operand reads per MMA (0), outputs of about a tile
// per SM the eight warps that hide each other's latency (3), smaller ones
// more blocks (2, 1).
template <bool AKF, bool BKF>
DtmaLaunch pick(int cfg) {
  switch (cfg) {
    case 1: return launch_dtma<32, 32, 16, 16, 6, 4, AKF, BKF>;
    case 2: return launch_dtma<64, 32, 32, 16, 4, 3, AKF, BKF>;
    case 3: return launch_dtma<64, 64, 32, 16, 4, 2, AKF, BKF>;
    default: return launch_dtma<64, 64, 32, 32, 4, 3, AKF, BKF>;
  }
}
constexpr int CFG_BM[DTMA_CONFIGS] = {64, 32, 64, 64};
constexpr int CFG_BN[DTMA_CONFIGS] = {64, 32, 32, 64};

// Whole calls: a CCSD iteration of o=24, v=318 662 -> 626 ms (33.8 TF/s over
// its FP64 GEMMs; 628 ms with the shapes tuned one by one for the earlier
// kernel), of o=12, v=57 2.53 -> 2.18 ms, Lambda residual of o=16, v=76 9.15
// -> 7.7 ms.

// Share of the FP64 MMA rate that r resident blocks of a configuration reach
// on their SM (from the timings above and 1024^3, 2048^3).
constexpr int CFG_OCC[DTMA_CONFIGS] = {3, 4, 3, 2};
constexpr double CFG_EFF[DTMA_CONFIGS][4] = {
    {0.70, 0.88, 0.93, 0.93}, {0.45, 0.68, 0.73, 0.77}, {0.58, 0.80, 0.90, 0.90},
    {0.88, 0.94, 0.94, 0.94}};

}  // namespace

bool dgemm_tma_usable(const Gemm& q) {
  if (q.scm != 1 || q.m <= 0 || q.n <= 0 || q.k <= 0) return false;
  if (q.m >= ((int64_t)1 << 31) || q.n >= ((int64_t)1 << 31) || q.k >= ((int64_t)1 << 31))
    return false;
  return operand(q.A, q.m, q.k, q.sam, q.sak, q.batch, q.sab).ok &&
         operand(q.B, q.n, q.k, q.sbn, q.sbk, q.batch, q.sbb).ok;
}

// Estimated time (us) of configuration cfg with K in S slices: the busiest
// SM's blocks at the rate its residents reach (64x64x16 multiply-adds take
// 0.521 us of an SM), a launch, and the reduction of the partial products.
static double dgemm_tma_cost(const Gemm& q, int cfg, int64_t S) {
  const int64_t bm = CFG_BM[cfg], bn = CFG_BN[cfg];
  const int64_t kt = ((q.k + S - 1) / S + DK - 1) / DK;
  int64_t ctas = ((q.m + bm - 1) / bm) * ((q.n + bn - 1) / bn) * q.batch * S;
  if (q.tri > 0) ctas = (int64_t)((double)ctas * gemm_kept(q)) + 1;
  const int64_t x = (ctas + 147) / 148;
  const double eff = CFG_EFF[cfg][std::min<int64_t>(x, CFG_OCC[cfg]) - 1];
  double t = 3.0 + 0.521 * (double)(bm * bn) / 4096.0 * (double)(kt * x) / eff;
  if (S > 1) t += 3.0 + 8.0e-6 * (double)(S + 1) * (double)q.m * (double)q.n / 4.0;
  return t;
}

double dgemm_tma_rule(const Gemm& q, int* cfg, int* nsplit) {
  *cfg = 0;
  *nsplit = 1;
  double best = -1.0;
  for (int c = 0; c < DTMA_CONFIGS; ++c) {
    if ((q.n + CFG_BN[c] - 1) / CFG_BN[c] > 65535) continue;
    for (int64_t S : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64}) {
      // partial products within 128 MiB of scratch
      if (S > 1 && (q.batch != 1 || q.tri > 0 || q.k / S < 64 || S * q.m * q.n > ((int64_t)1 << 24))) break;
      const double t = dgemm_tma_cost(q, c, S);
      if (best < 0.0 || t < best) {
        best = t;
        *cfg = c;
        *nsplit = (int)S;
      }
    }
  }
  return best;
}

int dgemm_tma(stream_t s, const Gemm& q, int cfg, int nsplit) {
  if (cfg < 0 || cfg >= DTMA_CONFIGS) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)s;
  if (q.tri > 0) nsplit = 1;  // the reduction of partial products covers all of C
  if (q.scm != 1 || (nsplit > 1 && q.batch != 1)) return (int)cudaErrorInvalidValue;
  CUtensorMap ma, mb;
  bool akf = false, bkf = false;
  if (!operand_map(&ma, &akf, q.A, q.m, q.k, q.sam, q.sak, q.batch, q.sab, CFG_BM[cfg]) ||
      !operand_map(&mb, &bkf, q.B, q.n, q.k, q.sbn, q.sbk, q.batch, q.sbb, CFG_BN[cfg]))
    return -1;
  DtmaLaunch f = akf ? (bkf ? pick<true, true>(cfg) : pick<true, false>(cfg))
                     : (bkf ? pick<false, true>(cfg) : pick<false, false>(cfg));
  if (nsplit <= 1) {
    DOut o{q.C, q.m, q.n, q.scn, q.scb, q.alpha, q.beta, (int)q.tri};
    return f(st, ma, mb, o, q.k, q.k, (int)q.batch, 0);
  }
  int64_t kc = (q.k + nsplit - 1) / nsplit;
  kc = (kc + DK - 1) / DK * DK;
  const int64_t S = (q.k + kc - 1) / kc;
  double* P = splitk_buffer(s, (size_t)S * q.m * q.n);
  if (!P) return (int)cudaErrorMemoryAllocation;
  DOut o{P, q.m, q.n, q.m, q.m * q.n, 1.0, 0.0};
  if (int e = f(st, ma, mb, o, q.k, kc, (int)S, 1)) return e;
  return splitk_reduce(s, q.m, q.n, (int)S, P, q.alpha, q.beta, q.C, q.scm, q.scn);
}

}  // namespace dev
}  // namespace ecg
