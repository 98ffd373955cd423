// dev_kbuild.cu — the FP64 (T) K builds on the TMA-staged FP64 MMA tile
// (sm_100a):
//
//   C_z(r, c) = beta C_z(r, c) + sum_s sum_k A_s[r, k; a_s(z)] B_s[c, k; b_s(z)]
//
// for a batch of occupied triplets z in one launch: up to four K segments
// (the two vvvo and the two ovoo products that share an index map into K),
// each operand a 3-D array (row, k, item) whose item a per-triplet table
// names.  Staging, fragment orders and the release rule are those of the
// TMA-staged FP64 GEMM (dev_dgemm.cu).
//
// What bounds it: the FP64 MMA pipe (12 v^4 flops a triplet against five passes
// over its K cube; v = 200: the pipe 83 to 90% active, 33 TF/s executed, 27 useful,
// DRAM at 12%).  Measured, a (T) call: v = 76, o = 16 91.7 ms with nine GEMMs a
// triplet, 23.4 so; v = 318, o = 6 272.6 and 226.9.
// Why this tile: rows run over the v^2 side, where the last of many tiles is
// the only ragged one, and columns over the v side in a width BN that covers
// v in whole tiles with the least padding (kb_width): 64 x 64 tiles spent 41%
// of the MMAs at v = 76 on padding, BN = 80 spends 5%.  Four warps stand along
// the rows (16 rows x BN columns each), so any multiple of 16 is a width.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "dgemm_frag.cuh"
#include "ecg_dev.h"
#include "tma_util.cuh"

namespace ecg {
namespace dev {

namespace {

using namespace tma;
using namespace dfrag;

constexpr int KB_BM = 64, KB_WARPS = 4, KB_THREADS = 32 * KB_WARPS;

template <int BN, int STAGES>
struct KbCfg {
  static constexpr int A_BYTES = KB_BM * DK * 8;
  static constexpr int B_BYTES = BN * DK * 8;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 2 * STAGES * 8;
  static_assert(BN % 16 == 0 && B_BYTES % 1024 == 0, "16-column blocks on 1024 bytes");
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

struct KbMaps {
  CUtensorMap a[KB_MAX_SEG], b[KB_MAX_SEG];
};
// Segment s covers the 16-deep k-slabs [end[s-1], end[s]) (unused trailing
// segments repeat the total).
struct KbSegs {
  int end[KB_MAX_SEG];
};
struct KbOut {
  double* C;
  int64_t m, n, scm, dm, scm2, scn;
  double beta;
  int vec;  // scn == 1 and every row starts on 16 bytes: column pairs move as one
};

template <int BN, int STAGES, int MINB>
__global__ void __launch_bounds__(KB_THREADS, MINB)
    kbuild_kernel(const __grid_constant__ KbMaps maps, const KbOut out, const KbSegs segs,
                  const KbItem* __restrict__ items, int ntn, unsigned long long wait_ns, int* err) {
  using Cfg = KbCfg<BN, STAGES>;
  constexpr int MT = 2, NTL = BN / 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + STAGES;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // column tiles run fastest: the few that share a row tile of the large
  // operand run together and read it through L2
  const int m0 = (int)(blockIdx.x / (unsigned)ntn) * KB_BM;
  const int n0 = (int)(blockIdx.x % (unsigned)ntn) * BN;
  const KbItem it = items[blockIdx.y];
  const int KT = segs.end[KB_MAX_SEG - 1];

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], KB_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    asm volatile("fence.proxy.async.shared::cta;\n" ::);
  }
  __syncthreads();

  auto issue = [&](int t) {
    const int s = t % STAGES;
    uint8_t* a = smem + s * Cfg::STAGE_BYTES;
    uint8_t* b = a + Cfg::A_BYTES;
    int sg = 0, start = 0, za = it.a[0], zb = it.b[0];
#pragma unroll
    for (int q = 1; q < KB_MAX_SEG; ++q)
      if (t >= segs.end[q - 1]) {
        sg = q;
        start = segs.end[q - 1];
        za = it.a[q];
        zb = it.b[q];
      }
    const int kk = (t - start) * DK;
    mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
#pragma unroll
    for (int q = 0; q < KB_BM / 16; ++q)
      tma_load_3d(a + q * 2048, &maps.a[sg], &full[s], m0 + 16 * q, kk, za);
#pragma unroll
    for (int q = 0; q < BN / 16; ++q)
      tma_load_3d(b + q * 2048, &maps.b[sg], &full[s], n0 + 16 * q, kk, zb);
  };

  int issued = 0;
  if (tid == 0)
    for (; issued < KT && issued < STAGES; ++issued) issue(issued);

  const int g = lane >> 2, t4 = lane & 3;
  const FragOff<false, MT> fa(16 * warp, g, t4);
  const FragOff<false, NTL> fb(0, g, t4);

  double acc[MT][NTL][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  bool ok = true;
  int consumed = 0;
  for (int t = 0; t < KT; ++t) {
    const int s = t % STAGES;
    const bool ready = mbar_wait(&full[s], (uint32_t)((t / STAGES) & 1), wait_ns);
    if (!__all_sync(~0u, ready)) {
      ok = false;
      break;
    }
    consumed = t + 1;
    // tile t-1 is released behind the wait on tile t, when its MMAs have taken
    // every fragment as an operand (see dev_dgemm.cu)
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
    // thread 0 refills the stage of tile t-1 once every warp has released it
    bool refill_ok = true;
    if (tid == 0 && t >= 1 && issued < KT) {
      const int tp = t - 1;
      if (mbar_wait(&empty[tp % STAGES], (uint32_t)((tp / STAGES) & 1), wait_ns))
        issue(issued++);
      else
        refill_ok = false;
    }
    if (!__all_sync(~0u, refill_ok)) {
      ok = false;
      break;
    }
  }
  if (!ok) {
    if (lane == 0) *(volatile int*)err = 49;
    // nothing of this CTA's may be in flight when it exits
    if (tid == 0)
      for (int t = consumed; t < issued; ++t)
        mbar_wait(&full[t % STAGES], (uint32_t)((t / STAGES) & 1), WAIT_NS);
    return;
  }

  // Epilogue, one fragment row at a time: with beta = 1 all its C values are
  // loaded before any is stored, so the loads overlap.
  double* C = out.C + it.c;
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int row = m0 + frag_row<false>(16 * warp, i, g);
    if (row >= out.m) continue;
    const int64_t rq = out.dm > 0 ? row / (int)out.dm : 0;
    double* Cr = C + (row - rq * out.dm) * out.scm + rq * out.scm2;
    // the lane's columns 2 t4, 2 t4 + 1 of block j are neighbours
    auto col_of = [&](int j) { return n0 + frag_row<false>(0, j, 2 * t4); };
    if (out.vec) {
      double2 cv[NTL];
      if (out.beta != 0.0) {
#pragma unroll
        for (int j = 0; j < NTL; ++j)
          cv[j] = col_of(j) < out.n ? *reinterpret_cast<const double2*>(Cr + col_of(j))
                                    : make_double2(0.0, 0.0);
      } else {
#pragma unroll
        for (int j = 0; j < NTL; ++j) cv[j] = make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int j = 0; j < NTL; ++j)
        if (col_of(j) < out.n)
          *reinterpret_cast<double2*>(Cr + col_of(j)) =
              make_double2(acc[i][j][0] + cv[j].x, acc[i][j][1] + cv[j].y);
      continue;
    }
    double cv[NTL][2];
    if (out.beta != 0.0) {
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          cv[j][h] = col_of(j) + h < out.n ? Cr[(col_of(j) + h) * out.scn] : 0.0;
    } else {
#pragma unroll
      for (int j = 0; j < NTL; ++j) cv[j][0] = cv[j][1] = 0.0;
    }
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (col_of(j) + h < out.n)
          Cr[(col_of(j) + h) * out.scn] = acc[i][j][h] + cv[j][h];
  }
}

template <int BN, int STAGES, int MINB>
int launch_kbuild(cudaStream_t st, const KbMaps& maps, const KbOut& out, const KbSegs& segs,
                  const KbItem* items, int nitems, unsigned long long wait_ns, int* err) {
  using Cfg = KbCfg<BN, STAGES>;
  auto kern = kbuild_kernel<BN, STAGES, MINB>;
  // cudaFuncSetAttribute acts on the current device only: one flag per device
  static std::atomic<bool> done[128] = {};
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess) cudaGetLastError();
  if (d < 0 || d >= 128 || !done[d].load(std::memory_order_acquire)) {
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return (int)e;
    }
    if (d >= 0 && d < 128) done[d].store(true, std::memory_order_release);
  }
  const int64_t mt = (out.m + KB_BM - 1) / KB_BM, nt = (out.n + BN - 1) / BN;
  if (mt * nt >= ((int64_t)1 << 31)) return (int)cudaErrorInvalidConfiguration;
  kern<<<dim3((unsigned)(mt * nt), (unsigned)nitems), KB_THREADS, Cfg::SMEM, st>>>(
      maps, out, segs, items, (int)nt, wait_ns, err);
  note_launches(1);
  return (int)cudaGetLastError();
}

// Column width for n columns: the one that pads n least, the wider of two
// that pad alike (fewer operand reads per MMA).  112 and 96 leave two blocks
// an SM where the others leave three.
int kb_width(int64_t n) {
  int best = 0;
  int64_t pad = 0;
  for (int w : {80, 64, 112, 96, 48, 32}) {
    const int64_t p = (n + w - 1) / w * w;
    if (best == 0 || p < pad) {
      best = w;
      pad = p;
    }
  }
  return best;
}

int kb_map(CUtensorMap* m, const KbOperand& o, int64_t nk) {
  if (((uintptr_t)o.X & 15) != 0 || !stride_ok(o.sk) || !stride_ok(o.sz) || o.ni <= 0 ||
      nk <= 0 || o.nz <= 0)
    return (int)cudaErrorInvalidValue;
  return dmap(m, o.X, o.ni, nk, o.sk, o.nz, o.sz, 16);
}

}  // namespace

int kbuild(stream_t s, const KbGemm& g, int nitems, const KbItem* items) {
  if (nitems <= 0) return 0;
  if (g.nseg < 1 || g.nseg > KB_MAX_SEG || g.m <= 0 || g.n <= 0 || !g.C || !items ||
      nitems > 65535 || g.m >= ((int64_t)1 << 31) || g.n >= ((int64_t)1 << 31) ||
      (g.beta != 0.0 && g.beta != 1.0))
    return (int)cudaErrorInvalidValue;
  KbMaps maps;
  KbSegs segs;
  int end = 0;
  double depth = 0.0;
  for (int q = 0; q < KB_MAX_SEG; ++q) {
    const int u = q < g.nseg ? q : 0;
    if (g.A[u].ni < g.m || g.B[u].ni < g.n) return (int)cudaErrorInvalidValue;
    if (int e = kb_map(&maps.a[q], g.A[u], g.k[u])) return e;
    if (int e = kb_map(&maps.b[q], g.B[u], g.k[u])) return e;
    if (q < g.nseg) {
      end += (int)((g.k[q] + DK - 1) / DK);
      depth += (double)g.k[q];
    }
    segs.end[q] = end;
  }
  const bool vec = g.scn == 1 && g.n % 2 == 0 && g.scm % 2 == 0 && g.scm2 % 2 == 0 &&
                   ((uintptr_t)g.C & 15) == 0 && g.even_items;
  const KbOut out{g.C, g.m, g.n, g.scm, g.dm, g.scm2, g.scn, g.beta, vec ? 1 : 0};
  cudaStream_t st = (cudaStream_t)s;
  const uint64_t w = tc_wait(s);
  const unsigned long long wns = w ? (unsigned long long)w : WAIT_NS;
  int* err = wait_error(s, WAIT_KBUILD);
  if (!err) return (int)cudaErrorMemoryAllocation;
  const int slot = ktime_begin(s, KT_DGEMM);
  int e;
  switch (kb_width(g.n)) {
    case 112: e = launch_kbuild<112, 4, 2>(st, maps, out, segs, items, nitems, wns, err); break;
    case 96: e = launch_kbuild<96, 4, 2>(st, maps, out, segs, items, nitems, wns, err); break;
    case 80: e = launch_kbuild<80, 4, 3>(st, maps, out, segs, items, nitems, wns, err); break;
    case 64: e = launch_kbuild<64, 4, 3>(st, maps, out, segs, items, nitems, wns, err); break;
    case 48: e = launch_kbuild<48, 4, 3>(st, maps, out, segs, items, nitems, wns, err); break;
    default: e = launch_kbuild<32, 4, 3>(st, maps, out, segs, items, nitems, wns, err); break;
  }
  ktime_end(s, KT_DGEMM, slot, 2.0 * (double)g.m * (double)g.n * depth * nitems);
  return e;
}

}  // namespace dev
}  // namespace ecg
