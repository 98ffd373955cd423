// dev_int3c.cu — three-centre Coulomb integrals (mn|P) over contracted real
// solid harmonics (replaces ElemCo.jl's libcint int3c2e calls,
// src/system/integrals_2e3idx.jl:108-158): the host plan, the Hermite
// expansions of the AO pairs and the launches; the kernel is in dev_int3c.cuh.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "dev_int3c.cuh"
#include "ecg_dev.h"

namespace ecg {
namespace dev {

using namespace int3c;

namespace {

constexpr int LMAX = INT_LMAX;
constexpr int ETSZ = (LMAX + 1) * (LMAX + 1) * (2 * LMAX + 1);  // one 1D E table

__device__ double g_boys[BN * BM];

// 1D Hermite coefficients E[(i*(lb+1)+j)*(la+lb+1)+t], i <= la, j <= lb.
__device__ void etab(int la, int lb, double p, double xpa, double xpb, double* E) {
  const int nt = la + lb + 1;
  const double h = 0.5 / p;
  for (int x = 0; x < (la + 1) * (lb + 1) * nt; ++x) E[x] = 0.0;
  auto at = [&](int i, int j, int t) -> double& { return E[(i * (lb + 1) + j) * nt + t]; };
  at(0, 0, 0) = 1.0;
  for (int i = 0; i <= la; ++i) {
    if (i > 0)
      for (int t = 0; t <= i; ++t) {
        double v = xpa * at(i - 1, 0, t);
        if (t > 0) v += h * at(i - 1, 0, t - 1);
        if (t + 1 <= i - 1) v += (t + 1) * at(i - 1, 0, t + 1);
        at(i, 0, t) = v;
      }
    for (int j = 1; j <= lb; ++j)
      for (int t = 0; t <= i + j; ++t) {
        double v = xpb * at(i, j - 1, t);
        if (t > 0) v += h * at(i, j - 1, t - 1);
        if (t + 1 <= i + j - 1) v += (t + 1) * at(i, j - 1, t + 1);
        at(i, j, t) = v;
      }
  }
}

// Hermite expansion of the spherical pair of each primitive pair, one warp a
// primitive pair: H[(ia + na*ib)*nt + tuv] = f sum S_a[i] S_b[j] Ex Ey Ez over the
// Cartesian components i, j of the two harmonics (sparse rows sh0[l*9 + m] ..
// of (x, y, z, coefficient)).  f holds coefficients, norms and the
// Gaussian-product factor; the harmonics' constants are in the rows.
struct HarmonicTerm {
  int x, y, z, pad;
  double c;
};
__global__ void __launch_bounds__(128)
    pair_hermite_kernel(const IntPairPrimSrc* __restrict__ src, int npp,
                        const HarmonicTerm* __restrict__ terms, const int* __restrict__ sh0,
                        double* __restrict__ Htab) {
  __shared__ double Es[4][3][ETSZ];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = blockIdx.x * 4 + warp;
  if (q >= npp) return;
  const IntPairPrimSrc g = src[q];
  const int la = g.la, lb = g.lb, nt1 = la + lb + 1, NT = tet(la + lb);
  if (lane < 3) etab(la, lb, g.p, g.pa[lane], g.pb[lane], Es[warp][lane]);
  __syncwarp();
  const double *Ex = Es[warp][0], *Ey = Es[warp][1], *Ez = Es[warp][2];
  const int na = 2 * la + 1, nab = na * (2 * lb + 1);
  for (int e = lane; e < nab * NT; e += 32) {
    const int ab = e / NT;
    int r = e - ab * NT, s = 0;
    while (tet(s) <= r) ++s;
    r -= s > 0 ? tet(s - 1) : 0;
    int w = 0;
    while ((w + 1) * (w + 2) / 2 <= r) ++w;
    const int v = r - w * (w + 1) / 2, u = w - v, t = s - w;
    const int ra = la * 9 + ab % na, rb = lb * 9 + ab / na;
    double sum = 0.0;
    for (int x = sh0[ra]; x < sh0[ra + 1]; ++x) {
      const HarmonicTerm A = terms[x];
      for (int y = sh0[rb]; y < sh0[rb + 1]; ++y) {
        const HarmonicTerm B = terms[y];
        if (t > A.x + B.x || u > A.y + B.y || v > A.z + B.z) continue;
        sum += A.c * B.c * Ex[(A.x * (lb + 1) + B.x) * nt1 + t] *
               Ey[(A.y * (lb + 1) + B.y) * nt1 + u] * Ez[(A.z * (lb + 1) + B.z) * nt1 + v];
      }
    }
    Htab[g.hoff + e] = g.f * sum;
  }
}

}  // namespace

namespace {

// F_m(T) tables on the current device, written on its first use.  The table goes
// up on the caller's stream, which is waited for before its address is handed
// out: the contexts' streams do not wait for the default stream, and a copy from
// pageable memory may return before the device has all of it.
int boys_table(cudaStream_t s, const double** out) {
  static std::mutex mu;
  static const double* at[128] = {};
  int d = 0;
  cudaError_t e = cudaGetDevice(&d);
  if (e != cudaSuccess) return (int)e;
  if (d < 0 || d >= 128) return (int)cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(mu);
  if (at[d]) {
    *out = at[d];
    return 0;
  }
  std::vector<double> tab((size_t)BN * BM);
  for (int i = 0; i < BN; ++i) {
    // F_top by its series, then downward recursion
    const long double T = (long double)i / BSTEP, et = expl(-T);
    long double term = 1.0L / (2 * BM - 1), sum = term;
    for (int k = 1; k < 1000 && term > 1e-22L * sum; ++k) {
      term *= 2.0L * T / (2 * BM - 1 + 2 * k);
      sum += term;
    }
    long double F = et * sum;
    for (int m = BM - 1; m >= 0; --m) {
      tab[(size_t)i * BM + m] = (double)F;
      if (m > 0) F = (2.0L * T * F + et) / (2 * m - 1);
    }
  }
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_boys);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(p, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) at[d] = (const double*)p;
  *out = at[d];
  return (int)e;
}

// The harmonics' constants 1 / sqrt(sum_{cc'} S_c S_c' prod (s_d - 1)!!): unit
// self-overlap once the radial part is normalised (int3c2e_sph's prologue).
double harmonic_norm(int l, int m) {
  double g = 0.0;
  for (int a = 0; a < (l + 1) * (l + 2) / 2; ++a)
    for (int b = 0; b < (l + 1) * (l + 2) / 2; ++b) {
      const int s[3] = {cart_i(l, a) + cart_i(l, b), cart_j(l, a) + cart_j(l, b),
                        2 * l - cart_i(l, a) - cart_i(l, b) - cart_j(l, a) - cart_j(l, b)};
      if ((s[0] | s[1] | s[2]) & 1) continue;
      double q = sh_coef(l, m, cart_i(l, a), cart_j(l, a)) *
                 sh_coef(l, m, cart_i(l, b), cart_j(l, b));
      for (int d = 0; d < 3; ++d)
        for (int x = s[d] - 1; x > 1; x -= 2) q *= x;
      g += q;
    }
  return 1.0 / std::sqrt(g);
}

// 1 / sqrt of a contracted shell's radial self-overlap sum c c' (pi/p)^{3/2}
// (2p)^{-l}, p = a + a'.
double radial_norm(const IntShell& s, const double* ex, const double* co) {
  double g = 0.0;
  for (int i = 0; i < s.nprim; ++i)
    for (int j = 0; j < s.nprim; ++j) {
      const double p = ex[s.poff + i] + ex[s.poff + j];
      g += co[s.poff + i] * co[s.poff + j] * std::pow(M_PI / p, 1.5) / std::pow(2.0 * p, s.l);
    }
  return g > 0.0 ? 1.0 / std::sqrt(g) : 0.0;
}

Kernel pick(int la, int lb) {
  if (la == 4) return lb <= 2 ? pick_g0(lb) : pick_g(lb);
  if (la == 3) return pick_f(lb);
  if (la == 2) return lb == 0 ? int3c_kernel<2, 0> : lb == 1 ? int3c_kernel<2, 1> : int3c_kernel<2, 2>;
  if (la == 1) return lb == 0 ? int3c_kernel<1, 0> : int3c_kernel<1, 1>;
  return int3c_kernel<0, 0>;
}

}  // namespace

int Int3cPlan::build(const IntShell* ao, int nao_sh, const double* aoex, const double* aoco,
                     const IntShell* fit, int nfit_sh, const double* fex, const double* fco) {
  *this = Int3cPlan();
  std::vector<double> nrm(nao_sh);
  for (int s = 0; s < nao_sh; ++s)
    if ((nrm[s] = radial_norm(ao[s], aoex, aoco)) == 0.0) return -1;
  for (int la = 0; la <= LMAX; ++la)
    for (int lb = 0; lb <= la; ++lb) {
      pair0[la * (LMAX + 1) + lb] = (int)pairs.size();
      const int nh = (2 * la + 1) * (2 * lb + 1) * tet(la + lb);
      std::vector<IntPair> rest;
      for (int x = 0; x < nao_sh; ++x)
        for (int y = 0; y < nao_sh; ++y) {
          if (ao[x].l != la || ao[y].l != lb || (la == lb && y > x)) continue;
          const IntShell &a = ao[x], &b = ao[y];
          IntPair pr{(int)prims.size(), 0, a.boff, b.boff, hlen};
          const double ab2 = (a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y) +
                             (a.z - b.z) * (a.z - b.z);
          for (int i = 0; i < a.nprim; ++i)
            for (int j = 0; j < b.nprim; ++j) {
              const double ea = aoex[a.poff + i], eb = aoex[b.poff + j], p = ea + eb;
              const double f = std::exp(-ea * eb / p * ab2) * aoco[a.poff + i] *
                               aoco[b.poff + j] * nrm[x] * nrm[y];
              if (f == 0.0) continue;
              const double P[3] = {(ea * a.x + eb * b.x) / p, (ea * a.y + eb * b.y) / p,
                                   (ea * a.z + eb * b.z) / p};
              prims.push_back({p, P[0], P[1], P[2]});
              src.push_back({p, {P[0] - a.x, P[1] - a.y, P[2] - a.z},
                             {P[0] - b.x, P[1] - b.y, P[2] - b.z}, f, hlen, la, lb});
              hlen += nh;
              ++pr.npp;
            }
          (pr.npp >= CONTRACTED ? pairs : rest).push_back(pr);
        }
      nsplit[la * (LMAX + 1) + lb] = (int)pairs.size() - pair0[la * (LMAX + 1) + lb];
      pairs.insert(pairs.end(), rest.begin(), rest.end());
      npair[la * (LMAX + 1) + lb] = (int)pairs.size() - pair0[la * (LMAX + 1) + lb];
    }
  // fitting shells by degree; their coefficients take the norm, the
  // 2 pi^{5/2} of the Coulomb integral and the (-1)^l (2c)^{-l} of the harmonic
  // derivative (the sign from R's derivative with respect to P - C)
  const double two_pi52 = 2.0 * std::pow(M_PI, 2.5);
  for (int l = 0; l <= LMAX; ++l) {
    aux0[l] = (int)aux.size();
    for (int s = 0; s < nfit_sh; ++s) {
      if (fit[s].l != l) continue;
      const double n = radial_norm(fit[s], fex, fco);
      if (n == 0.0) return -1;
      IntShell q = fit[s];
      q.poff = (int)ex.size();
      for (int k = 0; k < q.nprim; ++k) {
        const double c = fex[fit[s].poff + k];
        ex.push_back(c);
        co.push_back(two_pi52 * n * fco[fit[s].poff + k] * (l & 1 ? -1.0 : 1.0) /
                     std::pow(2.0 * c, l));
      }
      aux.push_back(q);
    }
    naux[l] = (int)aux.size() - aux0[l];
  }
  return 0;
}

// Device words (doubles) run() needs for the plan's tables.
int64_t Int3cPlan::table_doubles() const {
  auto d = [](size_t bytes) { return (int64_t)((bytes + 15) / 16 * 2); };
  return d(pairs.size() * sizeof(IntPair)) + d(prims.size() * sizeof(IntPrimPair)) +
         d(src.size() * sizeof(IntPairPrimSrc)) + d(aux.size() * sizeof(IntShell)) +
         d(ex.size() * 8) + d(co.size() * 8) + d(256 * sizeof(HarmonicTerm)) +
         d((9 * (LMAX + 1) + 1) * sizeof(int)) + hlen + 2;
}

int Int3cPlan::run(stream_t st, double* tables, int64_t n, double* out) const {
  cudaStream_t s = (cudaStream_t)st;
  const double* boys = nullptr;
  if (int e = boys_table(s, &boys)) return e;
  char* at = (char*)tables;
  int err = 0;
  auto put = [&](const void* p, size_t bytes) {
    void* d = at;
    if (bytes && !err)
      err = (int)cudaMemcpyAsync(d, p, bytes, cudaMemcpyHostToDevice, s);
    at += (bytes + 15) / 16 * 16;
    return d;
  };
  const IntPair* dp = (const IntPair*)put(pairs.data(), pairs.size() * sizeof(IntPair));
  const IntPrimPair* dq = (const IntPrimPair*)put(prims.data(), prims.size() * sizeof(IntPrimPair));
  const IntPairPrimSrc* ds =
      (const IntPairPrimSrc*)put(src.data(), src.size() * sizeof(IntPairPrimSrc));
  const IntShell* da = (const IntShell*)put(aux.data(), aux.size() * sizeof(IntShell));
  const double* dex = (const double*)put(ex.data(), ex.size() * 8);
  const double* dco = (const double*)put(co.data(), co.size() * 8);
  std::vector<HarmonicTerm> terms;
  std::vector<int> sh0;
  for (int l = 0; l <= LMAX; ++l)
    for (int m = 0; m < 9; ++m) {
      sh0.push_back((int)terms.size());
      for (int c = 0; m <= 2 * l && c < (l + 1) * (l + 2) / 2; ++c) {
        const int i = cart_i(l, c), j = cart_j(l, c);
        const double v = sh_coef(l, m - l, i, j);
        if (v != 0.0) terms.push_back({i, j, l - i - j, 0, v * harmonic_norm(l, m - l)});
      }
    }
  sh0.push_back((int)terms.size());
  if (terms.size() > 256) return (int)cudaErrorInvalidValue;
  terms.resize(256);
  const HarmonicTerm* dt = (const HarmonicTerm*)put(terms.data(), 256 * sizeof(HarmonicTerm));
  const int* dsh = (const int*)put(sh0.data(), sh0.size() * sizeof(int));
  double* H = (double*)at;
  if (err) return err;
  const int npp = (int)src.size();
  if (npp > 0) {
    pair_hermite_kernel<<<(npp + 3) / 4, 128, 0, s>>>(ds, npp, dt, dsh, H);
    note_launches(1);
    if (int e = (int)cudaGetLastError()) return e;
  }
  Launch g{};
  for (int l = 0; l <= LMAX; ++l)
    for (int m = 0; m <= 2 * l; ++m) g.nm[l].c[m] = harmonic_norm(l, m - l);
  g.aux = da; g.prims = dq; g.H = H; g.ex = dex; g.co = dco; g.boys = boys; g.n = n; g.out = out;
  for (int la = LMAX; la >= 0; --la)
    for (int lb = la; lb >= 0; --lb) {
      const int c = la * (LMAX + 1) + lb;
      if (npair[c] == 0) continue;
      g.pairs = dp + pair0[c];
      int64_t blocks = 0;
      for (int l = 0; l <= LMAX; ++l)
        for (int k = 0; k < 2; ++k) {
          Part& p = g.part[k + 2 * l];
          p.pair0 = k ? nsplit[c] : 0;
          p.npairs = k ? npair[c] - nsplit[c] : nsplit[c];
          p.aux0 = aux0[l];
          p.naux = naux[l];
          p.block0 = (int)blocks;
          blocks += ((int64_t)p.npairs * p.naux * (k ? 1 : SPLIT) + THREADS - 1) / THREADS;
          if (blocks >= ((int64_t)1 << 31)) return (int)cudaErrorInvalidConfiguration;
        }
      if (blocks == 0) continue;
      pick(la, lb)<<<(unsigned)blocks, THREADS, 0, s>>>(g);
      note_launches(1);
      if (int e = (int)cudaGetLastError()) return e;
    }
  return 0;
}

}  // namespace dev
}  // namespace ecg
