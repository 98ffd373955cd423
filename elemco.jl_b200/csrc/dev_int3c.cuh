// dev_int3c.cuh — the three-centre Coulomb integral kernel (mn|P), one
// instantiation per class of angular momenta (dev_int3c*.cu share them out, so
// that they compile side by side).
//
// (ab|P_m) = sum over primitives of  pref * sum_{tuv} H_ab[tuv] W_m[tuv],
//   W_m[tuv] = (2c)^{-l} sum_{|k| = l} S_{lm}[k] R_{tuv + k}:
// a Gaussian times a real solid harmonic S_lm is S_lm(d/dC) / (2c)^l of the
// plain Gaussian (the terms of lower order vanish with the Laplacian of S_lm),
// so the fitting function needs the Hermite integrals of degree l to l + la +
// lb only, and no expansion table.  H_ab[tuv], the Hermite expansion of the
// spherical pair with its coefficients, norms and Gaussian-product factor, is
// made once per primitive pair (pair_hermite_kernel) and read by all fitting
// shells; integrals come out spherical and normalised, both orders of m, n.
//
// One thread takes an AO shell pair and a fitting shell (contracted pairs:
// eight); the classes (la >= lb, l) are instantiations, so that all loops over
// components are unrolled and R lives in registers, and the threads of a warp
// share the pair (H is read as a broadcast).  What bounds it: latency, of the
// longest contraction at small molecules and of the f and g classes, whose R and
// sums live in local memory and whose pairs are few, at large ones ((H2O)4 cc-pVTZ:
// 61% of the kernels' 4.2 ms in three classes of 29 to 301 blocks).  Measured, the
// factors' whole call (allocations and fitting product included): H2O cc-pVDZ/RI 1.0
// ms, (H2O)4 cc-pVTZ/RI 9.7; with run-time loops, expansion tables in local memory
// and Cartesian output the integrals alone took 2.9 and 34.8.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <utility>

#include "ecg_dev.h"

namespace ecg {
namespace dev {
namespace int3c {

__host__ __device__ constexpr int tet(int s) { return (s + 1) * (s + 2) * (s + 3) / 6; }

// Boys functions F_0..F_{BM-1} at T = i / BSTEP, from which F_m(T) follows by
// eight Taylor terms (|dT| <= 1/32: the ninth is below 3e-17 of F_0).
constexpr int BSTEP = 16, BTMAX = 36, BN = BSTEP * BTMAX + 2, BM = INT_LTOT + 8;

template <int M>
__device__ __forceinline__ void boys_t(const double* __restrict__ tab, double T,
                                       double (&F)[M + 1]) {
  const double et = exp(-T);
  if (T < (double)BTMAX) {
    const int i = (int)(T * BSTEP + 0.5);
    const double d = (double)i * (1.0 / BSTEP) - T;
    const double* f = tab + i * BM + M;
    double r = f[7];
#pragma unroll
    for (int k = 7; k > 0; --k) r = f[k - 1] + r * d * (1.0 / k);
    F[M] = r;
#pragma unroll
    for (int n = M; n > 0; --n) F[n - 1] = (2.0 * T * F[n] + et) * (1.0 / (2 * n - 1));
  } else {  // erf(sqrt T) is 1 to rounding
    const double ti = 0.5 / T;
    F[0] = sqrt(M_PI * 0.5 * ti);
#pragma unroll
    for (int n = 0; n < M; ++n) F[n + 1] = ((2 * n + 1) * F[n] - et) * ti;
  }
}

__host__ __device__ constexpr int hx(int t, int u, int v) {
  return (t + u + v) * (t + u + v + 1) * (t + u + v + 2) / 6 + (u + v) * (u + v + 1) / 2 + v;
}

// R_{tuv}, t + u + v <= L, in place level by level: totals descend, so that
// level n + 1 is still there where level n reads it.
template <int L>
__device__ __forceinline__ void hermite_t(const double* __restrict__ tab, double alpha, double X,
                                          double Y, double Z, double (&R)[tet(L)]) {
  double F[L + 1];
  boys_t<L>(tab, alpha * (X * X + Y * Y + Z * Z), F);
  double sc[L + 1];
  sc[0] = 1.0;
#pragma unroll
  for (int n = 1; n <= L; ++n) sc[n] = sc[n - 1] * (-2.0 * alpha);
#pragma unroll
  for (int n = L; n >= 0; --n) {
#pragma unroll
    for (int s = L - n; s > 0; --s)
#pragma unroll
      for (int w = 0; w <= s; ++w)
#pragma unroll
        for (int v = 0; v <= w; ++v) {
          const int u = w - v, t = s - w;
          double r;
          if (t > 0) {
            r = X * R[hx(t - 1, u, v)];
            if (t > 1) r += (double)(t - 1) * R[hx(t > 1 ? t - 2 : 0, u, v)];
          } else if (u > 0) {
            r = Y * R[hx(t, u - 1, v)];
            if (u > 1) r += (double)(u - 1) * R[hx(t, u > 1 ? u - 2 : 0, v)];
          } else {
            r = Z * R[hx(t, u, v - 1)];
            if (v > 1) r += (double)(v - 1) * R[hx(t, u, v > 1 ? v - 2 : 0)];
          }
          R[hx(t, u, v)] = r;
        }
    R[0] = sc[n] * F[n];
  }
}

// Coefficient of x^i y^j z^{l-i-j} in the real solid harmonic S_lm, m = -l..l
// (Helgaker, Jorgensen, Olsen, eq. 6.4.47), without its constant N_lm.
__host__ __device__ constexpr double sh_binom(int n, int k) {
  double r = k < 0 || k > n ? 0.0 : 1.0;
  for (int i = 1; i <= k && r != 0.0; ++i) r = r * (n - k + i) / i;
  return r;
}
__host__ __device__ constexpr double sh_coef(int l, int m, int i, int j) {
  const int am = m < 0 ? -m : m, dm = m < 0 ? 1 : 0;
  double c = 0.0;
  for (int t = 0; t <= (l - am) / 2; ++t)
    for (int u = 0; u <= t; ++u)
      for (int k = dm; k <= am; k += 2) {
        if (2 * t + am - 2 * u - k != i || 2 * u + k != j) continue;
        double q = sh_binom(l, t) * sh_binom(l - t, am + t) * sh_binom(t, u) * sh_binom(am, k);
        for (int e = 0; e < t; ++e) q *= 0.25;
        c += ((t + (k - dm) / 2) & 1) ? -q : q;
      }
  return c;
}
__host__ __device__ constexpr int cart_i(int l, int n) {
  int i = l, left = n;
  while (left > l - i) {
    left -= l - i + 1;
    --i;
  }
  return i;
}
__host__ __device__ constexpr int cart_j(int l, int n) {
  int i = l, left = n;
  while (left > l - i) {
    left -= l - i + 1;
    --i;
  }
  return l - i - left;
}

template <int LAB, int LC, int M, int K>
__device__ __forceinline__ void add_harmonic(double (&w)[tet(LAB)],
                                             const double (&R)[tet(LAB + LC)]) {
  constexpr int i = cart_i(LC, K), j = cart_j(LC, K), k = LC - i - j;
  constexpr double c = sh_coef(LC, M - LC, i, j);
  if constexpr (c != 0.0) {
#pragma unroll
    for (int s = 0; s <= LAB; ++s)
#pragma unroll
      for (int x = 0; x <= s; ++x)
#pragma unroll
        for (int v = 0; v <= x; ++v)
          w[hx(s - x, x - v, v)] += c * R[hx(s - x + i, x - v + j, v + k)];
  }
}
template <int LAB, int LC, int M, int... K>
__device__ __forceinline__ void harmonic(double (&w)[tet(LAB)], const double (&R)[tet(LAB + LC)],
                                         std::integer_sequence<int, K...>) {
  (add_harmonic<LAB, LC, M, K>(w, R), ...);
}

// acc[m][ab] += f * sum_tuv H[ab][tuv] W_m[tuv] for m = M, M+1, ..
template <int LAB, int LC, int NAB, int M>
__device__ __forceinline__ void contract_m(const double (&R)[tet(LAB + LC)],
                                           const double* __restrict__ H, double f,
                                           double* __restrict__ acc) {
  constexpr int NT = tet(LAB);
  double w[NT];
#pragma unroll
  for (int x = 0; x < NT; ++x) w[x] = 0.0;
  harmonic<LAB, LC, M>(w, R, std::make_integer_sequence<int, (LC + 1) * (LC + 2) / 2>{});
#pragma unroll 1
  for (int ab = 0; ab < NAB; ++ab) {
    double v0 = 0.0, v1 = 0.0;
#pragma unroll
    for (int x = 0; x < NT; ++x)
      if (x & 1) v1 += H[ab * NT + x] * w[x];
      else v0 += H[ab * NT + x] * w[x];
    acc[M * NAB + ab] += f * (v0 + v1);
  }
  if constexpr (M < 2 * LC) contract_m<LAB, LC, NAB, M + 1>(R, H, f, acc);
}

struct HarmonicNorm {
  double c[2 * INT_LMAX + 1];
};

// One launch covers the pairs of one (la, lb) with all fitting shells: parts of
// consecutive blocks, each the pairs of one kind with the shells of one degree.
// A pair of few primitives takes one thread per fitting shell; a contracted one
// (CONTRACTED or more primitive pairs) SPLIT lanes, which share them out and
// add their sums by shuffles: its loop is what a small molecule waits for, and
// the blocks of the other degrees run beside it.
constexpr int PARTS = 2 * (INT_LMAX + 1), SPLIT = 8, CONTRACTED = 6, THREADS = 64;
struct Part {
  int block0;         // its first block (parts ascend; an empty part has none)
  int pair0, npairs;  // in the pairs of the launch
  int aux0, naux;
};
struct Launch {
  Part part[PARTS];  // kind k (0 contracted, 1 others) and degree l at k + 2 l
  HarmonicNorm nm[INT_LMAX + 1];
  const IntPair* pairs;
  const IntShell* aux;
  const IntPrimPair* prims;
  const double *H, *ex, *co, *boys;
  int64_t n;
  double* out;
};

template <int LA, int LB, int LC>
__device__ __forceinline__ void int3c_part(const Launch& g, const Part& p, int G,
                                           const HarmonicNorm& nm) {
  constexpr int LAB = LA + LB, L = LAB + LC, NA = 2 * LA + 1, NB = 2 * LB + 1, NAB = NA * NB;
  constexpr int NT = tet(LAB), NC = 2 * LC + 1;
  const int64_t id = (int64_t)((int)blockIdx.x - p.block0) * THREADS + threadIdx.x;
  const int64_t it = id / G;
  const int lane = (int)(id - it * G);
  const bool on = it < (int64_t)p.npairs * p.naux;
  const int ip = on ? (int)(it / p.naux) : 0;
  const IntPair pr = g.pairs[p.pair0 + ip];
  const IntShell P = g.aux[p.aux0 + (on ? (int)(it - (int64_t)ip * p.naux) : 0)];
  double acc[NAB * NC];
#pragma unroll 1
  for (int x = 0; x < NAB * NC; ++x) acc[x] = 0.0;
  for (int q = on ? lane : pr.npp; q < pr.npp; q += G) {
    const IntPrimPair pp = g.prims[pr.pp0 + q];
    const double* H = g.H + pr.hoff + (int64_t)q * (NAB * NT);
    for (int kc = 0; kc < P.nprim; ++kc) {
      const double c = g.ex[P.poff + kc];
      const double s = pp.p + c, ps = pp.p * c;
      double R[tet(L)];
      hermite_t<L>(g.boys, ps / s, pp.x - P.x, pp.y - P.y, pp.z - P.z, R);
      contract_m<LAB, LC, NAB, 0>(R, H, g.co[P.poff + kc] / (ps * sqrt(s)), acc);
    }
  }
  if (G > 1) {
#pragma unroll 1
    for (int x = 0; x < NAB * NC; ++x) {
      double v = acc[x];
      for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
      acc[x] = v;
    }
  }
  if (!on) return;
  const int64_t n = g.n;
#pragma unroll 1
  for (int m = 0; m < NC; ++m) {
    double* o = g.out + n * n * (int64_t)(P.boff + m);
    const double f = nm.c[m];
#pragma unroll 1
    for (int x = lane; x < NAB; x += G) {
      const int a = pr.aoff + x % NA, b = pr.boff + x / NA;
      if (pr.aoff == pr.boff && a < b) continue;  // of a shell with itself: (b, a) writes both
      const double v = f * acc[m * NAB + x];
      o[a + n * b] = v;
      o[b + n * a] = v;
    }
  }
}

template <int LA, int LB>
__global__ void __launch_bounds__(THREADS) int3c_kernel(const __grid_constant__ Launch g) {
  int k = 0;
  for (int q = 1; q < PARTS; ++q)
    if ((int)blockIdx.x >= g.part[q].block0 && g.part[q].npairs > 0 && g.part[q].naux > 0) k = q;
  const Part& p = g.part[k];
  const int G = k & 1 ? 1 : SPLIT;
  switch (k >> 1) {
    case 0: int3c_part<LA, LB, 0>(g, p, G, g.nm[0]); break;
    case 1: int3c_part<LA, LB, 1>(g, p, G, g.nm[1]); break;
    case 2: int3c_part<LA, LB, 2>(g, p, G, g.nm[2]); break;
    case 3: int3c_part<LA, LB, 3>(g, p, G, g.nm[3]); break;
    default: int3c_part<LA, LB, 4>(g, p, G, g.nm[4]); break;
  }
}

typedef void (*Kernel)(const Launch);
Kernel pick_f(int lb);   // la = 3 (dev_int3c_f.cu)
Kernel pick_g0(int lb);  // la = 4, lb <= 2 (dev_int3c_g0.cu)
Kernel pick_g(int lb);   // la = 4, lb = 3, 4 (dev_int3c_g.cu)

}  // namespace int3c
}  // namespace dev
}  // namespace ecg
