// ecg_triples.cpp — closed-shell (T) and Lambda-(T).
//
// For each occupied triplet i <= j <= k (i = j = k skipped, weights 2/1 as in
// cc_triples.jl:62-72) the 12 contractions of cc_triples.jl:89-104 are
// regrouped as K = P[W]:
//   W^{xyz}[a,b,c] = sum_d T^{xy}_{ad} (bd|cz) - sum_l T^{xl}_{ab} (ly|cz)
//   K[a,b,c] = W^{ijk}[a,b,c] + W^{jik}[b,a,c] + W^{ikj}[a,c,b]
//            + W^{kji}[c,b,a] + W^{jki}[b,c,a] + W^{kij}[c,a,b]
// The six vvvo GEMMs (M=v, N=v^2, K=v) accumulate straight into K: each
// epilogue writes W^{xyz}[a',(b',c')] to its permuted position in K.  vvvo is
// held in two layouts, [b,c,d,k] and [c,b,d,k], chosen per permutation so
// that the (b',c') pair maps to K through at most one index split; with that
// choice the permutations pair up into three GEMMs of K depth 2v whose two
// halves write the same K positions.  With T^{xy}_{ab} = T^{yx}_{ba} the six
// ovoo GEMMs pair up too, and each ovoo pair writes K through the same index
// map, with the same rows and columns, as one vvvo pair, so every K
// orientation is one GEMM of four K segments (v, v, o, o; ovoo held negated):
// three launches per batch of triplets, each with a single pass over K, with
// rows over the pair index and columns over a'.  A fused kernel forms
// X and both energy sums (sum K X and the singles/Fock term sum X Y,
// cc_triples.jl:113-156); per-triplet energies are summed on the host in
// triplet order, so the result is deterministic.
//
// Mixed precision: every operand is split into two BF16 slices once per call
// (vvvo in both layouts, T^{xy} per pair, T2[:,:,x,:] and T2[:,:,:,x] per
// occupied index, -ovoo per pair; each kind one stack), the GEMMs run on the
// tensor cores and K is kept in FP32.
#include "ecg_triples.h"

#include <algorithm>
#include <cmath>
#include <tuple>
#include <vector>

namespace ecg {

namespace {

// BF16 slices of the (T) operands in mixed precision: two slices (products
// hi*hi + hi*lo + lo*hi, ~2^-16 relative per product) keep the (T) energy
// within ~1e-8 relative of FP64, since the element errors average out.
constexpr int kTriplesSlices = 2;

// One W of K = P[W]: amplitudes T^{xy} and the integrals of occupied z in the
// [b,c,d] (l2 = false) or [c,b,d] (l2 = true) layout.
struct PermW {
  int x, y, z;
  bool l2;
};

// W[a',n], n = b' + v c' in the [b,c,d] layout, n = c' + v b' in the [c,b,d]
// layout.  W^{ijk} and W^{ikj} land at K[a',n], W^{jik} and W^{jki} at K[b',a',c'],
// W^{kji} and W^{kij} at K[n,a'] (see k_map).
void perm_table(int i, int j, int k, PermW* P) {
  P[0] = {i, j, k, false};
  P[1] = {j, i, k, false};
  P[2] = {i, k, j, true};
  P[3] = {k, j, i, true};
  P[4] = {j, k, i, true};
  P[5] = {k, i, j, false};
}

constexpr int kGemms = 3;
// the permutations whose W land in K through one index map
constexpr int kPairs[kGemms][2] = {{0, 2}, {1, 4}, {3, 5}};

// Where orientation q puts (row n = n0 + v n1, column a') in K[a,b,c], which sits
// at a + vp b + vp v c (vp >= v: the padded pitch of the a index; vp = v for FP64
// K, a multiple of 4 for FP32 K so that the energy kernel's TMA copies start on
// 16 bytes): (n % dm)*scm + (n / dm)*scm2 + a'*scn (dm = 0: n*scm + a'*scn).
struct KMap {
  int64_t scm, dm, scm2, scn;
};
KMap k_map(int q, int64_t v, int64_t vp) {
  if (q == 0) return {vp, 0, 0, 1};                      // K[a',n0,n1]
  if (q == 1) return {1, v, vp * v, vp};                 // K[n0,a',n1]
  return vp == v ? KMap{1, 0, 0, vp * v} : KMap{1, v, vp, vp * v};  // K[n0,n1,a']
}

// Consecutive triplets whose tensor-core tiles are interleaved, and the block of
// (i, j) the sweep takes them in: a chunk of 32 shares one k, about four j and
// eight i, so it reads 13 vvvo slabs where triplet by triplet it read 64 (and
// holds 15 MB of T^{xy} at v = 209, well inside L2).  Measured at v = 209, all
// triplets of 31 orbitals: chunks of 2 800 ms, 32 749, 64 747; at v = 129 and 318
// within the runs' spread of one another.
constexpr int kChunk = 32, kBlockI = 8, kBlockJ = 4;

// BF16 operands of one amplitude tensor (T2 or covariant U2), as stacks.
struct SplitAmps {
  dev::TcStack pair;  // T^{xy}[a,d]: rows a, k d        (x + o*y)
  dev::TcStack G;     // T2[:,:,x,l]: rows (a,b), k l    (x)
  dev::TcStack C;     // T2[:,:,l,x]: rows (a,b), k l    (x)
};

uint16_t* alloc_bf16(Ctx& c, size_t elems, const char* what) {
  return reinterpret_cast<uint16_t*>(c.alloc((int64_t)((elems + 3) / 4), what));
}

void split_amps(Ctx& c, const double* T, SplitAmps& S) {
  const int64_t o = c.no, v = c.nv, v2 = v * v;
  dev::stream_t s = c.st;
  const size_t ep = dev::tc_operand_elems(v, v, kTriplesSlices);
  const size_t eg = dev::tc_operand_elems(v2, o, kTriplesSlices);
  uint16_t* bp = alloc_bf16(c, ep * o * o, "(T) T^{xy} BF16");
  uint16_t* bg = alloc_bf16(c, 2 * eg * o, "(T) T2 slices BF16");
  check(dev::tc_split_stack(s, T, v, v, 1, v, 0, o * o, o, v2, v2 * o, bp, &S.pair),
        "split T^{xy}");
  check(dev::tc_split_stack(s, T, v2, o, 1, v2 * o, 0, o, o, v2, 0, bg, &S.G), "split T2 G");
  check(dev::tc_split_stack(s, T, v2, o, 1, v2, 0, o, o, v2 * o, 0, bg + eg * o, &S.C),
        "split T2 C");
}

// Everything the K builds read: FP64 integrals, or their BF16 splits.  The
// FP64 operands have even pitches, so that TMA can address them at odd v.
struct TriplesOps {
  bool mixed = false;
  int64_t v2p = 0, vq = 0;     // pitches of a (b,c) pair and of a virtual index
  const double* V1 = nullptr;  // [b,c,d,k], (b,c) in pitch v2p
  const double* V2 = nullptr;  // [c,b,d,k], (c,b) in pitch v2p
  const double* On = nullptr;  // -(lj|ck) as [c,l,j,k], c in pitch vq
  dev::TcStack V1s, V2s, Ons;  // rows (b,c) / (c,b), k d (item k); rows c, k l (j + o*k)
};

// FP64 amplitudes (T2 or covariant U2) as the K builds read them.
struct FpAmps {
  const double* pair = nullptr;  // T^{xy}[a,d], a in pitch vq, per pair x + o*y
  const double* ab = nullptr;    // T2[(a,b)], pitch v2p, per pair
};

// A copy in even pitches where v is odd (or the array starts off 16 bytes).
FpAmps fp_amps(Ctx& c, const double* T, const TriplesOps& ops) {
  const int64_t o = c.no, v = c.nv, v2 = v * v;
  FpAmps f{T, T};
  if (v % 2 == 0 && ((uintptr_t)T & 15) == 0) return f;
  double* p = c.alloc(ops.vq * v * o * o, "(T) T^{xy} padded");
  double* ab = c.alloc(ops.v2p * o * o, "(T) T2 padded");
  check(dev::repitch(c.st, v, v * o * o, T, v, p, ops.vq), "pad T^{xy}");
  check(dev::repitch(c.st, v2, o * o, T, v2, ab, ops.v2p), "pad T2");
  f.pair = p;
  f.ab = ab;
  return f;
}

// One occupied triplet of the sweep: indices, weight (cc_triples.jl:62-72) and
// the denominator shift e_i + e_j + e_k.
struct Trip {
  int i, j, k;
  double f, eijk;
};

// Items of the K builds, [orientation][triplet]: the operand items of the four
// segments (alike for FP64 arrays and BF16 stacks) and the K slot.
std::vector<dev::KbItem> k_items(Ctx& c, const std::vector<Trip>& tr, int NB,
                                 int64_t kstride) {
  const int64_t o = c.no, nt = (int64_t)tr.size();
  std::vector<dev::KbItem> items(kGemms * nt);
  for (int64_t t = 0; t < nt; ++t) {
    const int i = tr[t].i, j = tr[t].j, k = tr[t].k;
    PermW P[6];
    perm_table(i, j, k, P);
    auto on = [&](int y, int z) { return (int32_t)(y + o * z); };
    // ovoo segments: the occupied index of the T2 slices (see build_K_batch)
    // and the pair of -ovoo
    const int32_t ov[3][4] = {{k, j, on(j, i), on(k, i)},
                              {i, k, on(k, j), on(i, j)},
                              {i, j, on(j, k), on(i, k)}};
    for (int q = 0; q < kGemms; ++q) {
      const PermW &p0 = P[kPairs[q][0]], &p1 = P[kPairs[q][1]];
      items[q * nt + t] = {{p0.z, p1.z, ov[q][0], ov[q][1]},
                           {(int32_t)(p0.x + o * p0.y), (int32_t)(p1.x + o * p1.y), ov[q][2],
                            ov[q][3]},
                           (t % NB) * kstride};
    }
  }
  return items;
}

// K^{ijk} = P[W] for triplets t0 .. t0+nb-1 into K slots 0 .. nb-1 (FP64 or
// FP32), one launch per K orientation.
void build_K_batch(Ctx& c, const TriplesOps& ops, const FpAmps& F, const SplitAmps& S,
                   const dev::KbItem* items, int64_t nt, int64_t t0, int nb, void* K,
                   int64_t kstride, int64_t vp) {
  const int64_t o = c.no, v = c.nv, v2 = v * v;
  dev::stream_t s = c.st;
  PermW P[6];
  perm_table(0, 0, 0, P);  // the layouts do not depend on i, j, k
  if (!ops.mixed) {
    const int64_t v2p = ops.v2p, vq = ops.vq;
    const dev::KbOperand V1{ops.V1, v2, v2p, o, v2p * v}, V2{ops.V2, v2, v2p, o, v2p * v};
    const dev::KbOperand Tp{F.pair, v, vq, o * o, vq * v};
    const dev::KbOperand G{F.ab, v2, v2p * o, o, v2p};  // T2[:,:,x,l]: k = l, item x
    const dev::KbOperand C{F.ab, v2, v2p, o, v2p * o};  // T2[:,:,l,x]
    const dev::KbOperand On{ops.On, v, vq, o * o, vq * o};
    // T2 slices of the two ovoo segments: rows (b,c), (a,c) and (a,b) of K
    const dev::KbOperand* ab[kGemms][2] = {{&C, &G}, {&G, &C}, {&G, &C}};
    for (int q = 0; q < kGemms; ++q) {
      const PermW &p0 = P[kPairs[q][0]], &p1 = P[kPairs[q][1]];
      dev::KbGemm g;
      g.m = v2; g.n = v; g.nseg = 4;
      g.k[0] = g.k[1] = v; g.k[2] = g.k[3] = o;
      g.A[0] = p0.l2 ? V2 : V1; g.A[1] = p1.l2 ? V2 : V1;
      g.A[2] = *ab[q][0]; g.A[3] = *ab[q][1];
      g.B[0] = g.B[1] = Tp; g.B[2] = g.B[3] = On;
      g.beta = q ? 1.0 : 0.0;
      g.C = (double*)K;
      const KMap m = k_map(q, v, vp);
      g.scm = m.scm; g.dm = m.dm; g.scm2 = m.scm2; g.scn = m.scn;
      g.even_items = kstride % 2 == 0;
      check(dev::kbuild(s, g, nb, items + q * nt + t0), "W");
    }
    return;
  }
  const dev::TcStack* ab[kGemms][2] = {{&S.C, &S.G}, {&S.G, &S.C}, {&S.G, &S.C}};
  for (int q = 0; q < kGemms; ++q) {
    const PermW &p0 = P[kPairs[q][0]], &p1 = P[kPairs[q][1]];
    dev::TcKbuild g;
    g.m = v2; g.n = v; g.nseg = 4;
    g.A[0] = p0.l2 ? ops.V2s : ops.V1s; g.A[1] = p1.l2 ? ops.V2s : ops.V1s;
    g.A[2] = *ab[q][0]; g.A[3] = *ab[q][1];
    g.B[0] = g.B[1] = S.pair; g.B[2] = g.B[3] = ops.Ons;
    g.beta = q > 0;
    g.C = (float*)K;
    const KMap m = k_map(q, v, vp);
    g.scm = m.scm; g.dm = m.dm; g.scm2 = m.scm2; g.scn = m.scn;
    g.pad4 = vp % 4 == 0 && kstride % 4 == 0;
    check(dev::tc_kbuild(s, g, nb, items + q * nt + t0, kChunk), "W");
  }
}

}  // namespace

void pert_triples(Ctx& c, const double* U1h, const double* U2h, double* et, double* etb) {
  const int64_t o = c.no, v = c.nv, v2 = v * v, v3 = v2 * v, n = c.n;
  const bool lam = (U1h != nullptr);
  const bool mixed = c.mixed_active;
  dev::stream_t s = c.st;
  if (o < 2) {  // no triplet
    *et = *etb = 0.0;
    return;
  }
  // everything allocated here is freed on exit
  struct Scope {
    Ctx& c;
    size_t n0;
    ~Scope() { c.release_to(n0); }
  } scope{c, c.allocs.size()};

  TriplesOps ops;
  ops.mixed = mixed;
  ops.vq = (v + 1) / 2 * 2;
  ops.v2p = (v2 + 1) / 2 * 2;
  Contractor con = c.con();
  // vvvo[b,c,d,k] = (bd|ck): per k one GEMM over rows (b,d) into a slab
  // [b,d,c], whose orders [b,c,d] and [c,b,d] the K builds read
  const int64_t d3[3] = {v, v, v};
  const int bcd[3] = {0, 2, 1}, cbd[3] = {2, 0, 1};
  const bool pad = ops.v2p != v2;  // odd v: factors and integrals in an even pitch
  uint16_t *bv = nullptr, *bo = nullptr;
  double *V1 = nullptr, *V2 = nullptr, *Onp = nullptr;
  const size_t evs = dev::tc_operand_elems(v2, v, kTriplesSlices);
  const size_t eos = dev::tc_operand_elems(v, o, kTriplesSlices);
  const int64_t slab = ops.v2p * v;
  if (mixed) {
    bv = alloc_bf16(c, 2 * evs * o, "(T) vvvo BF16");
    bo = alloc_bf16(c, eos * o * o, "(T) ovoo BF16");
  } else {
    V1 = c.alloc(slab * o, "(T) vvvo [b,c,d,k]");
    V2 = c.alloc(slab * o, "(T) vvvo [c,b,d,k]");
    Onp = c.alloc(ops.vq * o * o * o, "(T) -ovoo");
  }
  // -ovoo: the ovoo segments share the vvvo segments' sign
  const size_t mark = c.allocs.size();
  double* On = c.alloc(o * o * o * v, "(T) ovoo");
  con(1.0, c.Boo, "ljQ", c.Bvo, "ckQ", 0.0, On, "ljck");
  if (mixed) {
    check(dev::axpby(s, o * o * o * v, -1.0, On, 0.0, On), "-ovoo");
    check(dev::tc_split_stack(s, On, v, o, o * o, 1, 0, o * o, o, o, o * o * v, bo, &ops.Ons),
          "split ovoo");
  } else {  // as [c,l,j,k]
    const int64_t dl[4] = {o, o, v, o};
    const int pl[4] = {2, 0, 1, 3};
    double* Oc = c.alloc(o * o * o * v, "(T) ovoo [c,l,j,k]");
    check(dev::permute(s, 4, dl, pl, -1.0, On, 0.0, Oc), "-ovoo");
    check(dev::repitch(s, v, o * o * o, Oc, v, Onp, ops.vq), "-ovoo pitch");
  }
  c.release_to(mark);
  double* D = c.alloc(v3, "(T) vvvo slab");
  double* Dt = mixed || pad ? c.alloc(v3, "(T) vvvo slab") : nullptr;
  const double* Bl = c.Bvv;
  if (pad) {
    double* t = c.alloc(ops.v2p * c.nq, "(T) padded Bvv");
    check(dev::repitch(s, v2, c.nq, c.Bvv, v2, t, ops.v2p), "pad Bvv");
    Bl = t;
  }
  for (int64_t kk = 0; kk < o; ++kk) {
    dev::Gemm g;
    g.m = v2; g.n = v; g.k = c.nq;
    g.A = Bl; g.sam = 1; g.sak = ops.v2p;
    g.B = c.Bvo + v * kk; g.sbn = 1; g.sbk = v * o;
    g.C = D; g.scn = v2;
    check(dev::gemm_strided(s, g), "vvvo");
    if (mixed) {
      check(dev::tc_split_stack(s, D, v2, v, v2, v, v, 1, 1, 0, 0, bv + evs * kk, &ops.V1s),
            "split vvvo");
      check(dev::permute(s, 3, d3, cbd, 1.0, D, 0.0, Dt), "vvvo perm");
      check(dev::tc_split_stack(s, Dt, v2, v, 1, v2, 0, 1, 1, 0, 0, bv + evs * (o + kk),
                                &ops.V2s),
            "split vvvo");
      continue;
    }
    for (int w = 0; w < 2; ++w) {
      double* V = (w ? V2 : V1) + slab * kk;
      check(dev::permute(s, 3, d3, w ? cbd : bcd, 1.0, D, 0.0, pad ? Dt : V), "vvvo perm");
      if (pad) check(dev::repitch(s, v2, v, Dt, v2, V, ops.v2p), "pad vvvo");
    }
  }
  if (mixed) {
    ops.V1s.base = bv;
    ops.V2s.base = bv + evs * o;
    ops.V1s.items = ops.V2s.items = o;
  } else {
    ops.V1 = V1;
    ops.V2 = V2;
    ops.On = Onp;
  }
  c.release_to(mark);

  double* U2c = nullptr;
  if (lam) {
    double* U2 = c.alloc(c.n2(), "(T) U2");
    U2c = c.alloc(c.n2(), "(T) U2 covariant");
    check(dev::h2d(U2, U2h, c.n2() * 8, s), "h2d U2");
    // contra2covariant (cctools.jl:935-938): (2 U2[a,b,i,j] + U2[b,a,i,j]) / 3
    check(dev::axpby(s, c.n2(), 2.0 / 3.0, U2, 0.0, U2c), "U2c");
    con.permute(1.0 / 3.0, U2, "baij", 1.0, U2c, "abij");
  }
  SplitAmps ST, SU;
  FpAmps FT, FU;
  if (!mixed) {
    FT = fp_amps(c, c.T2(), ops);
    if (lam) FU = fp_amps(c, U2c, ops);
  }
  if (mixed) {
    split_amps(c, c.T2(), ST);
    if (lam) split_amps(c, U2c, SU);
  }

  // the sweep: triplet weights of cc_triples.jl:62-72, taken in blocks of (i, j)
  // that share integrals; energies are summed in the reference's order (k, j,
  // i outermost first)
  const double* eps = c.fock_host.data();
  std::vector<Trip> tr;
  for (int k = 0; k < o; ++k)
    for (int j0 = 0; j0 <= k; j0 += kBlockJ)
      for (int i0 = 0; i0 <= std::min(j0 + kBlockJ - 1, k); i0 += kBlockI)
        for (int j = j0; j < std::min(j0 + kBlockJ, k + 1); ++j)
          for (int i = i0; i < std::min(i0 + kBlockI, j + 1); ++i) {
            if (i == j && j == k) continue;
            const double f = (i == j) ? 1.0 : (j == k ? 1.0 : 2.0);
            tr.push_back({i, j, k, f, eps[i + i * n] + eps[j + j * n] + eps[k + k * n]});
          }
  const int64_t nt = (int64_t)tr.size();
  // batches of NB triplets, one K slot each, within a 4 GiB budget (fewer where
  // memory ends before: see the allocation of K)
  const int64_t esz = mixed ? 4 : 8;
  const int64_t vp = mixed ? (v + 3) / 4 * 4 : v;  // K's a pitch (see k_map)
  const int64_t kstride = (vp * v2 + 31) / 32 * 32;
  const int64_t per = kstride * esz * (lam ? 2 : 1);
  int64_t nbmax = std::min<int64_t>({256, nt, ((int64_t)4 << 30) / per});
  if (c.triples_batch > 0) nbmax = std::min(nbmax, c.triples_batch);
  int NB = (int)std::max<int64_t>(1, nbmax);

  // energy terms per triplet: g = T1 (or U1/2), f[a,i] = fock[i, o+a], <ij|ab>, T2 (or U2c)
  std::vector<double> gh(v * o), fh(v * o);
  {
    std::vector<double> T1h(v * o);
    if (!lam) {
      check(dev::d2h(T1h.data(), c.T1(), v * o * 8, s), "d2h");
      check(dev::sync(s), "sync");
    }
    for (int64_t i = 0; i < o; ++i)
      for (int64_t a = 0; a < v; ++a) {
        gh[a + v * i] = lam ? 0.5 * U1h[a + v * i] : T1h[a + v * i];
        fh[a + v * i] = c.fock_host[i + (o + a) * n];
      }
  }
  double* gf = c.alloc(2 * v * o, "(T) singles/Fock vectors");
  check(dev::h2d(gf, gh.data(), v * o * 8, s), "h2d");
  check(dev::h2d(gf + v * o, fh.data(), v * o * 8, s), "h2d");
  const double* Nsrc = lam ? U2c : c.T2();
  std::vector<double> eijk(nt);
  for (int64_t t = 0; t < nt; ++t) eijk[t] = tr[t].eijk;
  double* eijk_d = c.alloc(nt, "(T) denominators");
  check(dev::h2d(eijk_d, eijk.data(), nt * 8, s), "h2d");
  // energy terms per triplet.  FP64: g, f, M = <ij|ab>, N = T2 (or U2c) as
  // separate arrays.  Mixed precision: FP32 copies interleaved in pairs,
  // (g, f)[a] per occupied index and (M, N)[a + v b] per occupied pair, which
  // the FP32 energy kernel stages with one 8-byte copy per position (they
  // enter only the singles/Fock term sum X Y).
  dev::TriplesTerms* terms_d = nullptr;
  dev::TriplesTermsF* termsf_d = nullptr;
  float* MNp = nullptr;
  float* MNt = nullptr;
  if (mixed) {
    float* GF = reinterpret_cast<float*>(c.alloc(v * o, "(T) FP32 (g, f)"));  // float2 [occ][a]
    const int64_t mne = dev::triples_mn_elems((int)v, o * o);
    MNp = reinterpret_cast<float*>(c.alloc(mne, "(T) FP32 (M, N)"));
    MNt = reinterpret_cast<float*>(c.alloc(mne, "(T) FP32 (M, N) transposed"));
    check(dev::to_f32_pairs(s, v * o, gf, gf + v * o, GF), "FP32 (g, f)");
    check(dev::triples_mn_pack(s, (int)v, o * o, c.Kvvoo, Nsrc, MNp, MNt),
          "FP32 (<ij|ab>, amplitudes)");
    auto gfp = [&](int x) { return static_cast<const void*>(GF + 2 * v * x); };
    std::vector<dev::TriplesTermsF> terms(nt);
    for (int64_t t = 0; t < nt; ++t) {
      const int i = tr[t].i, j = tr[t].j, k = tr[t].k;
      dev::TriplesTermsF& tt = terms[t];
      tt.gf[0] = gfp(i); tt.gf[1] = gfp(j); tt.gf[2] = gfp(k);
      tt.mnpair[0] = (int32_t)(j + o * k);
      tt.mnpair[1] = (int32_t)(i + o * k);
      tt.mnpair[2] = (int32_t)(i + o * j);
    }
    termsf_d = reinterpret_cast<dev::TriplesTermsF*>(
        c.alloc((int64_t)((nt * sizeof(dev::TriplesTermsF) + 7) / 8), "(T) energy terms"));
    check(dev::h2d(termsf_d, terms.data(), nt * sizeof(dev::TriplesTermsF), s), "h2d");
  } else {
    auto at = [&](const double* p, int64_t off) { return static_cast<const void*>(p + off); };
    auto M = [&](int x, int y) { return at(c.Kvvoo, v2 * (x + o * y)); };
    auto N = [&](int x, int y) { return at(Nsrc, v2 * (x + o * y)); };
    std::vector<dev::TriplesTerms> terms(nt);
    for (int64_t t = 0; t < nt; ++t) {
      const int i = tr[t].i, j = tr[t].j, k = tr[t].k;
      dev::TriplesTerms& tt = terms[t];
      tt.g[0] = at(gf, v * i); tt.g[1] = at(gf, v * j); tt.g[2] = at(gf, v * k);
      tt.f[0] = at(gf, v * (o + i)); tt.f[1] = at(gf, v * (o + j)); tt.f[2] = at(gf, v * (o + k));
      tt.M[0] = M(j, k); tt.M[1] = M(i, k); tt.M[2] = M(i, j);
      tt.N[0] = N(j, k); tt.N[1] = N(i, k); tt.N[2] = N(i, j);
    }
    terms_d = reinterpret_cast<dev::TriplesTerms*>(
        c.alloc((int64_t)((nt * sizeof(dev::TriplesTerms) + 7) / 8), "(T) energy terms"));
    check(dev::h2d(terms_d, terms.data(), nt * sizeof(dev::TriplesTerms), s), "h2d");
  }
  const int64_t ncube = dev::triples_cube_count((int)v);
  std::vector<int> trih(3 * ncube);
  dev::triples_cube_table((int)v, trih.data());
  int* tri = reinterpret_cast<int*>(c.alloc((3 * ncube + 1) / 2, "(T) cube table"));
  check(dev::h2d(tri, trih.data(), 3 * ncube * sizeof(int), s), "h2d");
  double* part = c.alloc(dev::triples_energy_scratch_len((int)v, NB), "(T) partial sums");
  double* Et = c.alloc(2 * nt, "(T) energies");
  static_assert(sizeof(dev::KbItem) % 8 == 0, "whole doubles");
  dev::KbItem* items_d = reinterpret_cast<dev::KbItem*>(
      c.alloc((int64_t)(kGemms * nt * sizeof(dev::KbItem) / 8), "(T) item table"));
  void *K = nullptr, *KU = nullptr;
  while (!K) {
    const size_t slots = c.allocs.size();
    try {
      void* k = c.alloc((NB * kstride * esz + 7) / 8, "(T) K slots");
      if (lam) KU = c.alloc((NB * kstride * esz + 7) / 8, "(T) K(Lambda) slots");
      K = k;
    } catch (const Error& e) {
      c.release_to(slots);
      if (e.code != ECG_ERR_OOM || NB == 1) throw;
      NB /= 2;
    }
  }
  const std::vector<dev::KbItem> items = k_items(c, tr, NB, kstride);
  check(dev::h2d(items_d, items.data(), items.size() * sizeof(dev::KbItem), s), "h2d");

  // batch loop: the first batch runs directly (first-use set-up of the
  // kernels), the others are recorded as one CUDA graph and run once
  const int64_t nbatch = (nt + NB - 1) / NB;
  try {
    for (int64_t bi = 0; bi < nbatch; ++bi) {
      if (bi == 1) check(dev::graph_capture_begin(s), "graph capture");
      const int64_t t0 = bi * NB;
      const int nb = (int)std::min<int64_t>(NB, nt - t0);
      build_K_batch(c, ops, FT, ST, items_d, nt, t0, nb, K, kstride, vp);
      if (lam) build_K_batch(c, ops, FU, SU, items_d, nt, t0, nb, KU, kstride, vp);
      if (mixed)
        check(dev::triples_energy_f32_batched(s, (int)v, (int)vp, nb, NB,
                                              static_cast<const float*>(K),
                                              static_cast<const float*>(KU), kstride, MNp, MNt,
                                              o * o, eijk_d + t0, c.eps + o, termsf_d + t0, tri,
                                              part, Et + 2 * t0),
              "triples energy");
      else
        check(dev::triples_energy_batched(s, (int)v, nb, K, KU, kstride, false, eijk_d + t0,
                                          c.eps + o, terms_d + t0, tri, part, Et + 2 * t0),
              "triples energy");
    }
    if (nbatch > 1) {
      int64_t nodes = 0;
      check(dev::graph_capture_run(s, &nodes), "(T) graph");
    }
  } catch (...) {
    dev::graph_capture_abort(s);
    throw;
  }
  std::vector<double> Eh(2 * nt);
  check(dev::d2h(Eh.data(), Et, 2 * nt * 8, s), "d2h");
  sync_checked(c);
  // sum K X, and the singles / Fock term sum X Y (cc_triples.jl:143-156 / :286-294)
  double Enb3 = 0.0, Esf = 0.0;
  std::vector<int64_t> order(nt);
  for (int64_t q = 0; q < nt; ++q) order[q] = q;
  std::sort(order.begin(), order.end(), [&](int64_t x, int64_t y) {
    return std::tie(tr[x].k, tr[x].j, tr[x].i) < std::tie(tr[y].k, tr[y].j, tr[y].i);
  });
  for (int64_t q : order) {
    Enb3 += tr[q].f * Eh[2 * q];
    Esf += tr[q].f * Eh[2 * q + 1];
  }
  const double En3 = Enb3 + Esf;
  if (!std::isfinite(En3)) throw Error(ECG_ERR_NONFINITE, "non-finite (T) energy");
  *et = En3;
  *etb = Enb3;
}

}  // namespace ecg
