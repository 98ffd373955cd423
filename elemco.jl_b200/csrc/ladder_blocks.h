// ladder_blocks.h — sizes of the symmetric ladder's a-blocks, in plain C++ so that
// the rules can be tested without a device.
#pragma once
#include <algorithm>
#include <cstdint>

namespace ecg {

// At most 2 GiB of V a block.
inline int64_t ladder_na_limit(int64_t nv) {
  return std::max<int64_t>(1, ((int64_t)1 << 28) / std::max<int64_t>(nv * nv * nv, 1));
}

// An eighth of the virtual space (the size that the precision rule goes by).
inline int64_t ladder_eighth(int64_t nv) {
  return std::max<int64_t>(1, std::min({(nv + 7) / 8, ladder_na_limit(nv), nv}));
}

// Pairs a <= b of the first block, which has the most of them.
inline int64_t ladder_pairs(int64_t nv, int64_t na) { return na * nv - na * (na - 1) / 2; }

// Whether the copy of B in an even pitch (odd nv, FP64) fits V+'s place, which a
// single block leaves free until V is built.
inline bool ladder_pad_in_vp(int64_t nv, int64_t nq, int64_t na) {
  return na == nv && (nv * nv + 1) * nq <= (nv * (nv + 1) / 2 + 1) / 2 * 2 * ladder_pairs(nv, na);
}

// Doubles of workspace that ladder() takes with blocks of na.
inline int64_t ladder_need(int64_t no, int64_t nv, int64_t nq, int64_t na) {
  auto get = [](int64_t n) { return (std::max<int64_t>(n, 1) + 31) / 32 * 32; };
  const int64_t cdp = nv * (nv + 1) / 2, cdm = nv * (nv - 1) / 2;
  const int64_t ijp = no * (no + 1) / 2, ijm = no * (no - 1) / 2;
  const int64_t ldp = (cdp + 1) / 2 * 2, ldm = std::max<int64_t>((cdm + 1) / 2 * 2, 2);
  const int64_t pp = ladder_pairs(nv, na);
  return get(ldp * ijp) + get(ldm * ijm) +
         get(std::max(na * nv * nv * nv, pp * (ijp + ijm))) + get(ldp * pp) + get(ldm * pp) +
         (nv % 2 && !ladder_pad_in_vp(nv, nq, na) ? get((nv * nv + 1) * nq) : 0);
}

// Doubles of workspace of a system.
inline int64_t system_workspace(int64_t no, int64_t nv, int64_t nq) {
  const int64_t n = no + nv, n2 = no * no * nv * nv;
  return 15 * n2 + 6 * nv * no * nq + 3 * nv * nv * nq + 2 * n * n * nq + 4 * no * no * no * no +
         3 * ladder_eighth(nv) * nv * nv * nv + 6 * n * n + (1 << 15);
}

// a-block size of the symmetric ladder: Vblk holds v^2 na (v - a0) doubles.
// An eighth of the virtual space, but as much of it as 256 MiB of V hold: at
// small v a block's five launches cost more than they compute (CCSD iteration
// of o=12, v=57 in one block 1.17 ms, in two 1.21; with slower ring terms 1.76
// and, in eight, 2.01; o=14, v=100 in four 5.78, in eight 6.05), and the tiles
// with b < a are skipped inside a block.  The workspace is what eight blocks and the
// other terms were given, and larger blocks take what of it is free beside the o^4
// and n^2 matrices that the callers keep: they take no more memory.  Blocks are
// then made alike (o=16, v=76: 38 + 38).
inline int64_t ladder_na(int64_t no, int64_t nv, int64_t nq) {
  const int64_t lim = std::min(ladder_na_limit(nv), nv), n = no + nv;
  const int64_t least = std::min(((nv + 7) / 8 + 1) / 2 * 2, lim);
  const int64_t kept = no * no * no * no + 4 * n * n + 1024;
  int64_t na = std::min(std::max(least, ((int64_t)1 << 25) / (nv * nv * nv)), lim);
  while (na > 1 && kept + ladder_need(no, nv, nq, na) > system_workspace(no, nv, nq)) --na;
  if (na >= nv) return nv;
  // an even block start keeps the block's rows of B on 16 bytes for TMA
  const int64_t nb = (nv + na - 1) / na, alike = ((nv + nb - 1) / nb + 1) / 2 * 2;
  if (alike <= na) return alike;
  return na > 1 ? na - na % 2 : na;
}

}  // namespace ecg
