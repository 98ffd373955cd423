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

// a-block size of the symmetric ladder: Vblk holds v^2 na (v - a0) doubles.
// An eighth of the virtual space, but as much of it as 256 MiB of V hold: at
// small v a block's five launches cost more than they compute (CCSD iteration
// of o=12, v=57 with 256 / 64 / 32 MiB: 1.76 / 1.80 / 1.84 ms, eight blocks
// 2.01; o=14, v=100: 5.78 / 5.97 / 5.98, eight blocks 6.05), and the tiles with
// b < a are skipped inside a block.
inline int64_t ladder_na(int64_t nv) {
  int64_t na = ((nv + 7) / 8 + 1) / 2 * 2;
  na = std::max(na, ((int64_t)1 << 25) / (nv * nv * nv));
  na = std::max<int64_t>(1, std::min({na, ladder_na_limit(nv), nv}));
  // an even block start keeps the block's rows of B on 16 bytes for TMA
  return na < nv && na > 1 ? na - na % 2 : na;
}

}  // namespace ecg
