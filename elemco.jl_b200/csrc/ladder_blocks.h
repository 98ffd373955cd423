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

}  // namespace ecg
