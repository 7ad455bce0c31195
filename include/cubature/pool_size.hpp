// pool_size.hpp -- how much device memory the second phase's pools may take.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace cubature {

// What is known of a device about the pools (per workspace, until its memory
// is released).
struct PoolBound {
  size_t share = 0;           // an eighth of the memory free when first asked
  size_t refused = SIZE_MAX;  // the least that could not be allocated
};

// Blocks to make the pools for: `want` of them would fill the chip and a block
// takes block_bytes.  At the default 2048 bisections all of them fit an eighth
// of an idle device's memory; with a higher limit (65 536: 105 GB) or less
// memory free the pools stay within that eighth, so that the region lists and
// the caller keep theirs -- but for the `least` blocks that a warp per box
// would have in flight, which may take up to half.  A size that was refused
// is not asked for again, nor is a larger one.  At least 1.
inline long long pool_blocks(long long want, long long least, size_t block_bytes,
                             const PoolBound& b) {
  const double least_bytes = (double)least * (double)block_bytes;
  const double bytes = std::max((double)b.share, std::min(least_bytes, 4.0 * (double)b.share));
  long long n = std::min(want, (long long)(bytes / (double)block_bytes));
  while (n > 1 && (double)n * (double)block_bytes >= (double)b.refused) n /= 2;
  return std::max<long long>(n, 1);
}

}  // namespace cubature
