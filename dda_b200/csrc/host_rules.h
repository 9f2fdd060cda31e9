// host_rules.h -- rules of the host side that need no device: what an
// allocation shrinks to.
#pragma once

#include <algorithm>
#include <cstddef>

namespace dda {

// The first of want, want / 2, want / 4, ..., least that alloc(bytes) takes;
// 0 when it refuses the least too.
template <typename F> size_t shrink_to_fit(size_t want, size_t least, F&& alloc) {
  for (size_t bytes = want;; bytes = std::max(least, bytes / 2)) {
    if (alloc(bytes)) return bytes;
    if (bytes <= least) return 0;
  }
}

}  // namespace dda
