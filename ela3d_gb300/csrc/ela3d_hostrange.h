// ela3d_hostrange.h -- whether an array lies whole inside one range of memory
// (host code without CUDA, so that it can be tested anywhere).
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace ela3d {

// All of [p, p + bytes) inside [start, start + size), bytes > 0.
inline bool range_holds(uint64_t start, uint64_t size, uint64_t p, uint64_t bytes) {
  return bytes > 0 && p >= start && p - start <= size && bytes <= size - (p - start);
}

}  // namespace ela3d
