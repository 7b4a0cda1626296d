// extent.h -- whether a buffer lies inside an allocation.
#pragma once

#include <cstddef>
#include <cstdint>

namespace glasma {

// [p, p + bytes) within [base, base + size), without forming either end (which might wrap)
inline bool extent_holds(uintptr_t base, size_t size, uintptr_t p, size_t bytes) {
  return p >= base && p - base <= size && bytes <= size - (p - base);
}

}  // namespace glasma
