// tgmm_div.cuh -- unsigned division of a 32-bit number by a number known on the host, as a
// multiply-high and shifts (Granlund and Montgomery's method; exact for every 32-bit numerator).
#pragma once

#include <stdint.h>

namespace tgmm {

// The magic number m and the shift l of the division by d (1 <= d < 2^32): l = ceil(log2 d),
// m = floor(2^32 (2^l - d) / d) + 1.
inline void div_magic(uint32_t d, uint32_t* m, int32_t* l) {
  int32_t k = 0;
  while (((uint64_t)1 << k) < d) k++;
  *m = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << k) - d)) / d + 1);
  *l = k;
}

__device__ __forceinline__ uint32_t div_by_magic(uint32_t n, uint32_t m, int32_t l) {
  const uint32_t t = __umulhi(n, m);
  return l == 0 ? n : (t + ((n - t) >> 1)) >> (l - 1);
}

}  // namespace tgmm
