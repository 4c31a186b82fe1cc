// Division by a divisor that is known at launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace moba {

// x / d for 0 <= x < 2^31 as a product: the upper half of 2 x mul, >> shift, with mul = ceil(2^(31 + shift) / d) and 2^shift >= d.  mul d
// exceeds 2^(31 + shift) by less than d, and x times that stays below 2^(31 + shift): the quotient is never one too large.
struct FastDiv {
  uint32_t mul, shift;
};
inline FastDiv fast_div(int64_t d) {
  FastDiv f{0, 0};
  while ((1ll << f.shift) < d) ++f.shift;
  f.mul = (uint32_t)(((1ull << (31 + f.shift)) + (uint64_t)d - 1) / (uint64_t)d);
  return f;
}
__host__ __device__ __forceinline__ int operator/(int x, const FastDiv& f) {
#if defined(__CUDA_ARCH__)
  return (int)(__umulhi(2u * (uint32_t)x, f.mul) >> f.shift);
#else
  return (int)((uint32_t)(((uint64_t)(2u * (uint32_t)x) * f.mul) >> 32) >> f.shift);
#endif
}

}  // namespace moba
