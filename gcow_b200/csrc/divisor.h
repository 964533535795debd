// Division by a number that a launch knows and the compiler does not, as one multiplication: exact for numbers below 2^31.
// With 2^(s - 1) < d <= 2^s, mul = floor(2^(31 + s) / d) + 1 fits 32 bits and b mul / 2^(31 + s) exceeds b / d by at most b / 2^(31 + s), which
// for b < 2^31 is less than 1 / d: the quotient is exact.
#pragma once
#include <stdint.h>

namespace gcow {

struct Divisor {
  uint32_t mul, shift;
#if defined(__CUDACC__)
  __host__ __device__ __forceinline__
#else
  inline
#endif
  uint32_t under(uint32_t b) const {                           // b / d
#if defined(__CUDA_ARCH__)
    return __umulhi(2u * b, mul) >> shift;
#else
    return (uint32_t)((2ull * b * mul) >> 32) >> shift;
#endif
  }
};
inline Divisor divisor(uint32_t d) {                           // d > 0
  uint32_t s = 0;
  while ((1ull << s) < d) s++;
  return {(uint32_t)((1ull << (31 + s)) / d + 1), s};
}

}  // namespace gcow
