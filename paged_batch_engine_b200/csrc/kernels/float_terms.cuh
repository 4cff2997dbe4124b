// Float32 numbers as three bfloat16 terms, x = h + m + l, for the tensor cores: they hold all of its 24 bits, two numbers a word.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace pbe {
constexpr float SMALLEST = 0x1p-102f;              // its last bit, 2^-125, is a bfloat16 number
constexpr float LARGEST = 0x1p47f;                 // a sum of 2^31 products of two such numbers stays below 2^127

// Are numbers zero, or of a size from SMALLEST to LARGEST?  Without a branch a number: the largest size and the smallest that is
// not zero, as integers (zero less one is the largest integer; infinities and what is no number are above LARGEST).
struct Sizes {
  uint32_t largest = 0, smallest = 0xffffffffu;
  __device__ __forceinline__ void add(float x) {
    const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
    largest = max(largest, u);
    smallest = min(smallest, u - 1u);
  }
  __device__ __forceinline__ bool whole() const {
    return largest <= __float_as_uint(LARGEST) && smallest >= __float_as_uint(SMALLEST) - 1u;
  }
};

// two numbers' next terms; what is left of them stays in x and y (exact: it has fewer bits than they had)
__device__ __forceinline__ uint32_t next_term(float& x, float& y) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&p);
  x -= __uint_as_float(w << 16);
  y -= __uint_as_float(w & 0xffff0000u);
  return w;
}
}  // namespace pbe
