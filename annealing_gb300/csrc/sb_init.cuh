// The counter hash of every seeded draw, and the hash-mode initial state of the plain and the grouped kernels.
#pragma once
#include <stdint.h>

namespace sbk {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z ^= z >> 30;
  z *= 0xBF58476D1CE4E5B9ULL;
  z ^= z >> 27;
  z *= 0x94D049BB133111EBULL;
  z ^= z >> 31;
  return z;
}

__device__ __forceinline__ float uniform_value(uint64_t seed, uint64_t e) {
  const uint64_t z = mix64(seed + 0x9E3779B97F4A7C15ULL * (e + 1));
  const uint32_t u = (uint32_t)(z >> 40);
  const float f = __fmul_rn((float)u, 5.9604644775390625e-08f);
  const float t = __fadd_rn(__fmul_rn(f, 2.0f), -1.0f);
  return __fmul_rn(t, 0.1f);
}

}  // namespace sbk
