// Packed fp32 arithmetic: two values in a 64-bit register, one issue slot an
// instruction, each rounded to nearest like the single-precision instruction.
#pragma once

#include <stdint.h>

namespace lime {
namespace x2 {

__device__ __forceinline__ uint64_t pack(float a, float b) {
  return (uint64_t)__float_as_uint(b) << 32 | __float_as_uint(a);
}
__device__ __forceinline__ void unpack(uint64_t p, float& a, float& b) {
  a = __uint_as_float((uint32_t)p);
  b = __uint_as_float((uint32_t)(p >> 32));
}
__device__ __forceinline__ uint64_t both(float a) { return pack(a, a); }
__device__ __forceinline__ uint64_t add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a - b = a + (-1) b, rounded once
__device__ __forceinline__ uint64_t sub(uint64_t a, uint64_t b) { return fma(b, 0xBF800000BF800000ull, a); }

}  // namespace x2
}  // namespace lime
