// tsu_half2.cuh -- pairs of 16-bit values in one 32-bit word: per-halfword
// add-max, add-min, maxima and minima (DPX and SIMD intrinsics, 0.5 warp
// instructions per cycle and scheduler each, as plain integer ones), and the
// small pieces the kernels need around them; in plain C++ for the CPU warp
// emulation of the tests.
#pragma once

#include <algorithm>
#include <cstdint>

namespace tsu {

#ifdef TSU_WARP_EMU
template <class F>
inline uint32_t h2_each(uint32_t a, uint32_t b, uint32_t c, F f) {
  const uint16_t lo = f((uint16_t)a, (uint16_t)b, (uint16_t)c);
  const uint16_t hi = f((uint16_t)(a >> 16), (uint16_t)(b >> 16), (uint16_t)(c >> 16));
  return (uint32_t)lo | ((uint32_t)hi << 16);
}
inline uint32_t h2_addmax(uint32_t a, uint32_t b, uint32_t c) {
  return h2_each(a, b, c, [](uint16_t x, uint16_t y, uint16_t z) { return std::max<uint16_t>((uint16_t)(x + y), z); });
}
inline uint32_t h2_addmin(uint32_t a, uint32_t b, uint32_t c) {
  return h2_each(a, b, c, [](uint16_t x, uint16_t y, uint16_t z) { return std::min<uint16_t>((uint16_t)(x + y), z); });
}
inline uint32_t h2s_add(uint32_t a, uint32_t b) {
  return h2_each(a, b, 0, [](uint16_t x, uint16_t y, uint16_t) { return (uint16_t)(x + y); });
}
inline uint32_t h2s_max(uint32_t a, uint32_t b) {
  return h2_each(a, b, 0, [](uint16_t x, uint16_t y, uint16_t) { return (uint16_t)std::max((int16_t)x, (int16_t)y); });
}
inline uint32_t h2s_min(uint32_t a, uint32_t b) {
  return h2_each(a, b, 0, [](uint16_t x, uint16_t y, uint16_t) { return (uint16_t)std::min((int16_t)x, (int16_t)y); });
}
inline uint32_t h2_max(uint32_t a, uint32_t b) { return h2_addmax(a, 0, b); }
inline uint32_t h2_min(uint32_t a, uint32_t b) { return h2_addmin(a, 0, b); }
inline uint32_t h2_next(uint32_t a, uint32_t b) { return (a >> 16) | (b << 16); }
inline uint32_t h2_signmask(uint32_t a) { return ((a & 0x8000u) ? 0xffffu : 0u) | ((a & 0x80000000u) ? 0xffff0000u : 0u); }
inline int h2_tz(uint32_t d) { return d ? __builtin_ctz(d) : 32; }
inline uint32_t h2_sum(uint32_t a, uint32_t acc) { return acc + (a & 0xffffu) + (a >> 16); }
#else
// max(a + b, c), min(a + b, c) per halfword, the sum modulo 2^16
__device__ __forceinline__ uint32_t h2_addmax(uint32_t a, uint32_t b, uint32_t c) { return __viaddmax_u16x2(a, b, c); }
__device__ __forceinline__ uint32_t h2_addmin(uint32_t a, uint32_t b, uint32_t c) { return __viaddmin_u16x2(a, b, c); }
// sum modulo 2^16, signed maximum and minimum
__device__ __forceinline__ uint32_t h2s_add(uint32_t a, uint32_t b) { return __vadd2(a, b); }
__device__ __forceinline__ uint32_t h2s_max(uint32_t a, uint32_t b) { return __vmaxs2(a, b); }
__device__ __forceinline__ uint32_t h2s_min(uint32_t a, uint32_t b) { return __vmins2(a, b); }
__device__ __forceinline__ uint32_t h2_max(uint32_t a, uint32_t b) { return __vmaxu2(a, b); }
__device__ __forceinline__ uint32_t h2_min(uint32_t a, uint32_t b) { return __vminu2(a, b); }
// (high half of a, low half of b)
__device__ __forceinline__ uint32_t h2_next(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5432); }
// 0xffff in each half whose bit 15 is set (prmt replicates the sign of bytes 1 and 3)
__device__ __forceinline__ uint32_t h2_signmask(uint32_t a) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %1, 0xbb99;" : "=r"(r) : "r"(a));
  return r;
}
// trailing zero bits, 32 for 0
__device__ __forceinline__ int h2_tz(uint32_t d) { return __clz((int)__brev(d)); }
// acc + both halves (unsigned: twice the bases of a match run, up to 40,926)
__device__ __forceinline__ uint32_t h2_sum(uint32_t a, uint32_t acc) { return __dp2a_lo(a, 0x0101u, acc); }
#endif
__device__ __forceinline__ uint32_t h2_dup(uint32_t v) { return (v & 0xffffu) * 0x10001u; }

}  // namespace tsu
