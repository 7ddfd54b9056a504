// Values that CTAs of one launch hand to each other while it runs: self-validating packets of 32 bits of data and a
// 32-bit epoch per 64-bit word (FP64: two words per value), so data and its arrival travel in one store and one load.
// A reader repeats the load until the epochs match; the number of repetitions is bounded, and a reader that gives up
// sets *fail, which ends the other waits too, and carries on.
#pragma once
#include <cstdint>

namespace bsgpu {

constexpr unsigned kSpinLimit = 1u << 24;  // polls of a wait (several seconds)

__device__ __forceinline__ void st_words(uint64_t* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void st_word(uint64_t* p, uint64_t a) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}
__device__ __forceinline__ void ld_words(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ uint64_t ld_word(const uint64_t* p) {
  uint64_t a;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return a;
}
__device__ __forceinline__ void put_packet(uint64_t* w, double v, unsigned ep) {
  const uint64_t bits = (uint64_t)__double_as_longlong(v), e = (uint64_t)ep << 32;
  st_words(w, e | (bits & 0xffffffffull), e | (bits >> 32));
}
__device__ __forceinline__ void put_packet(uint64_t* w, float v, unsigned ep) {
  st_word(w, ((uint64_t)ep << 32) | (uint64_t)__float_as_uint(v));
}
__device__ __forceinline__ double packet_double(uint64_t lo, uint64_t hi) {
  return __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
}
__device__ __forceinline__ bool packet_is(uint64_t w, unsigned ep) { return (unsigned)(w >> 32) == ep; }

// true: give up waiting
__device__ __forceinline__ bool spin_over(unsigned& n, unsigned int* fail) {
  if ((++n & 255u) != 0) return false;
  unsigned f;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(fail) : "memory");
  if (f) return true;
  if (n < kSpinLimit) return false;
  atomicExch(fail, 1u);
  return true;
}

// waits for one value
__device__ __forceinline__ double get_packet(const uint64_t* w, unsigned ep, unsigned int* fail, double) {
  uint64_t lo, hi;
  unsigned n = 0;
  do {
    ld_words(w, lo, hi);
  } while (!(packet_is(lo, ep) && packet_is(hi, ep)) && !spin_over(n, fail));
  return packet_double(lo, hi);
}
__device__ __forceinline__ float get_packet(const uint64_t* w, unsigned ep, unsigned int* fail, float) {
  uint64_t a;
  unsigned n = 0;
  do {
    a = ld_word(w);
  } while (!packet_is(a, ep) && !spin_over(n, fail));
  return __uint_as_float((unsigned)a);
}

}  // namespace bsgpu
