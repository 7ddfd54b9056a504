// Values that CTAs of one launch hand to each other while it runs: self-validating packets of 32 bits of data and a
// 32-bit epoch per 64-bit word (FP64: two words per value), so data and its arrival travel in one store and one load.
// A reader repeats the load until the epochs match; the number of repetitions is bounded, and a warp that gives up
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

// A wait of single threads (true: give up), for code whose lanes go their own ways anyway.
__device__ __forceinline__ bool spin_over(unsigned& n, unsigned int* fail) {
  if ((++n & 255u) != 0) return false;
  unsigned f;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(fail) : "memory");
  if (f) return true;
  if (n < kSpinLimit) return false;
  atomicExch(fail, 1u);
  return true;
}

// A wait of whole warps: `poll` loads what a lane waits for and says whether it has arrived, and all lanes repeat it
// until all have what they need.  Lanes that wait on their own leave the warp diverged, and every shuffle after that
// costs a reconvergence: the ILU chain ran at 3.7 us per wavefront that way, 1.2 us with this.
template <class F>
__device__ __forceinline__ void warp_wait(unsigned int* fail, F&& poll) {
  unsigned n = 0;
  while (!__all_sync(0xffffffffu, poll())) {
    if ((++n & 255u) == 0) {
      unsigned f;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(fail) : "memory");
      if (n >= kSpinLimit) {
        atomicExch(fail, 1u);
        f = 1;
      }
      if (__any_sync(0xffffffffu, f != 0)) break;
    }
  }
}

// one value per lane that has a `w`
__device__ __forceinline__ bool load_packet(const uint64_t* w, unsigned ep, double& v) {
  uint64_t lo, hi;
  ld_words(w, lo, hi);
  v = packet_double(lo, hi);
  return packet_is(lo, ep) && packet_is(hi, ep);
}
__device__ __forceinline__ bool load_packet(const uint64_t* w, unsigned ep, float& v) {
  const uint64_t a = ld_word(w);
  v = __uint_as_float((unsigned)a);
  return packet_is(a, ep);
}

}  // namespace bsgpu
