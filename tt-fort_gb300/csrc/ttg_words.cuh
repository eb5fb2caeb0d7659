// Values handed between the CTAs of one resident (cooperative) grid through
// global memory without barriers or fences: each 32-bit half of a value travels
// in one 64-bit word together with the number of its exchange, so a reader
// knows from the word itself that it is there (64-bit accesses do not tear).
// Exchange numbers only grow; buffers start at zero or hold older numbers.
// Every wait is bounded and ends early once another CTA has given up (*flag).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ttg {
namespace words {

constexpr long long SPIN_LIMIT = 1ll << 24;
template <class T> constexpr int count = (int)(sizeof(T) / 4);   // words of a value

template <class T>
__device__ __forceinline__ void put(unsigned long long* w, const T& v, unsigned int epoch) {
  const unsigned int* h = reinterpret_cast<const unsigned int*>(&v);
  const unsigned long long tag = (unsigned long long)epoch << 32;
#pragma unroll
  for (int k = 0; k < count<T>; k += 2)
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w + k), "l"(tag | h[k]),
                 "l"(tag | h[k + 1])
                 : "memory");
}
// a first load; several of these in flight cost one trip to L2
template <class T>
__device__ __forceinline__ void load(const unsigned long long* w, unsigned long long (&x)[count<T>]) {
#pragma unroll
  for (int k = 0; k < count<T>; k += 2)
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x[k]), "=l"(x[k + 1]) : "l"(w + k) : "memory");
}
// x holds a first load of w: the value once its words carry `epoch`; false
// (nothing in v, *flag set) once the wait ran out here or elsewhere
template <class T>
__device__ __forceinline__ bool take(const unsigned long long* w, unsigned long long (&x)[count<T>],
                                     T& v, unsigned int epoch, unsigned int* flag) {
  unsigned int* h = reinterpret_cast<unsigned int*>(&v);
  for (long long spin = 0; spin < SPIN_LIMIT; ++spin) {
    bool all = true;
#pragma unroll
    for (int k = 0; k < count<T>; ++k) {
      h[k] = (unsigned int)x[k];
      all = all && (unsigned int)(x[k] >> 32) == epoch;
    }
    if (all) return true;
    if ((spin & 255) == 255 && *(volatile unsigned int*)flag != 0u) break;
    load<T>(w, x);
  }
  atomicExch(flag, 1u);
  return false;
}

}  // namespace words
}  // namespace ttg
