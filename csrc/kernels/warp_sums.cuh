// Sums over a warp of several values at once.
#pragma once
#include <cuda_runtime.h>

namespace nangila {

// The sum over the warp of each of P values (a power of two up to 32). The values are shared out among the lanes as they are added up, half of
// them going to the other half of the lanes at every step: P - 1 exchanges and one for each step that is left, where P sums one by one take 5 P.
// The sum of value i is returned in the 32 / P lanes from i * 32 / P on.
template <int P, typename T>
__device__ __forceinline__ T warp_sums_of_power(T (&a)[P]) {
  static_assert(P >= 1 && P <= 32 && (P & (P - 1)) == 0, "a power of two");
  const int lane = threadIdx.x & 31;
  int off = 16;
#pragma unroll
  for (int half = P / 2; half >= 1; half >>= 1, off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const T other = __shfl_xor_sync(0xffffffffu, upper ? a[i] : a[i + half], off);
      a[i] = (upper ? a[i + half] : a[i]) + other;
    }
  }
#pragma unroll
  for (; off > 0; off >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], off);
  return a[0];
}

// The sum over the warp of each of N values, given to store(i, sum) by one lane each. (Five values are added up as eight: the chain of exchanges is
// what a sum waits for, and four and one would be two of them.)
template <int FROM = 0, int N, typename T, typename Store>
__device__ __forceinline__ void warp_sums(const T (&v)[N], const Store& store) {
  if constexpr (FROM < N) {
    constexpr int left = N - FROM;
    constexpr int P = left > 16 ? 32 : left > 8 ? 16 : left > 4 ? 8 : left > 2 ? 4 : left > 1 ? 2 : 1;
    T a[P];
#pragma unroll
    for (int i = 0; i < P; ++i) a[i] = FROM + i < N ? v[FROM + i < N ? FROM + i : 0] : T(0);
    const T sum = warp_sums_of_power<P>(a);
    const int lane = threadIdx.x & 31, i = FROM + lane / (32 / P);
    if (lane % (32 / P) == 0 && i < N) store(i, sum);
    warp_sums<FROM + P>(v, store);
  }
}

}  // namespace nangila
