// What the kernels of the compression branch's forward share: key order, sorting in registers, the host's tensor maps.
#pragma once
#include "common.cuh"

namespace s3r {

struct CmpMaps {
  CUtensorMap q, k, v, ks, vs;
  int scattered;               // leading key tiles for which the first kernel uses ks and vs
};
#ifdef __CUDACC__
// Threshold for the float pre-filter `score > thr`: an equal score with a larger column loses to the entry whose key
// this is.  The one place where float order and key order disagree is -0.0 < +0.0: a kept -0.0 yields a threshold
// just below zero so that +0.0 still passes the pre-filter (the exact test is on the keys).
__device__ __forceinline__ float key_to_float(uint32_t key) {
  if (key == 0u) return -INFINITY;            // empty slot: every finite score qualifies
  if (key == 0x7fffffffu) return __uint_as_float(0x80000001u);   // -0.0 -> largest negative subnormal
  const uint32_t b = (key & 0x80000000u) ? (key ^ 0x80000000u) : ~key;
  return __uint_as_float(b);
}

template <typename T>
__device__ __forceinline__ void order_desc(T& a, T& b) {           // larger first
  const T x = a < b ? b : a, y = a < b ? a : b;
  a = x;
  b = y;
}
__device__ __forceinline__ void order_desc(float& a, float& b) {
  const float x = fmaxf(a, b), y = fminf(a, b);
  a = x;
  b = y;
}
// Descending sort in registers: Batcher's odd-even merge sort (191 exchanges for 32).
template <int N, typename T>
__device__ __forceinline__ void sort_desc(T (&v)[N]) {
#pragma unroll
  for (int p = 1; p < N; p <<= 1)
#pragma unroll
    for (int k = p; k > 0; k >>= 1)
#pragma unroll
      for (int i = 0; i < N - k; ++i)
        if (i >= k % p && ((i - k % p) / k) % 2 == 0 && i / (2 * p) == (i + k) / (2 * p)) order_desc(v[i], v[i + k]);
}
#endif

}  // namespace s3r
