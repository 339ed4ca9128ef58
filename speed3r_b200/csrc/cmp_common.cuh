// What the kernels of the compression branch's forward share: key order, sorting in registers, the host's tensor maps.
#pragma once
#include "common.cuh"

namespace s3r {

struct CmpMaps {
  CUtensorMap q, k, v;
};
// Dense attention; row r's lower bound of its 32nd largest logit goes to bound[r * bound_stride].
int cmp_attn_fwd(const CmpMaps& m, void* o_c, float* lse, float* bound, int64_t bound_stride, int BH, int Nq, int Nc, float scale,
                 uint32_t* status, cudaStream_t st);
// Best columns of every row; idx[row * topk] holds the row's bound on entry.
int cmp_topk_fwd(const CmpMaps& m, int32_t* idx, int topk, int BH, int Nq, int Nc, uint32_t* status, cudaStream_t st);

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

// Descending bitonic sort of 32 values in registers.
__device__ __forceinline__ void sort32_desc(float (&v)[32]) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int l = i ^ j;
        if (l > i) {
          const float hi = fmaxf(v[i], v[l]), lo = fminf(v[i], v[l]);
          const bool desc = (i & k) == 0;
          v[i] = desc ? hi : lo;
          v[l] = desc ? lo : hi;
        }
      }
}
#endif

}  // namespace s3r
