// fp32 -> bf16 of several tensors in one launch: what autocast does to a module's input and weights, one tensor at a time
// (six launches and 12 us for the attention module at 2048 tokens, and the input once per Linear that reads it).
// Bound: HBM, 6 bytes per element.
#include "common.cuh"

namespace s3r {

constexpr int kCastMax = 8, kCastPerThread = 8, kCastVecs = 4;
constexpr int kCastPerBlock = 256 * kCastPerThread * kCastVecs;

struct CastParams {
  const float* src[kCastMax];
  __nv_bfloat16* dst[kCastMax];
  int64_t count[kCastMax];
  int first_block[kCastMax + 1];
  uint32_t wide;               // bit i: both sides of tensor i begin at a multiple of 16 bytes
  int n;
};

__global__ void __launch_bounds__(256) cast_bf16_kernel(const __grid_constant__ CastParams p) {
  griddep_wait();
  griddep_launch();
  int i = 0;
  while (i + 1 < p.n && static_cast<int>(blockIdx.x) >= p.first_block[i + 1]) ++i;
  const float* src = p.src[i];
  __nv_bfloat16* dst = p.dst[i];
  const int64_t base = static_cast<int64_t>(blockIdx.x - p.first_block[i]) * kCastPerBlock, left = p.count[i] - base;
  if (!(p.wide >> i & 1u)) {                   // a view that begins anywhere: one element at a time
    for (int64_t e = threadIdx.x; e < min(left, static_cast<int64_t>(kCastPerBlock)); e += 256) dst[base + e] = __float2bfloat16_rn(src[base + e]);
    return;
  }
  float4 v[kCastVecs][2];
#pragma unroll
  for (int u = 0; u < kCastVecs; ++u) {
    const int64_t e = (static_cast<int64_t>(u) * 256 + threadIdx.x) * kCastPerThread;
    if (e + kCastPerThread <= left) {
      v[u][0] = *reinterpret_cast<const float4*>(src + base + e);
      v[u][1] = *reinterpret_cast<const float4*>(src + base + e + 4);
    }
  }
#pragma unroll
  for (int u = 0; u < kCastVecs; ++u) {
    const int64_t e = (static_cast<int64_t>(u) * 256 + threadIdx.x) * kCastPerThread;
    if (e + kCastPerThread <= left) {
      *reinterpret_cast<uint4*>(dst + base + e) = make_uint4(pack_bf16(v[u][0].x, v[u][0].y), pack_bf16(v[u][0].z, v[u][0].w),
                                                             pack_bf16(v[u][1].x, v[u][1].y), pack_bf16(v[u][1].z, v[u][1].w));
    } else {
      for (int64_t k = e; k < left && k < e + kCastPerThread; ++k) dst[base + k] = __float2bfloat16_rn(src[base + k]);
    }
  }
}

}  // namespace s3r

using namespace s3r;

extern "C" int s3r_cast_bf16(int n, const float* const* src, void* const* dst, const int64_t* counts, void* stream) {
  S3R_REQUIRE(src && dst && counts, S3R_ERR_NULL, "s3r_cast_bf16: NULL array");
  S3R_REQUIRE(n >= 1 && n <= kCastMax, S3R_ERR_SHAPE, "s3r_cast_bf16: %d tensors (1 to %d)", n, kCastMax);
  CastParams p;
  p.n = n;
  p.wide = 0;
  int64_t blocks = 0;
  for (int i = 0; i < n; ++i) {
    S3R_REQUIRE(src[i] && dst[i], S3R_ERR_NULL, "s3r_cast_bf16: NULL pointer");
    S3R_REQUIRE(counts[i] > 0, S3R_ERR_SHAPE, "s3r_cast_bf16: sizes must be positive");
    S3R_REQUIRE((reinterpret_cast<uintptr_t>(src[i]) & 3) == 0 && (reinterpret_cast<uintptr_t>(dst[i]) & 1) == 0, S3R_ERR_ALIGNMENT,
                "s3r_cast_bf16: elements must be aligned");
    if (((reinterpret_cast<uintptr_t>(src[i]) | reinterpret_cast<uintptr_t>(dst[i])) & 15) == 0) p.wide |= 1u << i;
    p.src[i] = src[i];
    p.dst[i] = static_cast<__nv_bfloat16*>(dst[i]);
    p.count[i] = counts[i];
    p.first_block[i] = static_cast<int>(blocks);
    blocks += (counts[i] + kCastPerBlock - 1) / kCastPerBlock;
    S3R_REQUIRE(blocks < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_cast_bf16: grid too large");
  }
  p.first_block[n] = static_cast<int>(blocks);
  return launch(cast_bf16_kernel, static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream), p);
}
