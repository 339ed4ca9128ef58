// Block pooling of q/k/v (the compression step) and its backward.  Both are pure streaming
// kernels bounded by HBM bandwidth: every thread moves 16-byte vectors (8 bf16 channels), a
// token row of one head is 128 contiguous bytes, and neighbouring threads walk neighbouring heads so
// that the packed qkv projection is read in 2 KB contiguous runs.
#include "common.cuh"

namespace s3r {

struct alignas(16) Bf16x8 {
  uint32_t w[4];
};

// One launch pools up to three tensors (blockIdx.y): three launches of a few microseconds each were a tenth of the
// op at 2048 tokens.
struct PoolTensor {
  const __nv_bfloat16* in;
  int64_t sb, sh, st;
  __nv_bfloat16* out;
  int Nc, kernel, stride;
};
struct PoolParams {
  PoolTensor t[3];
  int B, H, d;
};

// BATCH: so many loads of a window leave together (its length is a multiple of BATCH; one at a time, windows of 32 tokens at
// 252000 took 760 us instead of 263).
template <int BATCH>
__device__ __forceinline__ void pool_tensor(const PoolTensor& p, int B, int H, int d) {
  const int vec_per_row = d >> 3;
  const int64_t total = static_cast<int64_t>(B) * p.Nc * H * vec_per_row;
  const float inv = 1.0f / static_cast<float>(p.kernel);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    // fastest -> slowest: channel vector, head, pooled row, batch
    int c8 = static_cast<int>(i % vec_per_row);
    int64_t r = i / vec_per_row;
    int h = static_cast<int>(r % H);
    r /= H;
    int j = static_cast<int>(r % p.Nc);
    int b = static_cast<int>(r / p.Nc);
    const __nv_bfloat16* src = p.in + b * p.sb + h * p.sh + static_cast<int64_t>(j) * p.stride * p.st + c8 * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add = [&](const Bf16x8& v) {
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        acc[2 * w] += bf16_lo(v.w[w]);
        acc[2 * w + 1] += bf16_hi(v.w[w]);
      }
    };
#pragma unroll 1
    for (int t0 = 0; t0 < p.kernel; t0 += BATCH) {
      Bf16x8 v[BATCH];
#pragma unroll
      for (int t = 0; t < BATCH; ++t) v[t] = *reinterpret_cast<const Bf16x8*>(src + (t0 + t) * p.st);
#pragma unroll
      for (int t = 0; t < BATCH; ++t) add(v[t]);
    }
    Bf16x8 o;
#pragma unroll
    for (int w = 0; w < 4; ++w) o.w[w] = pack_bf16(acc[2 * w] * inv, acc[2 * w + 1] * inv);
    *reinterpret_cast<Bf16x8*>(p.out + ((static_cast<int64_t>(b) * H + h) * p.Nc + j) * d + c8 * 8) = o;
  }
}
__global__ void __launch_bounds__(256) pool_fwd_kernel(const PoolParams p) {
  griddep_wait();
  griddep_launch();
  const PoolTensor& t = p.t[blockIdx.y];
  if (t.kernel % 16 == 0) pool_tensor<16>(t, p.B, p.H, p.d);
  else pool_tensor<1>(t, p.B, p.H, p.d);
}

__global__ void __launch_bounds__(256)
pool_bwd_kernel(const __nv_bfloat16* __restrict__ d_out, __nv_bfloat16* __restrict__ d_in, int64_t sb, int64_t sh,
                int64_t st, int B, int H, int T, int d, int Nc, int kernel, int stride, int accumulate) {
  const int vec_per_row = d >> 3;
  const int64_t total = static_cast<int64_t>(B) * T * H * vec_per_row;
  const float inv = 1.0f / static_cast<float>(kernel);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int c8 = static_cast<int>(i % vec_per_row);
    int64_t r = i / vec_per_row;
    int h = static_cast<int>(r % H);
    r /= H;
    int t = static_cast<int>(r % T);
    int b = static_cast<int>(r / T);
    // windows j with j*stride <= t < j*stride + kernel
    int j_hi = min(Nc - 1, t / stride);
    int j_lo = (t - kernel + 1 <= 0) ? 0 : (t - kernel + stride) / stride;   // ceil((t-kernel+1)/stride)
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const __nv_bfloat16* src = d_out + (static_cast<int64_t>(b) * H + h) * Nc * d + c8 * 8;
    for (int j = j_lo; j <= j_hi; ++j) {
      Bf16x8 v = *reinterpret_cast<const Bf16x8*>(src + static_cast<int64_t>(j) * d);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        acc[2 * w] += bf16_lo(v.w[w]);
        acc[2 * w + 1] += bf16_hi(v.w[w]);
      }
    }
    __nv_bfloat16* dst = d_in + b * sb + h * sh + t * st + c8 * 8;
    Bf16x8 o;
    if (accumulate) {
      Bf16x8 old = *reinterpret_cast<const Bf16x8*>(dst);
#pragma unroll
      for (int w = 0; w < 4; ++w)
        o.w[w] = pack_bf16(bf16_lo(old.w[w]) + acc[2 * w] * inv, bf16_hi(old.w[w]) + acc[2 * w + 1] * inv);
    } else {
#pragma unroll
      for (int w = 0; w < 4; ++w) o.w[w] = pack_bf16(acc[2 * w] * inv, acc[2 * w + 1] * inv);
    }
    *reinterpret_cast<Bf16x8*>(dst) = o;
  }
}

static int pool_grid(int64_t total_threads) {
  int64_t blocks = (total_threads + 255) / 256;
  int64_t cap = static_cast<int64_t>(sm_count()) * 16;   // 16 resident CTAs of 256 threads fill an SM's 2048 threads... x2 waves
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return static_cast<int>(blocks);
}

}  // namespace s3r

using namespace s3r;

extern "C" int s3r_pool_multi_fwd(int n, const void* const* in, const int64_t* strides, void* const* out, const int* kernels,
                                  const int* pool_strides, int B, int H, int T, int d, void* stream) {
  S3R_REQUIRE(in && strides && out && kernels && pool_strides, S3R_ERR_NULL, "s3r_pool_fwd: NULL array");
  S3R_REQUIRE(n >= 1 && n <= 3, S3R_ERR_SHAPE, "s3r_pool_fwd: %d tensors (1 to 3)", n);
  PoolParams p;
  p.B = B; p.H = H; p.d = d;
  int64_t most = 0;
  for (int i = 0; i < n; ++i) {
    const int64_t* st = strides + 3 * i;
    S3R_REQUIRE(in[i] && out[i], S3R_ERR_NULL, "s3r_pool_fwd: NULL pointer");
    S3R_REQUIRE(B > 0 && H > 0 && T > 0 && d > 0 && kernels[i] > 0 && pool_strides[i] > 0, S3R_ERR_SHAPE,
                "s3r_pool_fwd: sizes must be positive (B=%d H=%d T=%d d=%d kernel=%d stride=%d)", B, H, T, d, kernels[i],
                pool_strides[i]);
    S3R_REQUIRE(d % 8 == 0, S3R_ERR_UNSUPPORTED, "s3r_pool_fwd: head_dim %d is not a multiple of 8", d);
    S3R_REQUIRE(T >= kernels[i], S3R_ERR_SHAPE, "s3r_pool_fwd: T=%d shorter than the pooling kernel %d", T, kernels[i]);
    S3R_REQUIRE((reinterpret_cast<uintptr_t>(in[i]) & 15) == 0 && (reinterpret_cast<uintptr_t>(out[i]) & 15) == 0 &&
                    st[0] % 8 == 0 && st[1] % 8 == 0 && st[2] % 8 == 0,
                S3R_ERR_ALIGNMENT, "s3r_pool_fwd: pointers and strides must keep 16-byte alignment");
    PoolTensor& t = p.t[i];
    t.in = static_cast<const __nv_bfloat16*>(in[i]);
    t.sb = st[0]; t.sh = st[1]; t.st = st[2];
    t.out = static_cast<__nv_bfloat16*>(out[i]);
    t.Nc = (T - kernels[i]) / pool_strides[i] + 1;
    t.kernel = kernels[i]; t.stride = pool_strides[i];
    const int64_t total = static_cast<int64_t>(B) * t.Nc * H * (d / 8);
    most = total > most ? total : most;
  }
  return launch(pool_fwd_kernel, dim3(pool_grid(most), n), 256, 0, static_cast<cudaStream_t>(stream), p);
}

extern "C" int s3r_pool_fwd(const void* in, int64_t stride_b, int64_t stride_h, int64_t stride_t, void* out, int B,
                            int H, int T, int d, int kernel, int stride, void* stream) {
  const int64_t strides[3] = {stride_b, stride_h, stride_t};
  return s3r_pool_multi_fwd(1, &in, strides, &out, &kernel, &stride, B, H, T, d, stream);
}

extern "C" int s3r_pool_bwd(const void* d_out, void* d_in, int64_t stride_b, int64_t stride_h, int64_t stride_t,
                            int B, int H, int T, int d, int kernel, int stride, int accumulate, void* stream) {
  S3R_REQUIRE(d_out && d_in, S3R_ERR_NULL, "s3r_pool_bwd: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && T > 0 && d > 0 && kernel > 0 && stride > 0 && T >= kernel, S3R_ERR_SHAPE,
              "s3r_pool_bwd: bad sizes (B=%d H=%d T=%d d=%d kernel=%d stride=%d)", B, H, T, d, kernel, stride);
  S3R_REQUIRE(d % 8 == 0, S3R_ERR_UNSUPPORTED, "s3r_pool_bwd: head_dim %d is not a multiple of 8", d);
  S3R_REQUIRE((reinterpret_cast<uintptr_t>(d_out) & 15) == 0 && (reinterpret_cast<uintptr_t>(d_in) & 15) == 0 &&
                  stride_b % 8 == 0 && stride_h % 8 == 0 && stride_t % 8 == 0,
              S3R_ERR_ALIGNMENT, "s3r_pool_bwd: pointers and strides must keep 16-byte alignment");
  int Nc = (T - kernel) / stride + 1;
  int64_t total = static_cast<int64_t>(B) * T * H * (d / 8);
  pool_bwd_kernel<<<pool_grid(total), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(d_out), static_cast<__nv_bfloat16*>(d_in), stride_b, stride_h, stride_t, B, H,
      T, d, Nc, kernel, stride, accumulate);
  S3R_CUDA(cudaGetLastError());
  return 0;
}
