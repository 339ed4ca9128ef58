// Column sums of a bf16 matrix in fp32: the bias gradients of the module's projections (PyTorch's reduction of the same three
// matrices took 64 us of a training step at 2 x 6144 tokens).  Bound: HBM, the matrix once.  Two stages in a fixed order:
// a CTA sums a slice of the rows of 256 columns (lane = 8 columns, warps take turns at rows), a second kernel the slices.
#include "common.cuh"

namespace s3r {

constexpr int kColWarps = 8;

__global__ void __launch_bounds__(kColWarps * 32) colsum_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ partial,
                                                                int64_t rows, int cols, int64_t rows_per_slice) {
  __shared__ float red[kColWarps][256];
  griddep_wait();
  griddep_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * 256 + lane * 8;
  const int64_t r0 = blockIdx.y * rows_per_slice, r1 = min(rows, r0 + rows_per_slice);
  float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  if (c < cols) {
#pragma unroll 4
    for (int64_t r = r0 + warp; r < r1; r += kColWarps) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(x + r * cols + c));
      acc[0] = fadd2(acc[0], make_float2(bf16_lo(v.x), bf16_hi(v.x)));
      acc[1] = fadd2(acc[1], make_float2(bf16_lo(v.y), bf16_hi(v.y)));
      acc[2] = fadd2(acc[2], make_float2(bf16_lo(v.z), bf16_hi(v.z)));
      acc[3] = fadd2(acc[3], make_float2(bf16_lo(v.w), bf16_hi(v.w)));
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(&red[warp][lane * 8 + 2 * i]) = acc[i];
  __syncthreads();
  const int o = blockIdx.x * 256 + threadIdx.x;
  if (o < cols) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kColWarps; ++w) s += red[w][threadIdx.x];
    partial[static_cast<int64_t>(blockIdx.y) * cols + o] = s;
  }
}

__global__ void __launch_bounds__(128) colsum_slices_kernel(const float* __restrict__ partial, float* __restrict__ out, int cols, int slices) {
  griddep_wait();
  griddep_launch();
  const int o = blockIdx.x * 128 + threadIdx.x;
  if (o >= cols) return;
  float s = 0.f;
#pragma unroll 8
  for (int i = 0; i < slices; ++i) s += __ldg(partial + static_cast<int64_t>(i) * cols + o);
  out[o] = s;
}

// slices of at least 64 rows, as many as give every SM four CTAs
static int colsum_slices(int64_t rows, int cols) {
  const int64_t per_row = (cols + 255) / 256, want = (4 * sm_count() + per_row - 1) / per_row, most = (rows + 63) / 64;
  return static_cast<int>(want < most ? want : most);
}

}  // namespace s3r

using namespace s3r;

extern "C" size_t s3r_colsum_workspace_bytes(int64_t rows, int cols) {
  return rows > 0 && cols > 0 ? static_cast<size_t>(colsum_slices(rows, cols)) * cols * sizeof(float) : 0;
}

extern "C" int s3r_colsum(const void* x, float* out, int64_t rows, int cols, void* workspace, size_t workspace_bytes, void* stream) {
  S3R_REQUIRE(x && out && workspace, S3R_ERR_NULL, "s3r_colsum: NULL pointer");
  S3R_REQUIRE(rows > 0 && cols > 0, S3R_ERR_SHAPE, "s3r_colsum: sizes must be positive");
  S3R_REQUIRE(cols % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0, S3R_ERR_ALIGNMENT, "s3r_colsum: rows must be 16-byte aligned");
  S3R_REQUIRE(workspace_bytes >= s3r_colsum_workspace_bytes(rows, cols), S3R_ERR_TOO_LARGE,
              "s3r_colsum: workspace of %zu bytes is smaller than the %zu needed", workspace_bytes, s3r_colsum_workspace_bytes(rows, cols));
  const int slices = colsum_slices(rows, cols);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* partial = static_cast<float*>(workspace);
  const int rc = launch(colsum_kernel, dim3(static_cast<unsigned>((cols + 255) / 256), static_cast<unsigned>(slices)), kColWarps * 32, 0, st,
                        static_cast<const __nv_bfloat16*>(x), partial, rows, cols, (rows + slices - 1) / slices);
  if (rc) return rc;
  return launch(colsum_slices_kernel, static_cast<unsigned>((cols + 127) / 128), 128, 0, st, partial, out, cols, slices);
}
