// Arguments that the kernels of the selection branch share.
#pragma once
#include "common.cuh"

namespace s3r {

struct SelParams {
  const __nv_bfloat16 *q, *k, *v;
  int64_t kv_chunk_stride;       // elements
  const int32_t* idx;
  __nv_bfloat16* o_s;
  float* lse_s;
  const __nv_bfloat16* gate;
  int64_t gsb, gsh, gst;
  const __nv_bfloat16* o_c;
  __nv_bfloat16* y;
  int B, H, Tq, Tk, Tc /*tokens per kv chunk*/, nqb, topk;
  float scale_log2e;
  uint32_t* status;
};
// Blocks of 32 and 64 tokens.
int sel_big_fwd(int kv_chunks, int block, const SelParams& p, cudaStream_t st);

struct SelBwdParams {
  const __nv_bfloat16 *q, *k, *v, *d_o;
  const int32_t *idx, *offsets, *qids;
  const float *lse, *delta;
  __nv_bfloat16 *dq, *dk, *dv;
  // gradient of the pooled branch, added to dq | dk, dv (null: none): element t of dq gets dq_c[j] / kernel of every
  // window j that contains it.  Kernel and stride are multiples of 16, so a warp's 16 rows share their windows.
  const __nv_bfloat16 *dq_c, *dk_c, *dv_c;
  int q_kernel, q_stride, q_windows, k_kernel, k_stride, k_windows;
  int B, H, Tq, Tk, block, block_shift, topk, nqb, nkb;     // block = 16 << block_shift
  float cs, scale;
  uint32_t* status;
};
// Blocks of 64 tokens.
int sel_bwd64(const SelBwdParams& p, cudaStream_t st);

}  // namespace s3r
