// Arguments that the kernels of the selection branch's forward share.
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

}  // namespace s3r
