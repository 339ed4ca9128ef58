// Arguments that the kernels of the selection branch's forward share.
#pragma once
#include "common.cuh"

namespace s3r {

struct SelParams {
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
// Blocks of 32 and 64 tokens; kv_chunk_stride in elements.
int sel_big_fwd(const void* q, const void* k, const void* v, int kv_chunks, int64_t kv_chunk_stride, int block, const SelParams& p,
                cudaStream_t st);

}  // namespace s3r
