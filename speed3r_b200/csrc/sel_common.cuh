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
// Whether sel_bwd64 is the faster of the two kernels that take blocks of 64, for `bh` heads of `nqb` query blocks with `topk` entries
// each and `nkb` key blocks.  A task (a query block or a key block) costs it 9.3 ns more than the other (tensor memory, half an SM per
// CTA), an entry 6.7 ns less, and on an idle GPU it is 11 us sooner done: it pays where 11 us + 6.7 ns entries >= 9.3 ns tasks.  It also
// pays where the other's longest lists (2 us per entry in one warp) take longer than this one's tasks (9.2 ns each).  Round numbers of
// both; measured with the index, sel_bwd_kernel | sel_bwd64_kernel, us: one entry per list, 1536 tasks 29.9 | 30.0, 1876 35.6 | 37.3,
// 4096 57 | 72, 30 016 355 | 522; two entries, 3752 78.5 | 76.4, 4096 80.4 | 82.3, 30 016 519 | 574; three, 30 016 684 | 662; sixteen,
// 30 016 2809 | 1523.  16 heads of 16 query blocks on 938 key blocks, sixteen entries 162 | 192; 2 heads 49 | 38, four entries 27 | 29;
// 16 heads of 938 query blocks on one key block 2634 | 762.
inline bool sel_bwd64_pays(int64_t bh, int64_t nqb, int64_t nkb, int64_t topk) {
  const int64_t tasks = bh * (nqb + nkb), entries = bh * nqb * topk, longest = topk * (nqb > nkb ? nqb / nkb : 1);
  return 7 * tasks <= 5 * (entries + 1600) || tasks < 540 + 220 * longest;
}

}  // namespace s3r
