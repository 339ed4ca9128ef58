// Compression branch, forward: tensor maps and launches of the attention with every row's bound (cmp_attn.cuh) and of the
// collection of the columns or blocks that reach it (cmp_topk.cuh).
#include "cmp_attn.cuh"
#include "cmp_topk.cuh"

namespace s3r {

template <int R, int RANK>
__global__ void __launch_bounds__(AtCfg<R>::kThreads, 1)
cmp_attn_kernel(const __grid_constant__ CmpMaps m, const __grid_constant__ AtParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ AtCtl ctl;
  cmp_attn_cta<R, RANK>(m.q, m.k, m.v, m.ks, m.vs, p, ctl, smem_raw, blockIdx.x);
}
template <int R, int RANK>
__global__ void __launch_bounds__(TkCfg<R>::kThreads, 1)
cmp_topk_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ TkParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ TkCtl ctl;
  cmp_topk_cta<R, RANK, false>(map_q, map_k, p, ctl, smem_raw, blockIdx.x);
}

// Both in one grid, all of the attention's CTAs first.  With more row tiles than SMs the last wave of either leaves SMs idle
// (496 tiles on 148 SMs: a sixth of both); so the second kind's CTAs fill the first kind's last wave.  They wait for rows
// whose CTA has been running since before them and waits for nobody.
// Measured (16 heads, two launches -> one): 2400 x 2400 154 -> 126 us, 5000 x 5000 373 -> 320, 7875 x 63000 4.11 -> 3.66 ms;
// where the waves are full anyway the same: 6300 x 6300 449, 15750 x 15750 2155 -> 2145 us.
template <int RANK>
__global__ void __launch_bounds__(TkCfg<2>::kThreads, 1)
cmp_both_kernel(const __grid_constant__ CmpMaps m, const __grid_constant__ AtParams pa, const __grid_constant__ TkParams pt,
                const int attn_ctas) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ union {
    AtCtl attn;
    TkCtl topk;
  } ctl;
  if (static_cast<int>(blockIdx.x) < attn_ctas)
    cmp_attn_cta<2, RANK>(m.q, m.k, m.v, m.ks, m.vs, pa, ctl.attn, smem_raw, blockIdx.x);
  else
    cmp_topk_cta<2, RANK, true>(m.q, m.k, pt, ctl.topk, smem_raw, static_cast<int>(blockIdx.x) - attn_ctas);
}
static_assert(AtCfg<2>::kThreads == TkCfg<2>::kThreads && AtCfg<2>::kSmem <= TkCfg<2>::kSmem, "one launch shape for both kinds");

// Two launches where all row tiles fit the GPU at once.
template <int R, int RANK>
static int launch_cmp_apart(const CmpMaps& m, const AtParams& a, const TkParams& t, int64_t ctas, cudaStream_t st) {
  S3R_CUDA(cudaFuncSetAttribute(cmp_attn_kernel<R, RANK>, cudaFuncAttributeMaxDynamicSharedMemorySize, AtCfg<R>::kSmem));
  const int rc = launch(cmp_attn_kernel<R, RANK>, static_cast<unsigned>(ctas), AtCfg<R>::kThreads, AtCfg<R>::kSmem, st, m, a);
  if (rc) return rc;
  S3R_CUDA(cudaFuncSetAttribute(cmp_topk_kernel<R, RANK>, cudaFuncAttributeMaxDynamicSharedMemorySize, TkCfg<R>::kSmem));
  return launch(cmp_topk_kernel<R, RANK>, static_cast<unsigned>(ctas), TkCfg<R>::kThreads, TkCfg<R>::kSmem, st, m.q, m.k, t);
}
template <int RANK>
static int launch_cmp(const CmpMaps& m, AtParams a, TkParams t, int64_t BH, cudaStream_t st) {
  const int64_t tiles1 = BH * ((t.Nq + 127) / 128), tiles2 = BH * ((t.Nq + 255) / 256);
  S3R_REQUIRE(2 * tiles2 < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_cmp_attn_topk_fwd: grid too large");
  if (tiles2 > sm_count()) {
    // all of the table, not only the words that are waited for: a strided fill takes ten times as long
    S3R_CUDA(cudaMemsetAsync(t.idx, 0xff, static_cast<size_t>(BH) * t.Nq * t.topk * sizeof(int32_t), st));
    S3R_CUDA(cudaFuncSetAttribute(cmp_both_kernel<RANK>, cudaFuncAttributeMaxDynamicSharedMemorySize, TkCfg<2>::kSmem));
    return launch(cmp_both_kernel<RANK>, static_cast<unsigned>(2 * tiles2), TkCfg<2>::kThreads, TkCfg<2>::kSmem, st, m, a, t, static_cast<int>(tiles2));
  }
  // One row tile per CTA while all of them fit the GPU at once, two row tiles sharing every key tile beyond that.  Attention
  // alone: 384 x 384, 16 heads: 8.7 instead of 12.2 us; 1512 x 1512: 35 instead of 25 us.
  return tiles1 <= sm_count() ? launch_cmp_apart<1, RANK>(m, a, t, tiles1, st) : launch_cmp_apart<2, RANK>(m, a, t, tiles2, st);
}

}  // namespace s3r

using namespace s3r;

static int launch_cmp_fwd(const char* who, const void* q_c, const void* k_c, const void* v_c, void* o_c, float* lse,
                          int32_t* idx, int B, int H, int Nq, int Nc, int d, int topk, float scale, int rank_take,
                          void* stream) {
  S3R_REQUIRE(q_c && k_c && v_c && o_c && lse && idx, S3R_ERR_NULL, "%s: NULL pointer", who);
  S3R_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nc > 0, S3R_ERR_SHAPE, "%s: sizes must be positive (B=%d H=%d Nq=%d Nc=%d)", who,
              B, H, Nq, Nc);
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "%s: head_dim %d not supported (64 only)", who, d);
  S3R_REQUIRE(topk >= 1 && topk <= 32, S3R_ERR_UNSUPPORTED, "%s: topk %d not in [1,32]", who, topk);
  S3R_REQUIRE(scale > 0.f, S3R_ERR_UNSUPPORTED, "%s: softmax scale must be positive", who);
  const uintptr_t al = reinterpret_cast<uintptr_t>(q_c) | reinterpret_cast<uintptr_t>(k_c) |
                       reinterpret_cast<uintptr_t>(v_c) | reinterpret_cast<uintptr_t>(o_c);
  S3R_REQUIRE((al & 15) == 0, S3R_ERR_ALIGNMENT, "%s: tensors must be 16-byte aligned", who);
  const int BH = B * H;
  CmpMaps m;
  uint32_t box[3] = {64, 128, 1};
  {
    uint64_t dims[3] = {64, static_cast<uint64_t>(Nq), static_cast<uint64_t>(BH)};
    uint64_t strides[2] = {128, static_cast<uint64_t>(Nq) * 128};
    int rc = make_tensor_map(&m.q, q_c, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t dims[3] = {64, static_cast<uint64_t>(Nc), static_cast<uint64_t>(BH)};
    uint64_t strides[2] = {128, static_cast<uint64_t>(Nc) * 128};
    int rc = make_tensor_map(&m.k, k_c, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_tensor_map(&m.v, v_c, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  // keys i and 64 + i of a tile to rows 16 (i / 8) + i mod 8 and 8 further: the box's rows of eight keys alternate between
  // the tile's halves.  Whole tiles only, so that no coordinate inside the map's extents leaves the tensor.  Below eight
  // tiles a row has few columns per group and the copy's finer pieces gain nothing.
  m.scattered = rank_take == 0 && Nc >= 1024 ? Nc / 128 : 0;
  if (m.scattered > 0) {
    const uint64_t dims[5] = {64, 8, 2, static_cast<uint64_t>(m.scattered) * 16 - 8, static_cast<uint64_t>(BH)};
    const uint64_t strides[4] = {128, 64 * 128, 8 * 128, static_cast<uint64_t>(Nc) * 128};
    const uint32_t box5[5] = {64, 8, 2, 8, 1};
    int rc = make_tensor_map(&m.ks, k_c, 5, dims, strides, box5, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_tensor_map(&m.vs, v_c, 5, dims, strides, box5, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  } else {
    m.ks = m.k;
    m.vs = m.v;
  }
  uint32_t* status = device_status_ptr();
  S3R_REQUIRE(status != nullptr, S3R_ERR_DRIVER, "%s: could not resolve the device status word", who);
  AtParams a;
  a.o = static_cast<__nv_bfloat16*>(o_c);
  a.lse = lse;
  a.bound = reinterpret_cast<float*>(idx);
  a.Nq = Nq; a.Nc = Nc; a.topk = topk;
  a.scattered = m.scattered;
  a.rank_take = rank_take;
  a.c_scale = scale * 1.4426950408889634f;
  a.status = status;
  TkParams t;
  t.idx = idx;
  t.Nq = Nq; t.Nc = Nc; t.topk = topk;
  t.rank_take = rank_take;
  t.n_rank = rank_take > 0 ? (Nc - rank_take) / 4 + 1 : 0;       // blocks of four columns with all counted columns present
  t.pad = (rank_take > 0 ? t.n_rank : Nc) - 1;
  t.c_scale = a.c_scale;
  t.vec = (topk & 3) == 0 && (reinterpret_cast<uintptr_t>(idx) & 15) == 0;
  t.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return rank_take > 0 ? launch_cmp<1>(m, a, t, BH, st) : launch_cmp<0>(m, a, t, BH, st);
}

extern "C" int s3r_cmp_attn_topk_fwd(const void* q_c, const void* k_c, const void* v_c, void* o_c, float* lse,
                                     int32_t* idx, int B, int H, int Nq, int Nc, int d, int topk, float scale,
                                     void* stream) {
  return launch_cmp_fwd("s3r_cmp_attn_topk_fwd", q_c, k_c, v_c, o_c, lse, idx, B, H, Nq, Nc, d, topk, scale, 0, stream);
}

extern "C" int s3r_cmp_attn_blocktopk_fwd(const void* q_c, const void* k_c, const void* v_c, void* o_c, float* lse,
                                          int32_t* idx, int B, int H, int Nq, int Nc, int d, int topk, float scale,
                                          int group, int take, void* stream) {
  S3R_REQUIRE(group == 4, S3R_ERR_UNSUPPORTED, "s3r_cmp_attn_blocktopk_fwd: %d compressed keys per block (4 only)", group);
  S3R_REQUIRE(take >= 1 && take <= 4 && Nc >= take, S3R_ERR_UNSUPPORTED,
              "s3r_cmp_attn_blocktopk_fwd: take=%d must be in [1,4] and <= Nc=%d", take, Nc);
  return launch_cmp_fwd("s3r_cmp_attn_blocktopk_fwd", q_c, k_c, v_c, o_c, lse, idx, B, H, Nq, Nc, d, topk, scale, take,
                        stream);
}
