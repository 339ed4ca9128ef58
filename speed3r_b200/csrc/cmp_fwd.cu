// Compression branch, forward: tensor maps and the two launches, attention with every row's bound (cmp_attn.cu) and the
// columns or blocks that reach it (cmp_topk.cu).
#include "common.cuh"
#include "cmp_common.cuh"

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
  const CmpSizes n = {BH, Nq, Nc, topk, rank_take};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = cmp_attn_fwd(m, o_c, lse, reinterpret_cast<float*>(idx), n, scale, status, st);
  if (rc) return rc;
  return cmp_topk_fwd(m, idx, n, scale, status, st);
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
