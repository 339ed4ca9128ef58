// Selection branch, forward: block-sparse flash attention over the K key blocks each query block
// selected, with the gated merge of the two branches fused into the epilogue.
//
// Bound: gather bandwidth.  A query block of BS rows reads topk*BS key rows and value rows
// (2*topk*BS*128 B) for 4*BS*topk*BS*64 flop, i.e. BS flop per byte (16 at the reference's block
// size) against a machine balance of ~250 flop/B, so the kernels are organised around keeping many
// independent TMA gathers in flight, not around tensor-core throughput: mma.sync m16n8k16, whose M tile
// is a 16-row query block, online softmax in registers, epilogue y = g0*o_c + g1*o_s in 128-byte rows.
// This is so for blocks of 16 (sel16_fwd_kernel); blocks of 32 and 64 tokens run on tcgen05 (sel_big.cu).
// CTAs are ordered head-major so that the CTAs resident at one time gather from one head's K/V.
#include "sel_common.cuh"

namespace s3r {

// ------------------------------------------------------------------------------------------------
// Blocks of 16 tokens (the reference's setting)
// ------------------------------------------------------------------------------------------------
// One warp = one CTA owns one query block (16 rows = one m16n8k16 M tile) and takes its selected key blocks
// two at a time from a ring of two 8 KB stages; one TMA copy brings a block's keys and values.
//   * All fragments of a stage go from shared memory to registers before the first product, so that no product
//     waits for a load (with loads and products alternating a warp spent 2700 cycles on a pair of blocks).
//   * The exponent offset of a row is its running maximum, pair by pair: the row's largest weights are 1 and lose nothing
//     when P is rounded to bf16.  An offset fixed by the first pair saved the maxima and their shuffles, but not the
//     rounding: error against 64 bits 2.33e-3 instead of 2.20e-3 at unit-scale logits, 2.20e-3 instead of 1.62e-3 where a
//     few keys hold a row's weight.
//   * O and l are rescaled with every pair, whether a row moved or not: among 16 rows one nearly always does (two in three
//     warps still do at the last pair), and the vote and the branch stood in the chain (64 views 536 -> 510 us).
//   * The thread that asks for copies is elected, so that the compiler knows it is one and coordinates need no loop over lanes
//     (548 -> 533 us); the list's entries are read where they are used (read a pair ahead 548 -> 568 us).
//   * CTAs of one warp: nothing is shared between query blocks, and a finished warp makes room at once.
// Bound: the gather, then the latency of a pair's chain that twelve warps per SM do not cover, then the power limit.  H = 16,
// top-32, uniformly random blocks, us at 1965 MHz - this kernel | its copies and waits alone | those and its fragment loads:
// 2048 tokens 24.8 | 17.9 | 19.8, 64 views 486 = 17.4 TB/s gathered | 397 | 404, 100 views 775 | 625 | 632; so shared memory's reads
// are 2 %.  In a long loop the clock falls under the power limit, to 1.75 GHz at 100 views (843 us), 1.6 at 250 (2.28 ms | 1.62 |
// 1.65) and 1.3 at 1000, where a head's 258 MB of keys and values miss L2 (15.0 ms = 8.9 TB/s | 13.1 | 13.3).  The op's own tables
// favour some blocks (with independent inputs a tenth of them has a third of the picks): at 1000 views 10.5 ms.
// Slots of single blocks in a ring of three, which let 15 warps instead of 12 onto an SM, lost more to a second wait per pair
// (64 views 592 us; 2048 tokens 25.2); refilling a slot before the products instead of after them changed nothing (lop3 of the
// fragments or a proxy fence in front: 600 and 612 us).
// Gathering straight into fragments with 16-byte loads instead (no shared memory) ran at 8.7 TB/s: a fragment load
// touches 8 rows, and L1 serves few lines per cycle.
struct Sel16Params {
  const __nv_bfloat16* q;
  const int32_t* idx;
  __nv_bfloat16* o_s;
  float* lse_s;
  const __nv_bfloat16* gate;
  int64_t gsb, gsh, gst;
  const __nv_bfloat16* o_c;
  __nv_bfloat16* y;
  int H, Tq, Tk, Tc, nqb, topk;
  float scale_log2e;
  uint32_t* status;
};

constexpr int kSel16StageBytes = 2 * 2 * 2048;                    // two blocks of keys, two of values
constexpr int kSel16Smem = 2 * kSel16StageBytes + 1024;

template <bool APART>
__global__ void __launch_bounds__(32, 12) sel16_fwd_kernel(const __grid_constant__ PairMap map_kv, const Sel16Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) int32_t list[64];        // first token of each valid key block, table order
  __shared__ uint64_t full[2];
  __shared__ uint32_t abort_word;
  const int lane = threadIdx.x, g = lane >> 2, c = lane & 3;
  const int64_t task = blockIdx.x;
  const int bh = static_cast<int>(task / p.nqb), qb = static_cast<int>(task - static_cast<int64_t>(bh) * p.nqb);
  volatile uint32_t* abort_flag = &abort_word;
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  if (lane == 0) {
    abort_word = 0;
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
  }
  griddep_wait();
  griddep_launch();

  int nvalid = 0;
  {
    const int32_t* row = p.idx + task * p.topk;
    for (int r0 = 0; r0 < p.topk; r0 += 32) {
      const int i = r0 + lane;
      const int n = (i < p.topk) ? row[i] : -1;
      const bool ok = (n >= 0) && (static_cast<int64_t>(n) * 16 < p.Tk);
      const uint32_t m = __ballot_sync(0xffffffffu, ok);
      if (ok) list[nvalid + __popc(m & ((1u << lane) - 1u))] = n * 16;
      nvalid += __popc(m);
    }
    __syncwarp();
  }
  // an odd list ends with its last block twice; the second copy's scores are masked
  if ((nvalid & 1) && lane == 0) list[nvalid] = list[nvalid - 1];
  __syncwarp();
  const bool chunked = p.Tc != p.Tk, leader = elect_one_sync();
  // a block's keys and its values together
  auto issue = [&](int pair, int s) {
    if (leader) {
      const int2 t = *reinterpret_cast<const int2*>(list + 2 * pair);
      int t0 = t.x, t1 = t.y, c0 = 0, c1 = 0;
      if (chunked) {
        c0 = t0 / p.Tc; t0 -= c0 * p.Tc;
        c1 = t1 / p.Tc; t1 -= c1 * p.Tc;
      }
      const uint32_t dst = ring + s * kSel16StageBytes;
      mbar_expect_tx(&full[s], map_kv.b_first < 0 ? 4096u : 8192u);
      tma_load_pair<APART>(dst, map_kv, &full[s], t0, bh, c0);
      tma_load_pair<APART>(dst + 4096, map_kv, &full[s], t1, bh, c1);
    }
  };
  const int npairs = (nvalid + 1) >> 1;
  if (npairs > 0) issue(0, 0);
  if (npairs > 1) issue(1, 1);

  uint32_t qf[4][4];
  {
    const uint32_t* q32 = reinterpret_cast<const uint32_t*>(p.q) + static_cast<int64_t>(bh) * p.Tq * 32;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t* src = q32 + static_cast<int64_t>(min(qb * 16 + g + 8 * r, p.Tq - 1)) * 32 + c;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        qf[ks][r] = __ldg(src + ks * 8);
        qf[ks][r + 2] = __ldg(src + ks * 8 + 4);
      }
    }
  }
  // shared-memory offsets of this lane's ldmatrix rows (128-byte swizzle), per k-step of Q K^T and per pair of d-tiles of P V
  uint32_t off_k[4], off_v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    off_k[i] = swz128((lane & 7) + (lane >> 4) * 8, 2 * i + ((lane >> 3) & 1)) + (map_kv.b_first > 0 ? 2048u : 0u);
    off_v[i] = swz128((lane & 7) + ((lane >> 3) & 1) * 8, 2 * i + (lane >> 4)) + (map_kv.b_first == 0 ? 2048u : 0u);
  }

  float o[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_used[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};        // l: this lane's share
  const float cs = p.scale_log2e;
  const bool ragged = (p.Tk & 15) != 0;
#pragma unroll 1
  for (int it = 0; it < npairs; ++it) {
    const int S = it & 1;
    if (!__all_sync(0xffffffffu, mbar_try_wait(&full[S], (it >> 1) & 1)) && !mbar_wait_warp(&full[S], (it >> 1) & 1, abort_flag)) {
      volatile uint32_t dummy = 0;               // a last bounded chance for the other stage's copies to land
      if (it + 1 < npairs) mbar_wait(&full[S ^ 1], ((it + 1) >> 1) & 1, &dummy);
      if (lane == 0) atomicOr(p.status, kStatusWaitTimeout);
      return;
    }
    const uint32_t st = ring + S * kSel16StageBytes;
    // every fragment of the stage goes to registers first: the products below then wait for no load
    uint32_t kf[2][4][4], vf[2][4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int j = 0; j < 2; ++j) ldsm_x4(kf[j][ks][0], kf[j][ks][1], kf[j][ks][2], kf[j][ks][3], st + off_k[ks] + j * 4096);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int dp = 0; dp < 4; ++dp) ldsm_x4_t(vf[j][dp][0], vf[j][dp][1], vf[j][dp][2], vf[j][dp][3], st + off_v[dp] + j * 4096);
    float s[2][2][4];                            // [block][key n-tile]
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (ks == 0) mma_bf16_z(s[j][t], qf[ks], kf[j][ks][2 * t], kf[j][ks][2 * t + 1]);
          else mma_bf16(s[j][t], qf[ks], kf[j][ks][2 * t], kf[j][ks][2 * t + 1]);
        }
    if (2 * it + 1 >= nvalid) {                  // the second block is the padding of an odd list: no scores, no values
#pragma unroll
      for (int t = 0; t < 2; ++t) s[1][t][0] = s[1][t][1] = s[1][t][2] = s[1][t][3] = -INFINITY;
#pragma unroll
      for (int dp = 0; dp < 4; ++dp) vf[1][dp][0] = vf[1][dp][1] = vf[1][dp][2] = vf[1][dp][3] = 0u;
    }
    if (ragged) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int left = p.Tk - list[2 * it + j];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (t * 8 + 2 * c + (e & 1) >= left) s[j][t][e] = -INFINITY;
      }
    }
    // the offsets follow the running maxima
    float mn[2], neg[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float m = fmax3(fmaxf(s[0][0][2 * r], s[0][0][2 * r + 1]), s[0][1][2 * r], s[0][1][2 * r + 1]);
      m = fmax3(fmax3(m, s[1][0][2 * r], s[1][0][2 * r + 1]), s[1][1][2 * r], s[1][1][2 * r + 1]);
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      mn[r] = fmaxf(m_used[r], m * cs);                               // scale > 0 keeps the order
      neg[r] = mn[r] == -INFINITY ? 0.f : -mn[r];                     // no finite score yet: P = 0
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float alpha = fast_exp2(m_used[r] + neg[r]);               // 1 where the row did not move
      m_used[r] = mn[r];
      l[r] *= alpha;
#pragma unroll
      for (int dt = 0; dt < 8; ++dt) {
        const float2 x = fmul2(make_float2(o[dt][2 * r], o[dt][2 * r + 1]), make_float2(alpha, alpha));
        o[dt][2 * r] = x.x;
        o[dt][2 * r + 1] = x.y;
      }
    }
    uint32_t pk[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float2 nm = make_float2(neg[r], neg[r]), cs2 = make_float2(cs, cs);
      float2 sum;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          float2 x = ffma2(make_float2(s[j][t][2 * r], s[j][t][2 * r + 1]), cs2, nm);
          x.x = fast_exp2(x.x);
          x.y = fast_exp2(x.y);
          sum = (j | t) ? fadd2(sum, x) : x;
          pk[j][2 * t + r] = pack_bf16(x.x, x.y);
        }
      l[r] += sum.x + sum.y;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int dp = 0; dp < 4; ++dp) {
        mma_bf16(o[2 * dp], pk[j], vf[j][dp][0], vf[j][dp][1]);
        mma_bf16(o[2 * dp + 1], pk[j], vf[j][dp][2], vf[j][dp][3]);
      }
    __syncwarp();
    if (it + 2 < npairs) issue(it + 2, S);       // every fragment of the stage has been consumed
  }
  // ---- epilogue -----------------------------------------------------------------------------
  float inv[2];
  const int t0 = qb * 16 + g;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float ls = l[r];
    ls += __shfl_xor_sync(0xffffffffu, ls, 1);
    ls += __shfl_xor_sync(0xffffffffu, ls, 2);
    const bool any = ls != 0.f;                          // no valid key, or none with a score above -inf: o = 0, lse = -inf
    inv[r] = any ? 1.0f / ls : 0.f;
    if (p.lse_s && c == 0 && t0 + 8 * r < p.Tq)
      p.lse_s[static_cast<int64_t>(bh) * p.Tq + t0 + 8 * r] = any ? (m_used[r] + log2f(ls)) * 0.6931471805599453f : -INFINITY;
  }
  // rows of 128 bytes leave through the warp's first stage (its copies have landed and been read)
  __syncwarp();
  uint8_t* stage = smem_raw + (ring - smem_u32(smem_raw));
  auto put = [&](const float (&a)[8][4], uint8_t* dst, int64_t row_bytes) {
#pragma unroll
    for (int dt = 0; dt < 8; ++dt) {
      *reinterpret_cast<uint32_t*>(stage + swz128(g, dt) + 4 * c) = pack_bf16(a[dt][0], a[dt][1]);
      *reinterpret_cast<uint32_t*>(stage + swz128(g + 8, dt) + 4 * c) = pack_bf16(a[dt][2], a[dt][3]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = (lane >> 3) + 4 * i;
      if (qb * 16 + r < p.Tq)
        *reinterpret_cast<uint4*>(dst + r * row_bytes + (lane & 7) * 16) = *reinterpret_cast<const uint4*>(stage + swz128(r, lane & 7));
    }
    __syncwarp();
  };
#pragma unroll
  for (int dt = 0; dt < 8; ++dt)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[dt][e] *= inv[e >> 1];
  if (p.o_s) put(o, reinterpret_cast<uint8_t*>(p.o_s + (static_cast<int64_t>(bh) * p.Tq + static_cast<int64_t>(qb) * 16) * 64), 128);
  if (p.y) {
    const int b = bh / p.H, h = bh - b * p.H;
    float g0[2], g1[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(p.gate + b * p.gsb + h * p.gsh + min(t0 + 8 * r, p.Tq - 1) * p.gst);
      g0[r] = bf16_lo(w); g1[r] = bf16_hi(w);
    }
    const uint32_t* oc = reinterpret_cast<const uint32_t*>(p.o_c) + task * 32 + c;
#pragma unroll
    for (int dt = 0; dt < 8; ++dt) {
      const uint32_t w = oc[dt * 4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[dt][e] = g0[e >> 1] * ((e & 1) ? bf16_hi(w) : bf16_lo(w)) + g1[e >> 1] * o[dt][e];
    }
    put(o, reinterpret_cast<uint8_t*>(p.y + ((static_cast<int64_t>(b) * p.Tq + static_cast<int64_t>(qb) * 16) * p.H + h) * 64),
        static_cast<int64_t>(p.H) * 128);
  }
}

static int launch_sel16_fwd(const PairMap& mkv, const Sel16Params& p, int64_t ntasks, cudaStream_t st) {
  S3R_REQUIRE(ntasks < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_sel_attn_fwd: grid of %lld CTAs is too large", (long long)ntasks);
  auto* kernel = mkv.apart ? sel16_fwd_kernel<true> : sel16_fwd_kernel<false>;
  S3R_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSel16Smem));
  return launch(kernel, static_cast<unsigned>(ntasks), 32, kSel16Smem, st, mkv, p);
}

}  // namespace s3r

using namespace s3r;

extern "C" int s3r_sel_attn_fwd(const void* q, const void* k, const void* v, int kv_chunks, int64_t kv_chunk_stride,
                                const int32_t* idx, void* o_s, float* lse_s, const void* gate,
                                int64_t gate_stride_b, int64_t gate_stride_h, int64_t gate_stride_t, const void* o_c,
                                void* y, int B, int H, int Tq, int Tk, int d, int block, int topk, float scale,
                                void* stream) {
  S3R_REQUIRE(q && k && v && idx, S3R_ERR_NULL, "s3r_sel_attn_fwd: q, k, v and idx are required");
  S3R_REQUIRE(o_s || y, S3R_ERR_NULL, "s3r_sel_attn_fwd: at least one of o_s and y must be given");
  S3R_REQUIRE((gate != nullptr) == (y != nullptr) && (o_c != nullptr) == (y != nullptr), S3R_ERR_NULL,
              "s3r_sel_attn_fwd: gate, o_c and y must be given together");
  S3R_REQUIRE(B > 0 && H > 0 && Tq > 0 && Tk > 0 && topk > 0 && kv_chunks > 0, S3R_ERR_SHAPE,
              "s3r_sel_attn_fwd: sizes must be positive (B=%d H=%d Tq=%d Tk=%d topk=%d chunks=%d)", B, H, Tq, Tk, topk,
              kv_chunks);
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_sel_attn_fwd: head_dim %d not supported (64 only)", d);
  S3R_REQUIRE(block == 16 || block == 32 || block == 64, S3R_ERR_UNSUPPORTED,
              "s3r_sel_attn_fwd: block %d not supported (16, 32, 64)", block);
  S3R_REQUIRE(topk <= 64, S3R_ERR_UNSUPPORTED, "s3r_sel_attn_fwd: topk %d exceeds 64", topk);
  S3R_REQUIRE(scale > 0.f, S3R_ERR_UNSUPPORTED, "s3r_sel_attn_fwd: softmax scale must be positive");
  S3R_REQUIRE(Tk % kv_chunks == 0 && (kv_chunks == 1 || (Tk / kv_chunks) % block == 0), S3R_ERR_SHAPE,
              "s3r_sel_attn_fwd: Tk=%d must split into %d chunks of whole blocks", Tk, kv_chunks);
  const uintptr_t al = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                       reinterpret_cast<uintptr_t>(o_s) | reinterpret_cast<uintptr_t>(y) |
                       reinterpret_cast<uintptr_t>(o_c);
  S3R_REQUIRE((al & 15) == 0 && (kv_chunk_stride % 8) == 0, S3R_ERR_ALIGNMENT,
              "s3r_sel_attn_fwd: tensors must be 16-byte aligned");
  S3R_REQUIRE(!gate || ((reinterpret_cast<uintptr_t>(gate) & 3) == 0 && gate_stride_b % 2 == 0 &&
                        gate_stride_h % 2 == 0 && gate_stride_t % 2 == 0),
              S3R_ERR_ALIGNMENT, "s3r_sel_attn_fwd: gate pairs must be 4-byte aligned");

  const int BH = B * H;
  const int Tc = Tk / kv_chunks;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* status = device_status_ptr();
  S3R_REQUIRE(status != nullptr, S3R_ERR_DRIVER, "s3r_sel_attn_fwd: could not resolve the device status word");
  if (block == 16) {
    Sel16Params p;
    p.q = static_cast<const __nv_bfloat16*>(q);
    p.idx = idx;
    p.o_s = static_cast<__nv_bfloat16*>(o_s);
    p.lse_s = lse_s;
    p.gate = static_cast<const __nv_bfloat16*>(gate);
    p.gsb = gate_stride_b; p.gsh = gate_stride_h; p.gst = gate_stride_t;
    p.o_c = static_cast<const __nv_bfloat16*>(o_c);
    p.y = static_cast<__nv_bfloat16*>(y);
    p.H = H; p.Tq = Tq; p.Tk = Tk; p.Tc = Tc;
    p.nqb = (Tq + 15) / 16;
    p.topk = topk;
    p.scale_log2e = scale * 1.4426950408889634f;
    p.status = status;
    PairMap mkv;
    const int rc = make_pair_map(&mkv, k, v, Tk, BH, kv_chunks, kv_chunk_stride * 2);
    if (rc) return rc;
    return launch_sel16_fwd(mkv, p, static_cast<int64_t>(BH) * p.nqb, st);
  }
  SelParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.kv_chunk_stride = kv_chunk_stride;
  p.idx = idx;
  p.o_s = static_cast<__nv_bfloat16*>(o_s);
  p.lse_s = lse_s;
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.gsb = gate_stride_b; p.gsh = gate_stride_h; p.gst = gate_stride_t;
  p.o_c = static_cast<const __nv_bfloat16*>(o_c);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.B = B; p.H = H; p.Tq = Tq; p.Tk = Tk; p.Tc = Tc;
  p.nqb = (Tq + block - 1) / block;
  p.topk = topk;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.status = status;
  return sel_big_fwd(kv_chunks, block, p, st);
}
