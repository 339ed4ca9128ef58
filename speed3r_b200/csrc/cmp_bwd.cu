// Compression branch, backward: dense flash-attention backward over the pooled tensors on the
// tensor-memory MMA (tcgen05), operands staged by TMA.
//
//   delta = sum_d o*do                                  (s3r_delta)
//   dK/dV: a CTA owns 128 key rows and streams all query tiles of 128 rows
//        S^T = K Q^T, dP^T = V dO^T                     (M=128 keys, N=128 queries, K=64)
//        P^T = exp2(S^T*c - lse[q]),  dS^T = P^T * (dP^T - delta[q])        thread = key row
//        dV += P^T dO,  dK += dS^T Q                    (M=128, N=64, K=128 queries; A from tensor memory)
//   dQ   : a CTA owns 128 query rows and streams all key tiles of 128 rows
//        S = Q K^T, dP = dO V^T;  dS = exp2(S*c - lse[row]) * (dP - delta[row]);  dQ += dS K
// P and dS are rounded to bf16 before the second products, like the reference kernels
// (flash_attention_topk.py:246-512); the softmax scale of dS is applied once, to the dK / dQ accumulators.
//
// One template covers both: the CTA's own tiles X0, X1 (K,V or Q,dO) are the A operands of the first
// products, the streamed tiles Y0, Y1 (Q,dO or K,V) their B operands (K-major) and, read with
// the other descriptor, the B operands of the second products (N contiguous).
// Tensor memory holds S twice, so that the next tile's scores are there when a tile's gradients are done, dP, and two accumulators of
// 64 columns.  dQ's own tiles live in tensor memory, where dK/dV has its second accumulators: a product with both operands in shared
// memory reads (128 + N) x 32 bytes of it per k-step at 128 a cycle, M=128 N=64 in 48 cycles instead of its 32, N=128 in its 64.
// Roles: warp 0 TMA producer, warp 1 tcgen05.mma issuer, warp 2 tensor-memory allocator, warp 3 loads the
// streamed rows' lse/delta (dK/dV), warps 4-19 compute: a row has four threads, each with 32 of a tile's columns.  P and dS are
// written in place, over the low half of a thread's own columns of S and dP (its bf16 chunk c covers its columns 8c..8c+7, all of
// which it has read by then).  A tile goes through two passes - P from S (kept in registers as fp32), then dS from
// dP - each with its own pair of barriers.
// Bound: up to 2400 rows the chain of a tile (1845 cycles for dK/dV, 1460 for dQ, of which the exponentials' unit is busy 1024 and the
// tensor pipe 1024 | 768), beyond that the power limit: the clock falls to 1.7 GHz.  Issuing a product blocks for as long as the pipe
// takes for it (its queue holds one), so that all that the issuing warp does in between - waits that are over, address arithmetic, the
// branch around an elected lane - is time in which the pipe idles.  Before (256 own rows, tiles of 64, one S: 1930 and 1410 cycles for
// half as many columns of twice as many rows) that warp was what a period took.  With delta, 16 heads, us: 2400 x 2400 125 -> 107,
// 4032 x 4032 268 -> 259, 6300 x 6300 633 -> 615, 15750 x 15750 3689 -> 3605.  Tried: two streams of tiles of 64 with S twice in each
// (6300: 670; asking ahead and without the branch 631), compute warps that ask for their barriers ahead too (637).
// Both kinds of CTA are in one grid, dK/dV first: they do not depend on each other, and a small grid of one kind leaves
// SMs idle.
#include "common.cuh"

namespace s3r {

constexpr int kCbThreads = 640;
// registers: the launch gives every thread 96, the utility warps hand some of theirs over (640 x 96 = 61440 >= 512 x 104 + 128 x 56)
constexpr int kCbComputeRegs = 104, kCbUtilityRegs = 56;
constexpr int kCbStages = 5;
constexpr int kCbTile = 128 * 128;            // 128 rows x 64 bf16, bytes
constexpr int kCbOffX = 0;                                    // own X0, X1 behind it
constexpr int kCbOffY = 2 * kCbTile;                          // ring of (Y0, Y1)
constexpr int kCbOffStat = kCbOffY + kCbStages * 2 * kCbTile; // ring of 128 x -lse2, 128 x -delta
constexpr int kCbSmemBytes = kCbOffStat + kCbStages * 1024 + 1024;
// tensor-memory columns: S buffer b at 128 b, dP at 256 (P and dS in the first 16 of each 32 columns), accumulators at 384 (dV; dQ:
// its own tiles, q and dO) and 448 (dK | dQ)
constexpr uint32_t kCbColDP = 256, kCbColAcc = 384, kCbColAcc1 = 448;

struct CbCtl {
  uint64_t x_full, o_full, drained;
  uint64_t y_full[kCbStages], y_empty[kCbStages], st_full[kCbStages];
  uint64_t s_full[2], p_full[2], dp_full, ds_full;
  uint32_t tmem_base;
  uint32_t abort_flag;
};

struct CbParams {
  const __nv_bfloat16 *x0, *x1;  // dQ: q and dO
  const float *lse, *delta;      // [BH, Nq]
  __nv_bfloat16 *out0, *out1;    // dK/dV kernel: dV, dK [BH, Nc, 64];  dQ kernel: unused, dQ [BH, Nq, 64]
  int n_own, n_str;              // rows of the owned and of the streamed tensors (Nc, Nq | Nq, Nc)
  int Nq;
  float cs, scale;               // softmax scale * log2(e), softmax scale
  uint32_t* status;
};

// MODE 0: dK/dV (own = K, V; streamed = Q, dO).  MODE 1: dQ (own = Q, dO; streamed = K, V).  `cta`: which 256 own rows.
template <int MODE>
__device__ __forceinline__ void cmp_bwd_cta(const CUtensorMap& map_x0, const CUtensorMap& map_x1, const CUtensorMap& map_y0,
                                            const CUtensorMap& map_y1, const CbParams& p, CbCtl& ctl, uint8_t* smem_raw, int cta) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int own_tiles = (p.n_own + 127) / 128;
  const int bh = cta / own_tiles;
  const int r0 = (cta % own_tiles) * 128;
  const int ntiles = (p.n_str + 127) / 128;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sptr = smem_raw + (sbase - smem_u32(smem_raw));
  float* stats = reinterpret_cast<float*>(sptr + kCbOffStat);        // [stage][-lse2 x 128 | -delta x 128]

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    mbar_init(&ctl.x_full, MODE == 0 ? 1 : 16);
    mbar_init(&ctl.o_full, 1);
    mbar_init(&ctl.drained, 1);
    for (int s = 0; s < kCbStages; ++s) {
      mbar_init(&ctl.y_full[s], 1);
      mbar_init(&ctl.y_empty[s], 1);
      mbar_init(&ctl.st_full[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl.s_full[b], 1);
      mbar_init(&ctl.p_full[b], 16);
    }
    mbar_init(&ctl.dp_full, 1);
    mbar_init(&ctl.ds_full, 16);
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(&ctl.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_wait();
  griddep_launch();
  const uint32_t tmem = ctl.tmem_base;
  volatile uint32_t* abort_flag = &ctl.abort_flag;

  if (warp < 4) {
  reg_dealloc<kCbUtilityRegs>();
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      if (MODE == 0) {
        mbar_expect_tx(&ctl.x_full, 2 * kCbTile);
        tma_load_3d(sbase + kCbOffX, &map_x0, &ctl.x_full, 0, r0, bh);
        tma_load_3d(sbase + kCbOffX + kCbTile, &map_x1, &ctl.x_full, 0, r0, bh);
      }
      int issued = 0;
      for (int i = 0; i < ntiles; ++i) {
        const int s = i % kCbStages;
        if (!mbar_wait(&ctl.y_empty[s], ((i / kCbStages) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(&ctl.y_full[s], 2 * kCbTile);
        tma_load_3d(sbase + kCbOffY + s * 2 * kCbTile, &map_y0, &ctl.y_full[s], 0, i * 128, bh);
        tma_load_3d(sbase + kCbOffY + s * 2 * kCbTile + kCbTile, &map_y1, &ctl.y_full[s], 0, i * 128, bh);
        issued = i + 1;
      }
      if (*abort_flag) {
        // give copies already in flight a bounded chance to land before the CTA's memory is released
        for (int i = max(0, issued - kCbStages); i < issued; ++i) {
          volatile uint32_t dummy = 0;
          mbar_wait(&ctl.y_full[i % kCbStages], (i / kCbStages) & 1, &dummy);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (converged warp, one elected lane issues)
    {
      const bool leader = elect_one_sync();
      const uint32_t lead = leader;
      constexpr uint32_t idesc_1 = umma_idesc_bf16(128, 128, 0, 0);   // both operands K-major
      constexpr uint32_t idesc_2 = umma_idesc_bf16(128, 64, 0, 1);    // B = streamed tile read as [rows][64]: N contiguous
      // descriptors are built once; a tile's descriptor is the base plus its byte offset / 16
      const uint64_t desc_x = umma_desc_sw128(sbase + kCbOffX), desc_y = umma_desc_sw128(sbase + kCbOffY);
      const uint32_t acc = tmem + kCbColAcc, acc1 = tmem + kCbColAcc1, dp = tmem + kCbColDP;
      // The MMAs of streamed tile i come in two groups:
      //   A(i): [P of tile i stored]   dV += P^T dO    then   S of tile i + 2, into the same buffer   -> s_full
      //   B(i): [dS of tile i stored]  dK += dS^T Q    then   dP of tile i + 1                        -> dp_full
      // S and dP are overwritten by MMAs issued behind the MMAs that read P and dS from the same columns; the tensor pipe runs
      // them in issue order.  Issuing blocks at the pipe's rate, so whatever this warp does between two groups is time in which
      // the pipe idles: what the next group waits for is asked before the present one is issued.
      auto ydesc = [&](int st) { return desc_y + static_cast<uint64_t>(st * (2 * kCbTile >> 4)); };
      // the CTA's own operand from shared memory, or from tensor memory
      auto issue_s = [&](int i, int st) {
        if (MODE == 0) umma_ss_k4_by<2, 2>(lead, tmem + (i & 1) * 128, desc_x, ydesc(st), idesc_1, 0u);
        else umma_ts_k4_by<2>(lead, tmem + (i & 1) * 128, acc, ydesc(st), idesc_1, 0u);
        umma_commit_by(lead, &ctl.s_full[i & 1]);
      };
      auto issue_dp = [&](int st) {
        const uint64_t y1 = ydesc(st) + (kCbTile >> 4);
        if (MODE == 0) umma_ss_k4_by<2, 2>(lead, dp, desc_x + (kCbTile >> 4), y1, idesc_1, 0u);
        else umma_ts_k4_by<2>(lead, dp, acc + 32, y1, idesc_1, 0u);
        umma_commit_by(lead, &ctl.dp_full);
      };
      auto accumulate = [&](uint32_t d, uint32_t a, uint64_t y, uint32_t go_on) {
        umma_ts_k4_by<128, 24>(lead, d, a, y, idesc_2, go_on);
        umma_ts_k4_by<128, 24>(lead, d, a + 64, y + 4 * 128, idesc_2, 1u);
      };
      bool ok = mbar_wait_warp(&ctl.x_full, 0, abort_flag);
      for (int i = 0; i < 2 && i < ntiles && ok; ++i) {
        ok = mbar_wait_warp(&ctl.y_full[i], 0, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_s(i, i);
        if (i == 0) issue_dp(0);
      }
      auto next_stage = [](int st) { return st + 1 == kCbStages ? 0 : st + 1; };
      int st = 0, st1 = 1, st2 = 2;                // ring stages of tiles i, i + 1, i + 2
      uint32_t ph2 = 0;                            // phase of the last
      bool p_done = false, y_done = false;
#pragma unroll 1
      for (int i = 0; i < ntiles && ok; ++i) {
        const bool more = i + 2 < ntiles;
        ok = mbar_settle(p_done, &ctl.p_full[i & 1], (i >> 1) & 1, abort_flag);
        if (ok && more) ok = mbar_settle(y_done, &ctl.y_full[st2], ph2, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const bool ds_done = mbar_test(&ctl.ds_full, i & 1);
        if (MODE == 0) accumulate(acc, tmem + (i & 1) * 128, ydesc(st) + (kCbTile >> 4), i > 0 ? 1u : 0u);
        if (more) issue_s(i + 2, st2);
        st2 = next_stage(st2);
        if (st2 == 0) ph2 ^= 1u;
        ok = mbar_settle(ds_done, &ctl.ds_full, i & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        p_done = i + 1 < ntiles && mbar_test(&ctl.p_full[(i + 1) & 1], ((i + 1) >> 1) & 1);
        y_done = i + 3 < ntiles && mbar_test(&ctl.y_full[st2], ph2);
        accumulate(acc1, dp, ydesc(st), i > 0 ? 1u : 0u);
        umma_commit_by(lead, &ctl.y_empty[st]);
        if (i + 1 < ntiles) issue_dp(st1);
        st = st1;
        st1 = next_stage(st1);
      }
      ok = __all_sync(0xffffffffu, ok);
      if (leader) umma_commit(ok ? &ctl.o_full : &ctl.drained);      // who waits for results gets none from a CTA that gave up
      __syncwarp();
      if (!ok) {
        volatile uint32_t dummy = 0;
        mbar_wait(&ctl.drained, 0, &dummy);       // let issued MMAs drain before tensor memory is freed
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ lse / delta of the streamed rows (dK/dV kernel)
    if (MODE == 0) {
      for (int i = 0; i < ntiles; ++i) {
        const int s = i % kCbStages;
        if (!mbar_wait_warp(&ctl.y_empty[s], ((i / kCbStages) & 1) ^ 1, abort_flag)) break;
        float* dst = stats + s * 256;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int q = i * 128 + h * 32 + lane;
          const bool in = q < p.n_str;
          // rows past the end: lse = +inf makes P exactly 0
          dst[h * 32 + lane] = in ? -(p.lse[static_cast<int64_t>(bh) * p.Nq + q] * 1.4426950408889634f) : -INFINITY;
          dst[128 + h * 32 + lane] = in ? -p.delta[static_cast<int64_t>(bh) * p.Nq + q] : 0.f;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.st_full[s]);
      }
    }
  }
  } else {
    // ------------------------------------------------------------------ compute, four threads per owned row
    reg_alloc<kCbComputeRegs>();
    const int cols = ((warp - 4) >> 2) * 32;                  // this warpgroup's columns of a tile
    const int quarter = warp & 3;
    const int row = r0 + quarter * 32 + lane;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_dp = lane_base + kCbColDP + cols;
    const float cs = p.cs;
    float my_lse2 = -INFINITY, my_delta = 0.f;      // dQ: this row's statistics, negated
    if (MODE == 1 && row < p.n_own) {
      my_lse2 = -(p.lse[static_cast<int64_t>(bh) * p.Nq + row] * 1.4426950408889634f);
      my_delta = -p.delta[static_cast<int64_t>(bh) * p.Nq + row];
    }
    if (MODE == 1) {
      // this thread's quarter of the own operands, 32 channels of q or dO, to where dK/dV has its first accumulators
      uint32_t x[16];
      const uint4* src = reinterpret_cast<const uint4*>((cols & 64 ? p.x1 : p.x0) + (static_cast<int64_t>(bh) * p.n_own + row) * 64 + (cols & 32));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 v = row < p.n_own ? __ldg(src + i) : make_uint4(0u, 0u, 0u, 0u);
        x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
      }
      tmem_st16(lane_base + kCbColAcc + cols / 2, x);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.x_full);
    }
    bool ok = true;
    float pf[32];                                   // P of this row against 32 of the tile's streamed rows
    auto arrive = [&](uint64_t* bar) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    for (int i = 0; i < ntiles; ++i) {
      const int s = i % kCbStages;
      const uint32_t t_s = lane_base + (i & 1) * 128 + cols;
      if (!mbar_wait_warp(&ctl.s_full[i & 1], (i >> 1) & 1, abort_flag)) { ok = false; break; }
      if (MODE == 0 && !mbar_wait_warp(&ctl.st_full[s], (i / kCbStages) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const float4* st4 = reinterpret_cast<const float4*>(stats + s * 256 + cols);
      // pass 1: P = exp2(S c - lse), kept in registers; dK/dV: bf16 P written over the low columns of S.  Tensor-memory
      // loads run one chunk ahead.
      auto pass1 = [&](const uint32_t (&xs)[16], int c) {
        uint32_t pk[8];
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) {
          float l4[4];
          if (MODE == 0) {
            const float4 a = st4[c * 4 + g4];         // same address in every lane: broadcast
            l4[0] = a.x; l4[1] = a.y; l4[2] = a.z; l4[3] = a.w;
          } else {
            l4[0] = l4[1] = l4[2] = l4[3] = my_lse2;
          }
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 x = ffma2(make_float2(__uint_as_float(xs[4 * g4 + e]), __uint_as_float(xs[4 * g4 + e + 1])), make_float2(cs, cs),
                             make_float2(l4[e], l4[e + 1]));
            pf[16 * c + 4 * g4 + e] = fast_exp2(x.x);
            pf[16 * c + 4 * g4 + e + 1] = fast_exp2(x.y);
          }
          if (MODE == 0) {
            pk[2 * g4] = pack_bf16(pf[16 * c + 4 * g4], pf[16 * c + 4 * g4 + 1]);
            pk[2 * g4 + 1] = pack_bf16(pf[16 * c + 4 * g4 + 2], pf[16 * c + 4 * g4 + 3]);
          }
        }
        if (MODE == 0) tmem_st8(t_s + c * 8, pk);
      };
      // pass 2: dS = P (dP - delta), written over the low columns of dP
      auto pass2 = [&](const uint32_t (&xd)[16], int c) {
        uint32_t dk[8];
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) {
          float d4[4];
          if (MODE == 0) {
            const float4 b = st4[32 + c * 4 + g4];
            d4[0] = b.x; d4[1] = b.y; d4[2] = b.z; d4[3] = b.w;
          } else {
            d4[0] = d4[1] = d4[2] = d4[3] = my_delta;
          }
          float dv[4];
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 d = fadd2(make_float2(__uint_as_float(xd[4 * g4 + e]), __uint_as_float(xd[4 * g4 + e + 1])),
                                   make_float2(d4[e], d4[e + 1]));
            const float2 m = fmul2(make_float2(pf[16 * c + 4 * g4 + e], pf[16 * c + 4 * g4 + e + 1]), d);
            dv[e] = m.x;
            dv[e + 1] = m.y;
          }
          dk[2 * g4] = pack_bf16(dv[0], dv[1]);
          dk[2 * g4 + 1] = pack_bf16(dv[2], dv[3]);
        }
        tmem_st8(t_dp + c * 8, dk);
      };
      uint32_t xa[16], xb[16];
      tmem_ld16(t_s, xa);
      tmem_ld16(t_s + 16, xb);
      tmem_ld_wait();
      if (MODE == 1) arrive(&ctl.p_full[i & 1]);
      // Streamed rows past the end.  dK/dV: P and dS are 0 for any scale, whatever the products with the zeros that stand for them are
      // (0 x inf, where a key is infinite): S becomes 0, from which the row's lse of +inf makes P = 0, and dP becomes 0.
      const int left = i == ntiles - 1 ? p.n_str - i * 128 - cols : 32;
      auto none_past = [&](uint32_t (&x)[16], int c) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (16 * c + e >= left) x[e] = 0u;
      };
      if (MODE == 0 && left < 32) {
        none_past(xa, 0);
        none_past(xb, 1);
      }
      pass1(xa, 0);
      pass1(xb, 1);
      // dQ: keys past the end have S = 0, whose P overflows where all of a row's logits are far below zero.  dS = P dP is 0 unless the
      // row's dO is infinite, which makes all of its dQ NaN through the other keys.
      if (MODE == 1 && left < 32) {
#pragma unroll
        for (int e = 0; e < 32; ++e)
          if (e >= left) pf[e] = 0.f;
      }
      if (MODE == 0) {
        tmem_st_wait();
        arrive(&ctl.p_full[i & 1]);
      }
      if (!mbar_wait_warp(&ctl.dp_full, i & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      tmem_ld16(t_dp, xa);
      tmem_ld16(t_dp + 16, xb);
      tmem_ld_wait();
      if (MODE == 0 && left < 32) {
        none_past(xa, 0);
        none_past(xb, 1);
      }
      pass2(xa, 0);
      pass2(xb, 1);
      tmem_st_wait();
      arrive(&ctl.ds_full);
    }
    // epilogue: accumulators -> bf16 (dK and dQ carry the softmax scale); dK/dV: the first two warpgroups have dV
    if (ok) ok = mbar_wait_warp(&ctl.o_full, 0, abort_flag);
    const int u = cols >> 6, half = (cols >> 5) & 1;
    if (ok && (MODE == 0 || u == 1)) {
      tc_fence_after();
      const float f = u == 0 ? 1.f : p.scale;
      __nv_bfloat16* out = (u == 0 ? p.out0 : p.out1) + (static_cast<int64_t>(bh) * p.n_own + row) * 64;
      uint32_t o[32];
      tmem_ld32(lane_base + (u == 0 ? kCbColAcc : kCbColAcc1) + half * 32, o);
      tmem_ld_wait();
      if (row < p.n_own) {
        uint4* dst = reinterpret_cast<uint4*>(out + half * 32);
#pragma unroll
        for (int v = 0; v < 4; ++v)
          dst[v] = make_uint4(pack_bf16(__uint_as_float(o[8 * v]) * f, __uint_as_float(o[8 * v + 1]) * f),
                              pack_bf16(__uint_as_float(o[8 * v + 2]) * f, __uint_as_float(o[8 * v + 3]) * f),
                              pack_bf16(__uint_as_float(o[8 * v + 4]) * f, __uint_as_float(o[8 * v + 5]) * f),
                              pack_bf16(__uint_as_float(o[8 * v + 6]) * f, __uint_as_float(o[8 * v + 7]) * f));
      }
    }
    if (!ok) {
      *abort_flag = 1u;
      if (lane == 0) atomicOr(p.status, kStatusWaitTimeout);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
}

struct CbMaps {
  CUtensorMap q, d_o, k, v;
};
__global__ void __launch_bounds__(kCbThreads, 1)
cmp_bwd_kernel(const __grid_constant__ CbMaps m, const CbParams kv, const CbParams q, const int kv_ctas) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ CbCtl ctl;
  if (static_cast<int>(blockIdx.x) < kv_ctas)
    cmp_bwd_cta<0>(m.k, m.v, m.q, m.d_o, kv, ctl, smem_raw, blockIdx.x);
  else
    cmp_bwd_cta<1>(m.q, m.d_o, m.k, m.v, q, ctl, smem_raw, static_cast<int>(blockIdx.x) - kv_ctas);
}

}  // namespace s3r

using namespace s3r;

extern "C" int s3r_cmp_attn_bwd_delta(const void* q_c, const void* k_c, const void* v_c, const float* lse, const void* do_c,
                                      const float* delta, void* dq_c, void* dk_c, void* dv_c, int B, int H, int Nq,
                                      int Nc, int d, float scale, void* stream) {
  S3R_REQUIRE(q_c && k_c && v_c && lse && do_c && delta && dq_c && dk_c && dv_c, S3R_ERR_NULL,
              "s3r_cmp_attn_bwd: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nc > 0, S3R_ERR_SHAPE, "s3r_cmp_attn_bwd: bad sizes");
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_cmp_attn_bwd: head_dim %d not supported (64 only)", d);
  const uintptr_t al = reinterpret_cast<uintptr_t>(q_c) | reinterpret_cast<uintptr_t>(k_c) | reinterpret_cast<uintptr_t>(v_c) |
                       reinterpret_cast<uintptr_t>(do_c) | reinterpret_cast<uintptr_t>(dq_c) |
                       reinterpret_cast<uintptr_t>(dk_c) | reinterpret_cast<uintptr_t>(dv_c);
  S3R_REQUIRE((al & 15) == 0, S3R_ERR_ALIGNMENT, "s3r_cmp_attn_bwd: tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = 0;
  const int BH = B * H;
  CbMaps m;
  {
    const uint32_t box[3] = {64, 128, 1};
    uint64_t dq_[3] = {64, static_cast<uint64_t>(Nq), static_cast<uint64_t>(BH)};
    uint64_t sq_[2] = {128, static_cast<uint64_t>(Nq) * 128};
    uint64_t dk_[3] = {64, static_cast<uint64_t>(Nc), static_cast<uint64_t>(BH)};
    uint64_t sk_[2] = {128, static_cast<uint64_t>(Nc) * 128};
    struct { CUtensorMap* m; const void* ptr; uint64_t* dims; uint64_t* strides; } maps[4] = {
        {&m.q, q_c, dq_, sq_}, {&m.d_o, do_c, dq_, sq_}, {&m.k, k_c, dk_, sk_}, {&m.v, v_c, dk_, sk_}};
    for (auto& e : maps) {
      rc = make_tensor_map(e.m, e.ptr, 3, e.dims, e.strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
      if (rc) return rc;
    }
  }
  CbParams p;
  p.x0 = p.x1 = nullptr;
  p.lse = lse; p.delta = delta;
  p.Nq = Nq;
  p.cs = scale * 1.4426950408889634f;
  p.scale = scale;
  p.status = device_status_ptr();
  S3R_REQUIRE(p.status != nullptr, S3R_ERR_DRIVER, "s3r_cmp_attn_bwd: could not resolve the device status word");
  S3R_CUDA(cudaFuncSetAttribute(cmp_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCbSmemBytes));
  // dK, dV: own = K, V (Nc rows), streamed = Q, dO (Nq rows); dQ: own = Q, dO (Nq rows), streamed = K, V (Nc rows)
  CbParams kv = p, q = p;
  kv.out0 = static_cast<__nv_bfloat16*>(dv_c);
  kv.out1 = static_cast<__nv_bfloat16*>(dk_c);
  kv.n_own = Nc; kv.n_str = Nq;
  q.x0 = static_cast<const __nv_bfloat16*>(q_c);
  q.x1 = static_cast<const __nv_bfloat16*>(do_c);
  q.out0 = nullptr;
  q.out1 = static_cast<__nv_bfloat16*>(dq_c);
  q.n_own = Nq; q.n_str = Nc;
  const int64_t g0 = static_cast<int64_t>(BH) * ((Nc + 127) / 128),
                g1 = static_cast<int64_t>(BH) * ((Nq + 127) / 128);
  S3R_REQUIRE(g0 + g1 < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_cmp_attn_bwd: grid too large");
  return launch(cmp_bwd_kernel, static_cast<unsigned>(g0 + g1), kCbThreads, kCbSmemBytes, st, m, kv, q, static_cast<int>(g0));
}

extern "C" int s3r_cmp_attn_bwd(const void* q_c, const void* k_c, const void* v_c, const void* o_c, const float* lse,
                                const void* do_c, float* delta, void* dq_c, void* dk_c, void* dv_c, int B, int H,
                                int Nq, int Nc, int d, float scale, void* stream) {
  S3R_REQUIRE(q_c && k_c && v_c && o_c && lse && do_c && delta && dq_c && dk_c && dv_c, S3R_ERR_NULL,
              "s3r_cmp_attn_bwd: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nc > 0, S3R_ERR_SHAPE, "s3r_cmp_attn_bwd: bad sizes");
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_cmp_attn_bwd: head_dim %d not supported (64 only)", d);
  const int rc = s3r_delta(o_c, do_c, delta, static_cast<int64_t>(B) * H * Nq, d, stream);
  if (rc) return rc;
  return s3r_cmp_attn_bwd_delta(q_c, k_c, v_c, lse, do_c, delta, dq_c, dk_c, dv_c, B, H, Nq, Nc, d, scale, stream);
}
