// Compression branch, backward: dense flash-attention backward over the pooled tensors on the
// tensor-memory MMA (tcgen05), operands staged by TMA.
//
//   delta = sum_d o*do                                  (s3r_delta)
//   dK/dV: a CTA owns 128 key rows and streams all query tiles of 128 rows (or owns 256 and streams tiles of 64)
//        S^T = K Q^T, dP^T = V dO^T                     (M=128 keys, N=128 | 64 queries, K=64)
//        P^T = exp2(S^T*c - lse[q]),  dS^T = P^T * (dP^T - delta[q])        thread = key row
//        dV += P^T dO,  dK += dS^T Q                    (M=128, N=64, K=128 | 64 queries; A from tensor memory)
//   dQ   : a CTA owns 128 | 256 query rows and streams all key tiles of 128 | 64 rows
//        S = Q K^T, dP = dO V^T;  dS = exp2(S*c - lse[row]) * (dP - delta[row]);  dQ += dS K
// P and dS are rounded to bf16 before the second products, like the reference kernels
// (flash_attention_topk.py:246-512); the softmax scale of dS is applied once, to the dK / dQ accumulators.
//
// One template covers both: the CTA's own tiles X0, X1 (K,V or Q,dO) are the A operands of the first
// products, the streamed tiles Y0, Y1 (Q,dO or K,V) their B operands (K-major) and, read with
// the other descriptor, the B operands of the second products (N contiguous).
// One own row tile (R = 1): tensor memory holds S twice, so that the next tile's scores are there when a tile's gradients are done, dP, and two accumulators of
// 64 columns.  dQ's own tiles live in tensor memory, where dK/dV has its second accumulators: a product with both operands in shared
// memory reads (128 + N) x 32 bytes of it per k-step at 128 a cycle, M=128 N=64 in 48 cycles instead of its 32, N=128 in its 64.
// Two (R = 2): S, dP and two accumulators of each, every one of 64 columns; while the warps of one row tile are in their exponentials,
// the other's multiply and pack.  A shorter grid for the same rows: two_row_tiles() has what it is for.
// Roles: warp 0 TMA producer, warp 1 tcgen05.mma issuer, warp 2 tensor-memory allocator, warp 3 loads the
// streamed rows' lse/delta (dK/dV), warps 4-19 compute: a row has four threads (R = 2: two), each with 32 of a tile's columns.  P and dS are
// written in place, over the low half of a thread's own columns of S and dP (its bf16 chunk c covers its columns 8c..8c+7, all of
// which it has read by then).  A tile goes through two passes - P from S (kept in registers as fp32), then dS from
// dP - each with its own pair of barriers.
// Bound: up to 2400 rows the chain of a tile (1845 cycles for dK/dV, 1460 for dQ, of which the exponentials' unit is busy 1024 and the
// tensor pipe 1024 | 768), beyond that the power limit: the clock falls to 1.7 GHz.  Issuing a product blocks for as long as the pipe
// takes for it (its queue holds one), so that all that the issuing warp does in between - waits that are over, address arithmetic, the
// branch around an elected lane - is time in which the pipe idles.  With two row tiles (1930 and 1410 cycles for half as many columns
// of twice as many rows) that warp is what a period takes.  Two row tiles throughout -> one, with delta, 16 heads, us: 2400 x 2400 125 -> 107,
// 4032 x 4032 268 -> 259, 6300 x 6300 633 -> 615, 15750 x 15750 3689 -> 3605.  Tried: two streams of tiles of 64 with S twice in each
// (6300: 670; asking ahead and without the branch 631), compute warps that ask for their barriers ahead too (637).
// Both kinds of CTA are in one grid, dK/dV first: they do not depend on each other, and a small grid of one kind leaves
// SMs idle.
#include "common.cuh"

namespace s3r {

constexpr int kCbThreads = 640;
// registers: the launch gives every thread 96, the utility warps hand some of theirs over (640 x 96 = 61440 >= 512 x 104 + 128 x 56)
constexpr int kCbComputeRegs = 104, kCbUtilityRegs = 56;
constexpr int kCbOwn = 128 * 128;             // 128 rows x 64 bf16, bytes
// R: own row tiles of 128 per CTA
template <int R>
struct CbCfg {
  static constexpr int kRows = 128 * R, kTile = 128 / R, kStages = R == 1 ? 5 : 6;      // own rows, rows of a streamed tile
  static constexpr int kStr = kTile * 128;                           // a streamed tile, bytes
  static constexpr int kOffX = 0;                                    // row tile t: X0 at t * 2 * kCbOwn, X1 behind it
  static constexpr int kOffY = 2 * R * kCbOwn;                       // ring of (Y0, Y1)
  static constexpr int kOffStat = kOffY + kStages * 2 * kStr;        // ring of kTile x -lse2, kTile x -delta
  static constexpr int kSmem = kOffStat + kStages * kTile * 8 + 1024;
  // tensor-memory columns: S buffer b (R = 1) or of row tile b (R = 2) at 128 b, dP (P and dS in the first 16 of each 32 columns),
  // accumulators: dV (dQ: its own tiles, q and dO) and dK | dQ; of row tile 1 all 128 further
  static constexpr uint32_t kColDP = R == 1 ? 256 : 64, kColAcc = R == 1 ? 384 : 256, kColAcc1 = kColAcc + 64;
};
constexpr int kCbMaxStages = 6;

struct CbCtl {
  uint64_t x_full, o_full, drained;
  uint64_t y_full[kCbMaxStages], y_empty[kCbMaxStages], st_full[kCbMaxStages];
  uint64_t s_full[2], p_full[2], dp_full[2], ds_full[2];       // R = 1: s and p per buffer, the others' first; R = 2: per row tile
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

// MODE 0: dK/dV (own = K, V; streamed = Q, dO).  MODE 1: dQ (own = Q, dO; streamed = K, V).  `cta`: which 128 R own rows.
template <int R, int MODE>
__device__ __forceinline__ void cmp_bwd_cta(const CUtensorMap& map_x0, const CUtensorMap& map_x1, const CUtensorMap& map_y0,
                                            const CUtensorMap& map_y1, const CbParams& p, CbCtl& ctl, uint8_t* smem_raw, int cta) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  using C = CbCfg<R>;
  constexpr int kStages = C::kStages;
  const int own_tiles = (p.n_own + C::kRows - 1) / C::kRows;
  const int bh = cta / own_tiles;
  const int r0 = (cta % own_tiles) * C::kRows;
  const int ntiles = (p.n_str + C::kTile - 1) / C::kTile;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sptr = smem_raw + (sbase - smem_u32(smem_raw));
  float* stats = reinterpret_cast<float*>(sptr + C::kOffStat);       // [stage][-lse2 x kTile | -delta x kTile]

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    mbar_init(&ctl.x_full, MODE == 0 ? 1 : 16);
    mbar_init(&ctl.o_full, 1);
    mbar_init(&ctl.drained, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl.y_full[s], 1);
      mbar_init(&ctl.y_empty[s], 1);
      mbar_init(&ctl.st_full[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl.s_full[b], 1);
      mbar_init(&ctl.dp_full[b], 1);
      mbar_init(&ctl.p_full[b], 16 / R);
      mbar_init(&ctl.ds_full[b], 16 / R);
    }
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
        mbar_expect_tx(&ctl.x_full, 2 * R * kCbOwn);
#pragma unroll
        for (int t = 0; t < R * R; ++t) {        // the maps' boxes are a streamed tile's rows
          const uint32_t at = sbase + C::kOffX + t / R * (2 * kCbOwn) + t % R * C::kStr;
          tma_load_3d(at, &map_x0, &ctl.x_full, 0, r0 + t * C::kTile, bh);
          tma_load_3d(at + kCbOwn, &map_x1, &ctl.x_full, 0, r0 + t * C::kTile, bh);
        }
      }
      int issued = 0;
      for (int i = 0; i < ntiles; ++i) {
        const int s = i % kStages;
        if (!mbar_wait(&ctl.y_empty[s], ((i / kStages) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(&ctl.y_full[s], 2 * C::kStr);
        tma_load_3d(sbase + C::kOffY + s * 2 * C::kStr, &map_y0, &ctl.y_full[s], 0, i * C::kTile, bh);
        tma_load_3d(sbase + C::kOffY + s * 2 * C::kStr + C::kStr, &map_y1, &ctl.y_full[s], 0, i * C::kTile, bh);
        issued = i + 1;
      }
      if (*abort_flag) {
        // give copies already in flight a bounded chance to land before the CTA's memory is released
        for (int i = max(0, issued - kStages); i < issued; ++i) {
          volatile uint32_t dummy = 0;
          mbar_wait(&ctl.y_full[i % kStages], (i / kStages) & 1, &dummy);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (converged warp, one elected lane issues)
    const bool leader = elect_one_sync();
    constexpr uint32_t idesc_1 = umma_idesc_bf16(128, C::kTile, 0, 0);    // both operands K-major
    constexpr uint32_t idesc_2 = umma_idesc_bf16(128, 64, 0, 1);          // B = streamed tile read as [rows][64]: N contiguous
    // descriptors are built once; a tile's descriptor is the base plus its byte offset / 16
    const uint64_t desc_x = umma_desc_sw128(sbase + C::kOffX), desc_y = umma_desc_sw128(sbase + C::kOffY);
    auto ydesc = [&](int st) { return desc_y + static_cast<uint64_t>(st * (2 * C::kStr >> 4)); };
    bool ok = mbar_wait_warp(&ctl.x_full, 0, abort_flag);
    if constexpr (R == 1) {
      const uint32_t lead = leader;
      const uint32_t acc = tmem + C::kColAcc, acc1 = tmem + C::kColAcc1, dp = tmem + C::kColDP;
      // The MMAs of streamed tile i come in two groups:
      //   A(i): [P of tile i stored]   dV += P^T dO    then   S of tile i + 2, into the same buffer   -> s_full
      //   B(i): [dS of tile i stored]  dK += dS^T Q    then   dP of tile i + 1                        -> dp_full
      // S and dP are overwritten by MMAs issued behind the MMAs that read P and dS from the same columns; the tensor pipe runs
      // them in issue order.  Issuing blocks at the pipe's rate, so whatever this warp does between two groups is time in which
      // the pipe idles: what the next group waits for is asked before the present one is issued.
      // the CTA's own operand from shared memory, or from tensor memory
      auto issue_s = [&](int i, int st) {
        if (MODE == 0) umma_ss_k4_by<2, 2>(lead, tmem + (i & 1) * 128, desc_x, ydesc(st), idesc_1, 0u);
        else umma_ts_k4_by<2>(lead, tmem + (i & 1) * 128, acc, ydesc(st), idesc_1, 0u);
        umma_commit_by(lead, &ctl.s_full[i & 1]);
      };
      auto issue_dp = [&](int st) {
        const uint64_t y1 = ydesc(st) + (C::kStr >> 4);
        if (MODE == 0) umma_ss_k4_by<2, 2>(lead, dp, desc_x + (kCbOwn >> 4), y1, idesc_1, 0u);
        else umma_ts_k4_by<2>(lead, dp, acc + 32, y1, idesc_1, 0u);
        umma_commit_by(lead, &ctl.dp_full[0]);
      };
      auto accumulate = [&](uint32_t d, uint32_t a, uint64_t y, uint32_t go_on) {
        umma_ts_k4_by<128, 24>(lead, d, a, y, idesc_2, go_on);
        umma_ts_k4_by<128, 24>(lead, d, a + 64, y + 4 * 128, idesc_2, 1u);
      };
      for (int i = 0; i < 2 && i < ntiles && ok; ++i) {
        ok = mbar_wait_warp(&ctl.y_full[i], 0, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_s(i, i);
        if (i == 0) issue_dp(0);
      }
      auto next_stage = [](int st) { return st + 1 == kStages ? 0 : st + 1; };
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
        const bool ds_done = mbar_test(&ctl.ds_full[0], i & 1);
        if (MODE == 0) accumulate(acc, tmem + (i & 1) * 128, ydesc(st) + (C::kStr >> 4), i > 0 ? 1u : 0u);
        if (more) issue_s(i + 2, st2);
        st2 = next_stage(st2);
        if (st2 == 0) ph2 ^= 1u;
        ok = mbar_settle(ds_done, &ctl.ds_full[0], i & 1, abort_flag);
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
    } else {
      // Per row tile t the MMAs come in two groups per streamed tile i:
      //   A(t,i): [P of tile i-1 stored]  dV += P^T dO (tile i-1)   then   S = X0 Y0^T (tile i)   -> s_full[t]
      //   B(t,i): [dS of tile i-1 stored] dK += dS^T Q (tile i-1)   then   dP = X1 Y1^T (tile i)  -> dp_full[t]
      // in the same order of overwriting as above, the two row tiles half a period apart -  A(0,i)  B(1,i-1)  B(0,i)  A(1,i).
      int st0 = 0, st1 = 0, st2 = 0;              // ring stages of tiles i, i-1, i-2
      uint32_t ph0 = 0;
      const uint64_t x_t0 = desc_x, x_t1 = desc_x + static_cast<uint64_t>(2 * kCbOwn >> 4);
      const uint32_t d0 = tmem + C::kColAcc, d1 = d0 + 128, b0 = tmem, b1 = tmem + 128;
      constexpr uint32_t kAcc1 = C::kColAcc1 - C::kColAcc;
      // S or dP of a row tile: its own operand from shared memory, or from tensor memory
      auto first_product = [&](uint32_t d, uint64_t x_smem, uint32_t x_tmem, uint64_t y) {
        if (MODE == 0) umma_ss_k4<2, 2>(d, x_smem, y, idesc_1, 0u);
        else umma_ts_k4<2>(d, x_tmem, y, idesc_1, 0u);
      };
#pragma unroll 1
      for (int i = 0; i <= ntiles && ok; ++i) {
        const bool more = i < ntiles;
        const uint64_t y0 = ydesc(st0), y1 = ydesc(st1), y2 = ydesc(st2);
        // A(0,i)
        if (more) ok = mbar_wait_warp(&ctl.y_full[st0], ph0, abort_flag);
        if (ok && i >= 1) ok = mbar_wait_warp(&ctl.p_full[0], (i - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          if (MODE == 0 && i >= 1) umma_ts_k4<128, 24>(d0, b0, y1 + (C::kStr >> 4), idesc_2, i > 1 ? 1u : 0u);
          if (more) {
            first_product(b0, x_t0, d0, y0);
            umma_commit(&ctl.s_full[0]);
          }
        }
        __syncwarp();
        // B(1,i-1)
        if (i >= 1) {
          if (i >= 2) {
            ok = mbar_wait_warp(&ctl.ds_full[1], i & 1, abort_flag);
            if (!ok) break;
          }
          tc_fence_after();
          if (leader) {
            if (i >= 2) umma_ts_k4<128, 24>(d1 + kAcc1, b1 + C::kColDP, y2, idesc_2, i > 2 ? 1u : 0u);
            first_product(b1 + C::kColDP, x_t1 + (kCbOwn >> 4), d1 + 32, y1 + (C::kStr >> 4));
            umma_commit(&ctl.dp_full[1]);
            if (i >= 2) umma_commit(&ctl.y_empty[st2]);
          }
          __syncwarp();
        }
        // B(0,i)
        if (i >= 1) {
          ok = mbar_wait_warp(&ctl.ds_full[0], (i - 1) & 1, abort_flag);
          if (!ok) break;
        }
        tc_fence_after();
        if (leader) {
          if (i >= 1) umma_ts_k4<128, 24>(d0 + kAcc1, b0 + C::kColDP, y1, idesc_2, i > 1 ? 1u : 0u);
          if (more) {
            first_product(b0 + C::kColDP, x_t0 + (kCbOwn >> 4), d0 + 32, y0 + (C::kStr >> 4));
            umma_commit(&ctl.dp_full[0]);
          }
        }
        __syncwarp();
        // A(1,i)
        if (i >= 1) {
          ok = mbar_wait_warp(&ctl.p_full[1], (i - 1) & 1, abort_flag);
          if (!ok) break;
        }
        tc_fence_after();
        if (leader) {
          if (MODE == 0 && i >= 1) umma_ts_k4<128, 24>(d1, b1, y1 + (C::kStr >> 4), idesc_2, i > 1 ? 1u : 0u);
          if (more) {
            first_product(b1, x_t1, d1, y0);
            umma_commit(&ctl.s_full[1]);
          }
        }
        __syncwarp();
        st2 = st1;
        st1 = st0;
        if (++st0 == kStages) { st0 = 0; ph0 ^= 1u; }
      }
      // the last dK of row tile 1: B(1, ntiles) without a next tile (after the shift st2 is the last tile's stage)
      if (ok) {
        ok = mbar_wait_warp(&ctl.ds_full[1], (ntiles - 1) & 1, abort_flag);
        if (ok) {
          tc_fence_after();
          if (leader) umma_ts_k4<128, 24>(d1 + kAcc1, b1 + C::kColDP, ydesc(st2), idesc_2, ntiles > 1 ? 1u : 0u);
          __syncwarp();
        }
      }
    }
    if (leader) umma_commit(ok ? &ctl.o_full : &ctl.drained);      // who waits for results gets none from a CTA that gave up
    __syncwarp();
    if (!ok) {
      volatile uint32_t dummy = 0;
      mbar_wait(&ctl.drained, 0, &dummy);       // let issued MMAs drain before tensor memory is freed
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ lse / delta of the streamed rows (dK/dV kernel)
    if (MODE == 0) {
      for (int i = 0; i < ntiles; ++i) {
        const int s = i % kStages;
        if (!mbar_wait_warp(&ctl.y_empty[s], ((i / kStages) & 1) ^ 1, abort_flag)) break;
        float* dst = stats + s * 2 * C::kTile;
#pragma unroll
        for (int h = 0; h < C::kTile / 32; ++h) {
          const int q = i * C::kTile + h * 32 + lane;
          const bool in = q < p.n_str;
          // rows past the end: lse = +inf makes P exactly 0
          dst[h * 32 + lane] = in ? -(p.lse[static_cast<int64_t>(bh) * p.Nq + q] * 1.4426950408889634f) : -INFINITY;
          dst[C::kTile + h * 32 + lane] = in ? -p.delta[static_cast<int64_t>(bh) * p.Nq + q] : 0.f;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.st_full[s]);
      }
    }
  }
  } else {
    // ------------------------------------------------------------------ compute, four or two threads per owned row
    reg_alloc<kCbComputeRegs>();
    const int t = R == 1 ? 0 : (warp - 4) >> 3, cols = ((warp - 4) >> 2) % (4 / R) * 32;     // this warpgroup's row tile and columns of a tile
    const int quarter = warp & 3;
    const int row = r0 + t * 128 + quarter * 32 + lane;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + t * 128;
    const uint32_t t_dp = lane_base + C::kColDP + cols;
    const float cs = p.cs;
    float my_lse2 = -INFINITY, my_delta = 0.f;      // dQ: this row's statistics, negated
    if (MODE == 1 && row < p.n_own) {
      my_lse2 = -(p.lse[static_cast<int64_t>(bh) * p.Nq + row] * 1.4426950408889634f);
      my_delta = -p.delta[static_cast<int64_t>(bh) * p.Nq + row];
    }
    if (MODE == 1) {
      // this thread's share of the own operands, 32 or 64 channels of q or dO, to where dK/dV has its first accumulators
      uint32_t x[16 * R];
      const int ch = cols * R;
      const uint4* src = reinterpret_cast<const uint4*>((ch & 64 ? p.x1 : p.x0) + (static_cast<int64_t>(bh) * p.n_own + row) * 64 + (ch & 32));
#pragma unroll
      for (int i = 0; i < 4 * R; ++i) {
        const uint4 v = row < p.n_own ? __ldg(src + i) : make_uint4(0u, 0u, 0u, 0u);
        x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
      }
      if constexpr (R == 1) tmem_st16(lane_base + C::kColAcc + ch / 2, x);
      else tmem_st32(lane_base + C::kColAcc + ch / 2, x);
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
      const int s = i % kStages, b = R == 1 ? i & 1 : t;                     // b: of S and P
      const uint32_t t_s = lane_base + (R == 1 ? b * 128 : 0) + cols;
      if (!mbar_wait_warp(&ctl.s_full[b], (R == 1 ? i >> 1 : i) & 1, abort_flag)) { ok = false; break; }
      if (MODE == 0 && !mbar_wait_warp(&ctl.st_full[s], (i / kStages) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const float4* st4 = reinterpret_cast<const float4*>(stats + s * 2 * C::kTile + cols);
      // pass 1: P = exp2(S c - lse), kept in registers; dK/dV: bf16 P written over the low columns of S
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
            const float4 a = st4[C::kTile / 4 + c * 4 + g4];
            d4[0] = a.x; d4[1] = a.y; d4[2] = a.z; d4[3] = a.w;
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
      if (MODE == 1) arrive(&ctl.p_full[b]);
      // Streamed rows past the end.  dK/dV: P and dS are 0 for any scale, whatever the products with the zeros that stand for them are
      // (0 x inf, where a key is infinite): S becomes 0, from which the row's lse of +inf makes P = 0, and dP becomes 0.
      const int left = i == ntiles - 1 ? p.n_str - i * C::kTile - cols : 32;
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
        arrive(&ctl.p_full[b]);
      }
      if (!mbar_wait_warp(&ctl.dp_full[t], i & 1, abort_flag)) { ok = false; break; }
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
      arrive(&ctl.ds_full[t]);
    }
    // epilogue: accumulators -> bf16 (dK and dQ carry the softmax scale); R = 1: the first two warpgroups have dV, the others dK | dQ
    if (ok) ok = mbar_wait_warp(&ctl.o_full, 0, abort_flag);
    if (ok) tc_fence_after();
    const int half = (cols >> 5) & 1;
#pragma unroll
    for (int u = max(R == 1 ? cols >> 6 : 0, MODE); ok && u <= (R == 1 ? cols >> 6 : 1); ++u) {
      const float f = u == 0 ? 1.f : p.scale;
      __nv_bfloat16* out = (u == 0 ? p.out0 : p.out1) + (static_cast<int64_t>(bh) * p.n_own + row) * 64;
      uint32_t o[32];
      tmem_ld32(lane_base + (u == 0 ? C::kColAcc : C::kColAcc1) + half * 32, o);
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
template <int R>
__global__ void __launch_bounds__(kCbThreads, 1)
cmp_bwd_kernel(const __grid_constant__ CbMaps m, const CbParams kv, const CbParams q, const int kv_ctas) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ CbCtl ctl;
  if (static_cast<int>(blockIdx.x) < kv_ctas)
    cmp_bwd_cta<R, 0>(m.k, m.v, m.q, m.d_o, kv, ctl, smem_raw, blockIdx.x);
  else
    cmp_bwd_cta<R, 1>(m.q, m.d_o, m.k, m.v, q, ctl, smem_raw, static_cast<int>(blockIdx.x) - kv_ctas);
}

// One own row tile per CTA, or two.  Starting a CTA, its first tile's chain and its epilogue take 4 us in which the tensor pipe idles;
// two row tiles halve how often that is, but a stream takes 1.9 times as long.  They pay where one row tile needs exactly twice the waves,
// the streams are short, and the last wave is not so empty that its CTAs follow the first ones to finish: the shorter the more
// CTAs there are.  One -> two, us: 32 heads 270 13.7 -> 12.0, 384 13.7 -> 12.9, 512 16.7 -> 15.7, 1024 46.2 -> 43.4, 1536 88.7 -> 85.1;
// 24 heads 768 20.5 and 20.5, 1536 63.2 -> 61.5; 48 heads 640 35.3 -> 31.7.  Beyond the line: 16 heads 640 17.1 and 18.0,
// 2048 75.0 and 74.8; 20 heads 512 15.4 and 15.6; 24 heads 2304 129 and 134; 12 heads 896 20.3 and 22.5.  In a single wave of two the
// streams of dK/dV, the longer ones where there are more queries than keys, are the end: 48 heads 430 x 111 10.5 and 12.6.
static bool two_row_tiles(int64_t BH, int64_t Nq, int64_t Nc) {
  const int64_t sms = sm_count(), tq = (Nq + 127) / 128, tc = (Nc + 127) / 128, longest = tq > tc ? tq : tc;
  const int64_t one = BH * (tq + tc), two = BH * ((tq + 1) / 2 + (tc + 1) / 2);
  return longest <= 16 && (two > sms || tq <= tc) && (one + sms - 1) / sms == 2 * ((two + sms - 1) / sms) && (longest + 1) * sms <= 4 * one;
}

template <int R>
static int launch_cmp_bwd(const void* q_c, const void* k_c, const void* v_c, const void* do_c, const CbParams& kv, const CbParams& q,
                          int BH, int Nq, int Nc, cudaStream_t st) {
  using C = CbCfg<R>;
  CbMaps m;
  const uint32_t box[3] = {64, C::kTile, 1};
  const uint64_t dq[3] = {64, static_cast<uint64_t>(Nq), static_cast<uint64_t>(BH)}, dk[3] = {64, static_cast<uint64_t>(Nc), static_cast<uint64_t>(BH)};
  const uint64_t sq[2] = {128, static_cast<uint64_t>(Nq) * 128}, sk[2] = {128, static_cast<uint64_t>(Nc) * 128};
  struct { CUtensorMap* m; const void* ptr; const uint64_t *dims, *strides; } maps[4] = {
      {&m.q, q_c, dq, sq}, {&m.d_o, do_c, dq, sq}, {&m.k, k_c, dk, sk}, {&m.v, v_c, dk, sk}};
  for (auto& e : maps) {
    const int rc = make_tensor_map(e.m, e.ptr, 3, e.dims, e.strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  S3R_CUDA(cudaFuncSetAttribute(cmp_bwd_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
  const int64_t g0 = static_cast<int64_t>(BH) * ((Nc + C::kRows - 1) / C::kRows),
                g1 = static_cast<int64_t>(BH) * ((Nq + C::kRows - 1) / C::kRows);
  S3R_REQUIRE(g0 + g1 < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_cmp_attn_bwd: grid too large");
  return launch(cmp_bwd_kernel<R>, static_cast<unsigned>(g0 + g1), kCbThreads, C::kSmem, st, m, kv, q, static_cast<int>(g0));
}

}  // namespace s3r

using namespace s3r;

static int cmp_attn_bwd(const void* q_c, const void* k_c, const void* v_c, const float* lse, const void* do_c, const float* delta,
                        void* dq_c, void* dk_c, void* dv_c, int B, int H, int Nq, int Nc, int d, float scale, bool alone, void* stream) {
  S3R_REQUIRE(q_c && k_c && v_c && lse && do_c && delta && dq_c && dk_c && dv_c, S3R_ERR_NULL,
              "s3r_cmp_attn_bwd: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nc > 0, S3R_ERR_SHAPE, "s3r_cmp_attn_bwd: bad sizes");
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_cmp_attn_bwd: head_dim %d not supported (64 only)", d);
  const uintptr_t al = reinterpret_cast<uintptr_t>(q_c) | reinterpret_cast<uintptr_t>(k_c) | reinterpret_cast<uintptr_t>(v_c) |
                       reinterpret_cast<uintptr_t>(do_c) | reinterpret_cast<uintptr_t>(dq_c) |
                       reinterpret_cast<uintptr_t>(dk_c) | reinterpret_cast<uintptr_t>(dv_c);
  S3R_REQUIRE((al & 15) == 0, S3R_ERR_ALIGNMENT, "s3r_cmp_attn_bwd: tensors must be 16-byte aligned");
  CbParams p;
  p.x0 = p.x1 = nullptr;
  p.lse = lse; p.delta = delta;
  p.Nq = Nq;
  p.cs = scale * 1.4426950408889634f;
  p.scale = scale;
  p.status = device_status_ptr();
  S3R_REQUIRE(p.status != nullptr, S3R_ERR_DRIVER, "s3r_cmp_attn_bwd: could not resolve the device status word");
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
  auto* go = alone && two_row_tiles(static_cast<int64_t>(B) * H, Nq, Nc) ? launch_cmp_bwd<2> : launch_cmp_bwd<1>;
  return go(q_c, k_c, v_c, do_c, kv, q, B * H, Nq, Nc, static_cast<cudaStream_t>(stream));
}

// With delta given this is the whole op's backward, beside which the table's inverse runs: it holds SMs until 5 us before this kernel's
// end, so that waves say little, and the shorter CTAs of one row tile end sooner behind it.  The op, forward and backward, 2 samples, 16
// heads, one row tile and two (where alone two are 6 % faster): 6144 tokens 497.4 and 498.8 us, 8192 656.3 and 658.4.
extern "C" int s3r_cmp_attn_bwd_delta(const void* q_c, const void* k_c, const void* v_c, const float* lse, const void* do_c,
                                      const float* delta, void* dq_c, void* dk_c, void* dv_c, int B, int H, int Nq,
                                      int Nc, int d, float scale, void* stream) {
  return cmp_attn_bwd(q_c, k_c, v_c, lse, do_c, delta, dq_c, dk_c, dv_c, B, H, Nq, Nc, d, scale, false, stream);
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
  return cmp_attn_bwd(q_c, k_c, v_c, lse, do_c, delta, dq_c, dk_c, dv_c, B, H, Nq, Nc, d, scale, true, stream);
}
