// Compression branch, forward, first of two kernels: dense attention of the pooled queries over the pooled keys, and
// for every row a lower bound of its topk-th largest raw logit (RANK 0) or score of a block of four columns (RANK 1),
// from which the second kernel (cmp_topk.cuh) picks the row's best columns or blocks.
//
// The two jobs want different things.  Attention is bound by the exponentials (one per score, 16 per cycle and SM);
// the top-k has to look at every score once but keeps 32 of tens of thousands, through branches that depend on the
// data.  Side by side in one kernel (softmax warps and top-k warps reading the same scores) each waited for the other
// tile by tile; the products, which the second kernel repeats, are cheap: the tensor pipe was a fifth busy.
// Measured (16 heads, one kernel before -> this one + cmp_topk.cuh): 6300 x 6300 1047 ->
// 223 + 244 us (scores that cluster by view and patch: 1923 -> 222 + 315), 7875 x 63000 5.81 -> 2.45 + 1.69 ms; both kernels
// 384 x 384 99 -> 19 to 34 us, depending on the inputs.
//
// The bound: a row keeps the running maxima of 64 groups of columns (half of S, piece of 16 in it and column mod 8).  topk of
// the maxima are >= the topk-th largest of the maxima, so at least topk logits are, and the topk-th largest logit is.  With
// topk = 32 about 64 ln 2 = 44 logits of a row with independent scores reach the bound, whatever the number of columns.
// The maxima cost half an instruction per score (three-input max) and no branch.
// Large scores come in runs of keys (the patches of a view the query looks at), which one group must not hold two of: the
// copies of whole tiles bring keys i and 64 + i to columns 16 (i / 8) + i mod 8 and 8 further, so that a group is the keys
// equal mod 64.  With the keys in order, 63 instead of 48 logits of one row in a hundred reached the bound and one list in four
// of the second kernel filled up (6300 x 6300, keys of a view alike: both kernels 1048 -> 425 us).
// RANK 1: compressed keys are finer than selection blocks (windows of Lc tokens every Sc, blocks of Bs = 4 * Sc), and a block's
// score is log2 of the sum of 2^(c * s) over its first rank_take columns.  The groups keep the largest sums of P instead,
// 16 groups per thread for even tiles and 16 for odd ones, keys in order.
//
// Roles (R row tiles of 128 queries per CTA, R = 1 or 2):
//   warp 0  TMA producer: Q tiles once, then K and V tiles of 128 keys into rings
//   warp 1  tcgen05.mma issuer (converged warp, one elected lane issues): S = Q K^T (M=128, N=128), O += P V (M=128, N=64)
//   warp 2  tensor-memory allocator
//   warps 4..: two softmax warpgroups per row tile; a row has two threads, each with half of every tile's columns
// (one thread per row leaves two warps per scheduler, whose dependent instructions nobody else's fill: 2.55 instead of
// 2.45 ms for 7875 x 63000).
// S of a tile is released as soon as its last columns are in registers, before their exponentials, so that the next
// Q K^T runs under the rest of the softmax; P has tensor memory of its own.  Tensor memory: R x (S 128, O 64, P 64) columns.
// An eighth of the exponentials (ranking blocks: a sixteenth) are polynomials on the FMA pipe: they relieve the exponentials' unit and
// cost issue slots, of which the running maxima and roundings leave few.  Both kernels, 15750 x 15750, 16 heads: none 2130 us, 1/16
// 2085, 1/8 2062, 1/4 2098, 5/16 2160; 7875 x 63000: 3763, 3653, 3610, 3688, 3742; ranking blocks, 3937 x 15747: 808, 810, 846, 848.
// The exponent offset of a row is the maximum of its first tile and does not move: P, O and l are floats, which keep their
// relative precision however far later scores outgrow the first tile's, up to their range.  A CTA in which some row's
// scores outgrew its offset by more than 2^64 takes its keys a second time with the rows' exact maxima, which the group
// maxima have found by then (rows beside such a row are then rounded from other offsets than in a launch that groups rows
// otherwise: results do not depend on the grouping only while no row is).  No maximum, vote or branch stands between one exponential and the next (a check per tile, with
// the tile redone: 2.90 ms; a check per 32 columns, with P rescaled: 3.40 ms).
#pragma once
#include <type_traits>

#include "common.cuh"
#include "cmp_common.cuh"

namespace s3r {

constexpr int kAtTile = 128 * 128;             // 128 rows x 64 bf16, bytes

template <int R>
struct AtCfg {
  static constexpr int kThreads = 128 + 256 * R;
  static constexpr int kStages = 3;
  static constexpr int kOffK = R * kAtTile;
  static constexpr int kOffV = kOffK + kStages * kAtTile;
  static constexpr int kOffXchg = kOffV + kStages * kAtTile;      // what the two threads of a row tell each other: R x 2 x 128 floats
  static constexpr int kSmem = kOffXchg + R * 1024 + 1024;
  static constexpr uint32_t kColO = R * 128, kColP = R * 192, kCols = R * 256;
  // registers: the launch gives every thread the same number, for R = 2 the utility warps hand some of theirs over
  // (640 x 96 at launch = 61440 = 512 x 112 + 128 x 32)
  static constexpr int kSoftmaxRegs = 112, kUtilityRegs = 32;
};

struct AtCtl {
  uint64_t q_full, o_full, drained;
  uint64_t k_full[3], k_empty[3], v_full[3], v_empty[3];
  uint64_t s_full[2], s_free[2], p_full[2], pv_done[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t again;               // some row's offset was too small: a second pass over the keys
};

struct AtParams {
  __nv_bfloat16* o;
  float* lse;
  float* bound;                // row r's bound goes to bound[r * topk]
  int Nq, Nc, topk;
  int scattered;               // leading tiles whose keys the copies spread over the column groups (map_ks, map_vs)
  int rank_take;               // RANK 1: columns of a block that count
  float c_scale;               // softmax scale * log2(e)
  uint32_t* status;
};

// `cta`: which R * 128 rows
template <int R, int RANK>
__device__ __forceinline__ void cmp_attn_cta(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v,
                                             const CUtensorMap& map_ks, const CUtensorMap& map_vs, const AtParams& p, AtCtl& ctl,
                                             uint8_t* smem_raw, int cta) {
  using C = AtCfg<R>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_per_bh = (p.Nq + R * 128 - 1) / (R * 128);
  const int bh = cta / tiles_per_bh;
  const int q0 = (cta % tiles_per_bh) * R * 128;
  const int ntiles = (p.Nc + 127) / 128;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float (*xchg)[2][128] = reinterpret_cast<float (*)[2][128]>(smem_raw + (sbase - smem_u32(smem_raw)) + C::kOffXchg);

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    ctl.again = 0;
    mbar_init(&ctl.q_full, 1);
    mbar_init(&ctl.o_full, 1);
    mbar_init(&ctl.drained, 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&ctl.k_full[s], 1);
      mbar_init(&ctl.k_empty[s], 1);
      mbar_init(&ctl.v_full[s], 1);
      mbar_init(&ctl.v_empty[s], 1);
    }
    for (int t = 0; t < R; ++t) {
      mbar_init(&ctl.s_full[t], 1);
      mbar_init(&ctl.s_free[t], 8);
      mbar_init(&ctl.p_full[t], 8);
      mbar_init(&ctl.pv_done[t], 1);
    }
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(&ctl.tmem_base, C::kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_wait();
  griddep_launch();
  const uint32_t tmem = ctl.tmem_base;
  volatile uint32_t* abort_flag = &ctl.abort_flag;

  // Tiles are counted through both passes (n = pass * ntiles + j): ring stages and phases follow n.  Every role meets the
  // others at the end of a pass and reads the same decision.
  auto another_pass = [&](int pass) {
    __syncthreads();
    return pass == 0 && *static_cast<volatile uint32_t*>(&ctl.again) != 0u && *abort_flag == 0u;
  };
  if (warp < 4) {
    if (R == 2) reg_dealloc<C::kUtilityRegs>();
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      int pass = 0;
      do {
        if (lane == 0) {
          if (pass == 0) {
            mbar_expect_tx(&ctl.q_full, R * kAtTile);
#pragma unroll
            for (int t = 0; t < R; ++t) tma_load_3d(sbase + t * kAtTile, &map_q, &ctl.q_full, 0, q0 + t * 128, bh);
          }
          int issued = pass * ntiles;
          for (int j = 0; j < ntiles; ++j) {
            const int n = pass * ntiles + j, s = n % C::kStages;
            const uint32_t ph = (n / C::kStages) & 1;
            if (!mbar_wait(&ctl.k_empty[s], ph ^ 1, abort_flag)) break;
            mbar_expect_tx(&ctl.k_full[s], kAtTile);
            const bool scattered = RANK == 0 && j < p.scattered;
            const uint32_t dst_k = sbase + C::kOffK + s * kAtTile, dst_v = sbase + C::kOffV + s * kAtTile;
            if (scattered) tma_load_5d(dst_k, &map_ks, &ctl.k_full[s], 0, 0, 0, j * 16, bh);
            else tma_load_3d(dst_k, &map_k, &ctl.k_full[s], 0, j * 128, bh);
            issued = n + 1;                                                 // K of tile n is in flight
            if (!mbar_wait(&ctl.v_empty[s], ph ^ 1, abort_flag)) break;
            mbar_expect_tx(&ctl.v_full[s], kAtTile);
            if (scattered) tma_load_5d(dst_v, &map_vs, &ctl.v_full[s], 0, 0, 0, j * 16, bh);
            else tma_load_3d(dst_v, &map_v, &ctl.v_full[s], 0, j * 128, bh);
          }
          if (*abort_flag) {
            // give copies already in flight a bounded chance to land before the CTA's memory is released
            for (int n = max(0, issued - C::kStages); n < issued; ++n) {
              volatile uint32_t dummy = 0;
              mbar_wait(&ctl.k_full[n % C::kStages], (n / C::kStages) & 1, &dummy);
            }
          }
        }
        __syncwarp();
      } while (another_pass(pass++));
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      const bool leader = elect_one_sync();
      constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, 64, 0, 1);         // V tile is [keys][d]: N contiguous
      const uint64_t desc_q = umma_desc_sw128(sbase), desc_k = umma_desc_sw128(sbase + C::kOffK),
                     desc_v = umma_desc_sw128(sbase + C::kOffV);
      auto issue_qk = [&](int t, int s) {
        umma_ss_k4<2, 2>(tmem + t * 128, desc_q + static_cast<uint64_t>(t * (kAtTile >> 4)),
                         desc_k + static_cast<uint64_t>(s * (kAtTile >> 4)), idesc_qk, 0u);
        umma_commit(&ctl.s_full[t]);
      };
      auto issue_pv = [&](int t, int s, uint32_t acc) {
        const uint64_t v = desc_v + static_cast<uint64_t>(s * (kAtTile >> 4));
        umma_ts_k4<128>(tmem + C::kColO + t * 64, tmem + C::kColP + t * 64, v, idesc_pv, acc);
        umma_ts_k4<128>(tmem + C::kColO + t * 64, tmem + C::kColP + t * 64 + 32, v + 4 * 128, idesc_pv, 1u);
        umma_commit(&ctl.pv_done[t]);
      };
      bool ok = mbar_wait_warp(&ctl.q_full, 0, abort_flag);
      int pass = 0, s = 0, n = 0;
      uint32_t ph = 0;
      do {
        ok = ok && mbar_wait_warp(&ctl.k_full[s], ph, abort_flag);
        if (ok) {
          tc_fence_after();
          if (leader) {
#pragma unroll
            for (int t = 0; t < R; ++t) issue_qk(t, s);
            umma_commit(&ctl.k_empty[s]);
          }
          __syncwarp();
        }
#pragma unroll 1
        for (int j = 0; j < ntiles && ok; ++j, ++n) {
          const bool nxt = j + 1 < ntiles;
          const int sn = s + 1 == C::kStages ? 0 : s + 1;
          const uint32_t phn = sn == 0 ? ph ^ 1u : ph;
          if (nxt) ok = mbar_wait_warp(&ctl.k_full[sn], phn, abort_flag);
          if (ok) ok = mbar_wait_warp(&ctl.v_full[s], ph, abort_flag);
          if (!ok) break;
#pragma unroll
          for (int t = 0; t < R; ++t) {
            if (nxt) {
              ok = mbar_wait_warp(&ctl.s_free[t], n & 1, abort_flag);       // S of tile n is in registers
              if (!ok) break;
              tc_fence_after();
              if (leader) issue_qk(t, sn);
              if (t == R - 1 && leader) umma_commit(&ctl.k_empty[sn]);
              __syncwarp();
            }
            ok = mbar_wait_warp(&ctl.p_full[t], n & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (leader) issue_pv(t, s, j > 0 ? 1u : 0u);
            if (t == R - 1 && leader) umma_commit(&ctl.v_empty[s]);
            __syncwarp();
          }
          s = sn;
          ph = phn;
        }
        if (leader) umma_commit(ok ? &ctl.o_full : &ctl.drained);           // who waits for results gets none from a CTA that gave up
        __syncwarp();
        if (!ok) {
          volatile uint32_t dummy = 0;
          mbar_wait(&ctl.drained, 0, &dummy);             // let issued MMAs drain before tensor memory is freed
        }
      } while (another_pass(pass++));
    } else {
      int pass = 0;
      while (another_pass(pass++)) {}
    }
  } else {
    // ------------------------------------------------------------------ softmax, two threads per row
    if (R == 2) reg_alloc<C::kSoftmaxRegs>();
    const int t = (warp - 4) >> 3, half = ((warp - 4) >> 2) & 1, quarter = warp & 3;
    const int r = quarter * 32 + lane, row = q0 + t * 128 + r;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_s = lane_base + t * 128 + half * 64, t_o = lane_base + C::kColO + t * 64 + half * 32,
                   t_p = lane_base + C::kColP + t * 64 + half * 32;
    const float cs = p.c_scale;
    float m_used = 0.f, l = 0.f;
    float gm[32];                               // running maxima of this half's 32 groups: raw logits, or sums of P
#pragma unroll
    for (int i = 0; i < 32; ++i) gm[i] = RANK ? 0.f : -INFINITY;
    float raw = -INFINITY;                      // RANK 1: largest raw logit
    auto half_max = [&]() {                     // of what is not NaN
      if (RANK) return fmaxf(raw, -INFINITY);
      float m[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        m[i] = fmax3(fmax3(gm[8 * i], gm[8 * i + 1], gm[8 * i + 2]), fmax3(gm[8 * i + 3], gm[8 * i + 4], gm[8 * i + 5]),
                     fmaxf(gm[8 * i + 6], gm[8 * i + 7]));
      return fmaxf(fmax3(m[0], m[1], m[2]), m[3]);
    };
    // the two warpgroups of a row tile; whatever has happened, every warp of both comes here
    auto meet = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + t) : "memory"); };
    auto both_max = [&]() {
      const float mine = half_max();
      xchg[t][half][r] = mine;
      meet();
      const float m = fmaxf(mine, xchg[t][half ^ 1][r]);
      meet();
      return m;
    };
    auto mask = [&](uint32_t (&x)[16], int c, int left) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (half * 64 + c * 16 + i >= left) x[i] = 0xff800000u;   // -inf
    };
    auto take_maxima = [&](const uint32_t (&x)[16], int c) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (RANK) raw = fmax3_nan(raw, __uint_as_float(x[i]), __uint_as_float(x[8 + i]));
        else gm[c * 8 + i] = fmax3_nan(gm[c * 8 + i], __uint_as_float(x[i]), __uint_as_float(x[8 + i]));
      }
    };
    const float2 w01 = make_float2(1.f, p.rank_take > 1 ? 1.f : 0.f),
                 w23 = make_float2(p.rank_take > 2 ? 1.f : 0.f, p.rank_take > 3 ? 1.f : 0.f);
    // one tile; TAIL: its columns from `left` on do not exist; RANK 1: the sums go to the 16 groups of parity ODD
    auto tile = [&](int n, bool first, auto tail, auto odd, int left) -> bool {
      constexpr bool TAIL = decltype(tail)::value;
      constexpr int ODD = decltype(odd)::value;
      if (!mbar_wait_warp(&ctl.s_full[t], n & 1, abort_flag)) return false;
      tc_fence_after();
      uint32_t xa[16], xb[16];
      tmem_ld16(t_s, xa);
      // P of the previous tile must have been consumed
      if (!first && !mbar_wait_warp(&ctl.pv_done[t], (n - 1) & 1, abort_flag)) return false;
      tc_fence_after();
      const float2 nm = make_float2(-m_used, -m_used), cs2 = make_float2(cs, cs);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      auto piece = [&](uint32_t (&x)[16], int c) {
        if (TAIL) mask(x, c, left);
        take_maxima(x, c);
        uint32_t pk[8];
        float2 counted = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float2 v = ffma2(make_float2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), cs2, nm);
          if (i == 0 && (RANK == 0 || (c & 1) == 0)) {
            v = exp2_fma2(v);
          } else {
            v.x = fast_exp2(v.x);
            v.y = fast_exp2(v.y);
          }
          sum[i & 1] = fadd2(sum[i & 1], v);
          if (RANK && (i & 1) == 0) counted = make_float2(v.x, v.y * w01.y);
          if (RANK && (i & 1) == 1) {
            counted = ffma2(v, w23, counted);
            const bool exists = !TAIL || half * 64 + c * 16 + 2 * (i - 1) + p.rank_take <= left;
            float& g = gm[ODD * 16 + c * 4 + i / 2];
            g = fmaxf(g, exists ? counted.x + counted.y : 0.f);
          }
          pk[i] = pack_bf16(v.x, v.y);
        }
        tmem_st8(t_p + c * 8, pk);
      };
      tmem_ld_wait();
      tmem_ld16(t_s + 16, xb);
      piece(xa, 0);
      tmem_ld_wait();
      tmem_ld16(t_s + 32, xa);
      piece(xb, 1);
      tmem_ld_wait();
      tmem_ld16(t_s + 48, xb);
      piece(xa, 2);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.s_free[t]);         // all of this half of S is in registers
      piece(xb, 3);
      l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.p_full[t]);
      return true;
    };
    // the offset: the maximum of the row's first tile
    bool ok = mbar_wait_warp(&ctl.s_full[t], 0, abort_flag);
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t x[16];
        tmem_ld16(t_s + c * 16, x);
        tmem_ld_wait();
        mask(x, c, p.Nc);
        take_maxima(x, c);
      }
    }
    m_used = both_max() * cs;
    int pass = 0;
    const int whole = p.Nc / 128;
    do {
      if (pass == 1) {
        l = 0.f;
        m_used = both_max() * cs;
        if (RANK) {
#pragma unroll
          for (int i = 0; i < 32; ++i) gm[i] = 0.f;
        }
      }
      int n = pass * ntiles;
#pragma unroll 1
      for (int j = 0; j < whole && ok; ++j, ++n) {
        if (RANK && (j & 1)) ok = tile(n, false, std::false_type(), std::integral_constant<int, RANK>(), 0);
        else ok = tile(n, j == 0, std::false_type(), std::integral_constant<int, 0>(), 0);
      }
      if (ok && whole < ntiles) {
        if (RANK && (whole & 1)) ok = tile(n, false, std::true_type(), std::integral_constant<int, RANK>(), p.Nc - whole * 128);
        else ok = tile(n, whole == 0, std::true_type(), std::integral_constant<int, 0>(), p.Nc - whole * 128);
      }
      if (ok) ok = mbar_wait_warp(&ctl.o_full, pass & 1, abort_flag);
      if (pass == 0 && !(half_max() * cs <= m_used + 64.f)) ctl.again = 1u;
    } while (another_pass(pass++));

    // A row with a NaN or an infinite score is NaN throughout; the polynomial exponentials have made numbers of them.  A
    // group with a NaN counts as empty: the bound stays one.
    bool bad = RANK && !(raw < INFINITY);
    if (!RANK) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        bad |= !(gm[i] < INFINITY);
        gm[i] = fmaxf(gm[i], -INFINITY);
      }
    }
    if (bad) l = __uint_as_float(0x7fffffffu);
    // epilogue: the bound (topk-th largest of the row's 64 maxima: with both threads' 32 sorted, the larger of a[i] and
    // b[topk - 1 - i] over i < topk are the upper topk), lse and O / l.  The K ring is free by now.
    sort_desc<32>(gm);
    float* other = reinterpret_cast<float*>(smem_raw + (sbase - smem_u32(smem_raw)) + C::kOffK) + t * (32 * 128) + r;     // [slot][row]
    if (half == 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i) other[i * 128] = gm[i];
    }
    xchg[t][half][r] = l;
    meet();
    l += xchg[t][half ^ 1][r];
    if (ok && half == 0 && row < p.Nq) {
      float bound = INFINITY;
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < p.topk) bound = fminf(bound, fmaxf(gm[i], other[(p.topk - 1 - i) * 128]));
      // a sum's logarithm, less what its exponentials and the second kernel's scores can differ by: 2^-20 from the
      // exponentials, and roundings of the arguments, each below 2^-24 of their size.  The polynomial exponentials are 2^-126
      // for anything smaller: a sum in which two of those are more than 2^-21 bounds nothing.
      if (RANK) bound = bound < 4.930380657631324e-32f /* 2^-104 */ ? -INFINITY
                                  : m_used + log2f(bound) - (6.103515625e-5f + 9.5367431640625e-7f * fabsf(m_used));
      p.bound[(static_cast<int64_t>(bh) * p.Nq + row) * p.topk] = bound;
      p.lse[static_cast<int64_t>(bh) * p.Nq + row] = (m_used + log2f(l)) * 0.6931471805599453f;
    }
    if (ok) {
      tc_fence_after();
      const float inv = 1.f / l;
      uint32_t o[32];
      tmem_ld32(t_o, o);
      tmem_ld_wait();
      if (row < p.Nq) {
        uint4* dst = reinterpret_cast<uint4*>(p.o + (static_cast<int64_t>(bh) * p.Nq + row) * 64 + half * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          dst[i] = make_uint4(pack_bf16(__uint_as_float(o[8 * i]) * inv, __uint_as_float(o[8 * i + 1]) * inv),
                              pack_bf16(__uint_as_float(o[8 * i + 2]) * inv, __uint_as_float(o[8 * i + 3]) * inv),
                              pack_bf16(__uint_as_float(o[8 * i + 4]) * inv, __uint_as_float(o[8 * i + 5]) * inv),
                              pack_bf16(__uint_as_float(o[8 * i + 6]) * inv, __uint_as_float(o[8 * i + 7]) * inv));
      }
    }
    if (!ok && lane == 0) atomicOr(p.status, kStatusWaitTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, C::kCols);
}

}  // namespace s3r
