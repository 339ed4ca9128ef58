// Selection branch, forward, blocks of 32 and 64 tokens: on tcgen05.
//
// A row tile of 128 queries is G = 128 / BS query blocks, each with its own list of key blocks.  A step takes the next key
// block of every list: a key tile of 128 rows, one BS x 64 copy per list.  S = Q K^T (M=128, N=128) holds G x G blocks, of
// which the diagonal ones are wanted: block g's queries against its own key block.  The softmax threads read those alone; P
// is written over the diagonal blocks of a zeroed tile, so that O += P V (K=128) adds the right keys to each row.  The
// G - 1 unwanted blocks beside each wanted one are cheaper than mma.sync without them: 16 heads, top-16 blocks of 64 at 250
// views 3.86 -> 2.51 ms, 64 views 1002 -> 585 us; top-32 blocks of 32, 60000 tokens 1073 -> 964 us.
// Bound: latency, with no unit more than half busy.  A CTA takes its place for 19.8 us (64 512 tokens, top-16, 8064 CTAs in 538 us), of
// which 16 steps of 1750 cycles beside another CTA (80 KB of shared-memory traffic each; below) are 14.5; the rest passes before its
// first S, at its end and until the next CTA runs in its place.  The merge's operands are loaded before the last product is waited
// for (1.6 us less at the end, 2 to 4 % of the whole).  Two threads per row instead of one changed nothing; several row tiles per CTA
// without a barrier between them cost more registers and instructions than the starts they saved (574 -> 670 us).
// Roles: warp 0 TMA producer, warp 1 tcgen05.mma issuer, warp 2 tensor-memory allocator, warps 4-7 softmax, thread = row.
// Two CTAs per SM: their steps fill each other's waits.
// The exponent offset of a row is its running maximum, step by step (O is rescaled in tensor memory with every step: among a
// warp's 32 rows one nearly always moves): the row's largest weights are 1 and lose nothing when P is rounded to bf16.  Offsets fixed
// by the first step saved the rescaling (64 views 544 instead of 585 us, 250 views 2.42 instead of 2.51 ms) but rounded those weights:
// error against 64 bits 2.33e-3 instead of 2.24e-3 at unit-scale logits, 2.28e-3 instead of 1.64e-3 where a few keys hold a row's
// weight.  All exponentials on their own unit, packed rescaling and no vote in front of it: blocks of 64 at 64 views 551 -> 538 us, at
// 250 views 2206 -> 2148 us (a quarter as polynomials, which this kernel's unit at half load does not need, 12 us of it).
// Of a step's 1750 cycles (beside another CTA) 110 pass until the scores are in registers, 1000 from there to P, 170 until the
// product before is known to be done, 330 for the rescaling and P's store.  Fetching the next step's scores before the
// rescaling needed 192 registers and lost (614 us).
// Zero times a value that is not finite is NaN, so one such value among a query block's keys reaches every row of the tile
// through O += P V.  A row with finite scores and an O that is not is therefore done again from its own keys alone, by its
// thread and out of line: taking the tile's lists one by one with the tensor cores instead needed the row's state in
// registers across the passes and cost every call a fifth (250 views 3.81 -> 4.64 ms).
#include "sel_common.cuh"

namespace s3r {

constexpr int kSbgTile = 128 * 128;            // 128 rows x 64 bf16, bytes
constexpr int kSbgStages = 3;
constexpr int kSbgOffK = kSbgTile;
constexpr int kSbgOffV = kSbgOffK + kSbgStages * kSbgTile;
constexpr int kSbgOffCtl = kSbgOffV + kSbgStages * kSbgTile;
constexpr int kSbgThreads = 256;
constexpr uint32_t kSbgColO = 128, kSbgColP = 192;

struct SbgCtl {
  uint64_t q_full, o_full, drained;
  uint64_t k_full[kSbgStages], k_empty[kSbgStages], v_full[kSbgStages], v_empty[kSbgStages];
  uint64_t s_full, s_free, p_full, pv_done;
  uint32_t tmem_base, abort_flag;
  int nvalid[4], steps;
};
constexpr int kSbgOffList = kSbgOffCtl + 256;  // [G][topk] int32: first token of each valid key block
// two CTAs fit an SM up to 115712 bytes each: lists of up to 64 entries for blocks of 64, 48 for blocks of 32
static_assert(sizeof(SbgCtl) <= 256, "control words");

// O of one row, normalised, from the row's own keys: `list` of `nv` first tokens, weights 2^(cs q.k - m) / l.
template <int BS>
__device__ __noinline__ void sbg_row_alone(const SelParams& p, int bh, int row, const int32_t* list, int nv, float m, float l) {
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p.q) + (static_cast<int64_t>(bh) * p.Tq + row) * 32;
  const int64_t chunk = static_cast<int64_t>(p.kv_chunk_stride) / 2, in_chunk = static_cast<int64_t>(bh) * p.Tc;
  float o[64];
#pragma unroll
  for (int i = 0; i < 64; ++i) o[i] = 0.f;
#pragma unroll 1
  for (int j = 0; j < nv; ++j) {
    const int t0 = list[j], ch = t0 / p.Tc, n = min(BS, p.Tk - t0);
    const int64_t at = ch * chunk + (in_chunk + t0 - ch * p.Tc) * 32;
    const uint32_t *k = reinterpret_cast<const uint32_t*>(p.k) + at, *v = reinterpret_cast<const uint32_t*>(p.v) + at;
#pragma unroll 1
    for (int t = 0; t < n; ++t, k += 32, v += 32) {
      float s = 0.f;
#pragma unroll 8
      for (int i = 0; i < 32; ++i) s += bf16_lo(q[i]) * bf16_lo(k[i]) + bf16_hi(q[i]) * bf16_hi(k[i]);
      const float w = exp2f(s * p.scale_log2e - m);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        o[2 * i] += w * bf16_lo(v[i]);
        o[2 * i + 1] += w * bf16_hi(v[i]);
      }
    }
  }
  const int b = bh / p.H, h = bh - b * p.H, qb = row / BS;
  const float inv = 1.f / l;
  if (p.o_s) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.o_s) + (static_cast<int64_t>(bh) * p.Tq + row) * 32;
#pragma unroll
    for (int i = 0; i < 32; ++i) dst[i] = pack_bf16(o[2 * i] * inv, o[2 * i + 1] * inv);
  }
  if (p.y) {
    const uint32_t gw = *reinterpret_cast<const uint32_t*>(p.gate + b * p.gsb + h * p.gsh + row * p.gst);
    const uint32_t* oc = reinterpret_cast<const uint32_t*>(p.o_c) + (static_cast<int64_t>(bh) * p.nqb + qb) * 32;
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.y) + ((static_cast<int64_t>(b) * p.Tq + row) * p.H + h) * 32;
    const float g0 = bf16_lo(gw), g1 = bf16_hi(gw) * inv;
#pragma unroll
    for (int i = 0; i < 32; ++i) dst[i] = pack_bf16(g0 * bf16_lo(oc[i]) + g1 * o[2 * i], g0 * bf16_hi(oc[i]) + g1 * o[2 * i + 1]);
  }
}

template <int BS>
__global__ void __launch_bounds__(kSbgThreads, 2)
sel_big_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ SelParams p) {
  constexpr int G = 128 / BS;                  // query blocks per row tile
  extern __shared__ __align__(1024) uint8_t smem[];
  SbgCtl& ctl = *reinterpret_cast<SbgCtl*>(smem + kSbgOffCtl);
  int32_t* lists = reinterpret_cast<int32_t*>(smem + kSbgOffList);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_per_bh = (p.nqb + G - 1) / G;
  const int bh = blockIdx.x / tiles_per_bh, qb0 = (blockIdx.x % tiles_per_bh) * G;
  const uint32_t sbase = smem_u32(smem);

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    mbar_init(&ctl.q_full, 1);
    mbar_init(&ctl.o_full, 1);
    mbar_init(&ctl.drained, 1);
    for (int s = 0; s < kSbgStages; ++s) {
      mbar_init(&ctl.k_full[s], 1);
      mbar_init(&ctl.k_empty[s], 1);
      mbar_init(&ctl.v_full[s], 1);
      mbar_init(&ctl.v_empty[s], 1);
    }
    mbar_init(&ctl.s_full, 1);
    mbar_init(&ctl.s_free, 4);
    mbar_init(&ctl.p_full, 4);
    mbar_init(&ctl.pv_done, 1);
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(&ctl.tmem_base, 256);
    tmem_relinquish();
  }
  griddep_wait();
  if (warp >= 4 && warp < 4 + G) {
    // valid entries of one query block's row of the table, table order
    const int g = warp - 4, qb = qb0 + g;
    int n = 0;
    if (qb < p.nqb) {
      const int32_t* row = p.idx + (static_cast<int64_t>(bh) * p.nqb + qb) * p.topk;
      for (int r0 = 0; r0 < p.topk; r0 += 32) {
        const int i = r0 + lane, e = i < p.topk ? row[i] : -1;
        const bool ok = e >= 0 && static_cast<int64_t>(e) * BS < p.Tk;
        const uint32_t m = __ballot_sync(0xffffffffu, ok);
        if (ok) lists[g * p.topk + n + __popc(m & ((1u << lane) - 1u))] = e * BS;
        n += __popc(m);
      }
    }
    if (lane == 0) ctl.nvalid[g] = n;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();                            // not before this CTA has its tensor memory: a CTA of the next kernel could take it
  const uint32_t tmem = ctl.tmem_base;
  volatile uint32_t* abort_flag = &ctl.abort_flag;
  int steps = ctl.nvalid[0];
#pragma unroll
  for (int g = 1; g < G; ++g) steps = max(steps, ctl.nvalid[g]);
  const bool aligned = (sbase & 1023u) == 0;   // the swizzled tiles need it; dynamic shared memory starts there
  if (!aligned) steps = 0;

  if (warp < 4) {
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      const bool chunked = p.Tc != p.Tk;
      // lane g copies for list g; a list that has ended, or is empty, gets zeros (rows past the end of the map)
      int issued = 0;
      if (steps > 0 && lane == 0) {
        mbar_expect_tx(&ctl.q_full, kSbgTile);
        tma_load_4d(sbase, &map_q, &ctl.q_full, 0, qb0 * BS, bh, 0);
      }
      const int nv = lane < G ? ctl.nvalid[lane] : 0;
      for (int j = 0; j < steps; ++j) {
        const int s = j % kSbgStages;
        const uint32_t ph = (j / kSbgStages) & 1;
        int tok = p.Tc, ch = 0;
        if (j < nv) {
          tok = lists[lane * p.topk + j];
          if (chunked) { ch = tok / p.Tc; tok -= ch * p.Tc; }
        }
        if (!mbar_wait_warp(&ctl.k_empty[s], ph ^ 1, abort_flag)) break;
        if (lane == 0) mbar_expect_tx(&ctl.k_full[s], kSbgTile);
        __syncwarp();
        if (lane < G) tma_load_4d(sbase + kSbgOffK + s * kSbgTile + lane * BS * 128, &map_k, &ctl.k_full[s], 0, tok, bh, ch);
        issued = j + 1;                                                   // K of step j is in flight
        if (!mbar_wait_warp(&ctl.v_empty[s], ph ^ 1, abort_flag)) break;
        if (lane == 0) mbar_expect_tx(&ctl.v_full[s], kSbgTile);
        __syncwarp();
        if (lane < G) tma_load_4d(sbase + kSbgOffV + s * kSbgTile + lane * BS * 128, &map_v, &ctl.v_full[s], 0, tok, bh, ch);
      }
      if (*abort_flag) {
        // give copies already in flight a bounded chance to land before the CTA's memory is released
        for (int n = max(0, issued - kSbgStages); n < issued; ++n) {
          volatile uint32_t dummy = 0;
          mbar_wait(&ctl.k_full[n % kSbgStages], (n / kSbgStages) & 1, &dummy);
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      const bool leader = elect_one_sync();
      constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, 64, 0, 1);         // V tile is [keys][d]: N contiguous
      const uint64_t desc_q = umma_desc_sw128(sbase), desc_k = umma_desc_sw128(sbase + kSbgOffK),
                     desc_v = umma_desc_sw128(sbase + kSbgOffV);
      auto issue_qk = [&](int s) {
        umma_ss_k4<2, 2>(tmem, desc_q, desc_k + static_cast<uint64_t>(s * (kSbgTile >> 4)), idesc_qk, 0u);
        umma_commit(&ctl.s_full);
        umma_commit(&ctl.k_empty[s]);
      };
      auto issue_pv = [&](int s, uint32_t acc) {
        const uint64_t v = desc_v + static_cast<uint64_t>(s * (kSbgTile >> 4));
        umma_ts_k4<128>(tmem + kSbgColO, tmem + kSbgColP, v, idesc_pv, acc);
        umma_ts_k4<128>(tmem + kSbgColO, tmem + kSbgColP + 32, v + 4 * 128, idesc_pv, 1u);
        umma_commit(&ctl.pv_done);
        umma_commit(&ctl.v_empty[s]);
      };
      bool ok = steps == 0 || mbar_wait_warp(&ctl.q_full, 0, abort_flag);
      int s = 0;
      uint32_t ph = 0;
      ok = ok && (steps == 0 || mbar_wait_warp(&ctl.k_full[s], ph, abort_flag));
      if (ok && steps > 0) {
        tc_fence_after();
        if (leader) issue_qk(s);
        __syncwarp();
      }
#pragma unroll 1
      for (int j = 0; j < steps && ok; ++j) {
        const bool nxt = j + 1 < steps;
        const int sn = s + 1 == kSbgStages ? 0 : s + 1;
        const uint32_t phn = sn == 0 ? ph ^ 1u : ph;
        if (nxt) {
          ok = mbar_wait_warp(&ctl.k_full[sn], phn, abort_flag) &&
               mbar_wait_warp(&ctl.s_free, j & 1, abort_flag);            // S of step j is in registers
          if (!ok) break;
          tc_fence_after();
          if (leader) issue_qk(sn);
          __syncwarp();
        }
        ok = mbar_wait_warp(&ctl.v_full[s], ph, abort_flag) && mbar_wait_warp(&ctl.p_full, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (leader) issue_pv(s, j > 0 ? 1u : 0u);
        __syncwarp();
        s = sn;
        ph = phn;
      }
      if (leader) umma_commit(ok ? &ctl.o_full : &ctl.drained);            // who waits for results gets none from a CTA that gave up
      __syncwarp();
      if (!ok) {
        volatile uint32_t dummy = 0;
        mbar_wait(&ctl.drained, 0, &dummy);             // let issued MMAs drain before tensor memory is freed
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, thread = row
    const int quarter = warp & 3, r = quarter * 32 + lane, g = (quarter * 32) / BS, row = qb0 * BS + r;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_s = lane_base + g * BS, t_o = lane_base + kSbgColO, t_p = lane_base + kSbgColP + g * (BS / 2);
    const float cs = p.scale_log2e;
    const int nv = ctl.nvalid[g];
    const int32_t* list = lists + g * p.topk;
    const bool ragged = p.Tk % BS != 0;
    {
      uint32_t z[32];                           // P outside the diagonal blocks is zero for good
#pragma unroll
      for (int i = 0; i < 32; ++i) z[i] = 0u;
      tmem_st32(lane_base + kSbgColP, z);
      tmem_st32(lane_base + kSbgColP + 32, z);
      tmem_st_wait();
    }
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    auto step = [&](int j) -> bool {
      if (!mbar_wait_warp(&ctl.s_full, j & 1, abort_flag)) return false;
      tc_fence_after();
      uint32_t x[BS / 32][32];
#pragma unroll
      for (int c = 0; c < BS / 32; ++c) tmem_ld32(t_s + c * 32, x[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.s_free);              // this row's part of S is in registers
      const int left = j >= nv ? 0 : (ragged ? p.Tk - list[j] : BS);
      if (left < BS) {                                      // scores that do not exist
#pragma unroll
        for (int c = 0; c < BS / 32; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= left) x[c][i] = 0xff800000u;  // -inf
      }
      float gm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < BS / 32; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          gm[(i >> 1) & 3] = fmax3_nan(gm[(i >> 1) & 3], __uint_as_float(x[c][i]), __uint_as_float(x[c][i + 1]));
      // scale > 0 keeps the order; a NaN, or a score of +infinity (0 x inf), makes the offset and with it the row NaN
      const float mn = fmax3_nan(m_used, fmax3_nan(gm[0], gm[1], gm[2]) * cs, gm[3] * cs);
      const float neg = mn == -INFINITY ? 0.f : fmaf(mn, 0.f, -mn), alpha = fast_exp2(m_used + neg);
      m_used = mn;
      const float2 nm = make_float2(neg, neg), cs2 = make_float2(cs, cs);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      uint32_t pk[BS / 32][16];
#pragma unroll
      for (int c = 0; c < BS / 32; ++c) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 v = ffma2(make_float2(__uint_as_float(x[c][2 * i]), __uint_as_float(x[c][2 * i + 1])), cs2, nm);
          v.x = fast_exp2(v.x);
          v.y = fast_exp2(v.y);
          sum[i & 1] = fadd2(sum[i & 1], v);
          pk[c][i] = pack_bf16(v.x, v.y);
        }
      }
      // P of the previous step must have been consumed: all of P waits in registers, so that its product has this long
      if (j > 0 && !mbar_wait_warp(&ctl.pv_done, (j - 1) & 1, abort_flag)) return false;
      tc_fence_after();
      if (j > 0) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t o[32];
          tmem_ld32(t_o + hf * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = fmul2(make_float2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), make_float2(alpha, alpha));
            o[i] = __float_as_uint(x.x);
            o[i + 1] = __float_as_uint(x.y);
          }
          tmem_st32(t_o + hf * 32, o);
        }
      }
#pragma unroll
      for (int c = 0; c < BS / 32; ++c) tmem_st16(t_p + c * 16, pk[c]);
      l = l * alpha + ((sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.p_full);
      return true;
    };
    const int b = bh / p.H, h = bh - b * p.H;
    const bool live = row < p.Tq;
    uint32_t gate_word = 0;
    uint4 merged[8];                            // the row's block of the other branch
#pragma unroll 1
    for (int j = 0; j < steps && ok; ++j) ok = step(j);
    // what the merge needs, on its way while the last product runs
    if (live && p.y) {
      gate_word = __ldg(reinterpret_cast<const uint32_t*>(p.gate + b * p.gsb + h * p.gsh + row * p.gst));
      const uint4* oc = reinterpret_cast<const uint4*>(p.o_c + (static_cast<int64_t>(bh) * p.nqb + qb0 + g) * 64);
#pragma unroll
      for (int i = 0; i < 8; ++i) merged[i] = __ldg(oc + i);
    }
    if (ok) ok = mbar_wait_warp(&ctl.o_full, 0, abort_flag);

    if (ok && aligned) {
      tc_fence_after();
      const bool any = m_used != -INFINITY || l != l;       // no valid key, or none with a score above -inf: o = 0, lse = -inf
      const float inv = any ? 1.f / l : 0.f;
      if (live && p.lse_s)
        p.lse_s[static_cast<int64_t>(bh) * p.Tq + row] = any ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      const float g0 = bf16_lo(gate_word), g1 = bf16_hi(gate_word);
      float2 off = make_float2(0.f, 0.f);                   // NaN where some value of O is not finite
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t o[32];
        if (steps > 0) {
          tmem_ld32(t_o + hf * 32, o);
          tmem_ld_wait();
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = any ? __float_as_uint(__uint_as_float(o[i]) * inv) : 0u;
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          off = ffma2(make_float2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), make_float2(0.f, 0.f), off);
        auto f = [&](int i) { return __uint_as_float(o[i]); };
        if (live && p.o_s) {
          uint4* dst = reinterpret_cast<uint4*>(p.o_s + (static_cast<int64_t>(bh) * p.Tq + row) * 64 + hf * 32);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            dst[i] = make_uint4(pack_bf16(f(8 * i), f(8 * i + 1)), pack_bf16(f(8 * i + 2), f(8 * i + 3)),
                                pack_bf16(f(8 * i + 4), f(8 * i + 5)), pack_bf16(f(8 * i + 6), f(8 * i + 7)));
        }
        if (live && p.y) {
          uint4* dst = reinterpret_cast<uint4*>(p.y + ((static_cast<int64_t>(b) * p.Tq + row) * p.H + h) * 64 + hf * 32);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 c = merged[hf * 4 + i];
            const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack_bf16(g0 * bf16_lo(cw[e]) + g1 * f(8 * i + 2 * e), g0 * bf16_hi(cw[e]) + g1 * f(8 * i + 2 * e + 1));
            dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      if (live && any && l - l == 0.f && !(off.x + off.y == 0.f)) sbg_row_alone<BS>(p, bh, row, list, nv, m_used, l);
    }
    if ((!ok || !aligned) && lane == 0) atomicOr(p.status, kStatusWaitTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 256);
}

template <int BS>
static int launch_sel_big(int kv_chunks, const SelParams& p, cudaStream_t st) {
  constexpr int G = 128 / BS;
  const int BH = p.B * p.H;
  CUtensorMap mq, mk, mv;
  const uint64_t bh = static_cast<uint64_t>(BH), tq = static_cast<uint64_t>(p.Tq), tc = static_cast<uint64_t>(p.Tc);
  {
    const uint64_t dims[4] = {64, tq, bh, 1}, strides[3] = {128, tq * 128, tq * 128 * bh};
    const uint32_t box[4] = {64, 128, 1, 1};
    const int rc = make_tensor_map(&mq, p.q, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    const uint64_t dims[4] = {64, tc, bh, static_cast<uint64_t>(kv_chunks)};
    const uint64_t strides[3] = {128, tc * 128, kv_chunks > 1 ? static_cast<uint64_t>(p.kv_chunk_stride) * 2 : tc * 128 * bh};
    const uint32_t box[4] = {64, static_cast<uint32_t>(BS), 1, 1};
    int rc = make_tensor_map(&mk, p.k, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_tensor_map(&mv, p.v, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  const int64_t grid = static_cast<int64_t>(BH) * ((p.nqb + G - 1) / G);
  S3R_REQUIRE(grid < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_sel_attn_fwd: grid of %lld CTAs is too large", (long long)grid);
  const int smem = kSbgOffList + G * p.topk * static_cast<int>(sizeof(int32_t));
  S3R_CUDA(cudaFuncSetAttribute(sel_big_kernel<BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSbgOffList + 1024));
  return launch(sel_big_kernel<BS>, static_cast<unsigned>(grid), kSbgThreads, smem, st, mq, mk, mv, p);
}

int sel_big_fwd(int kv_chunks, int block, const SelParams& p, cudaStream_t st) {
  return block == 32 ? launch_sel_big<32>(kv_chunks, p, st) : launch_sel_big<64>(kv_chunks, p, st);
}

}  // namespace s3r
