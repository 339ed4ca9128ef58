// Selection branch, backward, blocks of 64 tokens: on tcgen05.
//
//   dK/dV: a CTA owns a key block and takes the query blocks that selected it two at a time (128 query rows Y)
//        S = Q K^T, dP = dO V^T                 (M=128 queries, N=64 keys)          thread = query row
//        P = exp2(S c - lse), dS = P (dP - delta)  to shared memory, 128-byte rows
//        [P | dS]^T [dO | Q]                    (M=128, N=128, K=128): dV and dK are its diagonal 64 x 64 blocks
//   dQ   : a CTA owns a query block and takes its key blocks two at a time (128 key rows Y)
//        S^T = K Q^T, dP^T = V dO^T             (M=128 keys, N=64 queries)          thread = key row
//        [dS_a | dS_b]^T [K_a | K_b]            (M=128, N=128, K=64): dQ is the sum of its diagonal blocks
// The two blocks beside the diagonal are not read: an M=64 product takes as long as an M=128 one.  The softmax scale is applied
// once, to the accumulators; the pooled branch's gradient is added in the store.
// Blocks of 64 only, and there not where lists are next to empty (sel_bwd64_pays).  The warps of sel_bwd.cu own 16 rows each, so that a block's four warps gather and read all of its tiles four
// times (2800 cycles of shared memory per pair of blocks and SM, 1860 of mma.sync); here it is 1220 of shared memory and 640 of
// tensor pipe for a dK/dV and a dQ step.  With blocks of 32 the same products would be a quarter instead of half useful.
// 16 heads, top-16, both parts with the index: 8328 tokens 422 -> 229 us, 40 000 tokens 1812 -> 1027 us (random tables).
// Bound: the latency of a step's chain - copies, S and dP, P and dS, second product, 2250 cycles beside the SM's other CTA - with two
// stages and two CTAs per SM.  No unit is half busy: shared memory 47 % (176 KB of copies, stores and reads per dK/dV step, 112 of them
// read by the products; 128 and 80 per dQ step), tensor pipe 39 %, exponentials 31 %.  Two threads per row
// instead of one changed nothing (230 and 1050 us), tasks handed on to running CTAs, with copies and first products ahead across
// them, little (225 and 981 us).
// Roles: warp 0 TMA producer, warp 1 tcgen05.mma issuer, warp 2 tensor-memory allocator, warps 4-7 P and dS.
#include "sel_common.cuh"

namespace s3r {

constexpr int kS64Own = 64 * 128, kS64Tile = 128 * 128;        // 64 and 128 rows x 64 bf16, bytes
constexpr int kS64Stages = 2;
// own tiles X0, X1; ring of (Y1, Y0); P and dS.  X0, Y0 make S, X1, Y1 make dP.
constexpr int kS64OffY = 2 * kS64Own, kS64OffG = kS64OffY + kS64Stages * 2 * kS64Tile, kS64OffCtl = kS64OffG + 2 * kS64Tile;
constexpr int kS64OffList = kS64OffCtl + 128, kS64OffStat = kS64OffList + 256;
constexpr int kS64Smem = kS64OffStat + 512 + 128;              // two CTAs per SM up to 115712 bytes each
static_assert(kS64Smem <= 115712, "two CTAs per SM");
constexpr int kS64Threads = 256;
constexpr uint32_t kS64ColDP = 64, kS64ColAcc = 128;

struct S64Ctl {
  uint64_t x_full, o_full, drained;
  uint64_t y_full[kS64Stages], y_empty[kS64Stages];
  uint64_t s_full, s_free, g_full, g_free;
  uint32_t tmem_base, abort_flag;
};
static_assert(sizeof(S64Ctl) <= 128, "control words");

struct S64Maps {
  CUtensorMap q, d_o, k, v;      // boxes of 64 rows
};

// acc += the pooled branch's gradient of token t: g_c[j] / kernel of every window j that contains it.  g_c begins at a multiple of 4
// bytes; where that is one of 16, as from any allocation, its rows are read in a quarter of the loads.
__device__ __forceinline__ void s64_add_pooled(float (&acc)[64], const __nv_bfloat16* g_c, int bh, int t, int kernel, int stride,
                                               int windows) {
  if (g_c == nullptr) return;
  const int hi = min(windows - 1, t / stride), lo = t + 1 <= kernel ? 0 : (t - kernel) / stride + 1;
  const float inv = 1.0f / static_cast<float>(kernel);
  const bool vec = (reinterpret_cast<uintptr_t>(g_c) & 15) == 0;
  for (int j = lo; j <= hi; ++j) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(g_c + (static_cast<int64_t>(bh) * windows + j) * 64);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint4 v = vec ? __ldg(reinterpret_cast<const uint4*>(src) + i)
                          : make_uint4(__ldg(src + 4 * i), __ldg(src + 4 * i + 1), __ldg(src + 4 * i + 2), __ldg(src + 4 * i + 3));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[8 * i + 2 * e] += bf16_lo(w[e]) * inv;
        acc[8 * i + 2 * e + 1] += bf16_hi(w[e]) * inv;
      }
    }
  }
}
__device__ __forceinline__ void s64_store_row(const float (&acc)[64], __nv_bfloat16* dst) {
  uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    d[i] = make_uint4(pack_bf16(acc[8 * i], acc[8 * i + 1]), pack_bf16(acc[8 * i + 2], acc[8 * i + 3]),
                      pack_bf16(acc[8 * i + 4], acc[8 * i + 5]), pack_bf16(acc[8 * i + 6], acc[8 * i + 7]));
}

// MODE 0: dK/dV of key block `blk`.  MODE 1: dQ of query block `blk`.
template <int MODE>
__device__ __forceinline__ void sel_bwd64_cta(const S64Maps& m, const SelBwdParams& p, uint8_t* smem, int bh, int blk) {
  S64Ctl& ctl = *reinterpret_cast<S64Ctl*>(smem + kS64OffCtl);
  int32_t* list = reinterpret_cast<int32_t*>(smem + kS64OffList);          // dQ: first token of each valid key block, table order
  float* stats = reinterpret_cast<float*>(smem + kS64OffStat);             // dQ: -lse2 of the 64 queries, then -delta
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t sbase = smem_u32(smem);

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    mbar_init(&ctl.x_full, 1);
    mbar_init(&ctl.o_full, 1);
    mbar_init(&ctl.drained, 1);
    for (int s = 0; s < kS64Stages; ++s) {
      mbar_init(&ctl.y_full[s], 1);
      mbar_init(&ctl.y_empty[s], 1);
    }
    mbar_init(&ctl.s_full, 1);
    mbar_init(&ctl.s_free, 4);
    mbar_init(&ctl.g_full, 4);
    mbar_init(&ctl.g_free, 1);
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(&ctl.tmem_base, 256);
    tmem_relinquish();
  }
  griddep_wait();
  const int32_t* ql = nullptr;                 // dK/dV: the query blocks that selected this key block
  int cnt = 0;                                 // entries of the list
  if (MODE == 0) {
    const int32_t* off = p.offsets + static_cast<int64_t>(bh) * (p.nkb + 1) + blk;
    const int beg = __ldg(off);
    cnt = __ldg(off + 1) - beg;
    ql = p.qids + static_cast<int64_t>(bh) * p.nqb * p.topk + beg;
  } else {
    // every warp finds the length, warp 4 writes the list
    const int32_t* row = p.idx + (static_cast<int64_t>(bh) * p.nqb + blk) * p.topk;
    for (int r0 = 0; r0 < p.topk; r0 += 32) {
      const int i = r0 + lane, e = i < p.topk ? __ldg(row + i) : -1;
      const bool ok = e >= 0 && static_cast<int64_t>(e) * 64 < p.Tk;
      const uint32_t b = __ballot_sync(0xffffffffu, ok);
      if (warp == 4 && ok) list[cnt + __popc(b & ((1u << lane) - 1u))] = e * 64;
      cnt += __popc(b);
    }
    if (warp == 5 || warp == 6) {              // the queries' statistics; rows past the end: lse = +inf makes P exactly 0
      const int i = (warp - 5) * 32 + lane, t = blk * 64 + i;
      const bool in = t < p.Tq;
      stats[i] = in ? __ldg(p.lse + static_cast<int64_t>(bh) * p.Tq + t) * -1.4426950408889634f : -INFINITY;
      stats[64 + i] = in ? -__ldg(p.delta + static_cast<int64_t>(bh) * p.Tq + t) : 0.f;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();                            // not before this CTA has its tensor memory: a CTA of the next kernel could take it
  const uint32_t tmem = ctl.tmem_base;
  volatile uint32_t* abort_flag = &ctl.abort_flag;
  const bool aligned = (sbase & 1023u) == 0;   // the swizzled tiles need it; dynamic shared memory starts there
  const int steps = aligned ? (cnt + 1) >> 1 : 0;

  if (warp < 4) {
    reg_dealloc<56>();
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      const bool leader = elect_one_sync();
      const CUtensorMap *mx0 = MODE == 0 ? &m.k : &m.q, *mx1 = MODE == 0 ? &m.v : &m.d_o;
      const CUtensorMap *my0 = MODE == 0 ? &m.q : &m.k, *my1 = MODE == 0 ? &m.d_o : &m.v;
      const int past = MODE == 0 ? p.Tq : p.Tk;            // rows past the end of the map are zeros
      if (steps > 0 && leader) {
        mbar_expect_tx(&ctl.x_full, 2 * kS64Own);
        tma_load_3d(sbase, mx0, &ctl.x_full, 0, blk * 64, bh);
        tma_load_3d(sbase + kS64Own, mx1, &ctl.x_full, 0, blk * 64, bh);
      }
      int issued = 0, cur = MODE == 0 && lane < cnt ? __ldg(ql + lane) : 0;
      for (int j = 0; j < steps; ++j) {
        const int s = j % kS64Stages;
        int t0, t1;
        if (MODE == 0) {
          if (j > 0 && (j & 15) == 0) cur = 2 * j + lane < cnt ? __ldg(ql + 2 * j + lane) : 0;
          t0 = __shfl_sync(0xffffffffu, cur, (2 * j) & 31) * 64;
          t1 = __shfl_sync(0xffffffffu, cur, (2 * j + 1) & 31) * 64;
        } else {
          t0 = list[2 * j];
          t1 = 2 * j + 1 < cnt ? list[2 * j + 1] : 0;
        }
        if (2 * j + 1 >= cnt) t1 = past;
        if (!mbar_wait_warp(&ctl.y_empty[s], ((j / kS64Stages) & 1) ^ 1, abort_flag)) break;
        if (leader) {
          const uint32_t y1 = sbase + kS64OffY + s * 2 * kS64Tile, y0 = y1 + kS64Tile;
          mbar_expect_tx(&ctl.y_full[s], 2 * kS64Tile);
          tma_load_3d(y0, my0, &ctl.y_full[s], 0, t0, bh);
          tma_load_3d(y0 + kS64Own, my0, &ctl.y_full[s], 0, t1, bh);
          tma_load_3d(y1, my1, &ctl.y_full[s], 0, t0, bh);
          tma_load_3d(y1 + kS64Own, my1, &ctl.y_full[s], 0, t1, bh);
        }
        __syncwarp();
        issued = j + 1;
      }
      if (*abort_flag) {
        // give copies already in flight a bounded chance to land before the CTA's memory is released
        volatile uint32_t dummy = 0;
        if (steps > 0) mbar_wait(&ctl.x_full, 0, &dummy);
        for (int j = max(0, issued - kS64Stages); j < issued; ++j) {
          dummy = 0;
          mbar_wait(&ctl.y_full[j % kS64Stages], (j / kS64Stages) & 1, &dummy);
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      const bool leader = elect_one_sync();
      constexpr uint32_t idesc_1 = umma_idesc_bf16(128, 64, 0, 0), idesc_2 = umma_idesc_bf16(128, 128, 1, 1);
      // second products: both operands with M | N contiguous, in two pieces of 64 that lie `apart` bytes from each other
      constexpr uint32_t apart = MODE == 0 ? kS64Tile : kS64Own;
      const uint64_t x0 = umma_desc_sw128(sbase), x1 = umma_desc_sw128(sbase + kS64Own), y = umma_desc_sw128(sbase + kS64OffY);
      const uint64_t g2 = umma_desc_sw128(sbase + kS64OffG, 1024, apart), y2 = umma_desc_sw128(sbase + kS64OffY, 1024, apart);
      auto first = [&](int s) {
        const uint64_t y1 = y + static_cast<uint64_t>(s * (2 * kS64Tile >> 4)), y0 = y1 + (kS64Tile >> 4);
        umma_ss_k4<2, 2>(tmem, y0, x0, idesc_1, 0u);
        umma_ss_k4<2, 2>(tmem + kS64ColDP, y1, x1, idesc_1, 0u);
        umma_commit(&ctl.s_full);
      };
      auto second = [&](int s, uint32_t acc) {
        if (MODE == 0) {
          const uint64_t b = y2 + static_cast<uint64_t>(s * (2 * kS64Tile >> 4));
          umma_ss_k4<128, 128>(tmem + kS64ColAcc, g2, b, idesc_2, acc);
          umma_ss_k4<128, 128>(tmem + kS64ColAcc, g2 + 4 * 128, b + 4 * 128, idesc_2, 1u);
        } else {
          umma_ss_k4<128, 128>(tmem + kS64ColAcc, g2, y2 + static_cast<uint64_t>(s * (2 * kS64Tile >> 4) + (kS64Tile >> 4)), idesc_2, acc);
        }
        umma_commit(&ctl.g_free);
        umma_commit(&ctl.y_empty[s]);
      };
      bool ok = steps == 0 || (mbar_wait_warp(&ctl.x_full, 0, abort_flag) && mbar_wait_warp(&ctl.y_full[0], 0, abort_flag));
      if (ok && steps > 0) {
        tc_fence_after();
        if (leader) first(0);
        __syncwarp();
      }
#pragma unroll 1
      for (int j = 0; j < steps && ok; ++j) {
        const int s = j % kS64Stages, sn = (j + 1) % kS64Stages;
        if (j + 1 < steps) {
          ok = mbar_wait_warp(&ctl.y_full[sn], ((j + 1) / kS64Stages) & 1, abort_flag) &&
               mbar_wait_warp(&ctl.s_free, j & 1, abort_flag);             // S and dP of step j are in registers
          if (!ok) break;
          tc_fence_after();
          if (leader) first(sn);
          __syncwarp();
        }
        ok = mbar_wait_warp(&ctl.g_full, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (leader) second(s, j > 0 ? 1u : 0u);
        __syncwarp();
      }
      if (leader) umma_commit(ok ? &ctl.o_full : &ctl.drained);            // who waits for results gets none from a CTA that gave up
      __syncwarp();
      if (!ok) {
        volatile uint32_t dummy = 0;
        mbar_wait(&ctl.drained, 0, &dummy);             // let issued MMAs drain before tensor memory is freed
      }
    }
  } else {
    // ------------------------------------------------------------------ P and dS, thread = row of Y
    reg_alloc<200>();
    const int quarter = warp & 3, r = quarter * 32 + lane, upper = r >> 6;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const float2 cs2 = make_float2(p.cs, p.cs);
    const uint32_t g_row = sbase + kS64OffG + r * 128;
    // dK/dV: statistics of this row's query, one step ahead of their use, and its list entry, two steps ahead
    auto entry = [&](int j) { return 2 * j + upper < cnt ? __ldg(ql + 2 * j + upper) : -1; };
    auto stat = [&](int e, float& l, float& d) {
      const int t = e * 64 + (r & 63);
      const bool in = e >= 0 && t < p.Tq;
      const int64_t at = static_cast<int64_t>(bh) * p.Tq + (in ? t : 0);
      l = in ? __ldg(p.lse + at) * -1.4426950408889634f : -INFINITY;
      d = in ? -__ldg(p.delta + at) : 0.f;
      return in;
    };
    float nl = 0.f, nd = 0.f;
    int e2 = -1;
    bool nlive = true;
    if (MODE == 0) {
      nlive = stat(entry(0), nl, nd);
      e2 = entry(1);
    }
    bool ok = true;
#pragma unroll 1
    for (int j = 0; j < steps; ++j) {
      const float lse = nl, delta = nd;
      // this row's query (dQ: key) exists
      const bool live = MODE == 0 ? nlive : 2 * j + upper < cnt && list[2 * j + upper] + (r & 63) < p.Tk;
      if (MODE == 0) {
        nlive = stat(e2, nl, nd);
        e2 = entry(j + 2);
      }
      ok = mbar_wait_warp(&ctl.s_full, j & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t pk[32], dk[32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t s[32], dp[32];
        tmem_ld32(lane_base + h * 32, s);
        tmem_ld32(lane_base + kS64ColDP + h * 32, dp);
        tmem_ld_wait();
        if (h == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.s_free);
        }
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float2 l[2] = {make_float2(lse, lse), make_float2(lse, lse)}, d[2] = {make_float2(delta, delta), make_float2(delta, delta)};
          if (MODE == 1) {
            const float4 a = *reinterpret_cast<const float4*>(stats + h * 32 + 2 * i), b = *reinterpret_cast<const float4*>(stats + 64 + h * 32 + 2 * i);
            l[0] = make_float2(a.x, a.y); l[1] = make_float2(a.z, a.w);
            d[0] = make_float2(b.x, b.y); d[1] = make_float2(b.z, b.w);
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float2 x = ffma2(make_float2(__uint_as_float(s[2 * (i + u)]), __uint_as_float(s[2 * (i + u) + 1])), cs2, l[u]);
            x.x = fast_exp2(x.x);
            x.y = fast_exp2(x.y);
            if (MODE == 0) pk[h * 16 + i + u] = pack_bf16(x.x, x.y);
            x = fmul2(x, fadd2(make_float2(__uint_as_float(dp[2 * (i + u)]), __uint_as_float(dp[2 * (i + u) + 1])), d[u]));
            dk[h * 16 + i + u] = MODE == 0 || live ? pack_bf16(x.x, x.y) : 0u;
          }
        }
      }
      // dK/dV: rows of queries past the end, and of the half that a list of odd length leaves empty.  Their scores are products of
      // zeros, which are NaN, not zero, with a key or value that is not finite.
      if (MODE == 0 && !live) {
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = dk[i] = 0u;
      }
      // the products of the step before must have read P and dS
      if (j > 0) {
        ok = mbar_wait_warp(&ctl.g_free, (j - 1) & 1, abort_flag);
        if (!ok) break;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t at = g_row + ((i ^ (r & 7)) << 4);
        if (MODE == 0) sts128(at, pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
        sts128(at + (MODE == 0 ? kS64Tile : 0), dk[4 * i], dk[4 * i + 1], dk[4 * i + 2], dk[4 * i + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.g_full);
    }
    if (ok) ok = mbar_wait_warp(&ctl.o_full, 0, abort_flag);
    tc_fence_after();
    // rows 0-63: first 64 columns of the accumulators, rows 64-127: the others
    float acc[64];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t x[32];
      if (steps > 0) {
        tmem_ld32(lane_base + kS64ColAcc + upper * 64 + h * 32, x);
        tmem_ld_wait();
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[h * 32 + i] = steps > 0 ? __uint_as_float(x[i]) : 0.f;
    }
    const int t = blk * 64 + (r & 63);
    if (MODE == 0) {
      if (ok && t < p.Tk) {
        if (upper) {
#pragma unroll
          for (int i = 0; i < 64; ++i) acc[i] *= p.scale;
        }
        s64_add_pooled(acc, upper ? p.dk_c : p.dv_c, bh, t, p.k_kernel, p.k_stride, p.k_windows);
        s64_store_row(acc, (upper ? p.dk : p.dv) + (static_cast<int64_t>(bh) * p.Tk + t) * 64);
      }
    } else {
      float* other = reinterpret_cast<float*>(smem + kS64OffY) + (r & 63);               // [column][row]; the ring is idle by now
      if (upper) {
#pragma unroll
        for (int i = 0; i < 64; ++i) other[i * 64] = acc[i];
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ok && !upper && t < p.Tq) {
#pragma unroll
        for (int i = 0; i < 64; ++i) acc[i] = (acc[i] + other[i * 64]) * p.scale;
        s64_add_pooled(acc, p.dq_c, bh, t, p.q_kernel, p.q_stride, p.q_windows);
        s64_store_row(acc, p.dq + (static_cast<int64_t>(bh) * p.Tq + t) * 64);
      }
    }
    if ((!ok || !aligned) && lane == 0) atomicOr(p.status, kStatusWaitTimeout);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 256);
}

// all of dK/dV's tasks, then dQ's
__global__ void __launch_bounds__(kS64Threads, 2) sel_bwd64_kernel(const __grid_constant__ S64Maps m, const __grid_constant__ SelBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int kv_tasks = p.B * p.H * p.nkb, x = static_cast<int>(blockIdx.x);
  if (x < kv_tasks) sel_bwd64_cta<0>(m, p, smem, x / p.nkb, x % p.nkb);
  else sel_bwd64_cta<1>(m, p, smem, (x - kv_tasks) / p.nqb, (x - kv_tasks) % p.nqb);
}

int sel_bwd64(const SelBwdParams& p, cudaStream_t st) {
  const uint64_t bh = static_cast<uint64_t>(p.B) * p.H;
  const int64_t tasks = static_cast<int64_t>(bh) * (static_cast<int64_t>(p.nkb) + p.nqb);
  S3R_REQUIRE(tasks < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_sel_attn_bwd: grid too large");
  S64Maps m;
  auto map = [&](CUtensorMap* out, const void* base, int rows) {
    const uint64_t t = static_cast<uint64_t>(rows), dims[3] = {64, t, bh}, strides[2] = {128, t * 128};
    const uint32_t box[3] = {64, 64, 1};
    return make_tensor_map(out, base, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  int rc = map(&m.q, p.q, p.Tq);
  if (!rc) rc = map(&m.d_o, p.d_o, p.Tq);
  if (!rc) rc = map(&m.k, p.k, p.Tk);
  if (!rc) rc = map(&m.v, p.v, p.Tk);
  if (rc) return rc;
  S3R_CUDA(cudaFuncSetAttribute(sel_bwd64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kS64Smem));
  return launch(sel_bwd64_kernel, static_cast<unsigned>(tasks), kS64Threads, kS64Smem, st, m, p);
}

}  // namespace s3r
