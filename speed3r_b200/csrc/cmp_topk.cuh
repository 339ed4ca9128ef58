// Compression branch, forward, second of two kernels: the `topk` columns of every pooled query's largest RAW logits
// (RANK 0), ordered by (logit descending, column ascending), or the `topk` blocks of four columns (RANK 1) by
// log2 of the sum of 2^(c * s) over a block's first rank_take columns, which needs no row normaliser.
//
// RANK 0 compares its logits exactly with a bound that the first kernel took from products of another shape (N = 128 instead of
// 64) with the keys in another order.  An element of S is the sum over its own row and column alone, in the same k-steps of
// 16 channels of the same instruction, so neither its neighbours nor N should matter; nothing documents it, and one unit's
// difference would lose the entries at the bound.  test_cmp_topk_keeps_logits_at_the_bound has the bound on single logits.
//
// The first kernel (cmp_attn.cuh) leaves a lower bound of each row's topk-th largest logit, so this one repeats Q K^T on
// the tensor cores and only collects the logits that reach the bound - about 44 per row with independent scores - into
// lists of (logit, column) pairs in shared memory, [slot][lane] so that a thread's accesses never meet another's on a
// bank.  A row has two threads (in two warpgroups that take turns at its key tiles) and a list for each.  A list that
// fills up (structured scores can leave a loose bound; equal scores all reach it) is cut back to its best 32 there and
// then, and goes on with the 32nd of those as its bound.  At the end every thread sorts its list in registers, and one of
// the two merges them.  What is sorted is one 32-bit word per pair - the logit's key above the bound's, cut to 25 bits where it
// needs more, and the pair's place - with a minimum and a maximum per exchange (sorting (key, column) as 64-bit words: 12 us
// per CTA, most of the kernel up to 384 keys and 15 % of it at 6300).  Words of the same key - logits that are equal, or equal in
// those bits: one row in several thousand, so that most launches have some - are put in order by their pairs afterwards, as
// neighbours.  A row is sorted again with the columns where the last of the 32 and one that was lost share a key, and where one pass
// over the neighbours leaves a run of five or more out of order, which would take as many passes as it is long.  (All of a warp's rows
// sorted again for any equal pair: this kernel 28 to 30 us instead of 17.5 for 2 x 384 x 384, 16 heads, 40 instead of 28 for
// 1024 x 1024; both kernels 466 instead of 454 for 6300 x 6300.  Long runs pass by pass: 64 x 64 with all keys the same 84 us instead
// of 39, 6300 x 6300 with every key there 16 times 666 instead of 620.)
//
// Bound: instructions and their latency in the scan: a max tree and a vote per 16 columns of a warp, and for the chunks
// with a hit (three in four at 250 views, one in three at 1000) a mask and a store.  A chunk's only pair is appended under a predicate,
// not in a branch: both kernels, 16 heads, 4032 x 4032 206.5 -> 203.2 us, 6300 x 6300 446 -> 425; several pairs of a chunk as well for one
// row tile (512 x 512 29.8 -> 29.5), but not for two, whose 16 warps cover the branches (1400 x 1400 55.1 with predicates, 54.6 with
// branches, 6300 x 6300 426.0 and 425.2).  The products take half of the time that the tensor pipe alone would need.  S of a tile
// is two buffers of 64 columns, so that the next products run while a half is
// scanned (16 columns at a time, S held for a whole tile: 1.05 instead of 0.95 ms for 15750 x 15750, 16 heads), each taken into
// registers 32 columns at a time (all 64 at once spilled in the scan: both kernels 448 instead of 439 us for 6300 x 6300, 2140
// instead of 2098 for 15750 x 15750).
// RANK 1 sums exponentials relative to the bound, three in four of them needed where a block counts three columns, and
// only blocks that reach it get their logarithm: bound by the exponentials' unit.
// Roles: warp 0 TMA producer, warp 1 tcgen05.mma issuer, warp 2 tensor-memory allocator, warps 4-19 scan: R = 2 row tiles of
// 128 queries, two warpgroups each.  Tensor memory: R row tiles x 2 tiles x 128 columns.  R = 1 (warps 4-11) where that still
// leaves one CTA per SM at most: the sorts share the issue slots of half as many warps.  Both kernels, 16 heads: 128 x 128
// 16.1 -> 13.6 us, 384 x 384 (2 samples) 24.2 -> 19.6, 1152 x 1152 56.0 -> 49.5.
#pragma once
#include "common.cuh"
#include "cmp_common.cuh"

namespace s3r {

constexpr int kTkTile = 128 * 128;             // 128 rows x 64 bf16, bytes
constexpr int kTkCap = 40;                     // pairs a list holds before it is cut back to 32
constexpr int kTkStages = 2;
template <int R>
struct TkCfg {
  static constexpr int kRows = R * 128, kThreads = 128 + 256 * R;
  static constexpr int kOffK = R * kTkTile, kOffBuf = kOffK + kTkStages * kTkTile;
  static constexpr int kSmem = kOffBuf + 2 * kRows * kTkCap * 8 + 1024;
};
// With fewer tiles the two scans of a row take halves of every tile, not turns: with an odd or small number of tiles one of
// them would have more.  Both kernels, 16 heads, halves against turns: 384 x 896 (7 tiles) 43.6 and 45.0 us, 4096 x 1900 (15)
// 143.5 and 146.2, 1512 x 1512 (12) 70.4 and 70.9; beyond the line 4096 x 4096 (32) 218.8 and 221.4, 6300 x 6300 (50) 445.3 and
// 451.5, so that the line could lie higher; longer ones were not measured.
constexpr int kTkSplitTiles = 16;

struct TkCtl {
  uint64_t q_full, drained;
  uint64_t k_full[kTkStages], k_empty[kTkStages];
  uint64_t s_full[2][2][2], s_empty[2][2][2];  // [row tile][tile parity][half of the tile]
  uint32_t tmem_base;
  uint32_t abort_flag;
};

struct TkParams {
  int32_t* idx;
  int Nq, Nc, topk;
  int pad;                     // what an empty place decodes to: the last column or block, the reference's padding
  int n_rank, rank_take;       // RANK 1: blocks whose counted columns all exist, columns counted per block
  float c_scale;               // RANK 1: softmax scale * log2(e)
  int vec;                     // rows of idx can be written 16 bytes at a time
  uint32_t* status;
};

__device__ __forceinline__ uint64_t tk_entry(uint2 raw) {          // larger = better: (key of the logit, ~column)
  return (static_cast<uint64_t>(sortable_key(__uint_as_float(raw.x))) << 32) | static_cast<uint32_t>(~raw.y);
}

// Cuts this thread's list of `cnt` > 32 pairs back to its best 32 (in place, column order lost) and returns the bound
// to go on with.  A binary min-heap over slots 0..31 whose root is replaced by every better pair of the rest.
__device__ __noinline__ float tk_cut(uint2* buf, int cnt) {
  auto ld = [&](int i) { return tk_entry(buf[i * 32]); };
  auto sift = [&](int i, uint2 raw) {
    const uint64_t v = tk_entry(raw);
    while (true) {
      int c = 2 * i + 1;
      if (c >= 32) break;
      uint64_t e = ld(c);
      if (c + 1 < 32) {
        const uint64_t e2 = ld(c + 1);
        if (e2 < e) { e = e2; ++c; }
      }
      if (e >= v) break;
      buf[i * 32] = buf[c * 32];
      i = c;
    }
    buf[i * 32] = raw;
  };
  for (int i = 15; i >= 0; --i) sift(i, buf[i * 32]);
  for (int i = 32; i < cnt; ++i) {
    const uint2 raw = buf[i * 32];
    if (tk_entry(raw) > ld(0)) sift(0, raw);
  }
  return key_to_float(sortable_key(__uint_as_float(buf[0].x)));
}

// The hits of a chunk where some list of the warp may fill up: eight columns at a time, all lists that could be cut at once
// (one by one as each fills, a warp cut up to 32 times where neighbouring queries want the same keys).  Out of line, so that
// the registers of the scan are not laid out around the cuts.
struct TkChunk {
  uint32_t x[16];
};
__device__ __noinline__ void tk_append_checked(const TkChunk ch, uint2* buf, uint32_t col0, int& cnt, float& thr) {
#pragma unroll 1
  for (uint32_t h = 0; h < 16; h += 8) {
    int n = cnt;
#pragma unroll 1
    for (uint32_t i = 0; i < 8; ++i) n += __uint_as_float(ch.x[h + i]) > thr;
    if (__any_sync(0xffffffffu, n > kTkCap)) {
      if (cnt > 32) {
        thr = tk_cut(buf, cnt);
        cnt = 32;
      }
      __syncwarp();
    }
#pragma unroll 1
    for (uint32_t i = 0; i < 8; ++i) {
      if (__uint_as_float(ch.x[h + i]) > thr) {
        buf[cnt * 32] = make_uint2(ch.x[h + i], col0 + h + i);
        ++cnt;
      }
    }
  }
}
static_assert(kTkCap >= 40, "eight pairs fit into a list that has been cut");

// A bitonic sequence (what a[i] = max(a[i], b[31 - i]) of two descending lists leaves: the best 32 of both), sorted.
template <typename T>
__device__ __forceinline__ void tk_merge(T (&v)[32]) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1)
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if ((i ^ j) > i) order_desc(v[i], v[i ^ j]);
}
// The best 32 of a row's two lists with ties in column order: columns to out[i * 128], ~0 for an empty place.
__device__ __noinline__ void tk_exact(const uint2* la, int na, const uint2* lb, int nb, uint32_t* out) {
  uint64_t a[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) a[i] = i < na ? tk_entry(la[i * 32]) : 0ull;
  sort_desc<32>(a);
#pragma unroll 1
  for (int part = 0; part < 6; ++part) {       // the rest in pieces of eight: 32.. of the first list, all of the second
    uint64_t e[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int s = part == 0 ? 32 + i : (part - 1) * 8 + i;
      const bool in = part == 0 ? s < na : s < nb;
      e[i] = in ? tk_entry((part == 0 ? la : lb)[s * 32]) : 0ull;
    }
    sort_desc<8>(e);
#pragma unroll
    for (int i = 0; i < 8; ++i) a[31 - i] = a[31 - i] < e[i] ? e[i] : a[31 - i];
    tk_merge(a);
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) out[i * 128] = a[i] >> 32 ? ~static_cast<uint32_t>(a[i]) : ~0u;
}
static_assert(kTkCap == 40, "tk_exact takes lists of up to 40, the packed words a place below 80");

// Both kinds of CTA in one grid: a row's bound is there when its word is no longer what it was filled with (all bits set: a NaN
// that no arithmetic returns).  For at most a second, in which a CTA of the attention goes through some 2 x 10^8 keys; called by whole
// warps.  Fill and grid are in stream order; the bound and the word that it replaces are one aligned word, so that nothing else has to be seen
// with it.
__device__ __forceinline__ bool wait_bound(const int32_t* word, bool mine, uint32_t& v, volatile uint32_t* abort_flag) {
  const uint64_t start = globaltimer_ns();
  while (true) {
    v = 0;
    if (mine) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
    if (__all_sync(0xffffffffu, v != ~0u)) return true;
    const bool over = *abort_flag != 0u || globaltimer_ns() - start > 1000000000ull;
    if (__any_sync(0xffffffffu, over)) {
      *abort_flag = 1u;
      return false;
    }
    __nanosleep(200);
  }
}

// `cta`: which R * 128 rows.  WAIT: in one grid with the CTAs that find the bounds.
template <int R, int RANK, bool WAIT>
__device__ __forceinline__ void cmp_topk_cta(const CUtensorMap& map_q, const CUtensorMap& map_k, const TkParams& p, TkCtl& ctl,
                                             uint8_t* smem_raw, int cta) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  using C = TkCfg<R>;
  const int tiles_per_bh = (p.Nq + C::kRows - 1) / C::kRows;
  const int bh = cta / tiles_per_bh;
  const int q0 = (cta % tiles_per_bh) * C::kRows;
  const int ntiles = (p.Nc + 127) / 128;
  const bool split = ntiles < kTkSplitTiles;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    mbar_init(&ctl.q_full, 1);
    mbar_init(&ctl.drained, 1);
    for (int s = 0; s < kTkStages; ++s) {
      mbar_init(&ctl.k_full[s], 1);
      mbar_init(&ctl.k_empty[s], 1);
    }
    for (int i = 0; i < 8; ++i) {
      mbar_init(&ctl.s_full[0][0][0] + i, 1);
      mbar_init(&ctl.s_empty[0][0][0] + i, 4);
    }
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(&ctl.tmem_base, R * 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // In a launch of its own this kernel could begin with its copies and products before the attention has ended, and wait for the bounds
  // as they come, in places that the attention fills before it lets this launch start.  The op at 2048 tokens took 1.6 us less that way,
  // but nothing documents what a grid sees of others in front of this wait, and a place's old content taken for a bound is a wrong table.
  griddep_wait();
  griddep_launch();
  const uint32_t tmem = ctl.tmem_base;
  volatile uint32_t* abort_flag = &ctl.abort_flag;

  // registers: for R = 2 the launch gives every thread 96, the utility warps hand most of theirs to the scan
  // (640 x 96 = 61440 = 512 x 112 + 128 x 32)
  if (warp < 4) {
    if (R == 2) reg_dealloc<32>();
    if (warp == 0) {
      if (lane == 0) {
        mbar_expect_tx(&ctl.q_full, R * kTkTile);
#pragma unroll
        for (int t = 0; t < R; ++t) tma_load_3d(sbase + t * kTkTile, &map_q, &ctl.q_full, 0, q0 + t * 128, bh);
        int issued = 0;
        for (int j = 0; j < ntiles; ++j) {
          const int s = j % kTkStages;
          if (!mbar_wait(&ctl.k_empty[s], ((j / kTkStages) & 1) ^ 1, abort_flag)) break;
          mbar_expect_tx(&ctl.k_full[s], kTkTile);
          tma_load_3d(sbase + C::kOffK + s * kTkTile, &map_k, &ctl.k_full[s], 0, j * 128, bh);
          issued = j + 1;
        }
        if (*abort_flag) {
          // give copies already in flight a bounded chance to land before the CTA's memory is released
          for (int j = max(0, issued - kTkStages); j < issued; ++j) {
            volatile uint32_t dummy = 0;
            mbar_wait(&ctl.k_full[j % kTkStages], (j / kTkStages) & 1, &dummy);
          }
        }
      }
    } else if (warp == 1) {
      const bool leader = elect_one_sync();
      constexpr uint32_t idesc = umma_idesc_bf16(128, 64, 0, 0);
      const uint64_t desc_q = umma_desc_sw128(sbase), desc_k = umma_desc_sw128(sbase + C::kOffK);
      bool ok = mbar_wait_warp(&ctl.q_full, 0, abort_flag);
      int s = 0;
      uint32_t ph = 0;
#pragma unroll 1
      for (int j = 0; j < ntiles && ok; ++j) {
        const int b = j & 1;
        ok = mbar_wait_warp(&ctl.k_full[s], ph, abort_flag);
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) {
          const int t = i % R, h = i / R;
          if (ok) ok = mbar_wait_warp(&ctl.s_empty[t][b][h], ((j >> 1) & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (leader) {
            umma_ss_k4<2, 2>(tmem + t * 256 + b * 128 + h * 64, desc_q + static_cast<uint64_t>(t * (kTkTile >> 4)),
                             desc_k + static_cast<uint64_t>(s * (kTkTile >> 4) + h * (kTkTile >> 5)), idesc, 0u);
            umma_commit(&ctl.s_full[t][b][h]);
            if (i == 2 * R - 1) umma_commit(&ctl.k_empty[s]);
          }
          __syncwarp();
        }
        if (++s == kTkStages) { s = 0; ph ^= 1u; }
      }
      if (!ok) {
        if (leader) umma_commit(&ctl.drained);
        __syncwarp();
        volatile uint32_t dummy = 0;
        mbar_wait(&ctl.drained, 0, &dummy);      // let issued MMAs drain before tensor memory is freed
      }
    }
  } else {
    if (R == 2) reg_alloc<112>();
    const int t = (warp - 4) >> 3, par = ((warp - 4) >> 2) & 1, quarter = warp & 3;
    const int row = q0 + t * 128 + quarter * 32 + lane;
    const uint32_t t_s = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + t * 256;
    uint2* lists = reinterpret_cast<uint2*>(smem_raw + (sbase - smem_u32(smem_raw)) + C::kOffBuf);
    uint2* buf = lists + (warp - 4) * (kTkCap * 32) + lane;
    int32_t* out = p.idx + (static_cast<int64_t>(bh) * p.Nq + row) * p.topk;
    // `score > thr` for every score that reaches the bound (NaN and -inf never do); rows past the end collect nothing
    float thr = INFINITY;
    uint32_t base_key = 0;                       // every collected pair's key is at least this
    bool ok = true;
    uint32_t bound_word = 0;
    if (WAIT) ok = wait_bound(out, row < p.Nq, bound_word, abort_flag);
    else if (row < p.Nq) bound_word = static_cast<uint32_t>(*out);
    if (ok && row < p.Nq) {
      const float bound = fmaxf(__uint_as_float(bound_word), -3.402823466e38f);
      base_key = sortable_key(bound == 0.f ? -0.f : bound);
      thr = bound == 0.f ? __uint_as_float(0x80000001u) : key_to_float(sortable_key(bound) - 1u);
    }
    const uint32_t first = smem_u32(buf), end = first + kTkCap * 256;
    uint32_t at = first;                         // where the list's next pair goes

    // 16 columns: a max tree and a vote pass over chunks in which no row of the warp has a hit
    auto scan = [&](const uint32_t* x, int col0) {
      auto f = [&](int i) { return __uint_as_float(x[i]); };
      const float m = fmaxf(fmax3(fmax3(f(0), f(1), f(2)), fmax3(f(3), f(4), f(5)), fmax3(f(6), f(7), f(8))),
                            fmax3(fmax3(f(9), f(10), f(11)), fmax3(f(12), f(13), f(14)), f(15)));
      if (!__any_sync(0xffffffffu, m > thr)) return;
      // bit 15 - i of the mask = sign of thr - x[i]; two chains of shifts
      uint32_t m0 = 0, m1 = 0;
      const float2 minus = make_float2(-1.f, -1.f), thr2 = make_float2(thr, thr);
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const float2 d0 = ffma2(make_float2(f(i), f(i + 1)), minus, thr2), d1 = ffma2(make_float2(f(8 + i), f(9 + i)), minus, thr2);
        m0 = __funnelshift_l(__float_as_uint(d0.y), __funnelshift_l(__float_as_uint(d0.x), m0, 1), 1);
        m1 = __funnelshift_l(__float_as_uint(d1.y), __funnelshift_l(__float_as_uint(d1.x), m1, 1), 1);
      }
      const uint32_t mask = (m0 << 8) | m1;
      // one hit per row at most, and room for it: it is the chunk's maximum
      if (!__any_sync(0xffffffffu, (mask & (mask - 1)) != 0u || at == end)) {
        sts64_append<256>(mask, at, __float_as_uint(m), static_cast<uint32_t>(col0 - 16 + __clz(mask)));
      } else if (!__any_sync(0xffffffffu, at + 256 * __popc(mask) > end)) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (R == 1) {
            sts64_append<256>(mask & (0x8000u >> i), at, x[i], static_cast<uint32_t>(col0 + i));
          } else if (mask & (0x8000u >> i)) {
            sts64(at, x[i], static_cast<uint32_t>(col0 + i));
            at += 256;
          }
        }
      } else {
        TkChunk ch;
#pragma unroll
        for (int i = 0; i < 16; ++i) ch.x[i] = x[i];
        int cnt = static_cast<int>(at - first) >> 8;
        tk_append_checked(ch, buf, static_cast<uint32_t>(col0), cnt, thr);
        at = first + cnt * 256;
        __syncwarp();
      }
    };
    // 16 columns as four blocks
    const float cs = p.c_scale;
    float2 off01, off23;                         // minus the bound; columns that do not count: minus infinity
    float cutoff;                                // roundings of the sums stay well below 1e-3 up to |bound| = 8192
    auto set_offsets = [&](float bound) {
      off01 = make_float2(-bound, p.rank_take > 1 ? -bound : -INFINITY);
      off23 = make_float2(p.rank_take > 2 ? -bound : -INFINITY, p.rank_take > 3 ? -bound : -INFINITY);
      cutoff = bound == INFINITY ? INFINITY : fabsf(bound) < 8192.f ? 0.999f : 0.f;      // +inf: a row past the end takes nothing
    };
    if (RANK) set_offsets(fmaxf(thr, -3.402823466e38f));
    const bool four = p.rank_take > 3;
    auto scan_blocks = [&](const uint32_t* x, int col0) {
      auto f = [&](int i) { return __uint_as_float(x[i]); };
      const float2 cs2 = make_float2(cs, cs);
      float sum[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = ffma2(make_float2(f(4 * i), f(4 * i + 1)), cs2, off01), b = ffma2(make_float2(f(4 * i + 2), f(4 * i + 3)), cs2, off23);
        if (i) {
          sum[i] = fast_exp2(a.x) + fast_exp2(a.y) + fast_exp2(b.x);
        } else {
          const float2 e = exp2_fma2(make_float2(fminf(a.x, 126.f), fminf(a.y, 126.f)));
          sum[i] = e.x + e.y + fast_exp2(b.x);
        }
        if (four) sum[i] += fast_exp2(b.y);
      }
      if (!__any_sync(0xffffffffu, fmaxf(fmax3(sum[0], sum[1], sum[2]), sum[3]) >= cutoff)) return;
      if (__any_sync(0xffffffffu, at + 4 * 256 > end)) {                    // cut every list that has something to lose
        const int cnt = static_cast<int>(at - first) >> 8;
        if (cnt > 32) {
          thr = tk_cut(buf, cnt);
          at = first + 32 * 256;
          set_offsets(thr);
        }
        __syncwarp();
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (sum[i] >= cutoff) {
          float a[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = e < p.rank_take ? f(4 * i + e) * cs : -INFINITY;
          const float m = fmaxf(fmax3(a[0], a[1], a[2]), a[3]);
          const float r = m + fast_log2((fast_exp2(a[0] - m) + fast_exp2(a[1] - m)) + (fast_exp2(a[2] - m) + fast_exp2(a[3] - m)));
          const int n = (col0 >> 2) + i;
          if (n < p.n_rank && r > thr) {
            sts64(at, __float_as_uint(r), static_cast<uint32_t>(n));
            at += 256;
          }
        }
      }
    };
    // half h of tile j
    auto half_tile = [&](int j, int h) -> bool {
      const int b = j & 1;
      if (!mbar_wait_warp(&ctl.s_full[t][b][h], (j >> 1) & 1, abort_flag)) return false;
      tc_fence_after();
      const uint32_t src = t_s + b * 128 + h * 64;
      const int col0 = j * 128 + h * 64, left = p.Nc - col0;
      auto release = [&]() {                     // all of this half of S is in registers: the next Q K^T may overwrite it
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.s_empty[t][b][h]);
      };
      auto go = [&](const uint32_t* x, int c) {
        if (RANK) scan_blocks(x, c);
        else scan(x, c);
      };
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t x[32];
        tmem_ld32(src + 32 * q, x);
        tmem_ld_wait();
        if (q == 1) release();
        if (left < 64) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (32 * q + i >= left) x[i] = 0xff800000u;   // -inf
        }
        go(x, col0 + 32 * q);
        go(x + 16, col0 + 32 * q + 16);
      }
      return true;
    };
    if (split) {
#pragma unroll 1
      for (int j = 0; j < ntiles && ok; ++j) ok = half_tile(j, par);
    } else {
#pragma unroll 1
      for (int u = 2 * par; u < 2 * ntiles && ok; u = (u & 1) ? u + 3 : u + 1) ok = half_tile(u >> 1, u & 1);
    }

    const int cnt = static_cast<int>(at - first) >> 8;
    const int r = quarter * 32 + lane;
    // Q and the K ring are idle once every scan warp is here (whatever happened): per row tile 32 words per row for sorted
    // words and columns, and four per row for what its threads tell each other
    asm volatile("bar.sync 3, %0;" ::"n"(256 * R) : "memory");
    uint32_t* words = reinterpret_cast<uint32_t*>(smem_raw + (sbase - smem_u32(smem_raw))) + t * (36 * 128) + r;   // [place][row]
    static_assert(R * 36 * 128 * 4 <= C::kOffBuf, "the lists behind Q and the K ring are still in use");
    // [list][row] largest key (later [0]: whether the row's words are columns already), [2][row] the second list's length, [3][row] the
    // largest word that it lost.  Between two meetings no word is both written and read: nothing else orders a row's two threads.
    uint32_t* tell = words + 32 * 128;
    auto meet = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + t) : "memory"); };
    uint32_t a[32], e[kTkCap - 32];
    uint32_t top = 0;
    // keys above the bound's, plus one: an empty place is 0
    auto word = [&](int i) {
      const uint32_t d = i < cnt ? sortable_key(__uint_as_float(buf[i * 32].x)) - base_key + 1u : 0u;
      top = max(top, d);
      return d;
    };
#pragma unroll
    for (int i = 0; i < 32; ++i) a[i] = word(i);
#pragma unroll
    for (int i = 0; i < kTkCap - 32; ++i) e[i] = word(32 + i);
    tell[par * 128] = top;
    if (par == 1) tell[2 * 128] = static_cast<uint32_t>(cnt);
    meet();
    top = max(top, tell[(par ^ 1) * 128]);
    const int shift = max(0, 7 - __clz(top | 1u));        // bits of the keys beyond 25
    auto pack = [&](uint32_t& d, int i) { d = d ? ((d >> shift) << 7) | static_cast<uint32_t>(127 - par * kTkCap - i) : 0u; };
#pragma unroll
    for (int i = 0; i < 32; ++i) pack(a[i], i);
    sort_desc<32>(a);
    uint32_t lost = 0;                         // the largest word that is not among the row's 32
    if (__any_sync(0xffffffffu, cnt > 32)) {
#pragma unroll
      for (int i = 0; i < kTkCap - 32; ++i) pack(e[i], 32 + i);
      sort_desc<kTkCap - 32>(e);
#pragma unroll
      for (int i = 0; i < kTkCap - 32; ++i) {
        lost = max(lost, min(a[31 - i], e[i]));
        a[31 - i] = max(a[31 - i], e[i]);
      }
      tk_merge(a);
    }
    if (par == 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i) words[i * 128] = a[i];
      tell[3 * 128] = lost;
    }
    meet();
    if (par == 0) {
      lost = max(lost, tell[3 * 128]);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const uint32_t o = words[(31 - i) * 128];
        lost = max(lost, min(a[i], o));
        a[i] = max(a[i], o);
      }
      tk_merge(a);
      const bool cut_equal = lost != 0u && lost >> 7 >= a[31] >> 7;
      uint32_t equal = 0;                      // bit i: words i and i + 1 have the same key
#pragma unroll
      for (int i = 0; i < 31; ++i) equal |= a[i + 1] != 0u && a[i] >> 7 == a[i + 1] >> 7 ? 1u << i : 0u;
      const uint2* other = buf + 4 * (kTkCap * 32);
      const bool exact = __any_sync(0xffffffffu, cut_equal);
      bool moved = !exact && __any_sync(0xffffffffu, equal != 0u);
      if (moved) {
        // neighbours of the same key change places until their pairs are in order; once where five or more are in a row
        auto pair_of = [&](uint32_t w) {
          const int place = 127 - static_cast<int>(w & 127u);
          return tk_entry(place < kTkCap ? buf[place * 32] : other[(place - kTkCap) * 32]);
        };
        const bool run = __any_sync(0xffffffffu, (equal & (equal >> 1) & (equal >> 2) & (equal >> 3)) != 0u);
#pragma unroll 1
        do {
          moved = false;
#pragma unroll
          for (int i = 0; i < 31; ++i) {
            if ((equal >> i) & 1u) {
              if (pair_of(a[i]) < pair_of(a[i + 1])) {
                const uint32_t w = a[i];
                a[i] = a[i + 1];
                a[i + 1] = w;
                moved = true;
              }
            }
          }
          moved = __any_sync(0xffffffffu, moved);
        } while (moved && !run);
      }
      if (exact || moved) {
        tk_exact(buf, cnt, other, static_cast<int>(tell[2 * 128]), words);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) words[i * 128] = a[i];
      }
      tell[0] = exact || moved;                // columns already, not words
    }
    meet();
    // Words to columns, by both threads of a row, half of it each, in a loop: a CTA runs this code once, and what it takes is
    // the fetching of instructions (32 lookups and stores unrolled in one of the threads: 4400 to 8100 cycles; both kernels,
    // 16 heads, 2 x 384 x 384 22.5 -> 22.0 us, 1024 x 1024 40.6 -> 39.9).
    if (ok && *abort_flag == 0u && row < p.Nq) {           // neither of the row's threads gave up
      const bool columns = tell[0] != 0u;
      const uint2* list = buf - par * 4 * (kTkCap * 32);
#pragma unroll 1
      for (int i0 = par * 16; i0 < par * 16 + 16; i0 += 4) {
        int32_t c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t w = words[(i0 + u) * 128];
          // one address and one load for either list and for empty places
          const int place = w != 0u && !columns ? 127 - static_cast<int>(w & 127u) : 0;
          const uint32_t col = list[(place < kTkCap ? place : place + 3 * kTkCap) * 32].y;
          c[u] = w == (columns ? ~0u : 0u) ? p.pad : static_cast<int32_t>(columns ? w : col);
        }
        if (p.vec) {
          if (i0 < p.topk) *reinterpret_cast<int4*>(out + i0) = make_int4(c[0], c[1], c[2], c[3]);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (i0 + u < p.topk) out[i0 + u] = c[u];
        }
      }
    }
    if (!ok && lane == 0) atomicOr(p.status, kStatusWaitTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, R * 256);
}

}  // namespace s3r
