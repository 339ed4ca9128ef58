// Selection branch, backward: key-centric index (CSR) of the selection table built on the device,
// the fused backward of the gated merge, and the two sparse gradient kernels.
//
//   dQ    : one warp per 16 query rows, looping over the key blocks its query block selected
//   dK/dV : one warp per 16 key rows, looping over the query blocks that selected its key block
//           (CSR lists, ascending query block => a fixed summation order, no atomics on floats)
#include <mutex>

#include "sel_common.cuh"

namespace s3r {

// ------------------------------------------------------------------------------------------------
// key-centric CSR
// ------------------------------------------------------------------------------------------------
__global__ void csr_count_kernel(const int32_t* __restrict__ idx, int32_t* __restrict__ counts, int64_t per_bh,
                                 int64_t total, int Nkb) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int n = idx[i];
    if (n >= 0 && n < Nkb) atomicAdd(&counts[(i / per_bh) * (Nkb + 1) + n], 1);
  }
}

// One CTA per (b,h): exclusive scan of counts[0..Nkb) in place -> offsets[0..Nkb]; cursor = offsets.
__global__ void __launch_bounds__(1024) csr_scan_kernel(int32_t* __restrict__ offsets, int32_t* __restrict__ cursor,
                                                        int Nkb) {
  __shared__ int32_t warp_sums[32];
  __shared__ int32_t carry_s;
  int32_t* off = offsets + static_cast<int64_t>(blockIdx.x) * (Nkb + 1);
  int32_t* cur = cursor + static_cast<int64_t>(blockIdx.x) * Nkb;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int base = 0; base < Nkb; base += 1024) {
    const int i = base + threadIdx.x;
    const int32_t v = (i < Nkb) ? off[i] : 0;
    int32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int32_t w = warp_sums[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      warp_sums[lane] = w;   // inclusive
    }
    __syncthreads();
    const int32_t carry = carry_s;
    const int32_t excl = carry + (warp > 0 ? warp_sums[warp - 1] : 0) + x - v;
    if (i < Nkb) {
      off[i] = excl;
      cur[i] = excl;
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = carry + warp_sums[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) off[Nkb] = carry_s;
}

__global__ void csr_fill_kernel(const int32_t* __restrict__ idx, int32_t* __restrict__ cursor,
                                int32_t* __restrict__ tmp, int64_t per_bh, int64_t total, int Nkb, int topk) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int n = idx[i];
    if (n >= 0 && n < Nkb) {
      const int64_t bh = i / per_bh;
      const int32_t pos = atomicAdd(&cursor[bh * Nkb + n], 1);
      tmp[bh * per_bh + pos] = static_cast<int32_t>((i - bh * per_bh) / topk);   // query block
    }
  }
}

// The fill above leaves every segment complete but in arrival order; the gradient kernel needs ascending
// query blocks (a fixed summation order).  Segments are sorted by length class:
//   len <= 128     one warp ranks the segment with shuffles, up to four entries per lane (the mean length is top-k;
//                  with 32 as the limit half of all segments went to the class below: 0.72 of 0.97 ms at 250 views)
//   len <= 4096    one CTA, bitonic network in shared memory
//   longer         ("sink" key blocks that most query blocks select) one CTA walks the (b,h) slice of the
//                  table in order and compacts the matching query blocks: O(Nq*topk), no comparison sort
// The first kernel handles the short class and queues every other segment for the second.
constexpr int kCsrSmemSort = 4096;
constexpr int kCsrWarpSort = 128;

// Ranks len <= 32 * N entries; entry and position make one unsigned key, so that equal entries keep an order.
template <int N>
__device__ __forceinline__ void csr_rank_sort(const int32_t* src, int32_t* dst, int len, int lane) {
  uint32_t key[N];
  int rank[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int pos = lane + 32 * i;
    key[i] = pos < len ? static_cast<uint32_t>(src[pos]) * kCsrWarpSort + pos : 0xffffffffu;
    rank[i] = 0;
  }
#pragma unroll
  for (int ch = 0; ch < N; ++ch) {
    const int n = min(32, len - 32 * ch);
    for (int t = 0; t < n; ++t) {
      const uint32_t y = __shfl_sync(0xffffffffu, key[ch], t);
#pragma unroll
      for (int i = 0; i < N; ++i) rank[i] += y < key[i];
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (lane + 32 * i < len) dst[rank[i]] = static_cast<int32_t>(key[i] / kCsrWarpSort);
}

__global__ void __launch_bounds__(256) csr_sort_small_kernel(const int32_t* __restrict__ offsets,
                                                             const int32_t* __restrict__ tmp, int32_t* __restrict__ qids,
                                                             int64_t per_bh, int Nkb, int64_t nseg, int warp_max,
                                                             int32_t* __restrict__ queue) {
  const int lane = threadIdx.x & 31;
  const int64_t seg = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  if (seg >= nseg) return;
  const int64_t bh = seg / Nkb;
  const int n = static_cast<int>(seg - bh * Nkb);
  const int32_t* off = offsets + bh * (Nkb + 1);
  const int beg = off[n], len = off[n + 1] - beg;
  const int32_t* src = tmp + bh * per_bh + beg;
  int32_t* dst = qids + bh * per_bh + beg;
  if (len > warp_max) {
    if (lane == 0) queue[1 + atomicAdd(&queue[0], 1)] = static_cast<int32_t>(seg);
  } else if (len <= 32) {
    csr_rank_sort<1>(src, dst, len, lane);
  } else if (len <= 64) {
    csr_rank_sort<2>(src, dst, len, lane);
  } else {
    csr_rank_sort<4>(src, dst, len, lane);
  }
}

__global__ void __launch_bounds__(256) csr_sort_long_kernel(const int32_t* __restrict__ idx,
                                                            const int32_t* __restrict__ offsets,
                                                            const int32_t* __restrict__ tmp, int32_t* __restrict__ qids,
                                                            int64_t per_bh, int Nkb, int topk,
                                                            const int32_t* __restrict__ queue) {
  __shared__ int32_t buf[kCsrSmemSort];
  __shared__ int32_t warp_tot[8];
  __shared__ int32_t run_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nqueued = queue[0];
  for (int w = blockIdx.x; w < nqueued; w += gridDim.x) {
    const int64_t seg = queue[1 + w];
    const int64_t bh = seg / Nkb;
    const int n = static_cast<int>(seg - bh * Nkb);
    const int32_t* off = offsets + bh * (Nkb + 1);
    const int beg = off[n], len = off[n + 1] - beg;
    int32_t* dst = qids + bh * per_bh + beg;
    if (len <= kCsrSmemSort) {
      int P = 64;
      while (P < len) P <<= 1;
      const int32_t* src = tmp + bh * per_bh + beg;
      for (int i = tid; i < P; i += 256) buf[i] = (i < len) ? src[i] : 0x7fffffff;
      __syncthreads();
      for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
          for (int i = tid; i < P; i += 256) {
            const int l = i ^ j;
            if (l > i) {
              const int32_t a = buf[i], b = buf[l];
              const bool up = (i & k) == 0;
              if ((a > b) == up) { buf[i] = b; buf[l] = a; }
            }
          }
          __syncthreads();
        }
      }
      for (int i = tid; i < len; i += 256) dst[i] = buf[i];
      __syncthreads();
    } else {
      // ordered compaction over the (b,h) slice of the table: 8 consecutive entries per thread
      const int32_t* tab = idx + bh * per_bh;
      if (tid == 0) run_base = 0;
      __syncthreads();
      for (int64_t base = 0; base < per_bh; base += 256 * 8) {
        const int64_t i0 = base + static_cast<int64_t>(tid) * 8;
        int32_t e[8];
        int cnt = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          e[u] = (i0 + u < per_bh) ? tab[i0 + u] : -1;
          cnt += (e[u] == n);
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        int before = run_base + incl - cnt;
        int total = 0;
#pragma unroll
        for (int ww = 0; ww < 8; ++ww) {
          const int t = warp_tot[ww];
          before += (ww < warp) ? t : 0;
          total += t;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (e[u] == n) dst[before++] = static_cast<int32_t>((i0 + u) / topk);
        __syncthreads();
        if (tid == 0) run_base += total;
        __syncthreads();
      }
    }
  }
}

// Short tables: one CTA builds the whole index of a (b,h) in shared memory - one launch instead of two memsets and five
// kernels (68 us at 384 query blocks, top-32, 32 heads, most of it launches and the long-segment kernel).  The line at
// kCsrOneEntries entries per (b,h) is where a CTA's passes over its table begin to outlast them.  Where there are more SMs
// than (b,h), several CTAs count all of a table and each fills and sorts a range of its keys (gridDim.y of them).
constexpr int kCsrOneEntries = 24576, kCsrOneKeys = 8192;

__global__ void __launch_bounds__(1024) csr_one_kernel(const int32_t* __restrict__ idx, int32_t* __restrict__ offsets,
                                                       int32_t* __restrict__ qids, int per_bh, int Nkb, int topk) {
  extern __shared__ int32_t one_smem[];
  griddep_wait();
  griddep_launch();
  int32_t* cur = one_smem;                   // counts, then the fill's cursors (= end of each segment afterwards)
  int32_t* ent = one_smem + Nkb;             // query blocks by segment, arrival order
  __shared__ int32_t warp_sums[32];
  __shared__ int32_t carry_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t* tab = idx + static_cast<int64_t>(blockIdx.x) * per_bh;
  int32_t* off = offsets + static_cast<int64_t>(blockIdx.x) * (Nkb + 1);
  int32_t* out = qids + static_cast<int64_t>(blockIdx.x) * per_bh;
  for (int i = tid; i < Nkb; i += 1024) cur[i] = 0;
  if (tid == 0) carry_s = 0;
  __syncthreads();
  for (int i = tid; i < per_bh; i += 1024) {
    const int n = tab[i];
    if (n >= 0 && n < Nkb) atomicAdd(&cur[n], 1);
  }
  __syncthreads();
  for (int base = 0; base < Nkb; base += 1024) {             // exclusive scan in place
    const int i = base + tid;
    const int32_t v = i < Nkb ? cur[i] : 0;
    int32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int32_t w = warp_sums[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    const int32_t carry = carry_s, excl = carry + (warp > 0 ? warp_sums[warp - 1] : 0) + x - v;
    if (i < Nkb) {
      cur[i] = excl;
      if (blockIdx.y == 0) off[i] = excl;
    }
    __syncthreads();
    if (tid == 1023) carry_s = carry + warp_sums[31];
    __syncthreads();
  }
  if (tid == 0 && blockIdx.y == 0) off[Nkb] = carry_s;
  const int per_part = (Nkb + gridDim.y - 1) / gridDim.y, lo = blockIdx.y * per_part, hi = min(Nkb, lo + per_part);
  const int before = lo > 0 && lo < Nkb ? cur[lo] : 0;       // entries of the keys in front of this range
  __syncthreads();
  for (int i = tid; i < per_bh; i += 1024) {
    const int n = tab[i];
    if (n >= lo && n < hi) ent[atomicAdd(&cur[n], 1)] = i / topk;
  }
  __syncthreads();
  for (int n = lo + warp; n < hi; n += 32) {
    const int beg = n > lo ? cur[n - 1] : before, len = cur[n] - beg;
    if (len == 0) continue;
    if (len <= 32) csr_rank_sort<1>(ent + beg, out + beg, len, lane);
    else if (len <= 64) csr_rank_sort<2>(ent + beg, out + beg, len, lane);
    else if (len <= kCsrWarpSort) csr_rank_sort<4>(ent + beg, out + beg, len, lane);
    else {                                                   // ordered compaction over the table
      int at = beg;
      for (int base = 0; base < per_bh; base += 32) {
        const bool hit = base + lane < per_bh && tab[base + lane] == n;
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (hit) out[at + __popc(m & ((1u << lane) - 1u))] = (base + lane) / topk;
        at += __popc(m);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// delta = sum_d o * do  (8 lanes per row, 16-byte loads)
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) delta_kernel(const __nv_bfloat16* __restrict__ o,
                                                    const __nv_bfloat16* __restrict__ d_o, float* __restrict__ delta,
                                                    int64_t rows) {
  griddep_wait();
  griddep_launch();
  const int64_t gid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t row = gid >> 3;
  const int c8 = threadIdx.x & 7;
  float s = 0.f;
  if (row < rows) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + row * 64 + c8 * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(d_o + row * 64 + c8 * 8);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int w = 0; w < 4; ++w) s += bf16_lo(aw[w]) * bf16_lo(bw[w]) + bf16_hi(aw[w]) * bf16_hi(bw[w]);
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  if (row < rows && c8 == 0) delta[row] = s;
}

// ------------------------------------------------------------------------------------------------
// backward of the gated merge: one warp per (b,h,query block); 8 lanes per token, 4 U tokens a pass
// ------------------------------------------------------------------------------------------------
struct MergeBwdParams {
  const __nv_bfloat16* dy;
  const __nv_bfloat16* gate;
  int64_t gsb, gsh, gst;
  const __nv_bfloat16* o_c;
  const __nv_bfloat16* o_s;
  __nv_bfloat16* do_s;
  float* dgate;
  __nv_bfloat16* do_c;
  float* delta_s;
  float* delta_c;                // null: not wanted
  int B, H, Tq, block, nqb;
};

// Bound: HBM and the latency of a pass.  U = 4 has 16 tokens' loads under way before the first is used, in 80 registers: 16 heads,
// blocks of 16, U = 1 -> 4: 2 x 6144 tokens 15.0 -> 14.1 us, 64 512 93.8 -> 88.6, 252 000 353 -> 337 (0.76 of the copy rate).  A pass whose
// tokens do not all exist costs as much as a whole one, and fewer warps fit: 64 512 tokens in blocks of 1 540 and 895 us, 4 148 and 234,
// 8 110 and 141, 12 98 and 105, 15 98.7 and 92.5, 17 101 and 109, 24 90 and 93, 32 86.5 and 80.1, 33 91.1 and 90.6, 100 94.8 and 79.8.
static bool merge_bwd_whole_passes(int block) { return block > 32 || block % 16 == 0 || block % 16 == 15; }

template <int U>
__global__ void __launch_bounds__(256) merge_bwd_kernel(const MergeBwdParams p) {
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31;
  const int64_t wid = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  if (wid >= static_cast<int64_t>(p.B) * p.H * p.nqb) return;
  const int m = static_cast<int>(wid % p.nqb);
  const int bh = static_cast<int>(wid / p.nqb);
  const int b = bh / p.H, h = bh % p.H;
  const int sub = lane >> 3, c8 = lane & 7;
  float oc[8], acc[8];
  {
    const uint4 v = *reinterpret_cast<const uint4*>(p.o_c + (static_cast<int64_t>(bh) * p.nqb + m) * 64 + c8 * 8);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { oc[2 * i] = bf16_lo(w[i]); oc[2 * i + 1] = bf16_hi(w[i]); acc[2 * i] = acc[2 * i + 1] = 0.f; }
  }
  for (int base = 0; base < p.block; base += 4 * U) {
    uint4 a[U], s[U];
    uint32_t gw[U];
    bool live[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int in_block = base + 4 * u + sub, t = m * p.block + in_block;
      live[u] = in_block < p.block && t < p.Tq;
      a[u] = s[u] = make_uint4(0u, 0u, 0u, 0u);
      gw[u] = 0u;
      if (U > 1 || live[u]) {                                // several: loaded in any case, without a branch around each
        const int tc = min(t, p.Tq - 1);
        a[u] = __ldg(reinterpret_cast<const uint4*>(p.dy + ((static_cast<int64_t>(b) * p.Tq + tc) * p.H + h) * 64 + c8 * 8));
        s[u] = __ldg(reinterpret_cast<const uint4*>(p.o_s + (static_cast<int64_t>(bh) * p.Tq + tc) * 64 + c8 * 8));
        gw[u] = __ldg(reinterpret_cast<const uint32_t*>(p.gate + b * p.gsb + h * p.gsh + tc * p.gst));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = m * p.block + base + 4 * u + sub;
      const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, sw[4] = {s[u].x, s[u].y, s[u].z, s[u].w};
      float dyv[8], osv[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        dyv[2 * i] = live[u] ? bf16_lo(aw[i]) : 0.f; dyv[2 * i + 1] = live[u] ? bf16_hi(aw[i]) : 0.f;
        osv[2 * i] = bf16_lo(sw[i]); osv[2 * i + 1] = bf16_hi(sw[i]);
      }
      const float g0 = live[u] ? bf16_lo(gw[u]) : 0.f, g1 = bf16_hi(gw[u]);
      float d0 = 0.f, d1 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        d0 += dyv[i] * oc[i];
        d1 += dyv[i] * osv[i];
        acc[i] += g0 * dyv[i];
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        d0 += __shfl_xor_sync(0xffffffffu, d0, o);
        d1 += __shfl_xor_sync(0xffffffffu, d1, o);
      }
      if (live[u]) {
        uint4 out;
        out.x = pack_bf16(g1 * dyv[0], g1 * dyv[1]); out.y = pack_bf16(g1 * dyv[2], g1 * dyv[3]);
        out.z = pack_bf16(g1 * dyv[4], g1 * dyv[5]); out.w = pack_bf16(g1 * dyv[6], g1 * dyv[7]);
        *reinterpret_cast<uint4*>(p.do_s + (static_cast<int64_t>(bh) * p.Tq + t) * 64 + c8 * 8) = out;
        if (c8 == 0) {
          *reinterpret_cast<float2*>(p.dgate + (static_cast<int64_t>(bh) * p.Tq + t) * 2) = make_float2(d0, d1);
          p.delta_s[static_cast<int64_t>(bh) * p.Tq + t] = g1 * d1;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 8);
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
  }
  uint4 out;
  out.x = pack_bf16(acc[0], acc[1]); out.y = pack_bf16(acc[2], acc[3]);
  out.z = pack_bf16(acc[4], acc[5]); out.w = pack_bf16(acc[6], acc[7]);
  if (sub == 0) *reinterpret_cast<uint4*>(p.do_c + (static_cast<int64_t>(bh) * p.nqb + m) * 64 + c8 * 8) = out;
  if (p.delta_c) {                                         // of the rounded gradient, as s3r_delta takes it
    const uint32_t w[4] = {out.x, out.y, out.z, out.w};
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) d += oc[2 * i] * bf16_lo(w[i]) + oc[2 * i + 1] * bf16_hi(w[i]);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == 0) p.delta_c[static_cast<int64_t>(bh) * p.nqb + m] = d;
  }
}

// ------------------------------------------------------------------------------------------------
// sparse dQ and dK/dV
// ------------------------------------------------------------------------------------------------
// Both kernels: one warp = one CTA owns 16 rows (queries | keys) and meets tiles of 16 rows of the other side, two at
// a time, out of a ring of two 8 KB stages; one TMA copy brings a tile of two tensors (K and V | Q and dO).
// Fragments are loaded ahead of the products that use them.  Softmax scale: applied once, to the accumulators.
// Bound: latency that twelve warps per SM (registers, rings) do not cover, between shared memory (79 % busy: a tile is written once and
// read as three | four 2 KB fragment sets, 10 | 12 KB of traffic per 4 KB gathered, at 128 bytes per cycle) and mma.sync (57 %: 24 |
// 32 of 8 cycles per tile and sub-partition); busy at 100 views, top-32.  In the dQ kernel the
// second tile's loads run under the first tile's exponentials (919 -> 638 us at 64 views, H = 16, top-32); the same
// order in the dK/dV kernel needs more registers than it gains: with the tiles one after the other 1161 -> 937 us, with
// eight or nine warps and the tiles overlapped 1110 us.
// Packed pairs in the exponentials' arithmetic, an elected thread that asks for copies and a wait whose usual outcome is one vote:
// both parts 1650 -> 1621 us at 64 views, 6350 -> 6255 at 250.  What an iteration asks for next - tokens of its copies, statistics -
// is found at its start and nothing waits there for a load: 1621 -> 1596 and 6255 -> 6160.  Turning fragments in registers (movmatrix)
// instead of reading them a second time: dQ the same (1627), dK/dV slower (1697).
constexpr int kSbStageBytes = 8192;
constexpr int kSbSmem = 2 * kSbStageBytes + 1024;

// sum over the windows that contain rows row0..row0+15, this lane's columns (8 dt + 2c, +1)
__device__ __forceinline__ void add_pooled(float (&acc)[8][4], const __nv_bfloat16* g_c, int bh, int row0, int kernel,
                                           int stride, int windows, int c) {
  if (g_c == nullptr) return;
  const int hi = min(windows - 1, row0 / stride), lo = row0 + 16 <= kernel ? 0 : (row0 + 16 - kernel + stride - 1) / stride;
  const float inv = 1.0f / static_cast<float>(kernel);
  for (int j = lo; j <= hi; ++j) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(g_c + (static_cast<int64_t>(bh) * windows + j) * 64) + c;
#pragma unroll
    for (int dt = 0; dt < 8; ++dt) {
      const uint32_t w = __ldg(src + dt * 4);
      const float a = bf16_lo(w) * inv, b = bf16_hi(w) * inv;
      acc[dt][0] += a; acc[dt][1] += b; acc[dt][2] += a; acc[dt][3] += b;
    }
  }
}
// 16 x 64 accumulators -> bf16 rows of 128 bytes, through 2 KB of shared memory of this warp
__device__ __forceinline__ void store_rows16(const float (&acc)[8][4], uint32_t tile, uint8_t* dst, int nrows, int lane) {
  const int g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int dt = 0; dt < 8; ++dt) {
    sts32(tile + swz128(g, dt) + 4 * c, pack_bf16(acc[dt][0], acc[dt][1]));
    sts32(tile + swz128(g + 8, dt) + 4 * c, pack_bf16(acc[dt][2], acc[dt][3]));
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = (lane >> 3) + 4 * i;
    if (r < nrows) *reinterpret_cast<uint4*>(dst + r * 128 + (lane & 7) * 16) = lds128(tile + swz128(r, lane & 7));
  }
  __syncwarp();
}
// A-operand fragments of 16 rows straight from global memory (rows of 128 bytes; rows >= nrows repeat the last)
__device__ __forceinline__ void ldg_a_frags(uint32_t (&f)[4][4], const __nv_bfloat16* rows, int nrows, int lane) {
  const int g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(rows) + min(g + 8 * r, nrows - 1) * 32 + c;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      f[ks][r] = __ldg(src + ks * 8);
      f[ks][r + 2] = __ldg(src + ks * 8 + 4);
    }
  }
}
// B-operand fragments of a swizzled 16-row tile: rows as n (off_n) or, transposed, rows as k (off_k)
__device__ __forceinline__ void frags_n(uint32_t (&f)[4][4], uint32_t tile, const uint32_t (&off)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) ldsm_x4(f[i][0], f[i][1], f[i][2], f[i][3], tile + off[i]);
}
__device__ __forceinline__ void frags_k(uint32_t (&f)[4][4], uint32_t tile, const uint32_t (&off)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) ldsm_x4_t(f[i][0], f[i][1], f[i][2], f[i][3], tile + off[i]);
}
// x = X Y^T, y = Z W^T for 16 x 16 tiles over 64 channels: four independent chains of four
__device__ __forceinline__ void two_products(float (&x)[2][4], float (&y)[2][4], const uint32_t (&xa)[4][4],
                                             const uint32_t (&xb)[4][4], const uint32_t (&ya)[4][4], const uint32_t (&yb)[4][4]) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (ks == 0) {
        mma_bf16_z(x[t], xa[ks], xb[ks][2 * t], xb[ks][2 * t + 1]);
        mma_bf16_z(y[t], ya[ks], yb[ks][2 * t], yb[ks][2 * t + 1]);
      } else {
        mma_bf16(x[t], xa[ks], xb[ks][2 * t], xb[ks][2 * t + 1]);
        mma_bf16(y[t], ya[ks], yb[ks][2 * t], yb[ks][2 * t + 1]);
      }
    }
}
__device__ __forceinline__ void accumulate(float (&acc)[8][4], const uint32_t (&a)[4], const uint32_t (&b)[4][4]) {
#pragma unroll
  for (int dp = 0; dp < 4; ++dp) {
    mma_bf16(acc[2 * dp], a, b[dp][0], b[dp][1]);
    mma_bf16(acc[2 * dp + 1], a, b[dp][2], b[dp][3]);
  }
}
struct SbLane {                    // this lane's ldmatrix offsets inside a swizzled tile
  uint32_t off_n[4], off_k[4];
  __device__ __forceinline__ explicit SbLane(int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      off_n[i] = swz128((lane & 7) + (lane >> 4) * 8, 2 * i + ((lane >> 3) & 1));
      off_k[i] = swz128((lane & 7) + ((lane >> 3) & 1) * 8, 2 * i + (lane >> 4));
    }
  }
};

struct SbShared {
  uint4 handed;                  // the next task (cluster launch control)
  uint64_t full[2], handed_bar;
  float stats[2][32];            // dK/dV: [tile of the pair][lse2 x 16 | delta x 16]
  int32_t next_off[2];           // dK/dV: ends and first entries of the next task's list
  int32_t list[64];              // those entries; dQ: first token of each valid key block, table order
  uint32_t abort_word;
};

// dQ of 16 rows.  `taken` pairs have gone through the ring before: a pair is its n-th, stage n & 1, phase (n >> 1) & 1.
template <bool APART>
__device__ __forceinline__ void sel_bwd_dq(const PairMap& map_kv, const SelBwdParams& p, SbShared& sh, uint32_t ring,
                                           uint32_t task, uint32_t taken) {
  const int lane = threadIdx.x, g = lane >> 2, c = lane & 3;
  const uint32_t nslices = (p.Tq + 15) / 16;
  const int bh = static_cast<int>(task / nslices), row0 = static_cast<int>(task - static_cast<uint32_t>(bh) * nslices) * 16;
  const int nrows = min(16, p.Tq - row0);
  volatile uint32_t* abort_flag = &sh.abort_word;
  int32_t* list = sh.list;
  int nvalid = 0;
  {
    const int32_t* row = p.idx + (static_cast<int64_t>(bh) * p.nqb + (row0 >> (4 + p.block_shift))) * p.topk;
    for (int r0 = 0; r0 < p.topk; r0 += 32) {
      const int i = r0 + lane;
      const int n = (i < p.topk) ? row[i] : -1;
      const bool ok = (n >= 0) && (static_cast<int64_t>(n) * p.block < p.Tk);
      const uint32_t bal = __ballot_sync(0xffffffffu, ok);
      if (ok) list[nvalid + __popc(bal & ((1u << lane) - 1u))] = n * p.block;
      nvalid += __popc(bal);
    }
    __syncwarp();
  }
  const int ntiles = nvalid << p.block_shift, npairs = (ntiles + 1) >> 1, in_block = (1 << p.block_shift) - 1;
  auto tok_of = [&](int t) { return list[t >> p.block_shift] + ((t & in_block) << 4); };
  const bool leader = elect_one_sync();
  auto issue = [&](int t0, int t1, bool two, int s) {
    if (leader) {
      mbar_expect_tx(&sh.full[s], (two ? 8192u : 4096u) >> (map_kv.b_first < 0));
      tma_load_pair<APART>(ring + s * kSbStageBytes, map_kv, &sh.full[s], t0, bh, 0);
      if (two) tma_load_pair<APART>(ring + s * kSbStageBytes + 4096, map_kv, &sh.full[s], t1, bh, 0);
    }
  };
  if (npairs > 0) issue(tok_of(0), tok_of(min(1, ntiles - 1)), 1 < ntiles, taken & 1);
  if (npairs > 1) issue(tok_of(2), tok_of(min(3, ntiles - 1)), 3 < ntiles, (taken + 1) & 1);

  uint32_t qf[4][4], dof[4][4];
  ldg_a_frags(qf, p.q + (static_cast<int64_t>(bh) * p.Tq + row0) * 64, nrows, lane);
  ldg_a_frags(dof, p.d_o + (static_cast<int64_t>(bh) * p.Tq + row0) * 64, nrows, lane);
  float neg_lse2[2], neg_delta[2];
  const float2 cs2 = make_float2(p.cs, p.cs);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t t = static_cast<int64_t>(bh) * p.Tq + row0 + min(g + 8 * r, nrows - 1);
    neg_lse2[r] = p.lse[t] * -1.4426950408889634f;         // finite wherever the list is not empty
    neg_delta[r] = -p.delta[t];
  }
  const SbLane of(lane);
  const uint32_t k_at = map_kv.b_first > 0 ? 2048u : 0u, v_at = map_kv.b_first == 0 ? 2048u : 0u;
  const bool ragged = (p.Tk & 15) != 0 || (p.Tk & (p.block - 1)) != 0;

  float dq[8][4] = {};
#pragma unroll 1
  for (int it = 0; it < npairs; ++it, ++taken) {
    const int S = taken & 1;
    if (!__all_sync(0xffffffffu, mbar_try_wait(&sh.full[S], (taken >> 1) & 1)) && !mbar_wait_warp(&sh.full[S], (taken >> 1) & 1, abort_flag)) {
      volatile uint32_t dummy = 0;                    // a last bounded chance for the other stage's copies to land
      if (it + 1 < npairs) mbar_wait(&sh.full[S ^ 1], ((taken + 1) >> 1) & 1, &dummy);
      if (lane == 0) atomicOr(p.status, kStatusWaitTimeout);
      return;
    }
    const uint32_t st = ring + S * kSbStageBytes;
    const bool both = 2 * it + 1 < ntiles;
    uint32_t kn0[4][4], kn1[4][4], vn0[4][4], vn1[4][4], kk0[4][4], kk1[4][4];
    float s0[2][4], dp0[2][4], s1[2][4], dp1[2][4];
    auto grad = [&](float (&s)[2][4], const float (&dp)[2][4], int t, uint32_t (&a)[4]) {
      const int left = ragged ? p.Tk - tok_of(t) : 16;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float2 pr = ffma2(make_float2(s[nt][2 * r], s[nt][2 * r + 1]), cs2, make_float2(neg_lse2[r], neg_lse2[r]));
          pr.x = fast_exp2(pr.x);
          pr.y = fast_exp2(pr.y);
          if (ragged && nt * 8 + 2 * c >= left) pr.x = 0.f;
          if (ragged && nt * 8 + 2 * c + 1 >= left) pr.y = 0.f;
          const float2 ds = fmul2(pr, fadd2(make_float2(dp[nt][2 * r], dp[nt][2 * r + 1]), make_float2(neg_delta[r], neg_delta[r])));
          s[nt][2 * r] = ds.x;
          s[nt][2 * r + 1] = ds.y;
        }
      a[0] = pack_bf16(s[0][0], s[0][1]); a[1] = pack_bf16(s[0][2], s[0][3]);
      a[2] = pack_bf16(s[1][0], s[1][1]); a[3] = pack_bf16(s[1][2], s[1][3]);
    };
    uint32_t a0[4], a1[4];
    frags_n(kn0, st + k_at, of.off_n);
    frags_n(vn0, st + v_at, of.off_n);
    two_products(s0, dp0, qf, kn0, dof, vn0);
    frags_k(kk0, st + k_at, of.off_k);
    const int t0 = tok_of(min(2 * it + 4, ntiles - 1)), t1 = tok_of(min(2 * it + 5, ntiles - 1));      // of the copies asked for below
    if (both) {
      frags_n(kn1, st + 4096 + k_at, of.off_n);
      frags_n(vn1, st + 4096 + v_at, of.off_n);
      grad(s0, dp0, 2 * it, a0);
      two_products(s1, dp1, qf, kn1, dof, vn1);
      accumulate(dq, a0, kk0);
      frags_k(kk1, st + 4096 + k_at, of.off_k);
      grad(s1, dp1, 2 * it + 1, a1);
      accumulate(dq, a1, kk1);
    } else {
      grad(s0, dp0, 2 * it, a0);
      accumulate(dq, a0, kk0);
    }
    __syncwarp();
    if (it + 2 < npairs) issue(t0, t1, 2 * it + 5 < ntiles, S);            // every fragment of the stage has been consumed
  }
#pragma unroll
  for (int dt = 0; dt < 8; ++dt)
#pragma unroll
    for (int e = 0; e < 4; ++e) dq[dt][e] *= p.scale;
  add_pooled(dq, p.dq_c, bh, row0, p.q_kernel, p.q_stride, p.q_windows, c);
  __syncwarp();
  store_rows16(dq, ring, reinterpret_cast<uint8_t*>(p.dq + (static_cast<int64_t>(bh) * p.Tq + row0) * 64), nrows, lane);
}

// The list of query blocks that selected this warp's key block comes 32 entries at a time into a register per
// lane, the statistics of a tile's rows one load ahead of their use.
// A warp that has finished its rows takes over the rows of a CTA that has not started (cluster launch control) and has asked
// for them, their list and their first copies before it is done with its own: lists differ in length by a factor of
// five, and CTAs that came and went left a fifth of the warps' places empty (9.6 of 12 per SM).
// Tasks: first all of dK/dV, then all of dQ, whose lists are of one length; a warp that is handed one of those is done after it.
// (As two kernels the second could not start before the longest lists of the first had been worked off.)
template <bool APART>
__global__ void __launch_bounds__(32, 10) sel_bwd_kernel(const __grid_constant__ PairMap map_qdo,
                                                         const __grid_constant__ PairMap map_kv, const SelBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(16) SbShared sh;
  const int lane = threadIdx.x, c = lane & 3;
  const uint32_t nslices = (p.Tk + 15) / 16, kv_tasks = nslices * static_cast<uint32_t>(p.B * p.H);
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  volatile uint32_t* abort_flag = &sh.abort_word;
  if (lane == 0) {
    sh.abort_word = 0;
    mbar_init(&sh.full[0], 1);
    mbar_init(&sh.full[1], 1);
    mbar_init(&sh.handed_bar, 1);
    mbar_fence_init();
  }
  griddep_wait();
  griddep_launch();
  __syncwarp();
  if (blockIdx.x >= kv_tasks) {
    sel_bwd_dq<APART>(map_kv, p, sh, ring, blockIdx.x - kv_tasks, 0);
    return;
  }
  const int in_block = (1 << p.block_shift) - 1;
  const SbLane of(lane);
  const uint32_t q_at = map_qdo.b_first > 0 ? 2048u : 0u, do_at = map_qdo.b_first == 0 ? 2048u : 0u;

  int bh, row0, cnt, ntiles, npairs;
  const int32_t* ql;
  // list entries of chunk c (32 of them) live in `q_cur`, those of chunk c+1 in `q_nxt`; called with growing t only
  int q_chunk, q_cur, q_nxt;
  auto tok_of = [&](int t) {
    const int e = t >> p.block_shift;
    if ((e >> 5) != q_chunk) {                         // warp-uniform
      q_chunk = e >> 5;
      q_cur = q_nxt;
      const int j = (q_chunk + 1) * 32 + lane;
      q_nxt = (j < cnt) ? ql[j] : 0;
    }
    return (__shfl_sync(0xffffffffu, q_cur, e & 31) << (4 + p.block_shift)) + ((t & in_block) << 4);
  };
  const bool leader = elect_one_sync();
  auto issue = [&](int t0, int t1, bool both, int s) {
    if (leader) {
      mbar_expect_tx(&sh.full[s], (both ? 8192u : 4096u) >> (map_qdo.b_first < 0));
      tma_load_pair<APART>(ring + s * kSbStageBytes, map_qdo, &sh.full[s], t0, bh, 0);
      if (both) tma_load_pair<APART>(ring + s * kSbStageBytes + 4096, map_qdo, &sh.full[s], t1, bh, 0);
    }
  };
  // lanes 0-15 fetch lse, lanes 16-31 delta of a tile's rows, as they are: nothing here waits for the load
  auto stat = [&](int tok0) {
    return __ldg((lane < 16 ? p.lse : p.delta) + static_cast<int64_t>(bh) * p.Tq + min(tok0 + (lane & 15), p.Tq - 1));
  };
  // -lse2 and -delta; a row past the end gets lse = +inf: P is exactly 0
  const float stat_scale = lane < 16 ? -1.4426950408889634f : -1.f;
  auto stat_value = [&](float x, int tok0) { return lane < 16 && tok0 + lane >= p.Tq ? -INFINITY : x * stat_scale; };
  auto offsets_of = [&](uint32_t task) {
    const uint32_t h = task / nslices, slice = task - h * nslices;
    return p.offsets + static_cast<int64_t>(h) * (p.nkb + 1) + (slice >> p.block_shift);
  };
  // a pair is the ring's n-th: stage n & 1, phase (n >> 1) & 1
  uint32_t taken = 0;
  int na = 0, nb = 0;                                  // tokens of the next pair to be computed (its copies are under way)
  float sa = 0.f, sb = 0.f;                            // and its statistics
  uint32_t kf[4][4], vf[4][4];
  // the task's sizes, first copies and fragments; its list's first entries are in q_cur and q_nxt
  auto begin = [&](uint32_t task, int beg, int count) {
    bh = static_cast<int>(task / nslices);
    row0 = static_cast<int>(task - static_cast<uint32_t>(bh) * nslices) * 16;
    cnt = count;
    ql = p.qids + static_cast<int64_t>(bh) * p.nqb * p.topk + beg;
    q_chunk = 0;
    ntiles = cnt << p.block_shift;
    npairs = (ntiles + 1) >> 1;
    if (npairs > 0) {
      na = tok_of(0);
      nb = 1 < ntiles ? tok_of(1) : na;
      issue(na, nb, 1 < ntiles, taken & 1);
      sa = stat(na);
      sb = stat(nb);
    }
    const int64_t at = (static_cast<int64_t>(bh) * p.Tk + row0) * 64;
    const int nrows = min(16, p.Tk - row0);
    ldg_a_frags(kf, p.k + at, nrows, lane);
    ldg_a_frags(vf, p.v + at, nrows, lane);
  };
  {
    const int32_t* off = offsets_of(blockIdx.x);
    const int beg = off[0], count = off[1] - beg;
    const int32_t* src = p.qids + static_cast<int64_t>(blockIdx.x / nslices) * p.nqb * p.topk + beg;
    q_cur = (lane < count) ? src[lane] : 0;
    q_nxt = (32 + lane < count) ? src[32 + lane] : 0;
    begin(blockIdx.x, beg, count);
  }
  uint32_t asked = 0, answered = 0;                    // requests and answers so far
#pragma unroll 1
  while (true) {
    auto request = [&]() {
      if (lane == 0) clc_request(&sh.handed, &sh.handed_bar);
      ++asked;
    };
    if (npairs <= 3) request();
    int ta = 0, tb = 0;
    if (npairs > 1) {
      ta = tok_of(2);
      tb = 3 < ntiles ? tok_of(3) : ta;
      issue(ta, tb, 3 < ntiles, (taken + 1) & 1);
    }
    int next = -1;
    bool ok = true;
    // the next task, if there is one, and the ends of its list
    auto learn = [&]() {
      ok = mbar_wait_warp(&sh.handed_bar, answered++ & 1, abort_flag);
      next = ok ? clc_answer(&sh.handed) : -1;
      if (static_cast<uint32_t>(next) < kv_tasks && lane < 2) cp_async4(smem_u32(&sh.next_off[lane]), offsets_of(next) + lane);
      cp_async_commit();
    };
    // a pair later: the first entries of its list
    auto look = [&]() {
      cp_async_wait<0>();
      __syncwarp();
      if (static_cast<uint32_t>(next) >= kv_tasks) return;          // none, or dQ
      const int beg = sh.next_off[0], count = sh.next_off[1] - beg;
      const int32_t* src = p.qids + static_cast<int64_t>(static_cast<uint32_t>(next) / nslices) * p.nqb * p.topk + beg;
      if (lane < count) cp_async4(smem_u32(&sh.list[lane]), src + lane);
      if (32 + lane < count) cp_async4(smem_u32(&sh.list[32 + lane]), src + 32 + lane);
      cp_async_commit();
    };
    float dk[8][4] = {}, dv[8][4] = {};
#pragma unroll 1
    for (int it = 0; it < npairs; ++it, ++taken) {
      const int S = taken & 1;
      sh.stats[0][lane] = stat_value(sa, na);
      sh.stats[1][lane] = stat_value(sb, nb);
      __syncwarp();
      if (it + 1 < npairs) { sa = stat(ta); sb = stat(tb); na = ta; nb = tb; }
      ok = ok && (__all_sync(0xffffffffu, mbar_try_wait(&sh.full[S], (taken >> 1) & 1)) || mbar_wait_warp(&sh.full[S], (taken >> 1) & 1, abort_flag));
      if (!ok) {
        volatile uint32_t dummy = 0;                    // a last bounded chance for what is under way to land
        if (it + 1 < npairs) mbar_wait(&sh.full[S ^ 1], ((taken + 1) >> 1) & 1, &dummy);
        if (asked != answered) mbar_wait(&sh.handed_bar, answered & 1, &dummy);
        if (lane == 0) atomicOr(p.status, kStatusWaitTimeout);
        return;
      }
      const uint32_t st = ring + S * kSbStageBytes;
      // P^T and dS^T of a tile, packed as A operands
      auto grad = [&](const float (&s)[2][4], const float (&dp)[2][4], int j, uint32_t (&pa)[4], uint32_t (&da)[4]) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float2 l2 = *reinterpret_cast<const float2*>(&sh.stats[j][nt * 8 + 2 * c]);
          const float2 d2 = *reinterpret_cast<const float2*>(&sh.stats[j][16 + nt * 8 + 2 * c]);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float2 pr = ffma2(make_float2(s[nt][2 * r], s[nt][2 * r + 1]), make_float2(p.cs, p.cs), l2);
            pr.x = fast_exp2(pr.x);
            pr.y = fast_exp2(pr.y);
            const float2 ds = fmul2(pr, fadd2(make_float2(dp[nt][2 * r], dp[nt][2 * r + 1]), d2));
            pa[2 * nt + r] = pack_bf16(pr.x, pr.y);
            da[2 * nt + r] = pack_bf16(ds.x, ds.y);
          }
        }
      };
      auto tile = [&](int j) {
        uint32_t qn[4][4], dn[4][4], qk[4][4], dkk[4][4], pa[4], da[4];
        float s[2][4], dp[2][4];
        frags_n(qn, st + j * 4096 + q_at, of.off_n);
        frags_n(dn, st + j * 4096 + do_at, of.off_n);
        two_products(s, dp, kf, qn, vf, dn);
        frags_k(dkk, st + j * 4096 + do_at, of.off_k);
        frags_k(qk, st + j * 4096 + q_at, of.off_k);
        grad(s, dp, j, pa, da);
        accumulate(dv, pa, dkk);
        accumulate(dk, da, qk);
      };
      if (it + 2 < npairs) {                            // found here, where nothing waits for them
        ta = tok_of(2 * it + 4);
        tb = 2 * it + 5 < ntiles ? tok_of(2 * it + 5) : ta;
      }
      tile(0);
      if (2 * it + 1 < ntiles) tile(1);
      __syncwarp();
      if (it + 2 < npairs) issue(ta, tb, 2 * it + 5 < ntiles, S);        // every fragment of the stage has been consumed
      // a request takes a task from those who could start it now, so it is made no sooner than its answer is needed
      const int left = npairs - 1 - it;
      if (left == 3) request();
      else if (left == 2) learn();
      else if (left == 1 && it > 0) look();
    }
    if (npairs < 3) {
      learn();
      look();
    }
    if (!ok) {
      if (lane == 0) atomicOr(p.status, kStatusWaitTimeout);
      return;
    }
    const int bh_done = bh, row_done = row0;
    cp_async_wait<0>();
    __syncwarp();
    if (static_cast<uint32_t>(next) < kv_tasks) {
      q_cur = sh.list[lane];
      q_nxt = sh.list[32 + lane];
      begin(next, sh.next_off[0], sh.next_off[1] - sh.next_off[0]);
      __syncwarp();
    }
#pragma unroll
    for (int dt = 0; dt < 8; ++dt)
#pragma unroll
      for (int e = 0; e < 4; ++e) dk[dt][e] *= p.scale;
    add_pooled(dk, p.dk_c, bh_done, row_done, p.k_kernel, p.k_stride, p.k_windows, c);
    add_pooled(dv, p.dv_c, bh_done, row_done, p.k_kernel, p.k_stride, p.k_windows, c);
    const int64_t at = (static_cast<int64_t>(bh_done) * p.Tk + row_done) * 64;
    const int nrows = min(16, p.Tk - row_done);
    const uint32_t tile = ring + ((taken + 1) & 1) * kSbStageBytes;       // the next task's first pair is in the other stage
    store_rows16(dk, tile, reinterpret_cast<uint8_t*>(p.dk + at), nrows, lane);
    store_rows16(dv, tile, reinterpret_cast<uint8_t*>(p.dv + at), nrows, lane);
    if (next < 0) return;
    fence_proxy_async_smem();                           // copies and the next answer come after these reads and writes
    __syncwarp();
    if (static_cast<uint32_t>(next) >= kv_tasks) {
      sel_bwd_dq<APART>(map_kv, p, sh, ring, static_cast<uint32_t>(next) - kv_tasks, taken);
      return;
    }
  }
}

static int grid_for(int64_t threads, int block) {
  int64_t b = (threads + block - 1) / block;
  const int64_t cap = static_cast<int64_t>(sm_count()) * 32;
  if (b > cap) b = cap;
  return static_cast<int>(b < 1 ? 1 : b);
}

}  // namespace s3r

using namespace s3r;

extern "C" size_t s3r_csr_workspace_bytes(int B, int H, int Nq, int topk, int Nkb) {
  if (B <= 0 || H <= 0 || Nq <= 0 || topk <= 0 || Nkb <= 0) return 0;
  const size_t bh = static_cast<size_t>(B) * H;
  size_t cursor = (bh * Nkb * sizeof(int32_t) + 255) & ~static_cast<size_t>(255);
  size_t tmp = (bh * Nq * topk * sizeof(int32_t) + 255) & ~static_cast<size_t>(255);
  // queue of the segments that one warp does not sort: at most one per non-empty segment, plus its counter
  size_t queue = ((bh * (Nq > (1 << 25) ? static_cast<size_t>(Nkb) : static_cast<size_t>(Nq) * topk / (kCsrWarpSort + 1)) + 2) * sizeof(int32_t) + 255) & ~static_cast<size_t>(255);
  return cursor + tmp + queue;
}

extern "C" int s3r_build_key_csr(const int32_t* idx, int32_t* offsets, int32_t* qids, int B, int H, int Nq, int topk,
                                 int Nkb, void* workspace, size_t workspace_bytes, void* stream) {
  S3R_REQUIRE(idx && offsets && qids && workspace, S3R_ERR_NULL, "s3r_build_key_csr: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && Nq > 0 && topk > 0 && Nkb > 0, S3R_ERR_SHAPE, "s3r_build_key_csr: bad sizes");
  S3R_REQUIRE(workspace_bytes >= s3r_csr_workspace_bytes(B, H, Nq, topk, Nkb), S3R_ERR_TOO_LARGE,
              "s3r_build_key_csr: workspace of %zu bytes is smaller than the %zu needed", workspace_bytes,
              s3r_csr_workspace_bytes(B, H, Nq, topk, Nkb));
  S3R_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, S3R_ERR_ALIGNMENT,
              "s3r_build_key_csr: workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t bh = static_cast<int64_t>(B) * H;
  const int64_t per_bh = static_cast<int64_t>(Nq) * topk, total = bh * per_bh;
  int32_t* cursor = static_cast<int32_t*>(workspace);
  int32_t* tmp = reinterpret_cast<int32_t*>(static_cast<uint8_t*>(workspace) +
                                            ((bh * Nkb * sizeof(int32_t) + 255) & ~static_cast<size_t>(255)));
  const int64_t nseg = bh * Nkb;
  S3R_REQUIRE(nseg < (1ll << 31) && total < (1ll << 40), S3R_ERR_TOO_LARGE, "s3r_build_key_csr: table too large");
  if (per_bh <= kCsrOneEntries && Nkb <= kCsrOneKeys) {
    const int smem = (Nkb + static_cast<int>(per_bh)) * static_cast<int>(sizeof(int32_t));
    S3R_CUDA(cudaFuncSetAttribute(csr_one_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (kCsrOneEntries + kCsrOneKeys) * static_cast<int>(sizeof(int32_t))));
    const int64_t parts = bh < sm_count() ? sm_count() / bh : 1;
    return launch(csr_one_kernel, dim3(static_cast<unsigned>(bh), static_cast<unsigned>(parts < 8 ? parts : 8)), 1024, smem, st, idx, offsets, qids, static_cast<int>(per_bh), Nkb, topk);
  }
  int32_t* queue = reinterpret_cast<int32_t*>(reinterpret_cast<uint8_t*>(tmp) +
                                              ((bh * Nq * topk * sizeof(int32_t) + 255) & ~static_cast<size_t>(255)));
  S3R_CUDA(cudaMemsetAsync(offsets, 0, bh * (Nkb + 1) * sizeof(int32_t), st));
  S3R_CUDA(cudaMemsetAsync(queue, 0, sizeof(int32_t), st));
  // a query block and its position in the segment share a 32-bit sort key
  const int warp_max = Nq <= (1 << 25) ? kCsrWarpSort : 0;
  csr_count_kernel<<<grid_for(total, 256), 256, 0, st>>>(idx, offsets, per_bh, total, Nkb);
  csr_scan_kernel<<<static_cast<unsigned>(bh), 1024, 0, st>>>(offsets, cursor, Nkb);
  csr_fill_kernel<<<grid_for(total, 256), 256, 0, st>>>(idx, cursor, tmp, per_bh, total, Nkb, topk);
  csr_sort_small_kernel<<<static_cast<unsigned>((nseg * 32 + 255) / 256), 256, 0, st>>>(offsets, tmp, qids, per_bh, Nkb,
                                                                                        nseg, warp_max, queue);
  csr_sort_long_kernel<<<sm_count() * 4, 256, 0, st>>>(idx, offsets, tmp, qids, per_bh, Nkb, topk, queue);
  S3R_CUDA(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------------------------------------------
// The same index build for callers that cannot allocate device memory.
//
// Some hosts of this library have no allocator to ask: a plug-in running inside another runtime
// that handed out all device memory at start-up, or a latency-critical loop in which a
// cudaMalloc (which synchronises the device) is not acceptable.  For them the scratch of the
// index build lives in the library image itself: a fixed array that every GPU that loads the
// library keeps until the process exits.  Sizes whose scratch does not fit are refused.
//
// In host code the array's name is only a stand-in; its device address is obtained once per
// device with cudaGetSymbolAddress (with that device current) and handed to the kernels.
// ------------------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_csr_static_scratch[S3R_CSR_STATIC_SCRATCH_BYTES];

extern "C" int s3r_build_key_csr_static(const int32_t* idx, int32_t* offsets, int32_t* qids, int B, int H, int Nq,
                                        int topk, int Nkb, void* stream) {
  S3R_REQUIRE(idx && offsets && qids, S3R_ERR_NULL, "s3r_build_key_csr_static: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && Nq > 0 && topk > 0 && Nkb > 0, S3R_ERR_SHAPE, "s3r_build_key_csr_static: bad sizes");
  const size_t need = s3r_csr_workspace_bytes(B, H, Nq, topk, Nkb);
  S3R_REQUIRE(need <= static_cast<size_t>(S3R_CSR_STATIC_SCRATCH_BYTES), S3R_ERR_TOO_LARGE,
              "s3r_build_key_csr_static: this table needs %zu bytes of scratch, the built-in buffer holds %zu; "
              "use s3r_build_key_csr with a caller-provided workspace",
              need, static_cast<size_t>(S3R_CSR_STATIC_SCRATCH_BYTES));
  // set-up, once per device: resolve the device address of the built-in buffer
  static void* dev_ptr[64] = {};
  static std::mutex mu;
  int dev = -1;
  S3R_CUDA(cudaGetDevice(&dev));
  S3R_REQUIRE(dev >= 0 && dev < 64, S3R_ERR_UNSUPPORTED, "s3r_build_key_csr_static: device ordinal %d out of range", dev);
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!dev_ptr[dev]) {
      void* p = nullptr;
      S3R_CUDA(cudaGetSymbolAddress(&p, g_csr_static_scratch));
      dev_ptr[dev] = p;
    }
    scratch = dev_ptr[dev];
  }
  // What must start at zero (the counter of the long-segment queue) is cleared by the build itself; the scan
  // writes every cursor and the sorts only read slots the fill wrote, so nothing an earlier call left behind
  // is ever read.
  return s3r_build_key_csr(idx, offsets, qids, B, H, Nq, topk, Nkb, scratch, S3R_CSR_STATIC_SCRATCH_BYTES, stream);
}

extern "C" int s3r_delta(const void* o, const void* d_o, float* delta, int64_t rows, int d, void* stream) {
  S3R_REQUIRE(o && d_o && delta, S3R_ERR_NULL, "s3r_delta: NULL pointer");
  S3R_REQUIRE(rows > 0, S3R_ERR_SHAPE, "s3r_delta: rows must be positive");
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_delta: head_dim %d not supported (64 only)", d);
  S3R_REQUIRE(((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(d_o)) & 15) == 0, S3R_ERR_ALIGNMENT,
              "s3r_delta: tensors must be 16-byte aligned");
  const int64_t blocks = (rows * 8 + 255) / 256;
  return launch(delta_kernel, static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream),
                static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), delta, rows);
}

extern "C" int s3r_merge_bwd_deltas(const void* dy, const void* gate, int64_t gate_stride_b, int64_t gate_stride_h,
                                    int64_t gate_stride_t, const void* o_c, const void* o_s, void* do_s, float* dgate,
                                    void* do_c, float* delta_s, float* delta_c, int B, int H, int Tq, int d, int block,
                                    void* stream) {
  S3R_REQUIRE(dy && gate && o_c && o_s && do_s && dgate && do_c && delta_s, S3R_ERR_NULL, "s3r_merge_bwd: NULL pointer");
  S3R_REQUIRE(B > 0 && H > 0 && Tq > 0 && block > 0, S3R_ERR_SHAPE, "s3r_merge_bwd: bad sizes");
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_merge_bwd: head_dim %d not supported (64 only)", d);
  uintptr_t al = 0;
  for (const void* t : {dy, o_c, o_s, static_cast<const void*>(do_s), static_cast<const void*>(do_c)}) al |= reinterpret_cast<uintptr_t>(t);
  S3R_REQUIRE((al & 15) == 0 && (reinterpret_cast<uintptr_t>(dgate) & 7) == 0, S3R_ERR_ALIGNMENT,
              "s3r_merge_bwd: tensors must be 16-byte aligned, dgate 8-byte");
  S3R_REQUIRE((reinterpret_cast<uintptr_t>(gate) & 3) == 0 && gate_stride_b % 2 == 0 && gate_stride_h % 2 == 0 && gate_stride_t % 2 == 0,
              S3R_ERR_ALIGNMENT, "s3r_merge_bwd: gate pairs must be 4-byte aligned");
  MergeBwdParams p;
  p.dy = static_cast<const __nv_bfloat16*>(dy);
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.gsb = gate_stride_b; p.gsh = gate_stride_h; p.gst = gate_stride_t;
  p.o_c = static_cast<const __nv_bfloat16*>(o_c);
  p.o_s = static_cast<const __nv_bfloat16*>(o_s);
  p.do_s = static_cast<__nv_bfloat16*>(do_s);
  p.dgate = dgate;
  p.do_c = static_cast<__nv_bfloat16*>(do_c);
  p.delta_s = delta_s;
  p.delta_c = delta_c;
  p.B = B; p.H = H; p.Tq = Tq; p.block = block;
  p.nqb = (Tq + block - 1) / block;
  const int64_t warps = static_cast<int64_t>(B) * H * p.nqb;
  return launch(merge_bwd_whole_passes(block) ? merge_bwd_kernel<4> : merge_bwd_kernel<1>, static_cast<unsigned>((warps * 32 + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream), p);
}

extern "C" int s3r_merge_bwd(const void* dy, const void* gate, int64_t gate_stride_b, int64_t gate_stride_h,
                             int64_t gate_stride_t, const void* o_c, const void* o_s, void* do_s, float* dgate,
                             void* do_c, float* delta_s, int B, int H, int Tq, int d, int block, void* stream) {
  return s3r_merge_bwd_deltas(dy, gate, gate_stride_b, gate_stride_h, gate_stride_t, o_c, o_s, do_s, dgate, do_c, delta_s, nullptr,
                              B, H, Tq, d, block, stream);
}

static int launch_sel_bwd(SelBwdParams& p, int d, cudaStream_t st) {
  S3R_REQUIRE(p.q && p.k && p.v && p.idx && p.offsets && p.qids && p.lse && p.delta && p.d_o && p.dq && p.dk && p.dv, S3R_ERR_NULL,
              "s3r_sel_attn_bwd: NULL pointer");
  S3R_REQUIRE(p.B > 0 && p.H > 0 && p.Tq > 0 && p.Tk > 0 && p.topk > 0, S3R_ERR_SHAPE, "s3r_sel_attn_bwd: bad sizes");
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_sel_attn_bwd: head_dim %d not supported (64 only)", d);
  S3R_REQUIRE(p.block == 16 || p.block == 32 || p.block == 64, S3R_ERR_UNSUPPORTED,
              "s3r_sel_attn_bwd: block %d not supported (16, 32, 64)", p.block);
  S3R_REQUIRE(p.topk <= 64, S3R_ERR_UNSUPPORTED, "s3r_sel_attn_bwd: topk %d exceeds 64", p.topk);
  const uintptr_t al = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) |
                       reinterpret_cast<uintptr_t>(p.d_o) | reinterpret_cast<uintptr_t>(p.dq) |
                       reinterpret_cast<uintptr_t>(p.dk) | reinterpret_cast<uintptr_t>(p.dv);
  S3R_REQUIRE((al & 15) == 0, S3R_ERR_ALIGNMENT, "s3r_sel_attn_bwd: tensors must be 16-byte aligned");
  const uintptr_t al_c = reinterpret_cast<uintptr_t>(p.dq_c) | reinterpret_cast<uintptr_t>(p.dk_c) | reinterpret_cast<uintptr_t>(p.dv_c);
  S3R_REQUIRE((al_c & 3) == 0, S3R_ERR_ALIGNMENT, "s3r_sel_attn_bwd_pooled: gradients of the pooled branch must be 4-byte aligned");
  p.block_shift = p.block == 16 ? 0 : p.block == 32 ? 1 : 2;
  p.nqb = (p.Tq + p.block - 1) / p.block;
  p.nkb = (p.Tk + p.block - 1) / p.block;
  p.status = device_status_ptr();
  S3R_REQUIRE(p.status != nullptr, S3R_ERR_DRIVER, "s3r_sel_attn_bwd: could not resolve the device status word");
  const int64_t bh = static_cast<int64_t>(p.B) * p.H;
  if (p.block == 64 && sel_bwd64_pays(bh, p.nqb, p.nkb, p.topk)) return sel_bwd64(p, st);
  const int64_t tq = bh * ((p.Tq + 15) / 16), tk = bh * ((p.Tk + 15) / 16);
  S3R_REQUIRE(tq + tk < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_sel_attn_bwd: grid too large");
  PairMap mkv, mqdo;
  int rc = make_pair_map(&mkv, p.k, p.v, p.Tk, static_cast<int>(bh), 1, 0);
  if (rc) return rc;
  rc = make_pair_map(&mqdo, p.q, p.d_o, p.Tq, static_cast<int>(bh), 1, 0);
  if (rc) return rc;
  auto* kernel = mkv.apart || mqdo.apart ? sel_bwd_kernel<true> : sel_bwd_kernel<false>;
  S3R_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSbSmem));
  return launch(kernel, static_cast<unsigned>(tk + tq), 32, kSbSmem, st, mqdo, mkv, p);
}

extern "C" int s3r_sel_attn_bwd(const void* q, const void* k, const void* v, const int32_t* idx,
                                const int32_t* offsets, const int32_t* qids, const float* lse_s, const float* delta_s,
                                const void* do_s, void* dq, void* dk, void* dv, int B, int H, int Tq, int Tk, int d,
                                int block, int topk, float scale, void* stream) {
  return s3r_sel_attn_bwd_pooled(q, k, v, idx, offsets, qids, lse_s, delta_s, do_s, dq, dk, dv, nullptr, nullptr, nullptr, 16,
                                 16, 16, 16, B, H, Tq, Tk, d, block, topk, scale, stream);
}

extern "C" int s3r_sel_attn_bwd_pooled(const void* q, const void* k, const void* v, const int32_t* idx,
                                       const int32_t* offsets, const int32_t* qids, const float* lse_s,
                                       const float* delta_s, const void* do_s, void* dq, void* dk, void* dv,
                                       const void* dq_c, const void* dk_c, const void* dv_c, int q_kernel, int q_stride,
                                       int k_kernel, int k_stride, int B, int H, int Tq, int Tk, int d, int block, int topk,
                                       float scale, void* stream) {
  S3R_REQUIRE(q_kernel > 0 && q_stride > 0 && k_kernel > 0 && k_stride > 0, S3R_ERR_SHAPE, "s3r_sel_attn_bwd_pooled: bad pooling sizes");
  S3R_REQUIRE((q_kernel | q_stride | k_kernel | k_stride) % 16 == 0, S3R_ERR_UNSUPPORTED,
              "s3r_sel_attn_bwd_pooled: pooling kernels and strides must be multiples of 16");
  SelBwdParams p = {};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.d_o = static_cast<const __nv_bfloat16*>(do_s);
  p.idx = idx; p.offsets = offsets; p.qids = qids;
  p.lse = lse_s; p.delta = delta_s;
  p.dq = static_cast<__nv_bfloat16*>(dq);
  p.dk = static_cast<__nv_bfloat16*>(dk);
  p.dv = static_cast<__nv_bfloat16*>(dv);
  p.dq_c = static_cast<const __nv_bfloat16*>(dq_c);
  p.dk_c = static_cast<const __nv_bfloat16*>(dk_c);
  p.dv_c = static_cast<const __nv_bfloat16*>(dv_c);
  p.q_kernel = q_kernel; p.q_stride = q_stride; p.q_windows = Tq >= q_kernel ? (Tq - q_kernel) / q_stride + 1 : 0;
  p.k_kernel = k_kernel; p.k_stride = k_stride; p.k_windows = Tk >= k_kernel ? (Tk - k_kernel) / k_stride + 1 : 0;
  p.B = B; p.H = H; p.Tq = Tq; p.Tk = Tk; p.block = block; p.topk = topk;
  p.cs = scale * 1.4426950408889634f;
  p.scale = scale;
  return launch_sel_bwd(p, d, static_cast<cudaStream_t>(stream));
}
