// Prologue of the sparse global attention, one pass over the packed projection: everything the reference
// does between `qkv = self.qkv(x)` and its two attention calls
// (pi3/models/layers/sparse_attention.py:95-123): split into q, k, v in [B,H,N,d], per-head LayerNorm of q
// and k, 2-D rotary embedding at the token positions, and for the compression branch the block means of
// the RAW q, k, v followed by the same LayerNorm and the rotary embedding at the block's mean position.
// In PyTorch that is about fifteen elementwise passes over [B,H,N,d]; here the projection is read once
// (6 KB per token, contiguous) and each output written once, so the kernel is bounded by HBM:
// 2 * 3*N*H*d*2 bytes plus the pooled tensors.
//
// A CTA works on one block of `block` tokens of one batch element; eight lanes own one (q|k|v, head) row
// of 64 channels (16 bytes per lane) and walk the block's tokens, so a block's mean never leaves
// registers.  Rounding points follow the reference under bf16 autocast: LayerNorm in fp32 from bf16
// input, rounded to bf16; the rotary products and their sum each rounded to bf16; the block mean
// accumulated in fp32 and rounded once.  cos/sin come from the caller's table (angles rounded to bf16
// before cos/sin, pi3/models/layers/pos_embed.py:112-159), so they are bit-identical to the reference's.
#include "common.cuh"

namespace s3r {

struct PrologueParams {
  const __nv_bfloat16* qkv;          // [B,N,(3,H,64)], tokens tok_stride elements apart
  int64_t tok_stride;
  const __nv_bfloat16* gate_in;      // logits (h,2) of a token, tokens tok_stride apart; null: none
  uint32_t* gate;                    // [B,H,N] pairs: their sigmoid
  const int64_t* pos;                // [B,N,2] (y,x) or null: no rotary embedding
  const __nv_bfloat16* cos_tab;      // [tab_rows,32]
  const __nv_bfloat16* sin_tab;
  int tab_rows;
  const float* qw; const float* qb;  // LayerNorm affine of q (null: no normalisation)
  const float* kw; const float* kb;
  float eps;
  __nv_bfloat16 *q, *k, *v, *q_c, *k_c, *v_c;
  int B, H, N, Nc, block;
  uint32_t* status;                  // device status word: a position outside the tables sets kStatusBadIndex
};

struct alignas(16) Vec8 {
  uint32_t w[4];
};

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float sum8(float x, uint32_t gmask) {
  x += __shfl_xor_sync(gmask, x, 1);
  x += __shfl_xor_sync(gmask, x, 2);
  return x + __shfl_xor_sync(gmask, x, 4);
}
__device__ __forceinline__ float2 splat(float x) { return make_float2(x, x); }
__device__ __forceinline__ void unpack8(float2 (&x)[4], const Vec8& v) {
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = make_float2(bf16_lo(v.w[i]), bf16_hi(v.w[i]));
}
__device__ __forceinline__ Vec8 pack8(const float2 (&x)[4]) {
  Vec8 v;
#pragma unroll
  for (int i = 0; i < 4; ++i) v.w[i] = pack_bf16(x[i].x, x[i].y);
  return v;
}
__device__ __forceinline__ Vec8 ldg_vec8(const __nv_bfloat16* p) {
  const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
  return Vec8{{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ int table_row(int64_t pv, int tab_rows) {
  return static_cast<int>(min(max(pv, static_cast<int64_t>(0)), static_cast<int64_t>(tab_rows - 1)));
}
// Rows of the rotary tables for a block's mean position and, behind it, for its tokens: (y, x) pairs in this warp's shared
// memory, clamped and checked once per warp instead of once per (q|k, head) row of every token.  LONG: a block whose rows do
// not fit there; its tokens' rows are found where they are used.
template <bool LONG>
__device__ __forceinline__ void block_rows(int* r, const int64_t* pos, int block, int tab_rows, uint32_t* status, int lane) {
  bool bad = false;
  auto put = [&](int i, int64_t pv) {
    const int row = table_row(pv, tab_rows);
    bad |= pv != row;
    if (!LONG || i < 2) r[i] = row;
  };
  float sum = 0.f;                                    // of the coordinate lane % 2: whole numbers, any order is exact
  for (int i = lane; i < 2 * block; i += 32) {
    const int64_t pv = __ldg(pos + i);
    put(2 + i, pv);
    sum += static_cast<float>(pv);
  }
#pragma unroll
  for (int d = 2; d < 32; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  // float mean, truncated: xpos.view(..).float().mean(dim=2).int()
  if (lane < 2) put(lane, static_cast<int64_t>(static_cast<int>(sum / static_cast<float>(block))));
  if (bad && status) atomicOr(status, kStatusBadIndex);     // clamped: the result for this token is wrong
  __syncwarp();
}
__device__ __forceinline__ Vec8 lds_vec8(uint32_t a) {
  const uint4 v = lds128(a);
  return Vec8{{v.x, v.y, v.z, v.w}};
}

// LayerNorm over the 64 channels held by 8 lanes (8 each), fp32, two passes; the caller rounds to bf16.
// `gmask` names the 8 lanes of the row: rows of one warp may belong to different tensors (q, k or v) and
// take different paths, so every shuffle synchronises its own group only.
// G rows side by side: the shuffles and the root of one are a chain, which the other's instructions fill.
template <int G>
__device__ __forceinline__ void ln_rows(float2 (&x)[G][4], const float2 (&w)[4], const float2 (&b)[4], float eps, uint32_t gmask) {
  float m[G];
  auto sums8 = [&]() {
#pragma unroll
    for (int d = 1; d < 8; d <<= 1)
#pragma unroll
      for (int u = 0; u < G; ++u) m[u] += __shfl_xor_sync(gmask, m[u], d);
  };
#pragma unroll
  for (int u = 0; u < G; ++u) {
    const float2 s = fadd2(fadd2(x[u][0], x[u][1]), fadd2(x[u][2], x[u][3]));
    m[u] = s.x + s.y;
  }
  sums8();
#pragma unroll
  for (int u = 0; u < G; ++u) {
    const float mean = m[u] * (1.f / 64.f);
    float2 v = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[u][i] = fadd2(x[u][i], splat(-mean));
      v = ffma2(x[u][i], x[u][i], v);
    }
    m[u] = v.x + v.y;
  }
  sums8();
#pragma unroll
  for (int u = 0; u < G; ++u) {
    const float rstd = rsqrtf(m[u] * (1.f / 64.f) + eps);
#pragma unroll
    for (int i = 0; i < 4; ++i) x[u][i] = ffma2(fmul2(x[u][i], splat(rstd)), w[i], b[i]);   // rounded to bf16 when packed
  }
}

// 2-D rotary embedding of a row held by 8 lanes, on packed bf16 pairs: lanes 0-3 hold the y half (32
// channels), lanes 4-7 the x half; inside a half channel j pairs with j+16, i.e. lane l with lane l^2.
// out = bf16(bf16(t*cos) + bf16(rot*sin)),  rot = -t[j+16] for j < 16 and t[j-16] otherwise: the packed
// bf16 multiply and add (the _rn forms, which the compiler may not contract into one FMA) round exactly
// where the reference's bf16 tensor ops do.
__device__ __forceinline__ uint32_t bf2_mul(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf2_add(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hadd2_rn(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <int G>
__device__ __forceinline__ void rope_rows(Vec8 (&o)[G], const Vec8 (&c)[G], const Vec8 (&s)[G], int l8, uint32_t gmask) {
  const uint32_t flip = (l8 & 2) == 0 ? 0x80008000u : 0u;
#pragma unroll
  for (int wd = 0; wd < 4; ++wd)
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const uint32_t other = __shfl_xor_sync(gmask, o[u].w[wd], 2) ^ flip;
      o[u].w[wd] = bf2_add(bf2_mul(o[u].w[wd], c[u].w[wd]), bf2_mul(other, s[u].w[wd]));
    }
}

// A CTA has up to 16 of the block's 3H rows (8 lanes each: four warps, one per scheduler).  A thread's share of 16 tokens is on
// its way at once, 16 bytes a token in slots of its own in shared memory (cp.async; nobody else reads them): 32 KB per CTA.
// Bound: HBM on long sequences (0.8 of the copy rate), on short ones the chain of a token - two sums over eight lanes, a root, a
// rotation - of which one after the other takes 980 cycles with two or three warps per scheduler.  Three forms:
// kProSide: four tokens go through it side by side, with their table rows in shared memory, in four CTAs of 128 registers per SM (two
//   in five of 102 as fast but for the short ones).
// kProOne: one by one, in six CTAs of 80 registers.  For blocks that fill no four or no chunk (prologue_side_by_side).
// kProLong: blocks whose rows of the tables do not fit shared memory; four side by side, each looking its row up.
// 16 heads, blocks of 16, one by one -> side by side: 2048 tokens 13.3 -> 10.7 us, 6144 18.6 -> 18.2, 64 512 183.7 -> 176.7, 252 000
// 697 -> 671.  One block of 6400 tokens, by itself or not, one by one -> four: 3.9 -> 2.7 ms.  Earlier forms, 252 000 tokens: six CTAs
// 628 us (without the gate), 24 KB in flight, the next tokens' loads in registers 759, four tokens ahead and the tables' rows found by
// every row 908, 24 rows per CTA 656, eight CTAs of 64 registers 804.
constexpr int kProRows = 16, kProThreads = kProRows * 8, kProChunk = 16, kProCtas = 4, kProOneCtas = 6, kProBwdCtas = 4;
constexpr int kProRingBytes = kProChunk * kProThreads * 16;
constexpr int kProTabBytes = (kProChunk + 1) * 256;    // cos (y, x) and sin (y, x) of a chunk's tokens and of the block's mean, 64 bytes each

enum ProForm { kProSide, kProOne, kProLong };
template <ProForm FORM>
__global__ void __launch_bounds__(kProThreads, FORM == kProOne ? kProOneCtas : kProCtas) prologue_fwd_kernel(const PrologueParams p) {
  constexpr bool LONG = FORM == kProLong, TAB = FORM == kProSide;
  constexpr int G = FORM == kProOne ? 1 : 4;               // tokens side by side
  extern __shared__ __align__(16) uint8_t smem[];      // [token of the chunk][thread] 16 bytes; [warp] rows of the tables
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31, l8 = threadIdx.x & 7;
  const int g = blockIdx.y * kProRows + (threadIdx.x >> 3);           // row of the token: (q|k|v, head)
  const uint32_t gmask = 0xffu << (threadIdx.x & 24);
  const bool live = g < 3 * p.H;
  const int which = g / p.H, h = g - which * p.H;
  const int b = blockIdx.x / p.Nc, j = blockIdx.x - b * p.Nc;
  const float* lw = which == 0 ? p.qw : p.kw;
  const float* lb = which == 0 ? p.qb : p.kb;
  const bool norm = which < 2 && lw != nullptr, rope = which < 2 && p.pos != nullptr;
  __nv_bfloat16* out = which == 0 ? p.q : (which == 1 ? p.k : p.v);
  __nv_bfloat16* out_c = which == 0 ? p.q_c : (which == 1 ? p.k_c : p.v_c);
  const int64_t bh = static_cast<int64_t>(b) * p.H + h;
  const int n0 = j * p.block;
  const int64_t tok0 = static_cast<int64_t>(b) * p.N + n0;
  const __nv_bfloat16* src = p.qkv + tok0 * p.tok_stride + g * 64 + l8 * 8;
  __nv_bfloat16* dst = out + (bh * p.N + n0) * 64 + l8 * 8;
  const uint32_t slots = smem_u32(smem) + threadIdx.x * 16;
  const uint32_t tab = smem_u32(smem) + kProRingBytes;
  int* rows = reinterpret_cast<int*>(smem + kProRingBytes + (TAB ? kProTabBytes : 0)) + (threadIdx.x >> 5) * 2 * (LONG ? 1 : p.block + 1);
  // two groups of loads per chunk: the first half is worked on while the second arrives
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < kProChunk; ++i) {
      if (live && t0 + i < p.block) cp_async16(slots + i * (kProThreads * 16), src + (t0 + i) * p.tok_stride);
      if (i == kProChunk / 2 - 1) cp_async_commit();
    }
    cp_async_commit();
  };
  fetch(0);
  // the gate's logits, as many as two per thread, are asked for here and used behind the rows' positions
  const int gates = p.gate_in != nullptr && blockIdx.y == 0 ? p.block * p.H : 0;
  auto gate_logits = [&](int i) { return __ldg(reinterpret_cast<const uint32_t*>(p.gate_in + (tok0 + i % p.block) * p.tok_stride) + i / p.block); };
  uint32_t logits[2] = {0u, 0u};
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = threadIdx.x + u * kProThreads;
    if (i < gates) logits[u] = gate_logits(i);
  }
  float2 w[4], bias[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[i] = norm ? __ldg(reinterpret_cast<const float2*>(lw) + l8 * 4 + i) : splat(1.f);
    bias[i] = norm ? __ldg(reinterpret_cast<const float2*>(lb) + l8 * 4 + i) : splat(0.f);
  }
  if (p.pos != nullptr) block_rows<LONG>(rows, p.pos + tok0 * 2, p.block, p.tab_rows, p.status, lane);
  auto put_gate = [&](int i, uint32_t v) {
    const float g0 = 1.f / (1.f + __expf(-bf16_lo(v))), g1 = 1.f / (1.f + __expf(-bf16_hi(v)));
    p.gate[(static_cast<int64_t>(b) * p.H + i / p.block) * p.N + n0 + i % p.block] = pack_bf16(g0, g1);
  };
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = threadIdx.x + u * kProThreads;
    if (i < gates) put_gate(i, logits[u]);
  }
  for (int i = threadIdx.x + 2 * kProThreads; i < gates; i += kProThreads) put_gate(i, gate_logits(i));
  // Table rows of a chunk's tokens to shared memory, for all rows of the CTA: asked for by every row as it came to a token, they
  // were a trip to L2 per pair of tokens on a grid too small to fill it with others' work.
  auto tables = [&](int t0) {
    const int n = min(kProChunk, p.block - t0);
    for (int i = threadIdx.x; i < 16 * (n + (t0 == 0)); i += kProThreads) {
      const bool mean = i >= 16 * n;
      const int row = rows[(mean ? 0 : 2 + 2 * (t0 + (i >> 4))) + ((i >> 2) & 1)];
      const uint4 v = __ldg(reinterpret_cast<const uint4*>((i & 8 ? p.sin_tab : p.cos_tab) + row * 32 + (i & 3) * 8));
      sts128(tab + (mean ? kProChunk : i >> 4) * 256 + (i & 15) * 16, v.x, v.y, v.z, v.w);
    }
  };
  const int* my_row = rows + (l8 >> 2);                // y for lanes 0-3, x for 4-7
  const __nv_bfloat16 *cos_l = p.cos_tab + (l8 & 3) * 8, *sin_l = p.sin_tab + (l8 & 3) * 8;
  auto row_of = [&](int t) { return LONG ? table_row(__ldg(p.pos + (tok0 + t) * 2 + (l8 >> 2)), p.tab_rows) : my_row[2 + 2 * t]; };

  float2 acc[4] = {splat(0.f), splat(0.f), splat(0.f), splat(0.f)};
  // G tokens of this row: accumulate the raw block sum, normalise, rotate, store
  auto tokens = [&](int t, int slot) {
    Vec8 c[G], s[G], o[G];
    float2 x[G][4];
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int at = min(slot + u, kProChunk - 1);
      o[u] = lds_vec8(slots + at * (kProThreads * 16));
      if (rope && !TAB) {
        const int row = row_of(min(t + u, p.block - 1)) * 32;
        c[u] = ldg_vec8(cos_l + row);
        s[u] = ldg_vec8(sin_l + row);
      } else if (rope) {
        c[u] = lds_vec8(tab + at * 256 + l8 * 16);
        s[u] = lds_vec8(tab + at * 256 + 128 + l8 * 16);
      }
    }
#pragma unroll
    for (int u = 0; u < G; ++u) {
      unpack8(x[u], o[u]);
      if (t + u < p.block) {
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = fadd2(acc[i], x[u][i]);
      }
    }
    if (norm) {
      ln_rows<G>(x, w, bias, p.eps, gmask);
#pragma unroll
      for (int u = 0; u < G; ++u) o[u] = pack8(x[u]);
    }
    if (rope) rope_rows<G>(o, c, s, l8, gmask);
#pragma unroll
    for (int u = 0; u < G; ++u)
      if (t + u < p.block) *reinterpret_cast<Vec8*>(dst + (t + u) * 64) = o[u];
  };
  for (int t0 = 0; t0 < p.block; t0 += kProChunk) {
    const int n = min(kProChunk, p.block - t0);
    if (TAB && p.pos != nullptr) {
      if (t0 > 0) __syncthreads();                     // the chunk before has been used
      tables(t0);
      __syncthreads();
    }
    if (live) {
      cp_async_wait<1>();
#pragma unroll (FORM == kProOne ? 2 : 1)
      for (int i = 0; i < n; i += G) {
        if (i == kProChunk / 2) cp_async_wait<0>();
        tokens(t0 + i, i);
      }
      if (t0 + kProChunk < p.block) fetch(t0 + kProChunk);
    }
  }
  if (!live) return;
  // compression branch: mean of the raw rows, then the same norm and the rotary embedding at the block's
  // mean position
  const float inv = 1.f / static_cast<float>(p.block);
  float2 x[1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) x[0][i] = make_float2(bf16r(acc[i].x * inv), bf16r(acc[i].y * inv));
  if (norm) ln_rows<1>(x, w, bias, p.eps, gmask);
  Vec8 o[1] = {pack8(x[0])};
  if (rope) {
    const int row = my_row[0] * 32;
    const Vec8 c[1] = {TAB ? lds_vec8(tab + kProChunk * 256 + l8 * 16) : ldg_vec8(cos_l + row)},
               s[1] = {TAB ? lds_vec8(tab + kProChunk * 256 + 128 + l8 * 16) : ldg_vec8(sin_l + row)};
    rope_rows<1>(o, c, s, l8, gmask);
  }
  *reinterpret_cast<Vec8*>(out_c + (bh * p.Nc + j) * 64 + l8 * 8) = o[0];
}

// ------------------------------------------------------------------------------------------------
// backward
// ------------------------------------------------------------------------------------------------
// One pass as well: the gradients of the six outputs and the projection are read once (the projection a second time out of
// L2: a block's mean comes before its tokens' gradients), the gradient of the packed projection is written once; in
// PyTorch it was about eighty elementwise passes (2.6 of 4.1 ms of a training step at 2 x 6144 tokens).  Arithmetic in fp32
// from the bf16 tensors, one rounding.  Same ownership as the forward; CTAs walk over blocks, so that the LayerNorm
// parameters' gradients stay in registers until the end: per-CTA sums, added up by prologue_bwd_reduce_kernel in a fixed
// order.
struct PrologueBwdParams {
  const __nv_bfloat16* qkv;
  int64_t tok_stride;                // of qkv and dqkv
  const uint32_t* gate;              // [B,H,N] pairs, sigmoid of the logits (null: no gate)
  const float2* dgate;               // [B,H,N] gradient of those
  __nv_bfloat16* dgate_in;           // gradient of the logits, inside dqkv's rows
  const int64_t* pos;
  const __nv_bfloat16* cos_tab;
  const __nv_bfloat16* sin_tab;
  int tab_rows;
  const float* qw; const float* kw;
  float eps;
  const __nv_bfloat16 *dq, *dk, *dv, *dq_c, *dk_c, *dv_c;
  __nv_bfloat16* dqkv;
  float* partial;                    // [CTA][q|k][weight|bias][64], null without norms
  int B, H, N, Nc, block;
};

// transposed rotary embedding: dt[j] = dy[j] cos[j] + dy[j+16] sin[j+16] for j < 16, dy[j] cos[j] - dy[j-16] sin[j-16] otherwise
__device__ __forceinline__ void rope_row_t(float2 (&dy)[4], const Vec8& cw, const Vec8& sw, int l8, uint32_t gmask) {
  float2 c[4], s[4];
  unpack8(c, cw);
  unpack8(s, sw);
  const float2 sign = splat((l8 & 2) == 0 ? 1.f : -1.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 o = fmul2(dy[i], s[i]);
    o.x = __shfl_xor_sync(gmask, o.x, 2);
    o.y = __shfl_xor_sync(gmask, o.y, 2);
    dy[i] = ffma2(o, sign, fmul2(dy[i], c[i]));
  }
}
// dx of y = LayerNorm(x) w + b in place of dy; adds to the parameters' gradients
__device__ __forceinline__ void ln_row_bwd(float2 (&x)[4], float2 (&dy)[4], const float2 (&w)[4], float2 (&gw)[4],
                                           float2 (&gb)[4], float eps, uint32_t gmask) {
  float2 s = fadd2(fadd2(x[0], x[1]), fadd2(x[2], x[3])), sg = splat(0.f), g[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    g[i] = fmul2(dy[i], w[i]);
    sg = fadd2(sg, g[i]);
  }
  const float mean = sum8(s.x + s.y, gmask) * (1.f / 64.f), mg = sum8(sg.x + sg.y, gmask) * (1.f / 64.f);
  float2 v = splat(0.f), sx = splat(0.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i] = fadd2(x[i], splat(-mean));
    v = ffma2(x[i], x[i], v);
    sx = ffma2(g[i], x[i], sx);
  }
  const float rstd = rsqrtf(sum8(v.x + v.y, gmask) * (1.f / 64.f) + eps);
  const float mgx = sum8(sx.x + sx.y, gmask) * (1.f / 64.f) * rstd;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i] = fmul2(x[i], splat(rstd));
    gw[i] = ffma2(dy[i], x[i], gw[i]);
    gb[i] = fadd2(gb[i], dy[i]);
    dy[i] = fmul2(splat(rstd), ffma2(x[i], splat(-mgx), fadd2(g[i], splat(-mg))));
  }
}

// Same rows per CTA and the same private slots: a block's 16 tokens of the projection stay in shared memory for both uses (its
// mean, then its tokens; longer blocks are read again), the gradients come through eight slots.  252000 tokens: 1272 us
// (registers instead of slots, everybody waiting for a block's rows: 1903), 64512: 338.
constexpr int kProBwdAhead = 8;
constexpr int kProBwdRingBytes = (kProChunk + kProBwdAhead) * kProThreads * 16;

template <bool LONG>
__global__ void __launch_bounds__(kProThreads, kProBwdCtas) prologue_bwd_kernel(const PrologueBwdParams p) {
  extern __shared__ __align__(16) uint8_t smem[];      // [token][thread] 16 bytes: projection, gradients; [warp] rows of the tables
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31, l8 = threadIdx.x & 7;
  const int g = blockIdx.y * kProRows + (threadIdx.x >> 3);
  const uint32_t gmask = 0xffu << (threadIdx.x & 24);
  const bool live = g < 3 * p.H;
  const int which = g / p.H, h = g - which * p.H;
  const float* lw = which == 0 ? p.qw : p.kw;
  const bool norm = which < 2 && lw != nullptr, rope = which < 2 && p.pos != nullptr;
  const __nv_bfloat16* dout = which == 0 ? p.dq : (which == 1 ? p.dk : p.dv);
  const __nv_bfloat16* dout_c = which == 0 ? p.dq_c : (which == 1 ? p.dk_c : p.dv_c);
  float2 w[4], gw[4], gb[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[i] = norm ? __ldg(reinterpret_cast<const float2*>(lw) + l8 * 4 + i) : splat(1.f);
    gw[i] = gb[i] = splat(0.f);
  }
  const float inv = 1.f / static_cast<float>(p.block);
  const uint32_t xs = smem_u32(smem) + threadIdx.x * 16, ds = xs + kProChunk * (kProThreads * 16);
  int* rows = reinterpret_cast<int*>(smem + kProBwdRingBytes) + (threadIdx.x >> 5) * 2 * (LONG ? 1 : p.block + 1);
  const int* my_row = rows + (l8 >> 2);                // y for lanes 0-3, x for 4-7
  const __nv_bfloat16 *cos_l = p.cos_tab + (l8 & 3) * 8, *sin_l = p.sin_tab + (l8 & 3) * 8;
  const bool resident = p.block <= kProChunk;
  const int nblocks = p.B * p.Nc;
  for (int blk = blockIdx.x; blk < nblocks; blk += gridDim.x) {
    const int b = blk / p.Nc, j = blk - b * p.Nc;
    const int64_t bh = static_cast<int64_t>(b) * p.H + h, tok0 = static_cast<int64_t>(b) * p.N + static_cast<int64_t>(j) * p.block;
    const __nv_bfloat16* src = p.qkv + tok0 * p.tok_stride + g * 64 + l8 * 8;
    const __nv_bfloat16* dsrc = dout + (bh * p.N + static_cast<int64_t>(j) * p.block) * 64 + l8 * 8;
    __nv_bfloat16* dst = p.dqkv + tok0 * p.tok_stride + g * 64 + l8 * 8;
    Vec8 raw_c;
    if (live) {
      if (norm && resident)
        for (int t = 0; t < p.block; ++t) cp_async16(xs + t * (kProThreads * 16), src + t * p.tok_stride);
      cp_async_commit();
#pragma unroll
      for (int t = 0; t < kProBwdAhead; ++t) {
        if (t < p.block) cp_async16(ds + t * (kProThreads * 16), dsrc + t * 64);
        cp_async_commit();
      }
      raw_c = ldg_vec8(dout_c + (bh * p.Nc + j) * 64 + l8 * 8);
    }
    __syncwarp();                                      // the previous block's rows have been used
    if (p.pos != nullptr) block_rows<LONG>(rows, p.pos + tok0 * 2, p.block, p.tab_rows, nullptr, lane);
    if (live) {
      // the pooled branch's gradient of every token of the block
      float2 dc[4];
      unpack8(dc, raw_c);
      if (rope) {
        const int row = my_row[0] * 32;
        rope_row_t(dc, ldg_vec8(cos_l + row), ldg_vec8(sin_l + row), l8, gmask);
      }
      cp_async_wait<kProBwdAhead>();
      if (norm) {
        float2 xc[4] = {splat(0.f), splat(0.f), splat(0.f), splat(0.f)};
#pragma unroll 4
        for (int t = 0; t < p.block; ++t) {
          float2 x[4];
          unpack8(x, resident ? lds_vec8(xs + t * (kProThreads * 16)) : ldg_vec8(src + t * p.tok_stride));
#pragma unroll
          for (int i = 0; i < 4; ++i) xc[i] = fadd2(xc[i], x[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) xc[i] = make_float2(bf16r(xc[i].x * inv), bf16r(xc[i].y * inv));
        ln_row_bwd(xc, dc, w, gw, gb, p.eps, gmask);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) dc[i] = fmul2(dc[i], splat(inv));

#pragma unroll 2
      for (int t = 0; t < p.block; ++t) {
        Vec8 c, s;
        if (rope) {
          const int row = (LONG ? table_row(__ldg(p.pos + (tok0 + t) * 2 + (l8 >> 2)), p.tab_rows) : my_row[2 + 2 * t]) * 32;
          c = ldg_vec8(cos_l + row);
          s = ldg_vec8(sin_l + row);
        }
        cp_async_wait<kProBwdAhead - 1>();
        const uint32_t slot = ds + (t % kProBwdAhead) * (kProThreads * 16);
        float2 dy[4];
        unpack8(dy, lds_vec8(slot));
        if (t + kProBwdAhead < p.block) cp_async16(slot, dsrc + (t + kProBwdAhead) * 64);
        cp_async_commit();
        if (rope) rope_row_t(dy, c, s, l8, gmask);
        if (norm) {
          float2 x[4];
          unpack8(x, resident ? lds_vec8(xs + t * (kProThreads * 16)) : ldg_vec8(src + t * p.tok_stride));
          ln_row_bwd(x, dy, w, gw, gb, p.eps, gmask);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) dy[i] = fadd2(dy[i], dc[i]);
        *reinterpret_cast<Vec8*>(dst + t * p.tok_stride) = pack8(dy);
      }
    }
    if (p.gate != nullptr && blockIdx.y == 0) {
      for (int i = threadIdx.x; i < p.block * p.H; i += kProThreads) {
        const int t = i % p.block, hd = i / p.block;
        const int64_t at = (static_cast<int64_t>(b) * p.H + hd) * p.N + static_cast<int64_t>(j) * p.block + t;
        const uint32_t v = __ldg(p.gate + at);
        const float2 d = __ldg(p.dgate + at);
        const float g0 = bf16_lo(v), g1 = bf16_hi(v);
        *(reinterpret_cast<uint32_t*>(p.dgate_in + (tok0 + t) * p.tok_stride) + hd) = pack_bf16(d.x * g0 * (1.f - g0), d.y * g1 * (1.f - g1));
      }
    }
  }
  if (p.partial == nullptr) return;
  cp_async_wait<0>();
  __syncthreads();
  float* red = reinterpret_cast<float*>(smem);         // [row][weight|bias][64]
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int at = (threadIdx.x >> 3) * 128 + l8 * 8 + 2 * i;
    *reinterpret_cast<float2*>(&red[at]) = gw[i];
    *reinterpret_cast<float2*>(&red[at + 64]) = gb[i];
  }
  __syncthreads();
  for (int o = threadIdx.x; o < 256; o += kProThreads) {     // (q|k, weight|bias, channel)
    float s = 0.f;
    for (int r = 0; r < kProRows; ++r)
      if ((blockIdx.y * kProRows + r) / p.H == (o >> 7)) s += red[r * 128 + (o & 127)];
    p.partial[(blockIdx.y * gridDim.x + blockIdx.x) * 256 + o] = s;
  }
}

// out[o] = sum over CTAs of partial[cta][o]; a warp per output
__global__ void __launch_bounds__(256) prologue_bwd_reduce_kernel(const float* __restrict__ partial, float* __restrict__ out, int ctas) {
  griddep_wait();
  griddep_launch();
  const int o = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  float s = 0.f;
  for (int c = lane; c < ctas; c += 32) s += partial[c * 256 + o];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (lane == 0) out[o] = s;
}

// The kernels' limit of dynamic shared memory is set to the most a CTA can have, the same in every call: set to a call's own
// need, two threads with blocks of different lengths could lower it for one another between setting and launching.
constexpr int kProMaxSmem = 227 * 1024;

// Shared memory of a CTA; `lengthy`: not even the rows of a block of that many tokens fit beside the slots (more than 5000: no
// setting of the model, but the kernel takes any).
static int prologue_smem(int ring, int block, bool* lengthy) {
  const int64_t warps = kProThreads / 32, all = ring + warps * 2 * (static_cast<int64_t>(block) + 1) * static_cast<int64_t>(sizeof(int));
  *lengthy = all > kProMaxSmem;
  return *lengthy ? ring + static_cast<int>(warps * 2 * sizeof(int)) : static_cast<int>(all);
}
static int prologue_parts(int H) { return (3 * H + kProRows - 1) / kProRows; }
// Whether the forward takes four tokens side by side.  What is left of a block beyond whole fours and whole chunks costs as much as they
// do; where the GPU is not filled the shorter chain counts for more.  16 heads, one by one and side by side, us: 60 000 tokens in blocks of 1
// 680 and 1130, 4 247 and 313, 8 182 and 213, 12 169 and 183, 17 173 and 191, 25 166 and 172, 28 162 and 161, 33 162 and 167 (20 000: 62 and
// 59); of 15 by CTAs 450: 13.9 and 10.9, 720: 15.5 and 13.0, 999: 15.5 and 16.7.
static bool prologue_side_by_side(int block, int64_t ctas) {
  return block % 16 == 0 || block >= 28 || (block >= 14 && 2 * ctas <= 3 * kProCtas * sm_count());
}
// CTAs along the blocks: four per SM over all parts
static int prologue_bwd_ctas(int B, int Nc, int H) {
  const int64_t n = static_cast<int64_t>(B) * Nc, parts = prologue_parts(H), cap = (kProBwdCtas * sm_count() + parts - 1) / parts;
  return static_cast<int>(n < cap ? n : cap);
}

}  // namespace s3r

using namespace s3r;

static int prologue_fwd(const void* qkv, int64_t tok_stride, const void* gate_in, void* gate, const int64_t* pos, const void* cos_tab, const void* sin_tab,
                                    int tab_rows, const float* q_weight, const float* q_bias, const float* k_weight,
                                    const float* k_bias, float eps, void* q, void* k, void* v, void* q_c, void* k_c,
                                    void* v_c, int B, int H, int N, int d, int block, void* stream) {
  S3R_REQUIRE(qkv && q && k && v && q_c && k_c && v_c, S3R_ERR_NULL, "s3r_qkv_prologue_fwd: NULL tensor");
  S3R_REQUIRE(B > 0 && H > 0 && N > 0 && block > 0, S3R_ERR_SHAPE,
              "s3r_qkv_prologue_fwd: sizes must be positive (B=%d H=%d N=%d block=%d)", B, H, N, block);
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_qkv_prologue_fwd: head_dim %d not supported (64 only)", d);
  S3R_REQUIRE(N % block == 0, S3R_ERR_SHAPE, "s3r_qkv_prologue_fwd: N=%d is not a multiple of the block %d", N, block);
  S3R_REQUIRE(3 * H * 8 <= 1024, S3R_ERR_UNSUPPORTED, "s3r_qkv_prologue_fwd: %d heads not supported (42 at most)", H);
  S3R_REQUIRE((q_weight != nullptr) == (q_bias != nullptr) && (k_weight != nullptr) == (k_bias != nullptr) &&
                  (q_weight != nullptr) == (k_weight != nullptr),
              S3R_ERR_NULL, "s3r_qkv_prologue_fwd: LayerNorm weights and biases of q and k come together or not at all");
  S3R_REQUIRE(pos == nullptr || (cos_tab && sin_tab && tab_rows > 0), S3R_ERR_NULL,
              "s3r_qkv_prologue_fwd: positions need the cos/sin tables");
  const uintptr_t al = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
                       reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(q_c) |
                       reinterpret_cast<uintptr_t>(k_c) | reinterpret_cast<uintptr_t>(v_c) |
                       reinterpret_cast<uintptr_t>(cos_tab) | reinterpret_cast<uintptr_t>(sin_tab);
  S3R_REQUIRE((al & 15) == 0, S3R_ERR_ALIGNMENT, "s3r_qkv_prologue_fwd: tensors must be 16-byte aligned");
  const uintptr_t al8 = reinterpret_cast<uintptr_t>(q_weight) | reinterpret_cast<uintptr_t>(q_bias) |
                        reinterpret_cast<uintptr_t>(k_weight) | reinterpret_cast<uintptr_t>(k_bias);
  S3R_REQUIRE((al8 & 7) == 0, S3R_ERR_ALIGNMENT, "s3r_qkv_prologue_fwd: LayerNorm parameters must be 8-byte aligned");
  const int Nc = N / block;
  const int64_t grid = static_cast<int64_t>(B) * Nc;
  S3R_REQUIRE(grid < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_qkv_prologue_fwd: grid of %lld CTAs is too large",
              (long long)grid);
  PrologueParams p;
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.tok_stride = tok_stride;
  p.gate_in = static_cast<const __nv_bfloat16*>(gate_in);
  p.gate = static_cast<uint32_t*>(gate);
  p.pos = pos;
  p.cos_tab = static_cast<const __nv_bfloat16*>(cos_tab);
  p.sin_tab = static_cast<const __nv_bfloat16*>(sin_tab);
  p.tab_rows = tab_rows;
  p.qw = q_weight; p.qb = q_bias; p.kw = k_weight; p.kb = k_bias;
  p.eps = eps;
  p.q = static_cast<__nv_bfloat16*>(q); p.k = static_cast<__nv_bfloat16*>(k); p.v = static_cast<__nv_bfloat16*>(v);
  p.q_c = static_cast<__nv_bfloat16*>(q_c); p.k_c = static_cast<__nv_bfloat16*>(k_c);
  p.v_c = static_cast<__nv_bfloat16*>(v_c);
  p.B = B; p.H = H; p.N = N; p.Nc = Nc; p.block = block;
  p.status = device_status_ptr();
  S3R_REQUIRE(p.status != nullptr, S3R_ERR_DRIVER, "s3r_qkv_prologue_fwd: could not resolve the device status word");
  const int64_t ctas = grid * prologue_parts(H);
  bool side = prologue_side_by_side(block, ctas), lengthy;
  int smem = prologue_smem(kProRingBytes + (side ? kProTabBytes : 0), block, &lengthy);
  if (side && lengthy) {
    // 6104 to 6239 tokens' rows fit beside the slots alone, in one CTA per SM.  20 such blocks, 16 heads: one by one 3.2 ms, as long blocks
    // 3.4, without a norm 2.6 and 3.0, but without positions 2.6 and 1.9, and 300 blocks of 4 heads 8.1 and 3.2
    side = false;
    if (pos != nullptr && ctas <= sm_count()) smem = prologue_smem(kProRingBytes, block, &lengthy);
  }
  auto* kernel = side ? prologue_fwd_kernel<kProSide> : lengthy ? prologue_fwd_kernel<kProLong> : prologue_fwd_kernel<kProOne>;
  S3R_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kProMaxSmem));
  return launch(kernel, dim3(static_cast<unsigned>(grid), prologue_parts(H)), kProThreads, smem,
                static_cast<cudaStream_t>(stream), p);
}

extern "C" int s3r_qkv_prologue_fwd(const void* qkv, const int64_t* pos, const void* cos_tab, const void* sin_tab,
                                    int tab_rows, const float* q_weight, const float* q_bias, const float* k_weight,
                                    const float* k_bias, float eps, void* q, void* k, void* v, void* q_c, void* k_c,
                                    void* v_c, int B, int H, int N, int d, int block, void* stream) {
  return prologue_fwd(qkv, static_cast<int64_t>(3) * H * d, nullptr, nullptr, pos, cos_tab, sin_tab, tab_rows, q_weight, q_bias, k_weight,
                      k_bias, eps, q, k, v, q_c, k_c, v_c, B, H, N, d, block, stream);
}

extern "C" int s3r_qkv_gate_prologue_fwd(const void* proj, const int64_t* pos, const void* cos_tab, const void* sin_tab,
                                         int tab_rows, const float* q_weight, const float* q_bias, const float* k_weight,
                                         const float* k_bias, float eps, void* q, void* k, void* v, void* q_c, void* k_c,
                                         void* v_c, void* gate, int B, int H, int N, int d, int block, void* stream) {
  S3R_REQUIRE(proj && gate, S3R_ERR_NULL, "s3r_qkv_gate_prologue_fwd: NULL tensor");
  S3R_REQUIRE(H > 0 && H % 4 == 0, S3R_ERR_UNSUPPORTED, "s3r_qkv_gate_prologue_fwd: %d heads are not a multiple of 4", H);
  const int64_t C3 = static_cast<int64_t>(3) * H * d;
  return prologue_fwd(proj, C3 + 2 * H, static_cast<const __nv_bfloat16*>(proj) + C3, gate, pos, cos_tab, sin_tab, tab_rows, q_weight,
                      q_bias, k_weight, k_bias, eps, q, k, v, q_c, k_c, v_c, B, H, N, d, block, stream);
}

extern "C" size_t s3r_qkv_prologue_bwd_workspace_bytes(int B, int H, int N, int block) {
  if (B <= 0 || H <= 0 || N <= 0 || block <= 0 || N < block) return 0;
  return static_cast<size_t>(prologue_bwd_ctas(B, N / block, H)) * prologue_parts(H) * 256 * sizeof(float);
}

static int prologue_bwd(const void* qkv, int64_t tok_stride, const void* gate, const float* dgate, void* dgate_in, const int64_t* pos, const void* cos_tab, const void* sin_tab, int tab_rows,
                                    const float* q_weight, const float* k_weight, float eps, const void* dq, const void* dk,
                                    const void* dv, const void* dq_c, const void* dk_c, const void* dv_c, void* dqkv,
                                    float* dparams, void* workspace, size_t workspace_bytes, int B, int H, int N, int d,
                                    int block, void* stream) {
  S3R_REQUIRE(qkv && dq && dk && dv && dq_c && dk_c && dv_c && dqkv, S3R_ERR_NULL, "s3r_qkv_prologue_bwd: NULL tensor");
  S3R_REQUIRE(B > 0 && H > 0 && N > 0 && block > 0, S3R_ERR_SHAPE,
              "s3r_qkv_prologue_bwd: sizes must be positive (B=%d H=%d N=%d block=%d)", B, H, N, block);
  S3R_REQUIRE(d == 64, S3R_ERR_UNSUPPORTED, "s3r_qkv_prologue_bwd: head_dim %d not supported (64 only)", d);
  S3R_REQUIRE(N % block == 0, S3R_ERR_SHAPE, "s3r_qkv_prologue_bwd: N=%d is not a multiple of the block %d", N, block);
  S3R_REQUIRE(3 * H * 8 <= 1024, S3R_ERR_UNSUPPORTED, "s3r_qkv_prologue_bwd: %d heads not supported (42 at most)", H);
  S3R_REQUIRE((q_weight != nullptr) == (k_weight != nullptr) && (q_weight != nullptr) == (dparams != nullptr), S3R_ERR_NULL,
              "s3r_qkv_prologue_bwd: LayerNorm weights of q and k and their gradients come together or not at all");
  S3R_REQUIRE(pos == nullptr || (cos_tab && sin_tab && tab_rows > 0), S3R_ERR_NULL,
              "s3r_qkv_prologue_bwd: positions need the cos/sin tables");
  S3R_REQUIRE(!dparams || (workspace && workspace_bytes >= s3r_qkv_prologue_bwd_workspace_bytes(B, H, N, block)), S3R_ERR_TOO_LARGE,
              "s3r_qkv_prologue_bwd: workspace of %zu bytes is smaller than the %zu needed", workspace_bytes,
              s3r_qkv_prologue_bwd_workspace_bytes(B, H, N, block));
  uintptr_t al = reinterpret_cast<uintptr_t>(cos_tab) | reinterpret_cast<uintptr_t>(sin_tab) | reinterpret_cast<uintptr_t>(dqkv);
  for (const void* t : {qkv, dq, dk, dv, dq_c, dk_c, dv_c}) al |= reinterpret_cast<uintptr_t>(t);
  S3R_REQUIRE((al & 15) == 0, S3R_ERR_ALIGNMENT, "s3r_qkv_prologue_bwd: tensors must be 16-byte aligned");
  S3R_REQUIRE(((reinterpret_cast<uintptr_t>(q_weight) | reinterpret_cast<uintptr_t>(k_weight)) & 7) == 0, S3R_ERR_ALIGNMENT,
              "s3r_qkv_prologue_bwd: LayerNorm parameters must be 8-byte aligned");
  const int Nc = N / block;
  S3R_REQUIRE(static_cast<int64_t>(B) * Nc < (1ll << 31), S3R_ERR_TOO_LARGE, "s3r_qkv_prologue_bwd: too many blocks");
  PrologueBwdParams p;
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.tok_stride = tok_stride;
  p.gate = static_cast<const uint32_t*>(gate);
  p.dgate = reinterpret_cast<const float2*>(dgate);
  p.dgate_in = static_cast<__nv_bfloat16*>(dgate_in);
  p.pos = pos;
  p.cos_tab = static_cast<const __nv_bfloat16*>(cos_tab);
  p.sin_tab = static_cast<const __nv_bfloat16*>(sin_tab);
  p.tab_rows = tab_rows;
  p.qw = q_weight; p.kw = k_weight;
  p.eps = eps;
  p.dq = static_cast<const __nv_bfloat16*>(dq); p.dk = static_cast<const __nv_bfloat16*>(dk);
  p.dv = static_cast<const __nv_bfloat16*>(dv); p.dq_c = static_cast<const __nv_bfloat16*>(dq_c);
  p.dk_c = static_cast<const __nv_bfloat16*>(dk_c); p.dv_c = static_cast<const __nv_bfloat16*>(dv_c);
  p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.partial = dparams ? static_cast<float*>(workspace) : nullptr;
  p.B = B; p.H = H; p.N = N; p.Nc = Nc; p.block = block;
  const int ctas = prologue_bwd_ctas(B, Nc, H), parts = prologue_parts(H);
  bool lengthy;
  const int smem = prologue_smem(kProBwdRingBytes, block, &lengthy);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto* kernel = lengthy ? prologue_bwd_kernel<true> : prologue_bwd_kernel<false>;
  S3R_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kProMaxSmem));
  const int rc = launch(kernel, dim3(static_cast<unsigned>(ctas), parts), kProThreads, smem, st, p);
  if (rc || !dparams) return rc;
  return launch(prologue_bwd_reduce_kernel, 32, 256, 0, st, p.partial, dparams, ctas * parts);
}

extern "C" int s3r_qkv_prologue_bwd(const void* qkv, const int64_t* pos, const void* cos_tab, const void* sin_tab, int tab_rows,
                                    const float* q_weight, const float* k_weight, float eps, const void* dq, const void* dk,
                                    const void* dv, const void* dq_c, const void* dk_c, const void* dv_c, void* dqkv,
                                    float* dparams, void* workspace, size_t workspace_bytes, int B, int H, int N, int d,
                                    int block, void* stream) {
  return prologue_bwd(qkv, static_cast<int64_t>(3) * H * d, nullptr, nullptr, nullptr, pos, cos_tab, sin_tab, tab_rows, q_weight, k_weight,
                      eps, dq, dk, dv, dq_c, dk_c, dv_c, dqkv, dparams, workspace, workspace_bytes, B, H, N, d, block, stream);
}

extern "C" int s3r_qkv_gate_prologue_bwd(const void* proj, const int64_t* pos, const void* cos_tab, const void* sin_tab,
                                         int tab_rows, const float* q_weight, const float* k_weight, float eps, const void* dq,
                                         const void* dk, const void* dv, const void* dq_c, const void* dk_c, const void* dv_c,
                                         const void* gate, const float* dgate, void* dproj, float* dparams, void* workspace,
                                         size_t workspace_bytes, int B, int H, int N, int d, int block, void* stream) {
  S3R_REQUIRE(proj && gate && dgate && dproj, S3R_ERR_NULL, "s3r_qkv_gate_prologue_bwd: NULL tensor");
  S3R_REQUIRE(H > 0 && H % 4 == 0, S3R_ERR_UNSUPPORTED, "s3r_qkv_gate_prologue_bwd: %d heads are not a multiple of 4", H);
  const int64_t C3 = static_cast<int64_t>(3) * H * d;
  return prologue_bwd(proj, C3 + 2 * H, gate, dgate, static_cast<__nv_bfloat16*>(dproj) + C3, pos, cos_tab, sin_tab, tab_rows, q_weight,
                      k_weight, eps, dq, dk, dv, dq_c, dk_c, dv_c, dproj, dparams, workspace, workspace_bytes, B, H, N, d, block,
                      stream);
}
