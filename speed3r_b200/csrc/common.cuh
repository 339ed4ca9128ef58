// Shared device/host helpers for the sm_100a kernels of the sparse global-attention path:
// status codes, bf16 packing, and thin wrappers over the PTX this library issues by hand
// (mbarrier, TMA tiled copies, ldmatrix / mma.sync, tcgen05 + tensor memory).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/speed3r_b200.h"

namespace s3r {

// ---------------------------------------------------------------------------------------------
// host-side error plumbing (thread-local message returned by s3r_last_error)
// ---------------------------------------------------------------------------------------------
int set_error(int code, const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

#define S3R_REQUIRE(cond, code, ...)                                  \
  do {                                                                \
    if (!(cond)) return ::s3r::set_error((code), __VA_ARGS__);        \
  } while (0)

#define S3R_CUDA(call)                                                \
  do {                                                                \
    int _rc = ::s3r::check_cuda((call), #call);                       \
    if (_rc != 0) return _rc;                                         \
  } while (0)

// Per-device status word the kernels write when a bounded wait runs out or an index is out of
// range.  It lives in a file-scope __device__ variable; the host reads it on request
// (s3r_device_status), never implicitly, so no call synchronises.
uint32_t* device_status_ptr();   // device address of the status word of the current device

// TMA descriptors (CUtensorMap) are built on the host per call; encode through the driver entry
// point obtained at run time, so the library does not link libcuda directly.
// dims/strides are innermost-first; strides in BYTES for dims 1..rank-1.
int make_tensor_map(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                    const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle,
                    CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);

// Two tensors of the same shape (`chunks` chunks of [BH, T / chunks, 64] bf16) whose 16-row tiles travel together, 2 KB of
// each: where the distance between them fits a tensor map's stride, as ONE map whose outermost dimension of two steps from
// one to the other, so that one copy brings both.
struct PairMap {
  CUtensorMap both, second;      // second: b's own map, where they are apart
  int b_first;                   // b's tile lies in front of a's; -1: a == b, one tile serves as both
  int apart;                     // two copies
};
// (b_first, apart) of two addresses: strides are below 2^40 bytes, and device memory of different origin (virtual-memory
// reservations, peers' and symmetric buffers) can be further apart.
struct PairOrder {
  int b_first, apart;
};
PairOrder pair_order(uint64_t a, uint64_t b);
int make_pair_map(PairMap* out, const void* a, const void* b, int T, int BH, int chunks, int64_t chunk_stride_bytes);

int sm_count();

#ifdef __CUDACC__
// Launch of a kernel whose CTAs may start while the kernel before it in the stream is still finishing (programmatic
// stream serialisation).  Every thread of such a kernel calls griddep_wait() before its first access to global memory;
// what comes before - barriers, tensor memory, index arithmetic - then overlaps the other kernel's last CTAs.  On a short
// sequence a call is a chain of kernels of 3 to 25 us, whose starts and ends are a good part of it.
template <typename... P, typename... A>
inline int launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(static_cast<unsigned>(threads));
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = a;
  c.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...), "kernel launch");
}
// All of the kernels before this one have completed and what they wrote is visible.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel's CTAs may start where there is room (they wait for this kernel's end themselves).
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kStatusWaitTimeout = 1u;   // a bounded mbarrier wait gave up
constexpr uint32_t kStatusBadIndex    = 2u;   // a rotary position was outside the cos/sin tables

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float fast_log2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 operations in one instruction (packed pairs in a 64-bit register).
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "add.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// 2^x of a pair on the FMA pipe, for kernels whose exponentials saturate their own unit (16 results per cycle and SM):
// x = n + f with n the nearest integer (the 1.5 * 2^23 shift), 2^f by a polynomial of degree 5 on [-1/2, 1/2], n added
// to the exponent field.  The coefficients are a least-squares fit of the relative error with the last one fixed at 1,
// reweighted until it levelled out: 1.6e-7, 2.2e-7 with fp32 rounding (ex2.approx: 2.4e-7).  x < 127; below -126, and for
// NaN, the result is 2^-126: whoever calls it looks for NaN among the scores (keeping NaN here, with 2^n as a factor, cost
// the long forward 2.5 %).
__device__ __forceinline__ float2 exp2_fma2(float2 x) {
  x.x = fmaxf(x.x, -126.f);
  x.y = fmaxf(x.y, -126.f);
  const float2 shift = make_float2(12582912.f, 12582912.f), unshift = make_float2(-12582912.f, -12582912.f);
  const float2 t = fadd2(x, shift), n = fadd2(t, unshift), f = fadd2(x, make_float2(-n.x, -n.y));
  float2 r = make_float2(1.327647012e-3f, 1.327647012e-3f);
  r = ffma2(r, f, make_float2(9.675541319e-3f, 9.675541319e-3f));
  r = ffma2(r, f, make_float2(5.550713279e-2f, 5.550713279e-2f));
  r = ffma2(r, f, make_float2(2.402211972e-1f, 2.402211972e-1f));
  r = ffma2(r, f, make_float2(6.931469671e-1f, 6.931469671e-1f));
  r = ffma2(r, f, make_float2(1.f, 1.f));
  r.x = __uint_as_float((__float_as_uint(t.x) << 23) + __float_as_uint(r.x));
  r.y = __uint_as_float((__float_as_uint(t.y) << 23) + __float_as_uint(r.y));
  return r;
}

// max of three in one instruction (three-operand max of sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// the same, NaN if any of them is
__device__ __forceinline__ float fmax3_nan(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Order-preserving float -> uint32 map: flip every bit of a negative value, set the sign bit of
// a non-negative one.  Larger float <=> larger key; -0.0 < +0.0.
__device__ __forceinline__ uint32_t sortable_key(float v) {
  uint32_t b = __float_as_uint(v);
  return b ^ (static_cast<uint32_t>(static_cast<int32_t>(b) >> 31) | 0x80000000u);
}

// ---- mbarrier -------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Whether the phase is complete, without waiting for it.  Asking takes about a hundred cycles even where it is, so that a warp
// with something else to issue asks before that and looks at the answer afterwards.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Per-warpgroup register re-partition (every warp of the group of four executes the same one).
template <int N>
__device__ __forceinline__ void reg_alloc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_dealloc() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
// Probe that lets the hardware park the thread for up to `hint_ns` while the phase is pending: a parked
// warp issues nothing, whereas a spinning one competes for issue slots with the warps doing the work.
__device__ __forceinline__ bool mbar_try_wait_parked(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait.  Returns false when the phase did not complete within `limit_ns` (about a second in
// the kernels) or when another thread of the CTA has already given up (*abort_flag != 0); the caller
// then unwinds instead of spinning for ever.  (Kept inline on purpose: a call at a site that holds a
// whole row of scores in registers cannot be register-allocated.)
__device__ __forceinline__ bool mbar_wait_limit(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                                uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (true) {
    if (mbar_try_wait_parked(bar, parity, 20000u)) return true;
    if (*abort_flag) return false;
    if (globaltimer_ns() - t0 > limit_ns) break;
  }
  *abort_flag = 1u;
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  return mbar_wait_limit(bar, parity, abort_flag, 1000000000ull);
}

// Same, called by all 32 lanes of a converged warp; the result is warp-uniform.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                               uint64_t limit_ns = 1000000000ull) {
  const bool ok = mbar_wait_limit(bar, parity, abort_flag, limit_ns);
  return __all_sync(0xffffffffu, ok);
}

// The rest of a wait that mbar_test began.  No vote: lanes may part where one of them gives up.
__device__ __forceinline__ bool mbar_settle(bool done, uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  return done || mbar_wait(bar, parity, abort_flag);
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- cp.async --------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst_smem), "l"(src) : "memory");
}

// ---- cluster launch control: a running CTA takes over the work of one that has not been launched yet ----
// One thread asks; the answer (16 bytes) lands in shared memory and completes `bar`.  After an answer without a CTA none
// may be asked for again.
__device__ __forceinline__ void clc_request(uint4* answer, uint64_t* bar) {
  mbar_expect_tx(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(answer)), "r"(smem_u32(bar)) : "memory");
}
// blockIdx.x of the CTA whose work was handed over, -1: none left
__device__ __forceinline__ int clc_answer(const uint4* answer) {
  int x;
  asm volatile(
      "{\n\t.reg .b128 r;\n\t.reg .pred p;\n\t.reg .b32 y, z, w;\n\t"
      "ld.shared.b128 r, [%1];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "mov.b32 %0, -1;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, y, z, w}, r;\n\t}"
      : "=r"(x) : "r"(smem_u32(answer)) : "memory");
  return x;
}

// ---- TMA tiled loads (no multicast anywhere in this library) --------------------------------
__device__ __forceinline__ void tma_load_3d(uint32_t dst_smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst_smem), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst_smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst_smem), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst_smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst_smem), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
// the tiles of 16 rows from `tok` on of both tensors, 2 KB each (one of them serves as both: 2 KB)
// APART: kernels are compiled for both, so that the usual form does not ask
template <bool APART>
__device__ __forceinline__ void tma_load_pair(uint32_t dst_smem, const PairMap& m, uint64_t* bar, int tok, int bh, int chunk) {
  tma_load_5d(dst_smem, &m.both, bar, 0, tok, bh, chunk, 0);
  if (APART && m.apart) tma_load_5d(dst_smem + 2048, &m.second, bar, 0, tok, bh, chunk, 0);
}

// ---- ldmatrix / mma.sync (m16n8k16, bf16 x bf16 -> fp32) ------------------------------------
__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Same with a zero accumulator on input.
__device__ __forceinline__ void mma_bf16_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
// Appends a pair at `at` where `on` is not 0, and moves `at` by STEP bytes: predicated, where the compiler would branch.
template <int STEP>
__device__ __forceinline__ void sts64_append(uint32_t on, uint32_t& at, uint32_t x, uint32_t y) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p st.shared.v2.b32 [%0], {%2, %3};\n\t@p add.u32 %0, %0, %4;\n\t}"
               : "+r"(at) : "r"(on), "r"(x), "r"(y), "n"(STEP) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}

// Byte offset of element (row, 16-byte chunk) inside a tile whose rows are 128 bytes and that
// was written with the 128-byte swizzle (TMA SWIZZLE_128B, tile base 1024-byte aligned):
// the chunk index is XORed with (row mod 8).
__device__ __forceinline__ uint32_t swz128(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

// ---- tcgen05 / tensor memory ----------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor for a bf16 operand tile stored with the 128-byte swizzle.
//   K-major  (rows = M or N, 64 contiguous K elements = 128 B per row): 8-row groups are
//            1024 B apart (stride byte offset); the leading offset is unused.
//   MN-major (rows = K, 64 contiguous M/N elements per row): 8-row (K) groups 1024 B apart.
// Start address, LBO and SBO are in 16-byte units; bits 46-47 hold the descriptor version (1),
// bits 61-63 the swizzle mode (2 = 128 B).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr, uint32_t sbo_bytes = 1024, uint32_t lbo_bytes = 16) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}
// Instruction descriptor, kind::f16, bf16 x bf16 -> fp32.  b_mn_major = 1 when B is stored with
// N contiguous (a [K][N] row-major tile).
__host__ __device__ constexpr uint32_t umma_idesc_bf16(uint32_t M, uint32_t N, uint32_t a_mn_major, uint32_t b_mn_major) {
  return (1u << 4)        // D format fp32
         | (1u << 7)      // A bf16
         | (1u << 10)     // B bf16
         | (a_mn_major << 15) | (b_mn_major << 16) | ((N >> 3) << 17) | ((M >> 4) << 24);
}
// One lane of a converged warp, the same one on every call.  The MMA warp stays converged (all lanes
// run the loop and the waits) and only the issuing instructions are predicated on the elected lane:
// descriptor arithmetic then stays on the warp-uniform datapath.  Measured on this part against an
// `if (lane == 0)` region around the whole loop: 42 instead of 52 cycles per M128 N64 K16 MMA.
__device__ __forceinline__ bool elect_one_sync() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
  return pred != 0;
}
// Four k-steps (K = 4 x 16) in one instruction sequence: the operand descriptors advance by constant
// numbers of 16-byte units (2 = 32 bytes along a K-major row, 128 = 2048 bytes = 16 rows of an MN-major
// tile), so one k-step costs the issuing thread one add per operand besides the MMA itself.  The issuing
// thread shares its scheduler with warps that do the arithmetic; every instruction it saves shortens the
// time from "operands ready" to "MMAs queued".
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_ss_k4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p, pt;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 pt, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "add.s64 a, %1, %5;\n\tadd.s64 b, %2, %6;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, pt;\n\t"
      "add.s64 a, a, %5;\n\tadd.s64 b, b, %6;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, pt;\n\t"
      "add.s64 a, a, %5;\n\tadd.s64 b, b, %6;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, pt;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accum), "n"(A_STEP), "n"(B_STEP)
      : "memory");
}
// Same with A in tensor memory (bf16 pairs: 8 columns per k-step; the third k-step starts A_JUMP columns after the second).
template <int B_STEP, int A_JUMP = 8>
__device__ __forceinline__ void umma_ts_k4(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p, pt;\n\t.reg .b64 b;\n\t.reg .b32 a;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 pt, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "add.u32 a, %1, 8;\n\tadd.s64 b, %2, %5;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, pt;\n\t"
      "add.u32 a, a, %6;\n\tadd.s64 b, b, %5;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, pt;\n\t"
      "add.u32 a, a, 8;\n\tadd.s64 b, b, %5;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, pt;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accum), "n"(B_STEP), "n"(A_JUMP)
      : "memory");
}
// Arrive on an mbarrier once every tcgen05 operation issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// The same for a warp that runs all of its loop converged: only the lane whose `lead` is set issues.  Without a branch around them
// there is nothing to converge after, and operands stay warp-uniform.
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_ss_k4_by(uint32_t lead, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p, pt, l;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 pt, 0, 0;\n\tsetp.ne.b32 l, %7, 0;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "add.s64 a, %1, %5;\n\tadd.s64 b, %2, %6;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, pt;\n\t"
      "add.s64 a, a, %5;\n\tadd.s64 b, b, %6;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, pt;\n\t"
      "add.s64 a, a, %5;\n\tadd.s64 b, b, %6;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, pt;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accum), "n"(A_STEP), "n"(B_STEP), "r"(lead)
      : "memory");
}
template <int B_STEP, int A_JUMP = 8>
__device__ __forceinline__ void umma_ts_k4_by(uint32_t lead, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p, pt, l;\n\t.reg .b64 b;\n\t.reg .b32 a;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 pt, 0, 0;\n\tsetp.ne.b32 l, %7, 0;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "add.u32 a, %1, 8;\n\tadd.s64 b, %2, %5;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, pt;\n\t"
      "add.u32 a, a, %6;\n\tadd.s64 b, b, %5;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, pt;\n\t"
      "add.u32 a, a, 8;\n\tadd.s64 b, b, %5;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, pt;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accum), "n"(B_STEP), "n"(A_JUMP), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void umma_commit_by(uint32_t lead, uint64_t* bar) {
  asm volatile("{\n\t.reg .pred l;\n\tsetp.ne.b32 l, %1, 0;\n\t"
               "@l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(lead)
               : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives lane (base_lane + i).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

#endif  // __CUDACC__
}  // namespace s3r
