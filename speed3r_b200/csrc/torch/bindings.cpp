// The torch.library operators of the package: argument checks, allocation and autograd wiring around the
// C ABI of include/speed3r_b200.h.  Everything between Python and the launches is native, because a call
// on a short sequence is bounded by host work: through torch.library.custom_op, Python autograd functions
// and ctypes the whole op at 2048 tokens took 243 us, of which the GPU worked 114 us.
//
// Two layers of operators:
//   base operators (pool_fwd, cmp_attn_topk_fwd, sel_attn_fwd, ...): one C-ABI call each, no autograd.
//     Registered for CUDA, and for CPU only to say that there is no CPU path.  Their shape functions for
//     torch.compile are registered from Python (ops.py).
//   differentiable operators (pool_tokens, flash_attn_topk, ..., sparse_attention): composite functions that
//     call the base operators through the dispatcher, inside a C++ autograd node when a gradient is needed.
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CachingHostAllocator.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/library.h>

#include <cmath>
#include <tuple>
#include <vector>

#include "../../../include/speed3r_b200.h"

namespace {

using at::Tensor;
using c10::optional;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

void need(const Tensor& t, const char* name, at::ScalarType dtype = at::kBFloat16, bool contiguous = true) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor: the speed3r_b200 kernels have no CPU path");
  TORCH_CHECK(t.scalar_type() == dtype, name, " must be ", dtype, ", got ", t.scalar_type());
  TORCH_CHECK(!contiguous || t.is_contiguous(), name, " must be contiguous");
}

// Sizes that are divided by: a division by zero ends the process in C++, where Python raised.
template <typename... N>
void need_positive(const char* what, N... n) {
  TORCH_CHECK(((n > 0) && ...), what, ": block, window and stride must be positive");
}

void check(int rc, const char* what) {
  if (rc == 0) return;
  char msg[512];
  s3r_last_error(msg, sizeof(msg));
  TORCH_CHECK(false, what, " failed with code ", rc, ": ", msg);
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
const int32_t* i32(const Tensor& t) { return static_cast<const int32_t*>(t.data_ptr()); }
int32_t* i32m(const Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); }
float* f32(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
Tensor fresh(at::IntArrayRef shape, const Tensor& like, at::ScalarType dtype) {
  return at::empty(shape, like.options().dtype(dtype));
}
// contiguous, whatever the strides of `t` (at::empty_like would keep a permuted layout)
Tensor fresh_like(const Tensor& t) { return at::empty(t.sizes(), t.options()); }
// The same values at a multiple of 16 bytes: a contiguous view may begin anywhere in its storage (a slice, a flattened
// parameter buffer), and the kernels load vectors.
Tensor aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone(); }
optional<Tensor> aligned(const optional<Tensor>& t) { return t.has_value() ? optional<Tensor>(aligned(*t)) : t; }
Tensor none(const Tensor& like) { return at::empty({0}, like.options()); }

// ------------------------------------------------------------------------------------------------
// base operators
// ------------------------------------------------------------------------------------------------
Tensor pool_fwd(const Tensor& x, int64_t kernel, int64_t stride) {
  need_positive("pool", kernel, stride);
  need(x, "x", at::kBFloat16, false);
  TORCH_CHECK(x.dim() == 4 && x.stride(3) == 1, "pool: x must be [B,H,T,d] and its channel dimension must have unit stride");
  const int64_t B = x.size(0), H = x.size(1), T = x.size(2), d = x.size(3);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = fresh({B, H, (T - kernel) / stride + 1, d}, x, at::kBFloat16);
  check(s3r_pool_fwd(x.data_ptr(), x.stride(0), x.stride(1), x.stride(2), out.data_ptr(), B, H, T, d, kernel, stride,
                     stream()), "s3r_pool_fwd");
  return out;
}

// q pooled per block, k and v with kernel/stride, in one launch where they are of one length
std::tuple<Tensor, Tensor, Tensor> pool_qkv_fwd(const Tensor& q, const Tensor& k, const Tensor& v, int64_t block,
                                                int64_t kernel, int64_t stride) {
  need_positive("pool", block, kernel, stride);
  const Tensor* x[3] = {&q, &k, &v};
  for (const Tensor* t : x) {
    need(*t, "x", at::kBFloat16, false);
    TORCH_CHECK(t->dim() == 4 && t->stride(3) == 1, "pool: q, k, v must be [B,H,T,d] and their channel dimension must have unit stride");
  }
  if (q.sizes() != k.sizes() || k.sizes() != v.sizes())            // queries against another sequence
    return {pool_fwd(q, block, block), pool_fwd(k, kernel, stride), pool_fwd(v, kernel, stride)};
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2), d = q.size(3);
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out[3];
  const void* in_p[3];
  void* out_p[3];
  int64_t st[9];
  int kernels[3], strides[3];
  for (int i = 0; i < 3; ++i) {
    kernels[i] = static_cast<int>(i == 0 ? block : kernel);
    strides[i] = static_cast<int>(i == 0 ? block : stride);
    out[i] = fresh({B, H, (T - kernels[i]) / strides[i] + 1, d}, q, at::kBFloat16);
    in_p[i] = x[i]->data_ptr();
    out_p[i] = out[i].data_ptr();
    for (int j = 0; j < 3; ++j) st[3 * i + j] = x[i]->stride(j);
  }
  check(s3r_pool_multi_fwd(3, in_p, st, out_p, kernels, strides, B, H, T, d, stream()), "s3r_pool_multi_fwd");
  return {out[0], out[1], out[2]};
}

Tensor pool_bwd(const Tensor& d_out_, int64_t T, int64_t kernel, int64_t stride) {
  need(d_out_, "d_out");
  const int64_t B = d_out_.size(0), H = d_out_.size(1), d = d_out_.size(3);
  c10::cuda::CUDAGuard guard(d_out_.device());
  const Tensor d_out = aligned(d_out_);
  Tensor d_in = fresh({B, H, T, d}, d_out, at::kBFloat16);
  check(s3r_pool_bwd(d_out.data_ptr(), d_in.data_ptr(), H * T * d, T * d, d, B, H, T, d, kernel, stride, 0, stream()),
        "s3r_pool_bwd");
  return d_in;
}

// group = 0: the table ranks columns; otherwise blocks of `group` columns by the mass of their first `take`
std::tuple<Tensor, Tensor, Tensor> cmp_fwd(const Tensor& q_c, const Tensor& k_c, const Tensor& v_c, int64_t topk,
                                           double scale, int64_t group, int64_t take) {
  need(q_c, "q_c");
  need(k_c, "k_c");
  need(v_c, "v_c");
  const int64_t B = q_c.size(0), H = q_c.size(1), Nq = q_c.size(2), d = q_c.size(3), Nc = k_c.size(2);
  const std::vector<int64_t> want = {B, H, Nc, d};
  TORCH_CHECK(k_c.sizes() == want && v_c.sizes() == want, "k_c/v_c shape mismatch: ", k_c.sizes(), " ", v_c.sizes(),
              " vs B=", B, " H=", H, " d=", d);
  c10::cuda::CUDAGuard guard(q_c.device());
  Tensor o = fresh({B, H, Nq, d}, q_c, at::kBFloat16), lse = fresh({B, H, Nq}, q_c, at::kFloat),
         idx = fresh({B, H, Nq, topk}, q_c, at::kInt);
  if (group == 0)
    check(s3r_cmp_attn_topk_fwd(q_c.data_ptr(), k_c.data_ptr(), v_c.data_ptr(), o.data_ptr(), f32(lse), i32m(idx), B, H,
                                Nq, Nc, d, topk, scale, stream()), "s3r_cmp_attn_topk_fwd");
  else
    check(s3r_cmp_attn_blocktopk_fwd(q_c.data_ptr(), k_c.data_ptr(), v_c.data_ptr(), o.data_ptr(), f32(lse), i32m(idx),
                                     B, H, Nq, Nc, d, topk, scale, group, take, stream()), "s3r_cmp_attn_blocktopk_fwd");
  return {o, lse, idx};
}
std::tuple<Tensor, Tensor, Tensor> cmp_attn_topk_fwd(const Tensor& q_c, const Tensor& k_c, const Tensor& v_c,
                                                     int64_t topk, double scale) {
  return cmp_fwd(q_c, k_c, v_c, topk, scale, 0, 0);
}
std::tuple<Tensor, Tensor, Tensor> cmp_attn_blocktopk_fwd(const Tensor& q_c, const Tensor& k_c, const Tensor& v_c,
                                                          int64_t topk, double scale, int64_t group, int64_t take) {
  TORCH_CHECK(group > 0, "s3r_cmp_attn_blocktopk_fwd: group must be positive");
  return cmp_fwd(q_c, k_c, v_c, topk, scale, group, take);
}

std::tuple<Tensor, Tensor, Tensor> cmp_bwd(const Tensor& q_c, const Tensor& k_c, const Tensor& v_c,
                                                const Tensor& o_c, const Tensor& lse, const Tensor& do_c_, double scale,
                                                const Tensor* have_delta) {
  need(q_c, "q_c");
  need(k_c, "k_c");
  need(v_c, "v_c");
  need(o_c, "o_c");
  need(do_c_, "do_c");
  need(lse, "lse", at::kFloat);
  const int64_t B = q_c.size(0), H = q_c.size(1), Nq = q_c.size(2), d = q_c.size(3), Nc = k_c.size(2);
  c10::cuda::CUDAGuard guard(q_c.device());
  const Tensor do_c = aligned(do_c_);
  Tensor dq = fresh_like(q_c), dk = fresh_like(k_c), dv = fresh_like(v_c);
  if (have_delta) {
    check(s3r_cmp_attn_bwd_delta(q_c.data_ptr(), k_c.data_ptr(), v_c.data_ptr(), f32(lse), do_c.data_ptr(), f32(*have_delta),
                                 dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, H, Nq, Nc, d, scale, stream()),
          "s3r_cmp_attn_bwd_delta");
    return {dq, dk, dv};
  }
  Tensor delta = fresh_like(lse);
  check(s3r_cmp_attn_bwd(q_c.data_ptr(), k_c.data_ptr(), v_c.data_ptr(), o_c.data_ptr(), f32(lse), do_c.data_ptr(),
                         f32(delta), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, H, Nq, Nc, d, scale, stream()),
        "s3r_cmp_attn_bwd");
  return {dq, dk, dv};
}
std::tuple<Tensor, Tensor, Tensor> cmp_attn_bwd(const Tensor& q_c, const Tensor& k_c, const Tensor& v_c,
                                                const Tensor& o_c, const Tensor& lse, const Tensor& do_c, double scale) {
  return cmp_bwd(q_c, k_c, v_c, o_c, lse, do_c, scale, nullptr);
}

void need_gate(const Tensor& gate) {
  need(gate, "gate", at::kBFloat16, false);
  TORCH_CHECK(gate.dim() == 4 && gate.stride(3) == 1, "gate: the last dimension (g0,g1) must have unit stride");
}

// Returns (o_s, lse_s, y); tensors not asked for come back with zero elements.
std::tuple<Tensor, Tensor, Tensor> sel_attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                                const optional<Tensor>& gate, const optional<Tensor>& o_c, int64_t block,
                                                double scale, bool want_o, bool want_lse, int64_t kv_chunks) {
  need_positive("selection attention", block);
  need(q, "q");
  need(k, "k");
  need(v, "v");
  need(idx, "topk_idx", at::kInt);
  const int64_t B = q.size(0), H = q.size(1), Tq = q.size(2), d = q.size(3);
  int64_t Tk, chunk_stride = 0;
  if (kv_chunks == 1) {
    Tk = k.size(2);
    TORCH_CHECK(k.sizes() == std::vector<int64_t>({B, H, Tk, d}) && v.sizes() == k.sizes(), "k/v must be [B,H,Tk,d]");
  } else {                               // [chunks, B, H, Tk/chunks, d] as an all-gather leaves it
    TORCH_CHECK(k.dim() == 5 && k.size(0) == kv_chunks && v.sizes() == k.sizes(), "chunked k/v must be [chunks,B,H,Tk/chunks,d]");
    Tk = k.size(3) * kv_chunks;
    chunk_stride = k.stride(0);
  }
  const int64_t K = idx.size(-1), nqb = (Tq + block - 1) / block;
  TORCH_CHECK(idx.sizes() == std::vector<int64_t>({B, H, nqb, K}), "topk_idx must be [B,H,ceil(Tq/block),K] = [", B, ", ", H,
              ", ", nqb, ", ", K, "], got ", idx.sizes());
  const bool merge = gate.has_value();
  int64_t gs[3] = {0, 0, 0};
  if (merge) {
    need_gate(*gate);
    TORCH_CHECK(o_c.has_value(), "gate and o_c come together");
    need(*o_c, "o_c");
    TORCH_CHECK(gate->sizes() == std::vector<int64_t>({B, H, Tq, 2}) && o_c->sizes() == std::vector<int64_t>({B, H, nqb, d}),
                "gate must be [B,H,Tq,2] and o_c [B,H,ceil(Tq/block),d]");
    for (int i = 0; i < 3; ++i) gs[i] = gate->stride(i);
  }
  c10::cuda::CUDAGuard guard(q.device());
  Tensor o_s = want_o ? fresh({B, H, Tq, d}, q, at::kBFloat16) : none(q);
  Tensor lse = fresh(want_lse ? std::vector<int64_t>{B, H, Tq} : std::vector<int64_t>{0}, q, at::kFloat);
  Tensor y = merge ? fresh({B, Tq, H * d}, q, at::kBFloat16) : none(q);
  check(s3r_sel_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), kv_chunks, chunk_stride, i32(idx),
                         want_o ? o_s.data_ptr() : nullptr, want_lse ? f32(lse) : nullptr, merge ? gate->data_ptr() : nullptr,
                         gs[0], gs[1], gs[2], merge ? o_c->data_ptr() : nullptr, merge ? y.data_ptr() : nullptr, B, H, Tq, Tk,
                         d, block, K, scale, stream()), "s3r_sel_attn_fwd");
  return {o_s, lse, y};
}

// The table's inverse on a stream of its own, from construction to join(): it needs nothing of the backward that precedes
// the selection branch's (31 us at 2 x 6144 tokens, as long as the merge and the compression branch take).
struct CsrBeside {
  c10::cuda::CUDAStream main, side;
  at::cuda::CUDAEvent done;
  bool joined = false;
  // A stream of PyTorch's pool, which callers' streams come from as well: one that is in a capture which this work is not part
  // of is left alone, and the work goes where it would without a second stream.
  static c10::cuda::CUDAStream beside(const c10::cuda::CUDAStream& main) {
    const auto side = c10::cuda::getStreamFromPool();
    auto capture = [](const c10::cuda::CUDAStream& s) {      // 0: none
      cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
      unsigned long long id = 0;
      C10_CUDA_CHECK(cudaStreamGetCaptureInfo(s.stream(), &status, &id));
      return status == cudaStreamCaptureStatusNone ? 0ull : id;
    };
    const auto theirs = capture(side);
    return theirs != 0 && theirs != capture(main) ? main : side;
  }
  CsrBeside(const int32_t* idx, int32_t* offsets, int32_t* qids, int64_t B, int64_t H, int64_t Nq, int64_t K, int64_t nkb, void* ws,
            size_t bytes)
      : main(c10::cuda::getCurrentCUDAStream()), side(beside(main)) {
    at::cuda::CUDAEvent start;
    start.record(main);
    start.block(side);
    const int rc = s3r_build_key_csr(idx, offsets, qids, B, H, Nq, K, nkb, ws, bytes, side.stream());
    done.record(side);
    if (rc != 0) join();
    check(rc, "s3r_build_key_csr");
  }
  void join() {
    if (!joined) done.block(main);
    joined = true;
  }
  ~CsrBeside() {
    try { join(); } catch (...) {}
  }
};
std::tuple<Tensor, Tensor> csr(const Tensor& idx, int64_t nkb, bool fill) {
  need(idx, "topk_idx", at::kInt);
  const int64_t B = idx.size(0), H = idx.size(1), Nq = idx.size(2), K = idx.size(3);
  c10::cuda::CUDAGuard guard(idx.device());
  Tensor offsets = fresh({B, H, nkb + 1}, idx, at::kInt), qids = fresh({B, H, Nq * K}, idx, at::kInt);
  if (fill) qids.fill_(-1);
  const size_t nbytes = s3r_csr_workspace_bytes(B, H, Nq, K, nkb);
  Tensor ws = fresh({static_cast<int64_t>(nbytes)}, idx, at::kByte);
  check(s3r_build_key_csr(i32(idx), i32m(offsets), i32m(qids), B, H, Nq, K, nkb, ws.data_ptr(), nbytes, stream()),
        "s3r_build_key_csr");
  return {offsets, qids};
}
// slots behind the entries of the table that were dropped hold -1
std::tuple<Tensor, Tensor> build_key_csr(const Tensor& idx, int64_t num_key_blocks) { return csr(idx, num_key_blocks, true); }

// The selection branch's gradients; with dq_c, dk_c, dv_c (gradients of q pooled per block and of k, v pooled with
// kernel/stride) the pooled branch's share is added to them.
std::tuple<Tensor, Tensor, Tensor> sel_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                           const Tensor& lse, const Tensor& delta, const Tensor& do_s_, const Tensor* dq_c,
                                           const Tensor* dk_c, const Tensor* dv_c, int64_t block, int64_t kernel,
                                           int64_t stride, double scale, const std::tuple<Tensor, Tensor>* inverse = nullptr) {
  need_positive("selection attention", block, kernel, stride);
  need(q, "q");
  need(k, "k");
  need(v, "v");
  need(do_s_, "do_s");
  const int64_t B = q.size(0), H = q.size(1), Tq = q.size(2), d = q.size(3), Tk = k.size(2), K = idx.size(-1);
  c10::cuda::CUDAGuard guard(q.device());
  const Tensor do_s = aligned(do_s_);
  const Tensor pooled[3] = {dq_c ? aligned(*dq_c) : Tensor(), dq_c ? aligned(*dk_c) : Tensor(), dq_c ? aligned(*dv_c) : Tensor()};
  auto [offsets, qids] = inverse ? *inverse : csr(idx, (Tk + block - 1) / block, false);
  Tensor dq = fresh_like(q), dk = fresh_like(k), dv = fresh_like(v);
  const bool fused = dq_c != nullptr && block % 16 == 0 && kernel % 16 == 0 && stride % 16 == 0;
  auto ptr = [&](int i) -> const void* { return fused ? pooled[i].data_ptr() : nullptr; };
  check(s3r_sel_attn_bwd_pooled(q.data_ptr(), k.data_ptr(), v.data_ptr(), i32(idx), i32(offsets), i32(qids), f32(lse), f32(delta),
                                do_s.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), ptr(0), ptr(1), ptr(2),
                                fused ? block : 16, fused ? block : 16, fused ? kernel : 16, fused ? stride : 16, B, H, Tq, Tk,
                                d, block, K, scale, stream()), "s3r_sel_attn_bwd");
  if (dq_c != nullptr && !fused) {
    check(s3r_pool_bwd(pooled[0].data_ptr(), dq.data_ptr(), H * Tq * d, Tq * d, d, B, H, Tq, d, block, block, 1, stream()), "s3r_pool_bwd");
    check(s3r_pool_bwd(pooled[1].data_ptr(), dk.data_ptr(), H * Tk * d, Tk * d, d, B, H, Tk, d, kernel, stride, 1, stream()), "s3r_pool_bwd");
    check(s3r_pool_bwd(pooled[2].data_ptr(), dv.data_ptr(), H * Tk * d, Tk * d, d, B, H, Tk, d, kernel, stride, 1, stream()), "s3r_pool_bwd");
  }
  return {dq, dk, dv};
}
std::tuple<Tensor, Tensor, Tensor> sel_attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                                const Tensor& lse, const Tensor& delta, const Tensor& do_s, int64_t block,
                                                double scale) {
  return sel_bwd(q, k, v, idx, lse, delta, do_s, nullptr, nullptr, nullptr, block, 16, 16, scale);
}
std::tuple<Tensor, Tensor, Tensor> sel_attn_bwd_pooled(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                                       const Tensor& lse, const Tensor& delta, const Tensor& do_s,
                                                       const Tensor& dq_c, const Tensor& dk_c, const Tensor& dv_c,
                                                       int64_t block, int64_t kernel, int64_t stride, double scale) {
  need_positive("selection attention", block, kernel, stride);
  need(dq_c, "dq_c");
  need(dk_c, "dk_c");
  need(dv_c, "dv_c");
  return sel_bwd(q, k, v, idx, lse, delta, do_s, &dq_c, &dk_c, &dv_c, block, kernel, stride, scale);
}

Tensor delta(const Tensor& o_, const Tensor& d_o_) {
  need(o_, "o");
  need(d_o_, "do");
  c10::cuda::CUDAGuard guard(o_.device());
  const Tensor o = aligned(o_), d_o = aligned(d_o_);
  Tensor out = fresh(o.sizes().slice(0, o.dim() - 1), o, at::kFloat);
  check(s3r_delta(o.data_ptr(), d_o.data_ptr(), f32(out), out.numel(), o.size(-1), stream()), "s3r_delta");
  return out;
}

std::tuple<Tensor, Tensor, Tensor, Tensor> merge_bwd_deltas(const Tensor& dy_, const Tensor& gate, const Tensor& o_c,
                                                            const Tensor& o_s, int64_t block, Tensor* delta_c) {
  need(dy_, "dy");
  need_gate(gate);
  const int64_t B = o_s.size(0), H = o_s.size(1), Tq = o_s.size(2), d = o_s.size(3);
  c10::cuda::CUDAGuard guard(dy_.device());
  const Tensor dy = aligned(dy_);
  Tensor do_s = fresh_like(o_s), dgate = fresh({B, H, Tq, 2}, dy, at::kFloat), do_c = fresh_like(o_c),
         delta_s = fresh({B, H, Tq}, dy, at::kFloat);
  if (delta_c) *delta_c = fresh({B, H, o_c.size(2)}, dy, at::kFloat);
  check(s3r_merge_bwd_deltas(dy.data_ptr(), gate.data_ptr(), gate.stride(0), gate.stride(1), gate.stride(2), o_c.data_ptr(),
                             o_s.data_ptr(), do_s.data_ptr(), f32(dgate), do_c.data_ptr(), f32(delta_s),
                             delta_c ? f32(*delta_c) : nullptr, B, H, Tq, d, block, stream()), "s3r_merge_bwd");
  return {do_s, dgate, do_c, delta_s};
}
std::tuple<Tensor, Tensor, Tensor, Tensor> merge_bwd(const Tensor& dy, const Tensor& gate, const Tensor& o_c,
                                                     const Tensor& o_s, int64_t block) {
  return merge_bwd_deltas(dy, gate, o_c, o_s, block, nullptr);
}

const void* ptr_or_null(const optional<Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }
const float* f32_or_null(const optional<Tensor>& t) { return t.has_value() ? f32(*t) : nullptr; }

// What the prologue's arguments have to be; returns the rows of the rotary tables (0: no rotary embedding)
int64_t need_prologue(const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos, const optional<Tensor>& cos,
                      const optional<Tensor>& sin, std::initializer_list<const optional<Tensor>*> norms) {
  TORCH_CHECK(qkv.dim() >= 3 && heads > 0 && block > 0 && qkv.numel() > 0, "qkv_prologue: qkv must be [B,N,3*H*d] and not empty");
  need(qkv, "qkv");
  const int64_t B = qkv.size(0), N = qkv.size(1), C3 = qkv.numel() / (B * N), d = C3 / (3 * heads);
  TORCH_CHECK(C3 == 3 * heads * d && N % block == 0, "qkv_prologue: qkv ", qkv.sizes(), " does not split into 3 x ", heads,
              " heads, or N=", N, " is not a multiple of the block ", block);
  for (const auto* w : norms) {
    TORCH_CHECK(w->has_value() == (*norms.begin())->has_value(), "qkv_prologue: q_norm and k_norm come together or not at all");
    if (w->has_value()) need(**w, "norm parameter", at::kFloat);
  }
  if (!pos.has_value()) return 0;
  TORCH_CHECK(cos.has_value() && sin.has_value(), "qkv_prologue: positions need the cos/sin tables");
  need(*cos, "cos");
  need(*sin, "sin");
  TORCH_CHECK(cos->sizes() == sin->sizes() && cos->dim() == 2 && cos->size(1) == d / 2, "qkv_prologue: cos/sin tables must be [rows,",
              d / 2, "]");
  TORCH_CHECK(pos->sizes() == std::vector<int64_t>({B, N, 2}) && pos->device() == qkv.device(),
              "qkv_prologue: pos must be [B,N,2] = [", B, ", ", N, ", 2] on ", qkv.device());
  need(*pos, "pos", at::kLong);
  return cos->size(0);
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> prologue_fwd(
    const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos, const optional<Tensor>& cos,
    const optional<Tensor>& sin, const optional<Tensor>& qw_, const optional<Tensor>& qb_, const optional<Tensor>& kw_,
    const optional<Tensor>& kb_, double eps) {
  const int64_t rows = need_prologue(qkv, heads, block, pos, cos, sin, {&qw_, &qb_, &kw_, &kb_});
  const int64_t B = qkv.size(0), N = qkv.size(1), d = qkv.numel() / (B * N) / (3 * heads);
  c10::cuda::CUDAGuard guard(qkv.device());
  const auto qw = aligned(qw_), qb = aligned(qb_), kw = aligned(kw_), kb = aligned(kb_);
  Tensor t[6];
  for (int i = 0; i < 6; ++i) t[i] = fresh({B, heads, i < 3 ? N : N / block, d}, qkv, at::kBFloat16);
  const bool rope = pos.has_value();
  check(s3r_qkv_prologue_fwd(qkv.data_ptr(), static_cast<const int64_t*>(ptr_or_null(pos)), rope ? ptr_or_null(cos) : nullptr,
                             rope ? ptr_or_null(sin) : nullptr, rows, f32_or_null(qw), f32_or_null(qb), f32_or_null(kw),
                             f32_or_null(kb), eps, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(),
                             t[4].data_ptr(), t[5].data_ptr(), B, heads, N, d, block, stream()), "s3r_qkv_prologue_fwd");
  return {t[0], t[1], t[2], t[3], t[4], t[5]};
}

// (gradient of qkv, [4,64] gradients of q weight, q bias, k weight, k bias; no elements without norms)
std::tuple<Tensor, Tensor> prologue_bwd(const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos,
                                        const optional<Tensor>& cos, const optional<Tensor>& sin, const optional<Tensor>& qw_,
                                        const optional<Tensor>& kw_, double eps, const Tensor& dq_, const Tensor& dk_,
                                        const Tensor& dv_, const Tensor& dq_c_, const Tensor& dk_c_, const Tensor& dv_c_) {
  const int64_t rows = need_prologue(qkv, heads, block, pos, cos, sin, {&qw_, &kw_});
  for (const Tensor* g : {&dq_, &dk_, &dv_, &dq_c_, &dk_c_, &dv_c_}) need(*g, "gradient");
  const int64_t B = qkv.size(0), N = qkv.size(1), d = qkv.numel() / (B * N) / (3 * heads);
  c10::cuda::CUDAGuard guard(qkv.device());
  const auto qw = aligned(qw_), kw = aligned(kw_);
  const Tensor dq = aligned(dq_), dk = aligned(dk_), dv = aligned(dv_), dq_c = aligned(dq_c_), dk_c = aligned(dk_c_), dv_c = aligned(dv_c_);
  const bool norm = qw.has_value(), rope = pos.has_value();
  const size_t nbytes = norm ? s3r_qkv_prologue_bwd_workspace_bytes(B, heads, N, block) : 0;
  Tensor dqkv = fresh_like(qkv), ws = fresh({static_cast<int64_t>(nbytes)}, qkv, at::kByte),
         dparams = fresh(norm ? std::vector<int64_t>{4, d} : std::vector<int64_t>{0}, qkv, at::kFloat);
  check(s3r_qkv_prologue_bwd(qkv.data_ptr(), static_cast<const int64_t*>(ptr_or_null(pos)), rope ? ptr_or_null(cos) : nullptr,
                             rope ? ptr_or_null(sin) : nullptr, rows, f32_or_null(qw), f32_or_null(kw), eps, dq.data_ptr(),
                             dk.data_ptr(), dv.data_ptr(), dq_c.data_ptr(), dk_c.data_ptr(), dv_c.data_ptr(), dqkv.data_ptr(),
                             norm ? f32(dparams) : nullptr, norm ? ws.data_ptr() : nullptr, nbytes, B, heads, N, d, block,
                             stream()), "s3r_qkv_prologue_bwd");
  return {dqkv, dparams};
}

// ------------------------------------------------------------------------------------------------
// the base operators as the differentiable ones call them: through the dispatcher, so that fake tensors,
// functionalisation and dispatch modes see them
// ------------------------------------------------------------------------------------------------
#define S3R_DISPATCHED(fn)                                                                              \
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("speed3r_b200::" #fn, "").typed<decltype(fn)>(); \
  return op.call

Tensor call_pool_fwd(const Tensor& x, int64_t kernel, int64_t stride) { S3R_DISPATCHED(pool_fwd)(x, kernel, stride); }
Tensor call_pool_bwd(const Tensor& g, int64_t T, int64_t kernel, int64_t stride) { S3R_DISPATCHED(pool_bwd)(g, T, kernel, stride); }
std::tuple<Tensor, Tensor, Tensor> call_cmp_topk(const Tensor& q, const Tensor& k, const Tensor& v, int64_t topk, double scale) {
  S3R_DISPATCHED(cmp_attn_topk_fwd)(q, k, v, topk, scale);
}
std::tuple<Tensor, Tensor, Tensor> call_cmp_blocktopk(const Tensor& q, const Tensor& k, const Tensor& v, int64_t topk,
                                                      double scale, int64_t group, int64_t take) {
  S3R_DISPATCHED(cmp_attn_blocktopk_fwd)(q, k, v, topk, scale, group, take);
}
std::tuple<Tensor, Tensor, Tensor> call_cmp(const Tensor& q, const Tensor& k, const Tensor& v, int64_t topk, double scale,
                                            int64_t group, int64_t take) {
  return group == 0 ? call_cmp_topk(q, k, v, topk, scale) : call_cmp_blocktopk(q, k, v, topk, scale, group, take);
}
std::tuple<Tensor, Tensor, Tensor> call_cmp_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o,
                                                const Tensor& lse, const Tensor& d_o, double scale) {
  S3R_DISPATCHED(cmp_attn_bwd)(q, k, v, o, lse, d_o, scale);
}
std::tuple<Tensor, Tensor, Tensor> call_sel(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                            const optional<Tensor>& gate, const optional<Tensor>& o_c, int64_t block,
                                            double scale, bool want_o, bool want_lse, int64_t chunks) {
  S3R_DISPATCHED(sel_attn_fwd)(q, k, v, idx, gate, o_c, block, scale, want_o, want_lse, chunks);
}
std::tuple<Tensor, Tensor, Tensor> call_sel_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                                const Tensor& lse, const Tensor& dlt, const Tensor& d_o, int64_t block,
                                                double scale) {
  S3R_DISPATCHED(sel_attn_bwd)(q, k, v, idx, lse, dlt, d_o, block, scale);
}
std::tuple<Tensor, Tensor, Tensor> call_sel_bwd_pooled(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                                       const Tensor& lse, const Tensor& dlt, const Tensor& d_o,
                                                       const Tensor& dq_c, const Tensor& dk_c, const Tensor& dv_c,
                                                       int64_t block, int64_t kernel, int64_t stride, double scale) {
  S3R_DISPATCHED(sel_attn_bwd_pooled)(q, k, v, idx, lse, dlt, d_o, dq_c, dk_c, dv_c, block, kernel, stride, scale);
}
std::tuple<Tensor, Tensor, Tensor> call_pool_qkv(const Tensor& q, const Tensor& k, const Tensor& v, int64_t block,
                                                 int64_t kernel, int64_t stride) {
  S3R_DISPATCHED(pool_qkv_fwd)(q, k, v, block, kernel, stride);
}
Tensor call_delta(const Tensor& o, const Tensor& d_o) { S3R_DISPATCHED(delta)(o, d_o); }
std::tuple<Tensor, Tensor, Tensor, Tensor> call_merge_bwd(const Tensor& dy, const Tensor& gate, const Tensor& o_c,
                                                          const Tensor& o_s, int64_t block) {
  S3R_DISPATCHED(merge_bwd)(dy, gate, o_c, o_s, block);
}

using SixTensors = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor>;
SixTensors call_prologue(const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos, const optional<Tensor>& cos,
                         const optional<Tensor>& sin, const optional<Tensor>& qw, const optional<Tensor>& qb,
                         const optional<Tensor>& kw, const optional<Tensor>& kb, double eps) {
  S3R_DISPATCHED(prologue_fwd)(qkv, heads, block, pos, cos, sin, qw, qb, kw, kb, eps);
}
std::tuple<Tensor, Tensor> call_prologue_bwd(const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos,
                                             const optional<Tensor>& cos, const optional<Tensor>& sin, const optional<Tensor>& qw,
                                             const optional<Tensor>& kw, double eps, const Tensor& dq, const Tensor& dk,
                                             const Tensor& dv, const Tensor& dq_c, const Tensor& dk_c, const Tensor& dv_c) {
  S3R_DISPATCHED(prologue_bwd)(qkv, heads, block, pos, cos, sin, qw, kw, eps, dq, dk, dv, dq_c, dk_c, dv_c);
}

// ------------------------------------------------------------------------------------------------
// differentiable operators
// ------------------------------------------------------------------------------------------------
// Forward-mode derivatives are refused, in every operator and whether a gradient is wanted or not: past the nodes, the base
// operators would drop a tangent without a word.
bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); }
bool has_tangent(const optional<Tensor>& t) { return t.has_value() && has_tangent(*t); }
template <typename... T>
void no_tangents(const T&... t) {
  TORCH_CHECK_NOT_IMPLEMENTED(!(has_tangent(t) || ...), "speed3r_b200: forward mode AD is not implemented for the operators of this package");
}
template <typename... T>
bool wants_grad(const T&... t) {
  no_tangents(t...);
  return at::GradMode::is_enabled() && (t.requires_grad() || ...);
}

// A backward of a node.  It runs without recording; where its result is to be differentiated again (create_graph), the result
// raises when that is tried: no operator here has a second derivative, and without this one would be missing silently.
template <typename F>
variable_list once(const variable_list& incoming, F&& backward) {
  const bool again = at::GradMode::is_enabled();
  variable_list g;
  {
    at::NoGradGuard no_grad;
    g = backward();
  }
  if (!again) return g;
  // the error stands between the result and all it depends on: the node's own inputs and the incoming gradients
  torch::autograd::edge_list edges = torch::autograd::collect_next_edges(incoming);
  if (const auto node = torch::autograd::get_current_node()) edges.insert(edges.end(), node->next_edges().begin(), node->next_edges().end());
  const auto error = std::make_shared<torch::autograd::Error>("the backward of speed3r_b200 operators cannot be differentiated again",
                                                              std::move(edges));
  for (Tensor& t : g)
    if (t.defined()) {
      t = t.detach();
      torch::autograd::set_history(t, error);
    }
  return g;
}

struct PoolNode : torch::autograd::Function<PoolNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t kernel, int64_t stride) {
    ctx->saved_data["T"] = x.size(2);
    ctx->saved_data["kernel"] = kernel;
    ctx->saved_data["stride"] = stride;
    at::AutoDispatchBelowADInplaceOrView below;
    return call_pool_fwd(x, kernel, stride);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    return {call_pool_bwd(g[0].contiguous(), ctx->saved_data["T"].toInt(), ctx->saved_data["kernel"].toInt(),
                          ctx->saved_data["stride"].toInt()), Tensor(), Tensor()};
  }
};
Tensor pool_tokens(const Tensor& x, int64_t kernel, int64_t stride) {
  return wants_grad(x) ? PoolNode::apply(x, kernel, stride) : call_pool_fwd(x, kernel, stride);
}

struct CmpNode : torch::autograd::Function<CmpNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, int64_t topk,
                               double scale, int64_t group, int64_t take) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, lse, idx] = call_cmp(q, k, v, topk, scale, group, take);
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["scale"] = scale;
    ctx->mark_non_differentiable({idx});
    ctx->set_materialize_grads(false);      // no zeros for the table
    return {o, idx};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] = call_cmp_bwd(s[0], s[1], s[2], s[3], s[4],
                                     g[0].defined() ? g[0].contiguous() : at::zeros_like(s[3]), ctx->saved_data["scale"].toDouble());
    return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
std::tuple<Tensor, Tensor> flash_attn_topk(const Tensor& q_, const Tensor& k_, const Tensor& v_, int64_t topk, double scale,
                                           int64_t group, int64_t take) {
  const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
  if (!wants_grad(q, k, v)) {
    auto [o, lse, idx] = call_cmp(q, k, v, topk, scale, group, take);
    return {o, idx};
  }
  const auto r = CmpNode::apply(q, k, v, topk, scale, group, take);
  return {r[0], r[1]};
}

struct SelNode : torch::autograd::Function<SelNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                        int64_t block, double scale) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, lse, y] = call_sel(q, k, v, idx, {}, {}, block, scale, true, true, 1);
    ctx->save_for_backward({q, k, v, o, lse, idx});
    ctx->saved_data["block"] = block;
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const Tensor d_o = g[0].contiguous();
    auto [dq, dk, dv] = call_sel_bwd(s[0], s[1], s[2], s[5], s[4], call_delta(s[3], d_o), d_o,
                                     ctx->saved_data["block"].toInt(), ctx->saved_data["scale"].toDouble());
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};
Tensor topk_blocksparse(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, int64_t block, double scale) {
  if (wants_grad(q, k, v)) return SelNode::apply(q, k, v, idx, block, scale);
  return std::get<0>(call_sel(q, k, v, idx, {}, {}, block, scale, true, false, 1));
}

struct SelMergeNode : torch::autograd::Function<SelMergeNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                        const Tensor& gate, const Tensor& o_c, int64_t block, double scale) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o_s, lse, y] = call_sel(q, k, v, idx, gate, o_c, block, scale, true, true, 1);
    ctx->save_for_backward({q, k, v, idx, gate, o_c, o_s, lse});
    ctx->saved_data["block"] = block;
    ctx->saved_data["scale"] = scale;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const int64_t block = ctx->saved_data["block"].toInt();
    auto [do_s, dgate, do_c, dlt] = call_merge_bwd(g[0].contiguous(), s[4], s[5], s[6], block);
    auto [dq, dk, dv] = call_sel_bwd(s[0], s[1], s[2], s[3], s[7], dlt, do_s, block, ctx->saved_data["scale"].toDouble());
    return {dq, dk, dv, Tensor(), dgate.to(s[4].scalar_type()), do_c, Tensor(), Tensor()};
  }
};
Tensor sel_merge(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const Tensor& gate, const Tensor& o_c,
                 int64_t block, double scale) {
  if (wants_grad(q, k, v, gate, o_c)) return SelMergeNode::apply(q, k, v, idx, gate, o_c, block, scale);
  return std::get<2>(call_sel(q, k, v, idx, gate, o_c, block, scale, false, false, 1));
}

// The prologue with its backward.  Norm parameters are fp32 here (prologue() casts them, differentiably).
struct PrologueNode : torch::autograd::Function<PrologueNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos,
                               const optional<Tensor>& cos, const optional<Tensor>& sin, const optional<Tensor>& qw,
                               const optional<Tensor>& qb, const optional<Tensor>& kw, const optional<Tensor>& kb, double eps) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [q, k, v, q_c, k_c, v_c] = call_prologue(qkv, heads, block, pos, cos, sin, qw, qb, kw, kb, eps);
    auto or_none = [](const optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); };
    ctx->save_for_backward({qkv, or_none(pos), or_none(cos), or_none(sin), or_none(qw), or_none(kw)});
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["block"] = block;
    ctx->saved_data["eps"] = eps;
    return {q, k, v, q_c, k_c, v_c};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    auto opt = [](const Tensor& t) { return t.defined() ? optional<Tensor>(t) : optional<Tensor>(); };
    auto [dqkv, dp] = call_prologue_bwd(s[0], ctx->saved_data["heads"].toInt(), ctx->saved_data["block"].toInt(), opt(s[1]), opt(s[2]),
                                        opt(s[3]), opt(s[4]), opt(s[5]), ctx->saved_data["eps"].toDouble(), g[0].contiguous(),
                                        g[1].contiguous(), g[2].contiguous(), g[3].contiguous(), g[4].contiguous(),
                                        g[5].contiguous());
    const bool norm = s[4].defined();
    auto param = [&](int i) { return norm ? dp.select(0, i) : Tensor(); };
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), param(0), param(1), param(2), param(3), Tensor()};
  }
};
SixTensors prologue(const Tensor& qkv, int64_t heads, int64_t block, const optional<Tensor>& pos_, const optional<Tensor>& cos,
                    const optional<Tensor>& sin, const optional<Tensor>& qw_, const optional<Tensor>& qb_,
                    const optional<Tensor>& kw_, const optional<Tensor>& kb_, double eps) {
  auto as = [&](const optional<Tensor>& t, at::ScalarType type) {
    return t.has_value() ? optional<Tensor>(t->to(qkv.device(), type).contiguous()) : t;
  };
  no_tangents(qkv, qw_, qb_, kw_, kb_);
  TORCH_CHECK(!pos_.has_value() || pos_->device() == qkv.device(), "qkv_prologue: pos must be on ", qkv.device());
  const auto pos = as(pos_, at::kLong), qw = as(qw_, at::kFloat), qb = as(qb_, at::kFloat), kw = as(kw_, at::kFloat), kb = as(kb_, at::kFloat);
  auto grad = [](const optional<Tensor>& t) { return t.has_value() && t->requires_grad(); };
  if (at::GradMode::is_enabled() && (qkv.requires_grad() || grad(qw) || grad(qb) || grad(kw) || grad(kb))) {
    const auto r = PrologueNode::apply(qkv, heads, block, pos, cos, sin, qw, qb, kw, kb, eps);
    return {r[0], r[1], r[2], r[3], r[4], r[5]};
  }
  return call_prologue(qkv, heads, block, pos, cos, sin, qw, qb, kw, kb, eps);
}

// What the module's arguments have to be: the native forms copy by these sizes into one allocation.  Shapes come before
// devices, so that they can be checked without a GPU.
void need_module(const Tensor& x, const Tensor& w_qkv, const optional<Tensor>& b_qkv, const Tensor& w_gate, const optional<Tensor>& b_gate,
                 const Tensor& w_proj, const optional<Tensor>& b_proj, const optional<Tensor>& pos, const optional<Tensor>& cos,
                 const optional<Tensor>& sin, std::initializer_list<const optional<Tensor>*> norms, int64_t heads, int64_t block) {
  TORCH_CHECK(x.dim() == 3 && heads > 0 && block > 0, "attention module: x must be [B,N,C]");
  const int64_t B = x.size(0), N = x.size(1), C = x.size(2), d = C / heads;
  TORCH_CHECK(C == heads * d && N % block == 0, "attention module: x ", x.sizes(), " does not split into ", heads, " heads and blocks of ", block);
  auto shape = [&](const Tensor& t, at::IntArrayRef want, const char* name) {
    TORCH_CHECK(t.sizes() == want, "attention module: the shape of ", name, " must be ", want, ", got ", t.sizes());
  };
  auto linear = [&](const Tensor& w, const optional<Tensor>& b, int64_t out, const char* name) {
    shape(w, {out, C}, name);
    if (b.has_value()) shape(*b, {out}, name);
  };
  linear(w_qkv, b_qkv, 3 * C, "qkv");
  linear(w_gate, b_gate, 2 * heads, "gate");
  TORCH_CHECK(w_proj.dim() == 2, "attention module: the shape of proj must be [out,C]");
  linear(w_proj, b_proj, w_proj.size(0), "proj");
  for (const auto* w : norms) {
    TORCH_CHECK(w->has_value() == (*norms.begin())->has_value(), "attention module: q_norm and k_norm come together or not at all");
    if (w->has_value()) shape(**w, {d}, "norm parameter");
  }
  if (pos.has_value()) {
    shape(*pos, {B, N, 2}, "xpos");
    TORCH_CHECK(cos.has_value() && sin.has_value() && cos->dim() == 2, "attention module: positions need the cos/sin tables");
    shape(*cos, {cos->size(0), d / 2}, "cos");
    shape(*sin, cos->sizes(), "sin");
  }
  TORCH_CHECK(x.is_cuda(), "x must be a CUDA tensor: the speed3r_b200 kernels have no CPU path");
  TORCH_CHECK(!pos.has_value() || pos->device() == x.device(), "xpos must be on ", x.device());
  if (pos.has_value()) {
    need(*cos, "cos");
    need(*sin, "sin");
  }
}

// The whole attention module without gradients: projections (cuBLAS), prologue, the two attentions, output projection.
// fp32 input and parameters are rounded to bf16 as under autocast, all in one launch, with the weights of qkv and gate side
// by side so that one GEMM does both; everything between the GEMMs lives in one allocation and goes straight to the C ABI:
// at 2048 tokens the call is bound by host work (388 us at first, 178 with an operator for every step, 105 so).
std::tuple<Tensor, Tensor> module_infer(const Tensor& x_, const Tensor& w_qkv, const optional<Tensor>& b_qkv, const Tensor& w_gate,
                                        const optional<Tensor>& b_gate, const Tensor& w_proj, const optional<Tensor>& b_proj,
                                        const optional<Tensor>& pos_, const optional<Tensor>& cos, const optional<Tensor>& sin,
                                        const optional<Tensor>& qw_, const optional<Tensor>& qb_, const optional<Tensor>& kw_,
                                        const optional<Tensor>& kb_, double eps, int64_t heads, int64_t block, int64_t topk,
                                        double scale) {
  no_tangents(x_, w_qkv, b_qkv, w_gate, b_gate, w_proj, b_proj, qw_, qb_, kw_, kb_);
  at::AutoDispatchBelowAutograd below;
  c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
  need_module(x_, w_qkv, b_qkv, w_gate, b_gate, w_proj, b_proj, pos_, cos, sin, {&qw_, &qb_, &kw_, &kb_}, heads, block);
  c10::cuda::CUDAGuard guard(x_.device());
  void* st = stream();
  const int64_t B = x_.size(0), N = x_.size(1), C = x_.size(2), H = heads, d = C / heads, M = B * N, Nc = N / block;
  auto as = [&](const optional<Tensor>& t, at::ScalarType type) {
    return t.has_value() ? optional<Tensor>(t->to(x_.device(), type).contiguous()) : t;
  };
  const auto pos = as(pos_, at::kLong), qw = aligned(as(qw_, at::kFloat)), qb = aligned(as(qb_, at::kFloat)),
             kw = aligned(as(kw_, at::kFloat)), kb = aligned(as(kb_, at::kFloat));

  // one GEMM for qkv and gate when both weights have to be cast anyway
  const bool merged = w_qkv.scalar_type() == at::kFloat && w_gate.scalar_type() == at::kFloat && H % 4 == 0 &&
                      b_qkv.has_value() == b_gate.has_value();
  const int64_t P = merged ? 3 * C + 2 * H : 3 * C;          // columns of the first projection
  // the allocation, in elements of bf16, every part 256-byte aligned
  int64_t used = 0;
  auto part = [&](int64_t n) {
    const int64_t at = used;
    used += (n + 127) & ~static_cast<int64_t>(127);
    return at;
  };
  struct Cast {
    Tensor from;
    int64_t at;
  };
  std::vector<Cast> casts;
  const bool x_wide = x_.scalar_type() == at::kFloat;
  const int64_t at_x = x_wide ? part(M * C) : 0;
  if (x_wide) casts.push_back({x_.contiguous(), at_x});
  int64_t at_w = 0, at_b = 0;
  if (merged) {
    at_w = part(P * C);
    casts.push_back({w_qkv.contiguous(), at_w});
    casts.push_back({w_gate.contiguous(), at_w + 3 * C * C});
    if (b_qkv.has_value()) {
      at_b = part(P);
      casts.push_back({b_qkv->contiguous(), at_b});
      casts.push_back({b_gate->contiguous(), at_b + 3 * C});
    }
  }
  auto narrow = [&](const Tensor& t) {                       // place of a bf16 copy, -1 where t is bf16 already
    if (t.scalar_type() != at::kFloat) return static_cast<int64_t>(-1);
    const int64_t at = part(t.numel());
    casts.push_back({t.contiguous(), at});
    return at;
  };
  const int64_t at_wp = narrow(w_proj), at_bp = b_proj.has_value() ? narrow(*b_proj) : -1;
  int64_t at_wq = -1, at_bq = -1, at_wg = -1, at_bg = -1;
  if (!merged) {
    at_wq = narrow(w_qkv);
    at_wg = narrow(w_gate);
    if (b_qkv.has_value()) at_bq = narrow(*b_qkv);
    if (b_gate.has_value()) at_bg = narrow(*b_gate);
  }
  const int64_t at_p = part(M * P), at_gl = merged ? 0 : part(M * 2 * H), at_tok = part(0);
  const int64_t tok = (M * C + 127) & ~static_cast<int64_t>(127), pooled = (B * H * Nc * d + 127) & ~static_cast<int64_t>(127);
  part(3 * tok + 4 * pooled);                                // q, k, v, q_c, k_c, v_c, o_c
  const int64_t at_gate = merged ? part(M * 2 * H) : 0, at_y = part(M * C), at_lse = part(2 * B * H * Nc);
  const Tensor buf = at::empty({used}, x_.options().dtype(at::kBFloat16));
  char* base = static_cast<char*>(buf.data_ptr());
  auto ptr = [&](int64_t at) { return static_cast<void*>(base + 2 * at); };
  auto view = [&](int64_t at, int64_t r, int64_t c) { return buf.as_strided({r, c}, {c, 1}, at); };
  if (!casts.empty()) {
    TORCH_CHECK(casts.size() <= 8, "too many tensors to cast");
    const float* src[8];
    void* dst[8];
    int64_t counts[8];
    for (size_t i = 0; i < casts.size(); ++i) {
      src[i] = f32(casts[i].from);
      dst[i] = ptr(casts[i].at);
      counts[i] = casts[i].from.numel();
    }
    check(s3r_cast_bf16(static_cast<int>(casts.size()), src, dst, counts, st), "s3r_cast_bf16");
  }
  auto gemm = [&](Tensor& out, const Tensor& a, const Tensor& w, const optional<Tensor>& bias) {
    if (bias.has_value()) at::addmm_out(out, *bias, a, w.t());
    else at::mm_out(out, a, w.t());
  };
  auto weight = [&](int64_t at, const Tensor& t) { return at >= 0 ? view(at, t.size(0), t.size(1)) : t; };
  auto bias = [&](int64_t at, const optional<Tensor>& t) {
    return t.has_value() && at >= 0 ? optional<Tensor>(buf.as_strided({t->size(0)}, {1}, at)) : t;
  };
  const Tensor x = x_wide ? view(at_x, M, C) : x_.contiguous().view({M, C});
  Tensor proj = view(at_p, M, P), gate_logits;
  if (merged) {
    gemm(proj, x, view(at_w, P, C), b_qkv.has_value() ? optional<Tensor>(buf.as_strided({P}, {1}, at_b)) : optional<Tensor>());
  } else {
    gemm(proj, x, weight(at_wq, w_qkv), bias(at_bq, b_qkv));
    gate_logits = view(at_gl, M, 2 * H);
    gemm(gate_logits, x, weight(at_wg, w_gate), bias(at_bg, b_gate));
    gate_logits.sigmoid_();
  }
  const int64_t rows = pos.has_value() ? cos->size(0) : 0;
  const void *cp = pos.has_value() ? cos->data_ptr() : nullptr, *sp = pos.has_value() ? sin->data_ptr() : nullptr;
  const int64_t* pp = static_cast<const int64_t*>(ptr_or_null(pos));
  void* t[7];                                                // q, k, v, q_c, k_c, v_c, o_c
  for (int i = 0; i < 7; ++i) t[i] = ptr(at_tok + (i < 3 ? i * tok : 3 * tok + (i - 3) * pooled));
  if (merged)
    check(s3r_qkv_gate_prologue_fwd(ptr(at_p), pp, cp, sp, rows, f32_or_null(qw), f32_or_null(qb), f32_or_null(kw), f32_or_null(kb),
                                    eps, t[0], t[1], t[2], t[3], t[4], t[5], ptr(at_gate), B, H, N, d, block, st),
          "s3r_qkv_gate_prologue_fwd");
  else
    check(s3r_qkv_prologue_fwd(ptr(at_p), pp, cp, sp, rows, f32_or_null(qw), f32_or_null(qb), f32_or_null(kw), f32_or_null(kb), eps,
                               t[0], t[1], t[2], t[3], t[4], t[5], B, H, N, d, block, st), "s3r_qkv_prologue_fwd");
  const Tensor idx = at::empty({B, H, Nc, topk}, x_.options().dtype(at::kInt));
  check(s3r_cmp_attn_topk_fwd(t[3], t[4], t[5], t[6], static_cast<float*>(ptr(at_lse)), i32m(idx), B, H, Nc, Nc, d, topk, scale, st),
        "s3r_cmp_attn_topk_fwd");
  // gate [B,H,N,2] from the prologue, or a view of the [B,N,H,2] logits
  check(s3r_sel_attn_fwd(t[0], t[1], t[2], 1, 0, i32(idx), nullptr, nullptr, merged ? ptr(at_gate) : ptr(at_gl),
                         merged ? H * N * 2 : N * H * 2, merged ? N * 2 : 2, merged ? 2 : H * 2, t[6], ptr(at_y), B, H, N, N, d, block,
                         topk, scale, st), "s3r_sel_attn_fwd");
  Tensor out = at::empty({M, w_proj.size(0)}, x_.options().dtype(at::kBFloat16));
  gemm(out, view(at_y, M, C), weight(at_wp, w_proj), bias(at_bp, b_proj));
  return {out.view({B, N, w_proj.size(0)}), idx};
}

// The module with gradients as one node, for fp32 parameters under bf16 autocast.  The forward is that of module_infer (one
// cast, one GEMM for qkv and gate) and keeps its one allocation for the backward; the backward runs the GEMMs with fp32
// results where a parameter or input is fp32 (nothing is rounded to bf16 and cast back) and everything between them
// through the C ABI.  As separate nodes a step at 2 x 6144 tokens enqueued for 1.1 ms, as long as the GPU worked on it.
struct ModulePlan {                                          // places in the forward's allocation, elements of bf16
  int64_t B, N, C, H, d, M, P, Nc, topk, block, used = 0;
  int64_t x, w, b, wp, bp, proj, tok, pooled, t0, gate, y, o_s, lse_c, lse_s;
  int64_t part(int64_t n) {
    const int64_t at = used;
    used += (n + 127) & ~static_cast<int64_t>(127);
    return at;
  }
  ModulePlan(at::IntArrayRef shape, int64_t heads, int64_t block_, int64_t topk_, bool x_wide, int64_t out_features)
      : B(shape[0]), N(shape[1]), C(shape[2]), H(heads), d(shape[2] / heads), M(B * N), P(3 * C + 2 * H), Nc(N / block_), topk(topk_),
        block(block_) {
    x = x_wide ? part(M * C) : -1;
    w = part(P * C);
    b = part(P);
    wp = part(out_features * C);
    bp = part(out_features);
    proj = part(M * P);
    tok = (M * C + 127) & ~static_cast<int64_t>(127);
    pooled = (B * H * Nc * d + 127) & ~static_cast<int64_t>(127);
    t0 = part(3 * tok + 4 * pooled);                         // q, k, v, q_c, k_c, v_c, o_c
    gate = part(M * 2 * H);
    y = part(M * C);
    o_s = part(M * C);
    lse_c = part(2 * B * H * Nc);
    lse_s = part(2 * M * H);
  }
  int64_t t(int i) const { return t0 + (i < 3 ? i * tok : 3 * tok + (i - 3) * pooled); }
};

struct ModuleNode : torch::autograd::Function<ModuleNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x_, const Tensor& w_qkv, const optional<Tensor>& b_qkv,
                               const Tensor& w_gate, const optional<Tensor>& b_gate, const Tensor& w_proj,
                               const optional<Tensor>& b_proj, const optional<Tensor>& pos, const optional<Tensor>& cos,
                               const optional<Tensor>& sin, const optional<Tensor>& qw_, const optional<Tensor>& qb_,
                               const optional<Tensor>& kw_, const optional<Tensor>& kb_, double eps, int64_t heads, int64_t block,
                               int64_t topk, double scale) {
    at::AutoDispatchBelowAutograd below;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    c10::cuda::CUDAGuard guard(x_.device());
    void* st = stream();
    const auto qw = aligned(qw_), qb = aligned(qb_), kw = aligned(kw_), kb = aligned(kb_);
    const bool x_wide = x_.scalar_type() == at::kFloat;
    const ModulePlan m(x_.sizes(), heads, block, topk, x_wide, w_proj.size(0));
    const Tensor buf = at::empty({m.used}, x_.options().dtype(at::kBFloat16)), x = x_.contiguous();
    char* base = static_cast<char*>(buf.data_ptr());
    auto ptr = [&](int64_t at) { return static_cast<void*>(base + 2 * at); };
    auto view = [&](int64_t at, int64_t r, int64_t c) { return buf.as_strided({r, c}, {c, 1}, at); };
    std::vector<Tensor> keep;
    const float* src[8];
    void* dst[8];
    int64_t counts[8];
    int n = 0;
    auto cast = [&](const Tensor& t, int64_t at) {
      need(t, "parameter", at::kFloat, false);
      keep.push_back(t.contiguous());
      src[n] = f32(keep.back());
      dst[n] = ptr(at);
      counts[n++] = t.numel();
    };
    if (x_wide) cast(x, m.x);
    cast(w_qkv, m.w);
    cast(w_gate, m.w + 3 * m.C * m.C);
    if (b_qkv.has_value()) {
      cast(*b_qkv, m.b);
      cast(*b_gate, m.b + 3 * m.C);
    }
    cast(w_proj, m.wp);
    if (b_proj.has_value()) cast(*b_proj, m.bp);
    check(s3r_cast_bf16(n, src, dst, counts, st), "s3r_cast_bf16");
    auto gemm = [&](Tensor out, const Tensor& a, const Tensor& w, bool bias, int64_t at_bias) {
      if (bias) at::addmm_out(out, buf.as_strided({w.size(0)}, {1}, at_bias), a, w.t());
      else at::mm_out(out, a, w.t());
    };
    gemm(view(m.proj, m.M, m.P), x_wide ? view(m.x, m.M, m.C) : x.view({m.M, m.C}), view(m.w, m.P, m.C), b_qkv.has_value(), m.b);
    const int64_t rows = pos.has_value() ? cos->size(0) : 0;
    check(s3r_qkv_gate_prologue_fwd(ptr(m.proj), static_cast<const int64_t*>(ptr_or_null(pos)), pos.has_value() ? cos->data_ptr() : nullptr,
                                    pos.has_value() ? sin->data_ptr() : nullptr, rows, f32_or_null(qw), f32_or_null(qb), f32_or_null(kw),
                                    f32_or_null(kb), eps, ptr(m.t(0)), ptr(m.t(1)), ptr(m.t(2)), ptr(m.t(3)), ptr(m.t(4)), ptr(m.t(5)),
                                    ptr(m.gate), m.B, m.H, m.N, m.d, block, st), "s3r_qkv_gate_prologue_fwd");
    const Tensor idx = at::empty({m.B, m.H, m.Nc, topk}, x_.options().dtype(at::kInt));
    check(s3r_cmp_attn_topk_fwd(ptr(m.t(3)), ptr(m.t(4)), ptr(m.t(5)), ptr(m.t(6)), static_cast<float*>(ptr(m.lse_c)), i32m(idx), m.B,
                                m.H, m.Nc, m.Nc, m.d, topk, scale, st), "s3r_cmp_attn_topk_fwd");
    check(s3r_sel_attn_fwd(ptr(m.t(0)), ptr(m.t(1)), ptr(m.t(2)), 1, 0, i32(idx), ptr(m.o_s), static_cast<float*>(ptr(m.lse_s)), ptr(m.gate),
                           m.H * m.N * 2, m.N * 2, 2, ptr(m.t(6)), ptr(m.y), m.B, m.H, m.N, m.N, m.d, block, topk, scale, st),
          "s3r_sel_attn_fwd");
    Tensor out = at::empty({m.M, w_proj.size(0)}, x_.options().dtype(at::kBFloat16));
    gemm(out, view(m.y, m.M, m.C), view(m.wp, w_proj.size(0), m.C), b_proj.has_value(), m.bp);

    auto or_none = [](const optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); };
    ctx->save_for_backward({buf, x_wide ? Tensor() : x, idx, or_none(pos), or_none(cos), or_none(sin), or_none(qw_), or_none(kw_)});
    ctx->saved_data["shape"] = x_.sizes().vec();
    ctx->saved_data["ints"] = std::vector<int64_t>{heads, block, topk, w_proj.size(0), b_qkv.has_value(), b_proj.has_value()};
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["scale"] = scale;
    ctx->mark_non_differentiable({idx});
    ctx->set_materialize_grads(false);      // no zeros for the table
    return {out.view({m.B, m.N, w_proj.size(0)}), idx};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    if (!g[0].defined()) return variable_list(19);
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    const auto s = ctx->get_saved_variables();
    const Tensor &buf = s[0], &idx = s[2];
    const auto shape = ctx->saved_data["shape"].toIntVector(), ints = ctx->saved_data["ints"].toIntVector();
    const double eps = ctx->saved_data["eps"].toDouble(), scale = ctx->saved_data["scale"].toDouble();
    const int64_t out_features = ints[3];
    const bool x_wide = !s[1].defined(), rope = s[3].defined(), norm = s[6].defined();
    const Tensor qw = norm ? aligned(s[6]) : s[6], kw = norm ? aligned(s[7]) : s[7];
    const ModulePlan m(shape, ints[0], ints[1], ints[2], x_wide, out_features);
    const size_t e_gate = ints[4] ? 3 : 2, e_wp = e_gate + (ints[4] ? 2 : 1);      // edges: absent biases have none
    c10::cuda::CUDAGuard guard(buf.device());
    void* st = stream();
    char* base = static_cast<char*>(buf.data_ptr());
    auto ptr = [&](int64_t at) { return static_cast<void*>(base + 2 * at); };
    auto view = [&](int64_t at, int64_t r, int64_t c) { return buf.as_strided({r, c}, {c, 1}, at); };
    const Tensor dy = aligned(g[0].to(at::kBFloat16).contiguous()).view({m.M, out_features});

    // the output projection's own gradients; is anything before it wanted?
    auto colsum = [&](const void* x, int64_t cols, void* ws, size_t bytes) {
      Tensor o = at::empty({cols}, buf.options().dtype(at::kFloat));
      check(s3r_colsum(x, f32(o), m.M, cols, ws, bytes, st), "s3r_colsum");
      return o;
    };
    Tensor dwp, dbp;
    auto output_projection = [&]() {
      if (ctx->needs_input_grad(e_wp)) dwp = at::mm(dy.t(), view(m.y, m.M, m.C), at::kFloat);
      if (!ints[5] || !ctx->needs_input_grad(e_wp + 1)) return;
      if (out_features % 8 == 0) {
        const Tensor ws = fresh({static_cast<int64_t>(s3r_colsum_workspace_bytes(m.M, out_features))}, buf, at::kByte);
        dbp = colsum(dy.data_ptr(), out_features, ws.data_ptr(), ws.numel());
      } else {
        dbp = dy.sum(0, false, at::kFloat);                  // the kernel reads rows of whole vectors
      }
    };
    const size_t e_norm = e_wp + (ints[5] ? 2 : 1) + (rope ? 3 : 0);
    bool before = false;
    for (size_t e = 0; e < e_wp; ++e) before |= ctx->needs_input_grad(e);
    for (size_t e = e_norm; norm && e < e_norm + 4; ++e) before |= ctx->needs_input_grad(e);
    if (!before) {
      output_projection();
      variable_list out(19);
      out[5] = dwp;
      out[6] = dbp;
      return out;
    }

    // scratch of the backward, bytes
    int64_t used = 0;
    auto part = [&](int64_t bytes) {
      const int64_t at = used;
      used += (bytes + 255) & ~static_cast<int64_t>(255);
      return at;
    };
    const int64_t BH = m.B * m.H, tok = 2 * m.M * m.C, pooled = 2 * BH * m.Nc * m.d;
    const int64_t a_dy = part(tok), a_dos = part(tok), a_dq = part(tok), a_dk = part(tok), a_dv = part(tok), a_doc = part(pooled),
                  a_dqc = part(pooled), a_dkc = part(pooled), a_dvc = part(pooled), a_delc = part(4 * BH * m.Nc), a_dgate = part(8 * m.M * m.H),
                  a_dels = part(4 * m.M * m.H), a_dproj = part(2 * m.M * m.P), a_off = part(4 * BH * (m.Nc + 1)),
                  a_qids = part(4 * BH * m.Nc * m.topk);
    const size_t csr_bytes = s3r_csr_workspace_bytes(m.B, m.H, m.Nc, m.topk, m.Nc),
                 pro_bytes = norm ? s3r_qkv_prologue_bwd_workspace_bytes(m.B, m.H, m.N, m.block) : 0,
                 col_bytes = s3r_colsum_workspace_bytes(m.M, m.P);
    const int64_t a_csr = part(csr_bytes), a_pro = part(pro_bytes), a_col = part(col_bytes);
    const Tensor scratch = at::empty({used / 2}, buf.options());
    char* sb = static_cast<char*>(scratch.data_ptr());
    auto sp = [&](int64_t at) { return static_cast<void*>(sb + at); };
    auto sf = [&](int64_t at) { return reinterpret_cast<float*>(sb + at); };
    auto sview = [&](int64_t at, int64_t r, int64_t c) { return scratch.as_strided({r, c}, {c, 1}, at / 2); };

    int32_t *off = static_cast<int32_t*>(sp(a_off)), *qids = static_cast<int32_t*>(sp(a_qids));
    CsrBeside beside(i32(idx), off, qids, m.B, m.H, m.Nc, m.topk, m.Nc, sp(a_csr), csr_bytes);
    Tensor dya = sview(a_dy, m.M, m.C);
    at::mm_out(dya, dy, view(m.wp, out_features, m.C));
    output_projection();
    // merge, the two branches, prologue
    check(s3r_merge_bwd_deltas(sp(a_dy), ptr(m.gate), m.H * m.N * 2, m.N * 2, 2, ptr(m.t(6)), ptr(m.o_s), sp(a_dos), sf(a_dgate),
                               sp(a_doc), sf(a_dels), sf(a_delc), m.B, m.H, m.N, m.d, m.block, st), "s3r_merge_bwd");
    check(s3r_cmp_attn_bwd_delta(ptr(m.t(3)), ptr(m.t(4)), ptr(m.t(5)), static_cast<float*>(ptr(m.lse_c)), sp(a_doc), sf(a_delc),
                                 sp(a_dqc), sp(a_dkc), sp(a_dvc), m.B, m.H, m.Nc, m.Nc, m.d, scale, st), "s3r_cmp_attn_bwd_delta");
    beside.join();
    check(s3r_sel_attn_bwd(ptr(m.t(0)), ptr(m.t(1)), ptr(m.t(2)), i32(idx), off, qids, static_cast<float*>(ptr(m.lse_s)), sf(a_dels),
                           sp(a_dos), sp(a_dq), sp(a_dk), sp(a_dv), m.B, m.H, m.N, m.N, m.d, m.block, m.topk, scale, st),
          "s3r_sel_attn_bwd");
    const Tensor dparams = at::empty({norm ? 4 : 0, m.d}, buf.options().dtype(at::kFloat));
    check(s3r_qkv_gate_prologue_bwd(ptr(m.proj), rope ? static_cast<const int64_t*>(s[3].data_ptr()) : nullptr,
                                    rope ? s[4].data_ptr() : nullptr, rope ? s[5].data_ptr() : nullptr, rope ? s[4].size(0) : 0,
                                    norm ? f32(qw) : nullptr, norm ? f32(kw) : nullptr, eps, sp(a_dq), sp(a_dk), sp(a_dv), sp(a_dqc),
                                    sp(a_dkc), sp(a_dvc), ptr(m.gate), sf(a_dgate), sp(a_dproj), norm ? f32(dparams) : nullptr, sp(a_pro),
                                    pro_bytes, m.B, m.H, m.N, m.d, m.block, st), "s3r_qkv_gate_prologue_bwd");
    // first projection
    const Tensor dproj = sview(a_dproj, m.M, m.P);
    Tensor dx, dw_qkv, dw_gate, db_qkv, db_gate;
    if (ctx->needs_input_grad(0)) {
      const Tensor w = view(m.w, m.P, m.C);
      dx = (x_wide ? at::mm(dproj, w, at::kFloat) : at::mm(dproj, w)).view(shape);
    }
    if (ctx->needs_input_grad(1) || ctx->needs_input_grad(e_gate)) {
      const Tensor dw = at::mm(dproj.t(), x_wide ? view(m.x, m.M, m.C) : s[1].view({m.M, m.C}), at::kFloat);
      dw_qkv = dw.narrow(0, 0, 3 * m.C);
      dw_gate = dw.narrow(0, 3 * m.C, 2 * m.H);
    }
    if (ints[4] && (ctx->needs_input_grad(2) || ctx->needs_input_grad(e_gate + 1))) {
      const Tensor db = colsum(sp(a_dproj), m.P, sp(a_col), col_bytes);
      db_qkv = db.narrow(0, 0, 3 * m.C);
      db_gate = db.narrow(0, 3 * m.C, 2 * m.H);
    }
    auto param = [&](int i) { return norm ? dparams.select(0, i) : Tensor(); };
    return {dx, dw_qkv, db_qkv, dw_gate, db_gate, dwp, dbp, Tensor(), Tensor(), Tensor(), param(0), param(1), param(2), param(3),
            Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
std::tuple<Tensor, Tensor> module_train(const Tensor& x, const Tensor& w_qkv, const optional<Tensor>& b_qkv, const Tensor& w_gate,
                                        const optional<Tensor>& b_gate, const Tensor& w_proj, const optional<Tensor>& b_proj,
                                        const optional<Tensor>& pos_, const optional<Tensor>& cos, const optional<Tensor>& sin,
                                        const optional<Tensor>& qw_, const optional<Tensor>& qb_, const optional<Tensor>& kw_,
                                        const optional<Tensor>& kb_, double eps, int64_t heads, int64_t block, int64_t topk,
                                        double scale) {
  no_tangents(x, w_qkv, b_qkv, w_gate, b_gate, w_proj, b_proj, qw_, qb_, kw_, kb_);
  need_module(x, w_qkv, b_qkv, w_gate, b_gate, w_proj, b_proj, pos_, cos, sin, {&qw_, &qb_, &kw_, &kb_}, heads, block);
  TORCH_CHECK(heads % 4 == 0 && b_qkv.has_value() == b_gate.has_value(), "module_train: heads in fours, and biases of qkv and gate together");
  auto as = [&](const optional<Tensor>& t, at::ScalarType type) {
    return t.has_value() ? optional<Tensor>(t->to(x.device(), type).contiguous()) : t;
  };
  const auto pos = as(pos_, at::kLong);
  const auto r = ModuleNode::apply(x, w_qkv, b_qkv, w_gate, b_gate, w_proj, b_proj, pos, cos, sin, as(qw_, at::kFloat), as(qb_, at::kFloat),
                                   as(kw_, at::kFloat), as(kb_, at::kFloat), eps, heads, block, topk, scale);
  return {r[0], r[1]};
}

// Tells the pinned-memory allocator that the current stream of `device` works on `host`: what Tensor.copy_ does, and a copy on
// raw pointers does not.  The memory is not handed out again before the work enqueued so far is done.
void host_in_use(const Tensor& host, at::Device device) {
  TORCH_CHECK(host.device().is_cpu() && device.is_cuda(), "host_in_use: a host tensor and a CUDA device");
  c10::cuda::CUDAGuard guard(device);
  at::getHostAllocator(at::kCUDA)->record_event(host.data_ptr(), host.storage().data_ptr().get_context(), c10::cuda::getCurrentCUDAStream(device.index()));
}

// a tensor with memory, not one of those that a tracer runs the backward on
bool plain(const Tensor& t) {
  return t.is_cuda() && !t.key_set().has(c10::DispatchKey::Python) && !t.key_set().has(c10::DispatchKey::Functionalize) &&
         !c10::impl::dispatch_mode_enabled();
}

// The whole op.  group = 0 where compressed keys are the selection blocks.  As one node its backward adds the
// pooled branch's gradients inside the selection kernels' stores: separate nodes write them out as [B,H,T,d] and add
// two bf16 tensors three times (1.5 of 19.4 ms at 250 views).
struct SparseNode : torch::autograd::Function<SparseNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                               int64_t block, int64_t topk, int64_t kernel, int64_t stride, double scale, int64_t group,
                               int64_t take) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [q_c, k_c, v_c] = call_pool_qkv(q, k, v, block, kernel, stride);
    auto [o_c, lse_c, idx] = call_cmp(q_c, k_c, v_c, topk, scale, group, take);
    auto [o_s, lse_s, y] = call_sel(q, k, v, idx, gate, o_c, block, scale, true, true, 1);
    ctx->save_for_backward({q, k, v, gate, q_c, k_c, v_c, o_c, lse_c, idx, o_s, lse_s});
    ctx->saved_data["block"] = block;
    ctx->saved_data["kernel"] = kernel;
    ctx->saved_data["stride"] = stride;
    ctx->saved_data["scale"] = scale;
    ctx->mark_non_differentiable({idx});
    ctx->set_materialize_grads(false);      // no zeros for the table
    return {y, idx};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return once(g, [&] { return gradients(ctx, g); });
  }
  static variable_list gradients(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const int64_t block = ctx->saved_data["block"].toInt();
    const double scale = ctx->saved_data["scale"].toDouble();
    if (!g[0].defined()) return variable_list(11);
    if (!ctx->needs_input_grad(0) && !ctx->needs_input_grad(1) && !ctx->needs_input_grad(2)) {          // the gate alone
      variable_list out(11);
      out[3] = std::get<1>(call_merge_bwd(g[0].contiguous(), s[3], s[7], s[10], block)).to(s[3].scalar_type());
      return out;
    }
    if (plain(s[0]) && plain(g[0])) {
      c10::cuda::CUDAGuard guard(s[0].device());
      const Tensor& idx = s[9];
      const int64_t B = idx.size(0), H = idx.size(1), Nq = idx.size(2), K = idx.size(3), nkb = (s[1].size(2) + block - 1) / block;
      const size_t nbytes = s3r_csr_workspace_bytes(B, H, Nq, K, nkb);
      const std::tuple<Tensor, Tensor> inverse(fresh({B, H, nkb + 1}, idx, at::kInt), fresh({B, H, Nq * K}, idx, at::kInt));
      const Tensor ws = fresh({static_cast<int64_t>(nbytes)}, idx, at::kByte);
      CsrBeside beside(i32(idx), i32m(std::get<0>(inverse)), i32m(std::get<1>(inverse)), B, H, Nq, K, nkb, ws.data_ptr(), nbytes);
      Tensor dlt_c;
      auto [do_s, dgate, do_c, dlt] = merge_bwd_deltas(g[0].contiguous(), s[3], s[7], s[10], block, &dlt_c);
      auto [dq_c, dk_c, dv_c] = cmp_bwd(s[4], s[5], s[6], s[7], s[8], do_c, scale, &dlt_c);
      beside.join();
      auto [dq, dk, dv] = sel_bwd(s[0], s[1], s[2], idx, s[11], dlt, do_s, &dq_c, &dk_c, &dv_c, block,
                                  ctx->saved_data["kernel"].toInt(), ctx->saved_data["stride"].toInt(), scale, &inverse);
      return {dq, dk, dv, dgate.to(s[3].scalar_type()), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
    auto [do_s, dgate, do_c, dlt] = call_merge_bwd(g[0].contiguous(), s[3], s[7], s[10], block);
    auto [dq_c, dk_c, dv_c] = call_cmp_bwd(s[4], s[5], s[6], s[7], s[8], do_c, scale);
    auto [dq, dk, dv] = call_sel_bwd_pooled(s[0], s[1], s[2], s[9], s[11], dlt, do_s, dq_c, dk_c, dv_c, block,
                                            ctx->saved_data["kernel"].toInt(), ctx->saved_data["stride"].toInt(), scale);
    return {dq, dk, dv, dgate.to(s[3].scalar_type()), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
std::tuple<Tensor, Tensor> sparse_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                                            int64_t block, int64_t topk, int64_t kernel, int64_t stride, double scale,
                                            int64_t group, int64_t take) {
  if (wants_grad(q, k, v, gate)) {
    const auto r = SparseNode::apply(q, k, v, gate, block, topk, kernel, stride, scale, group, take);
    return {r[0], r[1]};
  }
  auto [q_c, k_c, v_c] = call_pool_qkv(q, k, v, block, kernel, stride);
  auto [o_c, lse, idx] = call_cmp(q_c, k_c, v_c, topk, scale, group, take);
  return {std::get<2>(call_sel(q, k, v, idx, gate, o_c, block, scale, false, false, 1)), idx};
}

}  // namespace

TORCH_LIBRARY(speed3r_b200, m) {
  m.def("pool_fwd(Tensor x, int kernel, int stride) -> Tensor");
  m.def("pool_bwd(Tensor d_out, int T, int kernel, int stride) -> Tensor");
  m.def("cmp_attn_topk_fwd(Tensor q_c, Tensor k_c, Tensor v_c, int topk, float scale) -> (Tensor, Tensor, Tensor)");
  m.def("cmp_attn_blocktopk_fwd(Tensor q_c, Tensor k_c, Tensor v_c, int topk, float scale, int group, int take) -> "
        "(Tensor, Tensor, Tensor)");
  m.def("cmp_attn_bwd(Tensor q_c, Tensor k_c, Tensor v_c, Tensor o_c, Tensor lse, Tensor do_c, float scale) -> "
        "(Tensor, Tensor, Tensor)");
  m.def("sel_attn_fwd(Tensor q, Tensor k, Tensor v, Tensor idx, Tensor? gate, Tensor? o_c, int block, float scale, "
        "bool want_o, bool want_lse, int kv_chunks) -> (Tensor, Tensor, Tensor)");
  m.def("build_key_csr(Tensor idx, int num_key_blocks) -> (Tensor, Tensor)");
  m.def("sel_attn_bwd(Tensor q, Tensor k, Tensor v, Tensor idx, Tensor lse, Tensor delta, Tensor do_s, int block, "
        "float scale) -> (Tensor, Tensor, Tensor)");
  m.def("sel_attn_bwd_pooled(Tensor q, Tensor k, Tensor v, Tensor idx, Tensor lse, Tensor delta, Tensor do_s, Tensor dq_c, "
        "Tensor dk_c, Tensor dv_c, int block, int kernel, int stride, float scale) -> (Tensor, Tensor, Tensor)");
  m.def("pool_qkv_fwd(Tensor q, Tensor k, Tensor v, int block, int kernel, int stride) -> (Tensor, Tensor, Tensor)");
  m.def("delta(Tensor o, Tensor d_o) -> Tensor");
  m.def("merge_bwd(Tensor dy, Tensor gate, Tensor o_c, Tensor o_s, int block) -> (Tensor, Tensor, Tensor, Tensor)");
  m.def("prologue_fwd(Tensor qkv, int heads, int block, Tensor? pos, Tensor? cos, Tensor? sin, Tensor? qw, Tensor? qb, "
        "Tensor? kw, Tensor? kb, float eps) -> (Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)");
  m.def("prologue_bwd(Tensor qkv, int heads, int block, Tensor? pos, Tensor? cos, Tensor? sin, Tensor? qw, Tensor? kw, "
        "float eps, Tensor dq, Tensor dk, Tensor dv, Tensor dq_c, Tensor dk_c, Tensor dv_c) -> (Tensor, Tensor)");

  m.def("prologue(Tensor qkv, int heads, int block, Tensor? pos, Tensor? cos, Tensor? sin, Tensor? qw, Tensor? qb, "
        "Tensor? kw, Tensor? kb, float eps) -> (Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)", &prologue);
  m.def("module_infer(Tensor x, Tensor w_qkv, Tensor? b_qkv, Tensor w_gate, Tensor? b_gate, Tensor w_proj, Tensor? b_proj, "
        "Tensor? pos, Tensor? cos, Tensor? sin, Tensor? qw, Tensor? qb, Tensor? kw, Tensor? kb, float eps, int heads, "
        "int block, int topk, float scale) -> (Tensor, Tensor)", &module_infer);
  m.def("module_train(Tensor x, Tensor w_qkv, Tensor? b_qkv, Tensor w_gate, Tensor? b_gate, Tensor w_proj, Tensor? b_proj, "
        "Tensor? pos, Tensor? cos, Tensor? sin, Tensor? qw, Tensor? qb, Tensor? kw, Tensor? kb, float eps, int heads, "
        "int block, int topk, float scale) -> (Tensor, Tensor)", &module_train);
  m.def("host_in_use(Tensor host, Device device) -> ()", &host_in_use);
  m.def("pool_tokens(Tensor x, int kernel, int stride) -> Tensor", &pool_tokens);
  m.def("flash_attn_topk(Tensor q, Tensor k, Tensor v, int topk, float scale, int group, int take) -> (Tensor, Tensor)",
        &flash_attn_topk);
  m.def("topk_blocksparse(Tensor q, Tensor k, Tensor v, Tensor idx, int block, float scale) -> Tensor", &topk_blocksparse);
  m.def("sel_merge(Tensor q, Tensor k, Tensor v, Tensor idx, Tensor gate, Tensor o_c, int block, float scale) -> Tensor",
        &sel_merge);
  m.def("sparse_attention(Tensor q, Tensor k, Tensor v, Tensor gate, int block, int topk, int kernel, int stride, "
        "float scale, int group, int take) -> (Tensor, Tensor)", &sparse_attention);
}

#define S3R_BASE_OPS(m)                                     \
  m.impl("pool_fwd", &pool_fwd);                            \
  m.impl("pool_bwd", &pool_bwd);                            \
  m.impl("cmp_attn_topk_fwd", &cmp_attn_topk_fwd);          \
  m.impl("cmp_attn_blocktopk_fwd", &cmp_attn_blocktopk_fwd); \
  m.impl("cmp_attn_bwd", &cmp_attn_bwd);                    \
  m.impl("sel_attn_fwd", &sel_attn_fwd);                    \
  m.impl("build_key_csr", &build_key_csr);                  \
  m.impl("sel_attn_bwd", &sel_attn_bwd);                    \
  m.impl("sel_attn_bwd_pooled", &sel_attn_bwd_pooled);      \
  m.impl("pool_qkv_fwd", &pool_qkv_fwd);                    \
  m.impl("prologue_fwd", &prologue_fwd);                    \
  m.impl("prologue_bwd", &prologue_bwd);                    \
  m.impl("delta", &delta);                                  \
  m.impl("merge_bwd", &merge_bwd)

TORCH_LIBRARY_IMPL(speed3r_b200, CUDA, m) { S3R_BASE_OPS(m); }
TORCH_LIBRARY_IMPL(speed3r_b200, CPU, m) { S3R_BASE_OPS(m); }      // every one of them refuses CPU tensors
