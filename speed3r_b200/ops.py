"""The package's operators over the C-ABI kernels.

Public functions mirror the reference's op signatures:

* ``flash_attn_topk_func(q_c, k_c, v_c, topk_val, bias=None, causal=False, softmax_scale=None)``
  -> ``(o_c, idx)``      (pi3/models/sparse_attn/flash_attention_topk.py:633-668)
* ``topk_blocksparse_attention(q, k, v, topk_idx, block_size, softmax_scale=None)`` -> ``o``
  (pi3/models/sparse_attn/topk_blocksparse_attention.py:1093-1121)

plus the pieces the reference leaves to eager PyTorch (sparse_attention.py:97-102, 127-136):

* ``pool_tokens(x, kernel, stride)``: mean pooling along the sequence
* ``sel_attn_merge(q, k, v, idx, gate, o_c, block_size)``: selection attention with the gated
  merge fused, returning ``[B,T,H*d]``

Allocation, argument checks and autograd wiring are native (``csrc/torch/bindings.cpp``, a ``torch.library``
namespace over the C ABI); this file holds the Python signatures and the shape functions for
``torch.compile``.  CPU tensors, fp32/fp16 inputs and a missing library raise: there is no fallback.
"""
from __future__ import annotations

import math
import threading
from typing import Optional, Tuple

import torch
from torch import Tensor

from . import _lib

_BF16 = torch.bfloat16
_lock = threading.Lock()
_ns = None


def _register_fakes() -> None:
    fake = torch.library.register_fake

    @fake("speed3r_b200::pool_fwd")
    def _(x, kernel, stride):
        B, H, T, d = x.shape
        return x.new_empty(B, H, (T - kernel) // stride + 1, d)

    @fake("speed3r_b200::pool_bwd")
    def _(d_out, T, kernel, stride):
        B, H, Nc, d = d_out.shape
        return d_out.new_empty(B, H, T, d)

    def cmp_fwd(q_c, k_c, v_c, topk, scale, group=0, take=0):
        B, H, Nq, d = q_c.shape
        return (q_c.new_empty(B, H, Nq, d), q_c.new_empty(B, H, Nq, dtype=torch.float32),
                q_c.new_empty(B, H, Nq, topk, dtype=torch.int32))

    fake("speed3r_b200::cmp_attn_topk_fwd", cmp_fwd)
    fake("speed3r_b200::cmp_attn_blocktopk_fwd", cmp_fwd)

    @fake("speed3r_b200::cmp_attn_bwd")
    def _(q_c, k_c, v_c, o_c, lse, do_c, scale):
        return tuple(t.new_empty(t.shape) for t in (q_c, k_c, v_c))

    @fake("speed3r_b200::sel_attn_fwd")
    def _(q, k, v, idx, gate, o_c, block, scale, want_o, want_lse, kv_chunks):
        B, H, Tq, d = q.shape
        return (q.new_empty(B, H, Tq, d) if want_o else q.new_empty(0),
                q.new_empty(B, H, Tq, dtype=torch.float32) if want_lse else q.new_empty(0, dtype=torch.float32),
                q.new_empty(B, Tq, H * d) if gate is not None else q.new_empty(0))

    @fake("speed3r_b200::build_key_csr")
    def _(idx, num_key_blocks):
        B, H, Nq, K = idx.shape
        return idx.new_empty(B, H, num_key_blocks + 1), idx.new_empty(B, H, Nq * K)

    @fake("speed3r_b200::sel_attn_bwd")
    def _(q, k, v, idx, lse, delta, do_s, block, scale):
        return tuple(t.new_empty(t.shape) for t in (q, k, v))

    @fake("speed3r_b200::sel_attn_bwd_pooled")
    def _(q, k, v, idx, lse, delta, do_s, dq_c, dk_c, dv_c, block, kernel, stride, scale):
        return tuple(t.new_empty(t.shape) for t in (q, k, v))

    @fake("speed3r_b200::pool_qkv_fwd")
    def _(q, k, v, block, kernel, stride):
        window = lambda x, kernel, stride: x.new_empty(*x.shape[:2], (x.shape[2] - kernel) // stride + 1, x.shape[3])
        return window(q, block, block), window(k, kernel, stride), window(v, kernel, stride)

    @fake("speed3r_b200::prologue_fwd")
    def _(qkv, heads, block, pos, cos, sin, qw, qb, kw, kb, eps):
        B, N = qkv.shape[:2]
        d = qkv.numel() // (B * N * 3 * heads)
        return tuple(qkv.new_empty(B, heads, n, d) for n in (N, N, N, N // block, N // block, N // block))

    @fake("speed3r_b200::prologue_bwd")
    def _(qkv, heads, block, pos, cos, sin, qw, kw, eps, dq, dk, dv, dq_c, dk_c, dv_c):
        return (qkv.new_empty(qkv.shape),
                qkv.new_empty((0,) if qw is None else (4, dq.shape[-1]), dtype=torch.float32))

    @fake("speed3r_b200::delta")
    def _(o, d_o):
        return o.new_empty(o.shape[:-1], dtype=torch.float32)

    @fake("speed3r_b200::merge_bwd")
    def _(dy, gate, o_c, o_s, block):
        B, H, Tq, d = o_s.shape
        return (o_s.new_empty(o_s.shape), o_s.new_empty(B, H, Tq, 2, dtype=torch.float32), o_c.new_empty(o_c.shape),
                o_s.new_empty(B, H, Tq, dtype=torch.float32))


def _ops():
    """The ``torch.ops`` namespace of the native operators, loaded (and built if need be) at first use."""
    global _ns
    if _ns is None:
        with _lock:
            if _ns is None:
                _lib.load()
                torch.ops.load_library(_lib.TORCH_LIB_PATH)
                _register_fakes()
                _ns = torch.ops.speed3r_b200
    return _ns


def _need(t: Tensor, name: str, dtype=_BF16, contiguous=True) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor: the speed3r_b200 kernels have no CPU path")
    if t.dtype != dtype:
        raise RuntimeError(f"{name} must be {dtype}, got {t.dtype}")
    if contiguous and not t.is_contiguous():
        raise RuntimeError(f"{name} must be contiguous")


def _scale(softmax_scale: Optional[float], q: Tensor) -> float:
    return 1.0 / math.sqrt(q.shape[-1]) if softmax_scale is None else float(softmax_scale)


# ------------------------------------------------------------------------------------------------
# raw kernels (no autograd)
# ------------------------------------------------------------------------------------------------
def _cmp_fwd(q_c: Tensor, k_c: Tensor, v_c: Tensor, topk: int, scale: float) -> Tuple[Tensor, Tensor, Tensor]:
    """(o, lse, idx) of the compression attention."""
    return _ops().cmp_attn_topk_fwd.default(q_c, k_c, v_c, topk, scale)


def _sel_fwd(q: Tensor, k: Tensor, v: Tensor, idx: Tensor, gate: Optional[Tensor], o_c: Optional[Tensor],
             block: int, scale: float, want_o: bool, want_lse: bool, kv_chunks: int) -> Tuple[Tensor, Tensor, Tensor]:
    """Returns (o_s, lse_s, y); tensors not asked for come back with zero elements."""
    return _ops().sel_attn_fwd.default(q, k, v, idx, gate, o_c, block, scale, want_o, want_lse, kv_chunks)


def build_key_csr(idx: Tensor, num_key_blocks: int) -> Tuple[Tensor, Tensor]:
    """Key-centric CSR of the selection table: (offsets [B,H,Nkb+1], qids [B,H,Nq*K]) int32."""
    return _ops().build_key_csr.default(idx, num_key_blocks)


def qkv_prologue(qkv: Tensor, num_heads: int, block: int, pos: Optional[Tensor] = None,
                 cos: Optional[Tensor] = None, sin: Optional[Tensor] = None,
                 q_norm: Optional[Tuple[Tensor, Tensor, float]] = None,
                 k_norm: Optional[Tuple[Tensor, Tensor, float]] = None):
    """Everything between the qkv projection and the two attention calls of the module
    (pi3/models/layers/sparse_attention.py:95-123) in one kernel, forward only:
    ``qkv [B,N,3*H*d]`` -> ``(q, k, v [B,H,N,d], q_c, k_c, v_c [B,H,N/block,d])`` with the per-head
    LayerNorm of q and k (``(weight, bias, eps)`` or None), the 2-D rotary embedding at ``pos
    [B,N,2]`` (``cos``/``sin`` = the bf16 tables RoPE2D caches) and, for the pooled tensors, at each
    block's truncated mean position."""
    _need(qkv, "qkv")
    if qkv.requires_grad and torch.is_grad_enabled():
        raise RuntimeError("qkv_prologue is forward-only; the module's training path uses its differentiable form")
    with torch.no_grad():
        return _prologue(qkv, num_heads, block, pos, cos, sin, q_norm, k_norm)


def _prologue(qkv, num_heads, block, pos, cos, sin, q_norm, k_norm):
    """``qkv_prologue`` with a backward."""
    if (q_norm is None) != (k_norm is None):
        raise RuntimeError("qkv_prologue: q_norm and k_norm come together or not at all")
    if q_norm is not None and abs(q_norm[2] - k_norm[2]) > 0:
        raise RuntimeError("qkv_prologue: q_norm and k_norm must share eps")
    qw, qb, eps = q_norm if q_norm is not None else (None, None, 1e-5)
    kw, kb, _ = k_norm if k_norm is not None else (None, None, 0.0)
    return _ops().prologue.default(qkv, num_heads, block, pos, cos, sin, qw, qb, kw, kb, float(eps))


# ------------------------------------------------------------------------------------------------
# differentiable operators
# ------------------------------------------------------------------------------------------------
def pool_tokens(x: Tensor, kernel: int = 16, stride: int = 16) -> Tensor:
    """Mean over ``kernel`` consecutive tokens every ``stride`` tokens of ``x [B,H,T,d]`` (any
    batch/head/token strides) -> ``[B,H,Nc,d]``.  sparse_attention.py:97-102 for one of q/k/v."""
    return _ops().pool_tokens.default(x, kernel, stride)


def flash_attn_blocktopk_func(q, k, v, topk_val, group, take, softmax_scale=None):
    """Compression attention whose table ranks selection BLOCKS by the softmax mass of their own compressed
    keys (columns ``group*n .. group*n+take-1``): for settings where compressed keys are finer than selection
    blocks.  Returns ``(o, idx)`` like ``flash_attn_topk_func``; ``idx`` holds block numbers."""
    if int(group) < 1:
        raise RuntimeError(f"flash_attn_blocktopk_func: {group} compressed keys per block")
    return _ops().flash_attn_topk.default(q, k, v, int(topk_val), _scale(softmax_scale, q), int(group), int(take))


def sparse_attention_op(q, k, v, gate, block_size=16, topk=32, kernel=16, stride=16):
    """The whole op on ``q,k,v [B,H,T,d]`` and ``gate [B,H,T,2]``: queries pooled per selection block
    (``block_size`` tokens), keys and values pooled with ``kernel``/``stride``, compression attention with the
    fused table, selection attention over the table's blocks, gated merge.  At 16/16/16 this is the
    reference's path (``sparse_attention.py:95-136`` without the norms and rotary embedding); when compressed
    keys are finer than selection blocks (e.g. kernel 32, stride 16, blocks of 64) the blocks are ranked by
    probability mass.  Returns ``(y [B,T,H*d], idx)``."""
    group = take = 0
    if (kernel, stride) != (block_size, block_size):
        if block_size % stride or kernel > block_size or (block_size - kernel) % stride:
            raise RuntimeError("need stride | block_size and kernel = block_size - i*stride")
        group, take = block_size // stride, (block_size - kernel) // stride + 1
    return _ops().sparse_attention.default(q, k, v, gate, int(block_size), int(topk), int(kernel), int(stride),
                                           _scale(None, q), group, take)


def flash_attn_topk_func(q, k, v, topk_val, bias=None, causal=False, softmax_scale=None):
    """Compression attention with fused top-k selection; drop-in for the reference's
    ``flash_attn_topk_func`` (flash_attention_topk.py:633-668).  Inputs ``[B,H,n,d]`` bf16."""
    assert bias is None, "bias is not supported (the reference ignores it as well)"
    assert not causal, "the sparse global attention is bidirectional; causal is not implemented"
    return _ops().flash_attn_topk.default(q, k, v, int(topk_val), _scale(softmax_scale, q), 0, 0)


def topk_blocksparse_attention(q, k, v, topk_idx, block_size, softmax_scale=None):
    """Block-sparse selection attention; drop-in for the reference's ``topk_blocksparse_attention``
    (topk_blocksparse_attention.py:1093-1121).  q,k,v ``[B,H,T,d]`` bf16 contiguous, ``topk_idx``
    ``[B,H,T/block,K]`` int32."""
    assert q.dtype == torch.bfloat16, "bf16 only"
    assert q.dtype == k.dtype and k.dtype == v.dtype
    assert topk_idx.dtype == torch.int32
    return _ops().topk_blocksparse.default(q, k, v, topk_idx, int(block_size), _scale(softmax_scale, q))


def sel_attn_merge(q, k, v, topk_idx, gate, o_c, block_size, softmax_scale=None):
    """Selection attention with the gated merge fused into its epilogue:
    ``y[b,t,(h d)] = gate[b,h,t,0] * o_c[b,h,t//block] + gate[b,h,t,1] * sel_attn(q,k,v)[b,h,t]``
    (topk_blocksparse_attention.py:35-128 + sparse_attention.py:127-136).  ``gate [B,H,T,2]`` may
    be a strided view of the ``[B,T,2H]`` projection."""
    return _ops().sel_merge.default(q, k, v, topk_idx, gate, o_c, int(block_size), _scale(softmax_scale, q))


def sel_attn_merge_chunked(q, k_chunks, v_chunks, topk_idx, gate, o_c, block_size, softmax_scale=None):
    """Forward-only form of ``sel_attn_merge`` for sequence-partitioned inference: the keys and
    values are the all-gathered ``[G,B,H,Tk/G,d]`` chunks (rank order = sequence order), read in
    place; ``q``, ``gate``, ``o_c`` and ``topk_idx`` are the local query rows; ``topk_idx`` holds
    GLOBAL key-block numbers."""
    with torch.no_grad():
        return _sel_fwd(q, k_chunks, v_chunks, topk_idx, gate, o_c, int(block_size), _scale(softmax_scale, q),
                        False, False, int(k_chunks.shape[0]))[2]
