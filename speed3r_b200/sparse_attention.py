"""Drop-in replacement for the reference's global-attention module.

``SparseFlashAttentionRope`` keeps the constructor signature, sub-module names (``qkv``, ``proj``,
``q_norm``, ``k_norm``, ``gate`` = Sequential(Linear, Sigmoid)), attributes and ``forward(x,
attn_bias=None, xpos=None)`` of pi3/models/layers/sparse_attention.py:60-141, so a checkpoint of
the reference loads unchanged and ``BlockRope(attn_class=SparseFlashAttentionRope)`` works
(pi3/models/layers/block.py:282-312).  The projections stay PyTorch (cuBLAS) code; pooling, the compression attention with its top-k
selection, the selection attention and the gated merge run in the CUDA library (speed3r_b200.ops).
The LayerNorms, the rotary embedding, the pooling and the q/k/v split run as one library kernel as well
(``ops.qkv_prologue``), with gradients as without; settings that kernel does not take stay PyTorch code around
the differentiable ops.

The reference's literals (pooling 16/16, top-k 32) are keyword arguments here with the same
defaults.
"""
from __future__ import annotations

import weakref
from typing import Optional

import torch
from torch import Tensor, nn

from . import ops


class _TableRows:
    """How many rows the rotary cos/sin tables need for a position tensor, without reading
    ``positions.max()`` back on every call.

    Row r of the tables depends on r alone (pos_embed.py:119-129), so a table that is longer than
    needed gives bit-identical results; only a table that is too SHORT is an error.  The size is
    therefore grow-only, and the maximum of a position tensor is read back once per tensor
    *object*: the entry is keyed on the storage-owning base tensor through a weak reference (all
    the reshaped views the decode loop passes down share one base) together with its in-place
    version counter, and is dropped when that tensor dies.  A new tensor that happens to reuse
    the address of an old one is a new object and is measured again."""

    def __init__(self, min_rows: int = 64):
        self.rows = min_rows
        self._seen = {}

    def __call__(self, positions: Tensor) -> int:
        base = positions._base if positions._base is not None else positions
        key = id(base)
        hit = self._seen.get(key)
        if hit is not None and hit[0]() is base and hit[1] == base._version:
            return self.rows
        need = int(base.max()) + 1 if base.numel() else 1        # one read-back per position tensor
        self.rows = max(self.rows, need)
        seen = self._seen
        self._seen[key] = (weakref.ref(base, lambda _r, k=key: seen.pop(k, None)), base._version)
        return self.rows


_WIDE = (torch.float32, torch.bfloat16)


def _global_hooks() -> bool:
    m = nn.modules.module
    return bool(m._global_forward_hooks or m._global_forward_pre_hooks or m._global_backward_hooks or m._global_backward_pre_hooks)


def _watched(m: nn.Module) -> bool:
    """Somebody wants to see this module called: a hook, or a ``forward`` of its own on the instance (as offloading and
    quantisation wrappers put there)."""
    return bool(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or "forward" in m.__dict__)


def _plain_rope(rope) -> bool:
    """A rotary module whose ``forward`` is the table look-up that the prologue does itself."""
    return rope is None or not (_watched(rope) or (isinstance(rope, RoPE2D) and type(rope).forward is not RoPE2D.forward))


def rope_tables(rope, D: int, rows: int, device, dtype):
    """cos/sin tables ``[rows, 2*(D/2)]`` with the reference's arithmetic (pos_embed.py:119-129: the
    angle is rounded to ``dtype`` before cos/sin).  ``rope`` is this package's ``RoPE2D`` or the
    reference's: for the latter its own ``get_cos_sin`` builds (and caches) the tables."""
    if hasattr(rope, "_cos_sin"):
        return rope._cos_sin(D, rows, device, dtype)
    return rope.get_cos_sin(D, rows, device, dtype)


def _is_rope2d(rope) -> bool:
    """This package's RoPE2D or the reference's pure-PyTorch one (same attributes and table builder)."""
    return isinstance(rope, RoPE2D) or (hasattr(rope, "base") and hasattr(rope, "F0") and
                                        callable(getattr(rope, "get_cos_sin", None)))


class RoPE2D(nn.Module):
    """2-D rotary embedding with the arithmetic of pi3/models/layers/pos_embed.py:112-159 (the
    angle table is rounded to the activation dtype before cos/sin).  Unlike the reference it does
    not read ``positions.max()`` back on every call: the tables only ever grow, and a position
    tensor is measured once (see ``_TableRows``)."""

    def __init__(self, freq: float = 100.0, F0: float = 1.0):
        super().__init__()
        self.base = freq
        self.F0 = F0
        self._tables = {}
        self._rows = _TableRows()

    def _cos_sin(self, D, seq_len, device, dtype):
        key = (D, seq_len, device, dtype)
        if key not in self._tables:
            inv_freq = 1.0 / (self.base ** (torch.arange(0, D, 2).float().to(device) / D))
            t = torch.arange(seq_len, device=device, dtype=inv_freq.dtype)
            freqs = torch.einsum("i,j->ij", t, inv_freq).to(dtype)
            freqs = torch.cat((freqs, freqs), dim=-1)
            self._tables[key] = (freqs.cos(), freqs.sin())
        return self._tables[key]

    get_cos_sin = _cos_sin          # the reference's name for the same builder

    def _seq_len(self, positions: Tensor) -> int:
        return self._rows(positions)

    @staticmethod
    def _rope1d(tokens, pos1d, cos, sin):
        cos = torch.nn.functional.embedding(pos1d, cos)[:, None, :, :]
        sin = torch.nn.functional.embedding(pos1d, sin)[:, None, :, :]
        x1, x2 = tokens[..., : tokens.shape[-1] // 2], tokens[..., tokens.shape[-1] // 2:]
        return tokens * cos + torch.cat((-x2, x1), dim=-1) * sin

    def forward(self, tokens: Tensor, positions: Tensor, seq_len: Optional[int] = None) -> Tensor:
        D = tokens.size(3) // 2
        if seq_len is None:
            seq_len = self._seq_len(positions)
        cos, sin = self._cos_sin(D, seq_len, tokens.device, tokens.dtype)
        y, x = tokens.chunk(2, dim=-1)
        y = self._rope1d(y, positions[:, :, 0], cos, sin)
        x = self._rope1d(x, positions[:, :, 1], cos, sin)
        return torch.cat((y, x), dim=-1)


class SparseFlashAttentionRope(nn.Module):
    def __init__(
        self,
        dim: int,
        num_heads: int = 16,
        qkv_bias: bool = False,
        proj_bias: bool = True,
        attn_drop: float = 0.0,
        proj_drop: float = 0.0,
        qk_norm: bool = False,
        norm_layer: nn.Module = nn.LayerNorm,
        rope=None,
        block_size: int = 4,
        topk: int = 32,
    ) -> None:
        super().__init__()
        self.num_heads = num_heads
        head_dim = dim // num_heads
        self.scale = head_dim ** -0.5
        self.qkv = nn.Linear(dim, dim * 3, bias=qkv_bias)
        self.attn_drop = nn.Dropout(attn_drop)
        self.proj = nn.Linear(dim, dim, bias=proj_bias)
        self.proj_drop = nn.Dropout(proj_drop)
        self.q_norm = norm_layer(head_dim) if qk_norm else nn.Identity()
        self.k_norm = norm_layer(head_dim) if qk_norm else nn.Identity()
        self.rope = rope
        gate_linear = nn.Linear(dim, num_heads * 2, bias=True)
        nn.init.zeros_(gate_linear.weight)
        gate_linear.bias.data.copy_(torch.tensor([-1.0, 1.0]).repeat(num_heads))
        self.gate = nn.Sequential(gate_linear, nn.Sigmoid())
        self.block_size = block_size
        self.topk = topk
        self.record_idx = False      # debugging aid: keep the last selected-block table in .last_idx
        self.last_idx = None
        self._rows = _TableRows()    # table length when the rotary module is the reference's own
        self.seq_parallel = None     # a seq_parallel.SequenceParallel: x holds this rank's slice of the views

    def _can_fuse_prologue(self, qkv, x, xpos, N, Bs, d) -> bool:
        """Inference (nothing to differentiate) in a setting the one-pass prologue takes."""
        if torch.is_grad_enabled() and (x.requires_grad or any(p.requires_grad for p in self.parameters())):
            return False
        return self._prologue_takes(xpos, N, Bs, d)

    def _prologue_takes(self, xpos, N, Bs, d) -> bool:
        """Norms that are LayerNorm(d) with affine or Identity, a 2-D rotary module (this package's or the
        reference's pure-PyTorch one) or none, whole blocks, head counts the kernel takes."""
        qn, kn = self._modules["q_norm"], self._modules["k_norm"]
        if not (isinstance(qn, nn.Identity) and isinstance(kn, nn.Identity)):
            for m in (qn, kn):
                if not (isinstance(m, nn.LayerNorm) and m.elementwise_affine and m._parameters.get("bias") is not None and
                        tuple(m.normalized_shape) == (d,)):
                    return False
            if qn.eps != kn.eps:
                return False
        if xpos is not None and not _is_rope2d(self.rope):
            return False
        return d == 64 and N % Bs == 0 and self.num_heads <= 42

    def _trains_through_prologue(self, xpos, N, Bs, d) -> bool:
        """``_prologue_takes``, and the norms and the rotary module are what they look like: with gradients they are called
        unless they are."""
        mods = self._modules
        return (all(type(m) in (nn.LayerNorm, nn.Identity) and not _watched(m) for m in (mods["q_norm"], mods["k_norm"])) and
                not _global_hooks() and (xpos is None or _plain_rope(self.rope)) and self._prologue_takes(xpos, N, Bs, d))

    def _native_op(self, x, xpos, N, Bs, d):
        """The native operator that runs the whole module, or None: plain Linear projections that nobody watches, bf16 (by
        autocast or by dtype), no sequence partition; with gradients fp32 parameters under autocast.  A dispatch mode (a
        tracer, a counter) sees no kernel of a native call, so under one the steps are taken apart.  Sub-modules and
        parameters are taken from their dictionaries: nn.Module's attribute look-up was half of the 12 us this took."""
        mods = self._modules
        qkv, gate, proj = mods["qkv"], mods["gate"], mods["proj"]
        if (self.seq_parallel is not None or not x.is_cuda or type(x) is not Tensor or type(gate) is not nn.Sequential or
                len(gate._modules) != 2 or _global_hooks() or torch.compiler.is_compiling() or torch._C._len_torch_dispatch_stack()):
            return None
        glin, act = gate._modules.values()
        if type(act) is not nn.Sigmoid:
            return None
        for m in (gate, act, mods["q_norm"], mods["k_norm"]):
            if _watched(m):
                return None
        dev, narrow, full = x.get_device(), 0, 0
        for m in (qkv, glin, proj):
            if type(m) is not nn.Linear or _watched(m):
                return None
            for p in m._parameters.values():
                if p is None:
                    continue
                if type(p) is not nn.Parameter or p.get_device() != dev:
                    return None
                if p.dtype == torch.float32:
                    full += 1
                elif p.dtype == torch.bfloat16:
                    narrow += 1
                else:
                    return None
            if m._parameters.get("weight") is None:
                return None
        autocast = torch.is_autocast_enabled("cuda")
        if autocast:
            if torch.get_autocast_dtype("cuda") != torch.bfloat16 or x.dtype not in _WIDE:
                return None
        elif x.dtype != torch.bfloat16 or full:
            return None
        if self._can_fuse_prologue(None, x, xpos, N, Bs, d):
            return ops._ops().module_infer.default
        if (torch.is_grad_enabled() and autocast and self.num_heads % 4 == 0 and not narrow and
                (qkv._parameters["bias"] is None) == (glin._parameters["bias"] is None) and self._trains_through_prologue(xpos, N, Bs, d)):
            return ops._ops().module_train.default
        return None

    def _rope_and_norms(self, xpos, d, device, dtype):
        """(cos, sin, q_norm, k_norm) as the one-pass prologue takes them."""
        cos = sin = qn = kn = None
        if xpos is not None:
            rows = self.rope._seq_len(xpos) if isinstance(self.rope, RoPE2D) else self._rows(xpos)
            cos, sin = rope_tables(self.rope, d // 2, rows, device, dtype)
        q_norm, k_norm = self._modules["q_norm"], self._modules["k_norm"]
        if isinstance(q_norm, nn.LayerNorm):
            qn = (q_norm.weight, q_norm.bias, q_norm.eps)
            kn = (k_norm.weight, k_norm.bias, k_norm.eps)
        return cos, sin, qn, kn

    def _forward_native(self, op, x, xpos, H, d, Bs) -> Tensor:
        cos, sin, qn, kn = self._rope_and_norms(xpos, d, x.device, torch.bfloat16)
        qw, qb, eps = qn if qn is not None else (None, None, 1e-5)
        kw, kb, _ = kn if kn is not None else (None, None, 0.0)
        mods = self._modules
        qkv, g, proj = mods["qkv"]._parameters, next(iter(mods["gate"]._modules.values()))._parameters, mods["proj"]._parameters
        y, idx = op(x, qkv["weight"], qkv["bias"], g["weight"], g["bias"], proj["weight"], proj["bias"], xpos, cos, sin,
                    qw, qb, kw, kb, eps, H, Bs, self.topk, 1.0 / d ** 0.5)
        if self.record_idx:
            self.last_idx = idx
        drop = mods["proj_drop"]
        if type(drop) is nn.Dropout and not _watched(drop) and (drop.p == 0.0 or not drop.training):
            return y
        return drop(y)

    def _forward_fused(self, qkv, gate, xpos, B, N, H, d, Bs, train=False) -> Tensor:
        cos, sin, qn, kn = self._rope_and_norms(xpos, d, qkv.device, qkv.dtype)
        q, k, v, q_c, k_c, v_c = ops._prologue(qkv, H, Bs, xpos, cos, sin, qn, kn)
        if self.seq_parallel is not None and train:
            # this rank's queries against the whole sequence; the backward reduce-scatters dK and dV
            y, idx = self.seq_parallel.attention_grad(q, k, v, q_c, k_c, v_c, gate, Bs, self.topk,
                                                      ops.flash_attn_topk_func, ops.sel_attn_merge)
            if self.record_idx:
                self.last_idx = idx.detach()
            return self.proj_drop(self.proj(y))
        if self.seq_parallel is not None:
            # this rank's query blocks against the whole sequence: pooled and token-level K/V are exchanged
            y, idx = self.seq_parallel.attention(q, k, v, q_c, k_c, v_c, gate, Bs, self.topk,
                                                 ops.flash_attn_topk_func, ops.sel_attn_merge_chunked)
            if self.record_idx:
                self.last_idx = idx.detach()
            return self.proj_drop(self.proj(y))
        o_c, idx = ops.flash_attn_topk_func(q_c, k_c, v_c, self.topk)
        if self.record_idx:
            self.last_idx = idx.detach()
        y = ops.sel_attn_merge(q, k, v, idx, gate, o_c, Bs)
        return self.proj_drop(self.proj(y))

    def forward(self, x: Tensor, attn_bias=None, xpos: Optional[Tensor] = None) -> Tensor:
        B, N, C = x.shape
        H = self.num_heads
        d = C // H
        Bs = self.block_size ** 2
        op = self._native_op(x, xpos, N, Bs, d)
        if op is not None:
            return self._forward_native(op, x, xpos, H, d, Bs)
        qkv = self.qkv(x)
        gate = self.gate(x).view(B, N, H, 2).permute(0, 2, 1, 3)          # [B,H,N,2] view, no copy
        if qkv.dtype != torch.bfloat16:
            raise RuntimeError("SparseFlashAttentionRope runs in bf16 (use torch.autocast(dtype=torch.bfloat16)); "
                               f"got {qkv.dtype}")
        gate = gate.to(qkv.dtype)
        if self._can_fuse_prologue(qkv, x, xpos, N, Bs, d):
            return self._forward_fused(qkv.detach(), gate, xpos, B, N, H, d, Bs)
        if torch.is_grad_enabled() and self._trains_through_prologue(xpos, N, Bs, d):
            return self._forward_fused(qkv, gate, xpos, B, N, H, d, Bs, train=True)
        if self.seq_parallel is not None and N % Bs != 0:
            raise RuntimeError("sequence-parallel attention needs whole 16-token blocks on every rank")
        qkv5 = qkv.view(B, N, 3, H, d)
        q_t, k_t, v_t = (qkv5[:, :, i].permute(0, 2, 1, 3) for i in range(3))   # [B,H,N,d] views of the projection

        # compression branch: pool raw q,k,v, then norm + rope with the block's mean position
        q_c, k_c, v_c = (ops.pool_tokens(t, Bs, Bs) for t in (q_t, k_t, v_t))
        q_c, k_c = self.q_norm(q_c).to(v_c.dtype), self.k_norm(k_c).to(v_c.dtype)
        rope_kw = {}
        if xpos is not None and isinstance(self.rope, RoPE2D):
            rope_kw = dict(seq_len=self.rope._seq_len(xpos))     # one table for token and block positions
        if xpos is not None:
            xpos_c = xpos.view(B, N // Bs, Bs, 2).float().mean(dim=2).int()
            q_c = self.rope(q_c, xpos_c, **rope_kw)
            k_c = self.rope(k_c, xpos_c, **rope_kw)
        # selection branch at token level, gated merge fused into its epilogue
        q, k = self.q_norm(q_t).to(qkv.dtype), self.k_norm(k_t).to(qkv.dtype)
        if xpos is not None:
            q = self.rope(q, xpos, **rope_kw)
            k = self.rope(k, xpos, **rope_kw)
        if self.seq_parallel is not None:
            # this rank's queries against the whole sequence; the backward reduce-scatters dK and dV
            y, idx = self.seq_parallel.attention_grad(q.contiguous(), k.contiguous(), v_t.contiguous(), q_c, k_c, v_c,
                                                      gate, Bs, self.topk, ops.flash_attn_topk_func, ops.sel_attn_merge)
        else:
            o_c, idx = ops.flash_attn_topk_func(q_c, k_c, v_c, self.topk)
            y = ops.sel_attn_merge(q.contiguous(), k.contiguous(), v_t.contiguous(), idx, gate, o_c, Bs)
        if self.record_idx:
            self.last_idx = idx.detach()
        y = self.proj(y)
        return self.proj_drop(y)
