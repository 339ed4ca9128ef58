"""The sparse global-attention op for callers whose q, k, v live in pinned HOST memory.

The reference keeps its tensors on the device (`SparseFlashAttentionRope.forward`,
pi3/models/layers/sparse_attention.py:88-143); a host that holds them in its own memory pays the
PCIe copies on top of the kernels.  `HostPipeline` hides most of that cost by cutting the op along
the two axes on which it is independent and running three streams:

* heads are independent, so the op runs head group by head group: a group's K and V arrive (a head of a
  `[1,H,T,d]` tensor is one contiguous span) and are pooled as they land, then its queries follow in
  chunks of query blocks.  The first group computes while the second is still on the bus, so the copy-in
  stream never waits for the kernels and the kernels only wait for data;
* compute stream: per (head group, query chunk), pool -> compression attention + top-k -> selection
  attention with the gated merge; a chunk needs the group's pooled K/V but only its own queries;
* copy-out stream: each chunk of a group's `y [1,T,Hg*d]` goes back while the next chunk computes, as a
  strided copy into the group's columns of the caller's `y [1,T,H*d]`.

The query chunk is sized so that one compression-attention launch fills whole waves of the GPU
(`Hg * ceil(rows/256)` CTAs a multiple of the SM count).  The last group's chunks are a quarter of the sequence at most:
what follows the last byte in is one chunk's kernels and its copy out, and nothing else hides them (64512 tokens, 16
heads: 8.55 -> 8.03 ms, of which 7.7 for the copies in).  Results are bit-identical to the unchunked
call: every query row sees the same keys in the same order.  One thing couples rows: where some row's compressed logits
outgrow its first 128 keys' by more than 2^64, all rows of its 128 or 256 take their exact maxima as exponent offsets, and
chunks group rows differently; such rows, which normalised queries and keys do not have, may round differently.
"""
from __future__ import annotations

import math
from typing import Optional

import torch
from torch import Tensor

from . import _lib, ops

_ROWS_PER_CTA = 256          # pooled query rows one compression-attention CTA owns
_Q_BUFFERS = 4
_GROUP_BYTES = 10 << 20      # q, k and v of a head group: about as long on the bus as the host takes to enqueue the group


def rows_per_chunk_for(num_heads: int, sm_count: int) -> int:
    """Pooled query rows per chunk such that one compression-attention launch (``num_heads *
    ceil(rows/256)`` CTAs, one CTA per SM at a time) fills whole waves of the GPU."""
    return _ROWS_PER_CTA * (sm_count // math.gcd(num_heads, sm_count))


def query_chunks(num_pooled_rows: int, rows_per_chunk: int):
    """[(first pooled row, last pooled row + 1)] covering ``num_pooled_rows`` in order; the last may be short."""
    rows = max(1, min(num_pooled_rows, rows_per_chunk))
    return [(r, min(num_pooled_rows, r + rows)) for r in range(0, num_pooled_rows, rows)]


def _pinned(t: Tensor, name: str) -> None:
    if t.device.type != "cpu" or not t.is_pinned():
        raise RuntimeError(f"{name}: expected a pinned host tensor")
    if t.dtype != torch.bfloat16 or not t.is_contiguous():
        raise RuntimeError(f"{name}: expected a contiguous bf16 tensor")


class HostPipeline:
    """Pre-allocated device buffers and streams for one problem size (B = 1).

    ``pipe = HostPipeline(H, T, device=...)`` then ``pipe(hq, hk, hv, hgate, hy)`` with pinned host
    tensors ``hq/hk/hv [1,H,T,d]``, ``hgate [1,H,T,2]`` and the result buffer ``hy [1,T,H*d]``.
    The call only enqueues work; the calling stream is made to wait for the last copy, so an event
    recorded on it (or a synchronize) covers the whole op.  ``heads_per_group`` heads travel and compute
    together (``heads_per_copy`` is the older name of the same argument)."""

    def __init__(self, H: int, T: int, d: int = 64, block_size: int = 16, topk: int = 32,
                 device: Optional[torch.device] = None, rows_per_chunk: Optional[int] = None,
                 heads_per_group: Optional[int] = None, heads_per_copy: Optional[int] = None):
        if T % block_size:
            raise RuntimeError(f"T={T} must be a multiple of the block size {block_size}")
        self.H, self.T, self.d, self.block, self.topk = H, T, d, block_size, topk
        self.dev = torch.device(device if device is not None else torch.cuda.current_device())
        if self.dev.type != "cuda":
            raise RuntimeError("HostPipeline needs a CUDA device")
        self.Nc = T // block_size
        hg = heads_per_group if heads_per_group is not None else heads_per_copy
        if hg is None:
            hg = 4
            while hg < H and hg * T * d * 6 < _GROUP_BYTES:
                hg *= 2
        self.hg = max(1, min(H, hg))
        whole_waves = rows_per_chunk is None
        if whole_waves:
            sms = torch.cuda.get_device_properties(self.dev).multi_processor_count
            rows_per_chunk = rows_per_chunk_for(self.hg, sms)
        self.rows = max(1, min(self.Nc, rows_per_chunk))
        quarter = -(-self.Nc // (4 * _ROWS_PER_CTA)) * _ROWS_PER_CTA
        self.rows_last = min(self.rows, quarter) if whole_waves else self.rows
        bf = dict(device=self.dev, dtype=torch.bfloat16)
        hg = self.hg
        # two sets of group buffers: group g+1 lands while group g computes
        self.k = [torch.empty(1, hg, T, d, **bf) for _ in range(2)]
        self.v = [torch.empty(1, hg, T, d, **bf) for _ in range(2)]
        self.gate = [torch.empty(1, hg, T, 2, **bf) for _ in range(2)]
        tc = self.rows * block_size
        # query chunks may run up to four ahead of the kernels: a chunk computes a little longer than it travels, and
        # the copy-in stream must not wait for a free buffer while the next group's K and V could be on the bus
        self.qbuf = [torch.empty(1, hg, tc, d, **bf) for _ in range(_Q_BUFFERS)]
        self.s_in, self.s_out = torch.cuda.Stream(self.dev), torch.cuda.Stream(self.dev)

    def chunks(self):
        """[(first pooled row, last pooled row + 1)] of the query chunks of every head group but the last."""
        return query_chunks(self.Nc, self.rows)

    def groups(self):
        """[(first head, last head + 1)] of the head groups; the last may be short."""
        return [(h, min(self.H, h + self.hg)) for h in range(0, self.H, self.hg)]

    @torch.no_grad()
    def __call__(self, hq: Tensor, hk: Tensor, hv: Tensor, hgate: Tensor, hy: Tensor) -> None:
        H, T, d = self.H, self.T, self.d
        for n, t, shape in (("hq", hq, (1, H, T, d)), ("hk", hk, (1, H, T, d)), ("hv", hv, (1, H, T, d)),
                            ("hgate", hgate, (1, H, T, 2)), ("hy", hy, (1, T, H * d))):
            _pinned(t, n)
            if tuple(t.shape) != shape:
                raise RuntimeError(f"{n}: expected shape {shape}, got {tuple(t.shape)}")
        main = torch.cuda.current_stream(self.dev)
        s_in, s_out = self.s_in, self.s_out
        s_in.wait_stream(main)            # device buffers may still be read by an earlier call
        s_out.wait_stream(main)
        try:
            self._enqueue(main, hq, hk, hv, hgate, hy)
        finally:
            # the caller may drop its tensors at once: their memory is not to be handed out before the copies are done
            in_use = ops._ops().host_in_use.default
            with torch.cuda.stream(s_in):
                for t in (hq, hk, hv, hgate):
                    in_use(t, self.dev)
            with torch.cuda.stream(s_out):
                in_use(hy, self.dev)
            main.wait_stream(s_out)
            main.wait_stream(s_in)

    def _enqueue(self, main, hq: Tensor, hk: Tensor, hv: Tensor, hgate: Tensor, hy: Tensor) -> None:
        H, T, d, bs = self.H, self.T, self.d, self.block
        s_in, s_out = self.s_in, self.s_out
        copy2d, in_stream, out_stream = _lib.load().s3r_copy2d_async, s_in.cuda_stream, s_out.cuda_stream
        esz = hy.element_size()
        tok = d * esz                     # bytes of a token of one head

        def fetch(dst: Tensor, src: Tensor, first: int, rows: int, width: int, pitch: int) -> None:
            """``rows`` spans of ``width`` bytes, ``pitch`` apart in host memory from byte ``first`` on, to ``dst``."""
            _lib.check(copy2d(dst.data_ptr(), width, src.data_ptr() + first, pitch, width, rows, in_stream), "s3r_copy2d_async")

        def mark(stream) -> torch.cuda.Event:
            e = torch.cuda.Event()
            e.record(stream)
            return e

        grp_free = [None, None]           # compute of the group that last used buffer set i is finished
        q_free = [None] * _Q_BUFFERS      # compute of the chunk that last used qbuf[i] is finished
        step = 0
        for gi, (h0, h1) in enumerate(self.groups()):
            b, n = gi & 1, h1 - h0
            k, v, gate = (buf[b][:, :n] for buf in (self.k, self.v, self.gate))
            if grp_free[b] is not None:
                s_in.wait_event(grp_free[b])
            fetch(k, hk, h0 * T * tok, n, T * tok, T * tok)
            k_in = mark(s_in)
            fetch(v, hv, h0 * T * tok, n, T * tok, T * tok)
            fetch(gate, hgate, h0 * T * 2 * esz, n, T * 2 * esz, T * 2 * esz)
            v_in = mark(s_in)
            main.wait_event(k_in)
            k_c = ops.pool_tokens(k, bs, bs)                      # pooled while V is still on the bus
            main.wait_event(v_in)
            v_c = ops.pool_tokens(v, bs, bs)
            done = None
            for r0, r1 in (self.chunks() if h1 < H else query_chunks(self.Nc, self.rows_last)):
                i = step % _Q_BUFFERS
                step += 1
                t0, t1 = r0 * bs, r1 * bs
                q_dev = self.qbuf[i].view(-1)[:n * (t1 - t0) * d].view(1, n, t1 - t0, d)
                if q_free[i] is not None:
                    s_in.wait_event(q_free[i])
                fetch(q_dev, hq, (h0 * T + t0) * tok, n, (t1 - t0) * tok, T * tok)
                main.wait_event(mark(s_in))
                q_c = ops.pool_tokens(q_dev, bs, bs)
                o_c, idx = ops.flash_attn_topk_func(q_c, k_c, v_c, self.topk)
                y = ops.sel_attn_merge(q_dev, k, v, idx, gate[:, :, t0:t1], o_c, bs)      # [1, t1-t0, n*d]
                done = q_free[i] = mark(main)
                y.record_stream(s_out)    # the allocator must not hand y out again before it has left
                s_out.wait_event(done)
                # this group's columns of the rows t0..t1 of hy [1,T,H*d]
                _lib.check(copy2d(hy.data_ptr() + t0 * H * tok + h0 * tok, H * tok, y.data_ptr(), n * tok, n * tok, t1 - t0,
                                  out_stream), "s3r_copy2d_async")
            grp_free[b] = done
