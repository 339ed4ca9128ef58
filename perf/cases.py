"""Timed cases of the sparse global attention: what a program that uses the package asks of it.

The path is reached in seven ways, and every case is one of them (``kind``):

``op_fwd``       ``ops.sparse_attention_op`` without gradients: the whole op on q, k, v, gate
``op_train``     the same op, forward and backward
``module_fwd``   the drop-in ``SparseFlashAttentionRope`` under bf16 autocast without gradients
``module_train`` the module, forward and backward with the gradients of its input and parameters
``sel_train``    ``ops.topk_blocksparse_attention`` on a caller's own table, forward and backward
``rank_share``   what one GPU of a sequence-partitioned forward runs between its collectives
``host``         ``HostPipeline``: the op on pinned host tensors, copies included

Sizes are numbers of tokens.  A view has 256 tokens (224 x 224 pixels) in training and 1008 (392 x 504) or
about 1041 in inference; sequences run from a handful of small views to 1000 large ones.
"""
import math

import torch

import speed3r_b200
from speed3r_b200 import HostPipeline, ops

D = 64               # head dimension of every configuration
LO_T, HI_T = 2048, 1008000


def listed():
    return [
        # 8 views of 256 tokens: the smallest scene, where launches and host work are the time
        dict(name="op fwd 8x256", kind="op_fwd", B=1, H=16, T=2048, setting="reference", inputs="iid"),
        # 100 views whose keys cluster by view and patch as trained features do
        dict(name="op fwd 100x1008 structured", kind="op_fwd", B=1, H=16, T=100800, setting="reference", inputs="structured"),
        # 1000 views: the longest sequence, the headline setting
        dict(name="op fwd 1000x1008", kind="op_fwd", B=1, H=16, T=1008000, setting="reference", inputs="iid"),
        # keys pooled 32/16, blocks of 64, top-16: the coarser selection, at 250 views (whole blocks of 64)
        dict(name="op fwd 250x1008 extension", kind="op_fwd", B=1, H=16, T=251968, setting="extension", inputs="iid"),
        # training: 2 samples of 24 views of 256 tokens
        dict(name="op fwd+bwd 2x24x256", kind="op_train", B=2, H=16, T=6144, setting="reference", inputs="iid"),
        # training on a long sequence
        dict(name="op fwd+bwd 250x1008", kind="op_train", B=1, H=16, T=252000, setting="reference", inputs="iid"),
        # one attention layer of the model on a small scene, activations already bf16
        dict(name="module fwd 8x256", kind="module_fwd", B=1, H=16, T=2048, x="bf16"),
        # one attention layer at 64 views; LayerNorm under autocast hands over fp32
        dict(name="module fwd 64x1008", kind="module_fwd", B=1, H=16, T=64512, x="fp32"),
        # one attention layer of a training step
        dict(name="module fwd+bwd 2x24x256", kind="module_train", B=2, H=16, T=6144, x="fp32"),
        # the selection op alone on 8 views of 1041 tokens, so that the last block is cut short
        dict(name="sel fwd+bwd 8x1041", kind="sel_train", B=1, H=16, T=8328, block=64, K=16),
        # one of 8 GPUs at 1000 views: its queries against everybody's keys
        dict(name="rank share 1000x1008 / 8", kind="rank_share", B=1, H=16, T=1008000, G=8),
        # tensors that live in host memory, 64 views
        dict(name="host 64x1008", kind="host", B=1, H=16, T=64512),
    ]


def _tokens(rng, lo, hi, step=16):
    """Log-uniform number of tokens, a multiple of `step` (of the block, not of any tile of a kernel)."""
    t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(round(t / step)) * step)


def draw(rng):
    kind = rng.choice(["op_fwd", "op_fwd", "op_train", "op_train", "module_fwd", "module_train", "sel_train",
                       "rank_share", "host"])
    H = rng.choice([6, 12, 16, 16])
    if kind == "op_fwd":
        setting = rng.choice(["reference", "reference", "extension"])
        return dict(kind=kind, B=1, H=H, T=_tokens(rng, LO_T, 700000, 16 if setting == "reference" else 64),
                    setting=setting, inputs=rng.choice(["iid", "structured"]))
    if kind == "op_train":
        B = rng.choice([1, 2])
        return dict(kind=kind, B=B, H=H, T=_tokens(rng, LO_T, 300000 if B == 1 else 100000), setting="reference",
                    inputs=rng.choice(["iid", "structured"]))
    if kind == "module_fwd":
        return dict(kind=kind, B=rng.choice([1, 2]), H=H, T=_tokens(rng, LO_T, 200000), x=rng.choice(["bf16", "fp32"]))
    if kind == "module_train":
        return dict(kind=kind, B=rng.choice([1, 2]), H=H, T=_tokens(rng, LO_T, 40000), x=rng.choice(["bf16", "fp32"]))
    if kind == "sel_train":
        block = rng.choice([16, 32, 64])
        T = int(math.exp(rng.uniform(math.log(4096), math.log(60000))))       # any length: the last block may be short
        return dict(kind=kind, B=rng.choice([1, 2]), H=H, T=T, block=block, K=rng.choice([8, 16, 32]))
    if kind == "rank_share":
        G = rng.choice([2, 4, 8])
        return dict(kind=kind, B=1, H=H, T=_tokens(rng, 65536, HI_T, 16 * G), G=G)
    return dict(kind=kind, B=1, H=H, T=_tokens(rng, 4096, 80000))


def _settings(case):
    """(selection block, top-k, pooling kernel, pooling stride)."""
    return (64, 16, 32, 16) if case.get("setting") == "extension" else (16, 32, 16, 16)


def _norm(x):
    return torch.nn.functional.layer_norm(x, (D,)).bfloat16()


def _features(g, B, H, T, inputs="iid"):
    """Queries or keys after the per-head LayerNorm.  ``structured``: a component per view plus one per patch
    position, mixed through a rank-16 map, plus noise, so that selections cluster on a few views."""
    if inputs == "iid":
        return _norm(torch.randn(B, H, T, D, device="cuda", generator=g))
    tok = 1008 if T >= 8 * 1008 else 256
    views, r = -(-T // tok), 16
    view = torch.randn(B, H, views, 1, r, device="cuda", generator=g)
    patch = torch.randn(B, H, 1, tok, r, device="cuda", generator=g)
    mix = torch.randn(B, H, r, D, device="cuda", generator=g) / 4.0
    low = (view + patch).reshape(B, H, views * tok, r)[:, :, :T] @ mix
    return _norm(low + 0.5 * torch.randn(B, H, T, D, device="cuda", generator=g))


def _positions(B, T):
    """(y, x) of every token: views of 28 x 36 or 16 x 16 patches in a row."""
    h, w = (28, 36) if T >= 8 * 1008 else (16, 16)
    tok = torch.arange(T, device="cuda") % (h * w)
    return torch.stack((tok // w, tok % w), -1)[None].expand(B, -1, -1).contiguous()


def _gate(g, B, H, T):
    return torch.sigmoid(torch.randn(B, H, T, 2, device="cuda", generator=g)).bfloat16()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind, B, H, T = case["kind"], case["B"], case["H"], case["T"]
    s = dict(case)
    if kind in ("op_fwd", "op_train"):
        s["q"], s["k"] = (_features(g, B, H, T, case["inputs"]) for _ in range(2))
        s["v"], s["gate"] = _features(g, B, H, T), _gate(g, B, H, T)
        if kind == "op_train":
            for n in ("q", "k", "v", "gate"):
                s[n].requires_grad_(True)
            s["dy"] = (0.1 * torch.randn(B, T, H * D, device="cuda", generator=g)).bfloat16()
    elif kind in ("module_fwd", "module_train"):
        m = speed3r_b200.SparseFlashAttentionRope(H * D, num_heads=H, qkv_bias=True, proj_bias=True, qk_norm=True,
                                                  rope=speed3r_b200.RoPE2D(100.0)).cuda()
        with torch.no_grad():
            for lin in (m.qkv, m.proj, m.gate[0]):
                lin.weight.normal_(0.0, 0.02, generator=g)
            for lin in (m.qkv, m.proj):                       # the gate keeps its (-1, +1) bias
                lin.bias.normal_(0.0, 0.02, generator=g)
            for ln in (m.q_norm, m.k_norm):
                ln.weight.add_(0.1 * torch.randn(D, device="cuda", generator=g))
                ln.bias.normal_(0.0, 0.1, generator=g)
        s["m"], s["xpos"] = m, _positions(B, T)
        x = torch.randn(B, T, H * D, device="cuda", generator=g)
        s["x"] = x.bfloat16() if case["x"] == "bf16" else x
        if kind == "module_train":
            s["x"].requires_grad_(True)
            s["dy"] = (0.1 * torch.randn(B, T, H * D, device="cuda", generator=g)).bfloat16()
            s["wrt"] = [s["x"]] + list(m.parameters())
        else:
            m.eval()
    elif kind == "sel_train":
        nb, K = -(-T // case["block"]), case["K"]
        # distinct blocks spread over the sequence: one in each K-th of it
        u = torch.rand(B, H, nb, K, device="cuda", generator=g)
        s["idx"] = ((torch.arange(K, device="cuda") + u) * (nb / K)).int().clamp_(0, nb - 1)
        s["q"], s["k"], s["v"] = (_features(g, B, H, T).requires_grad_(True) for _ in range(3))
        s["do"] = (0.1 * torch.randn(B, H, T, D, device="cuda", generator=g)).bfloat16()
    elif kind == "rank_share":
        G, n = case["G"], T // case["G"]
        s["q"], s["gate"] = _features(g, B, H, n), _gate(g, B, H, n)
        for x in ("k", "v"):
            dense = _features(g, B, H, T)
            s[x + "_c"] = ops.pool_tokens(dense, 16, 16)
            s[x] = dense.view(B, H, G, n, D).permute(2, 0, 1, 3, 4).contiguous()
    else:
        s["pipe"] = HostPipeline(H, T, D, device=torch.device("cuda", torch.cuda.current_device()))
        dev = [_features(g, 1, H, T) for _ in range(3)] + [_gate(g, 1, H, T)]
        s["host"] = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in dev]
        s["hy"] = torch.empty(1, T, H * D, dtype=torch.bfloat16, pin_memory=True)
    return s


def run(s):
    kind = s["kind"]
    if kind == "op_fwd":
        with torch.no_grad():
            y, idx = ops.sparse_attention_op(s["q"], s["k"], s["v"], s["gate"], *_settings(s))
        return {"y": y, "idx": idx}
    if kind == "op_train":
        y, idx = ops.sparse_attention_op(s["q"], s["k"], s["v"], s["gate"], *_settings(s))
        grads = torch.autograd.grad(y, (s["q"], s["k"], s["v"], s["gate"]), s["dy"])
        return {"y": y.detach(), "idx": idx, "grads": grads}
    if kind == "module_fwd":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return s["m"](s["x"], xpos=s["xpos"])
    if kind == "module_train":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = s["m"](s["x"], xpos=s["xpos"])
        return {"y": y.detach(), "grads": torch.autograd.grad(y, s["wrt"], s["dy"])}
    if kind == "sel_train":
        o = ops.topk_blocksparse_attention(s["q"], s["k"], s["v"], s["idx"], s["block"])
        return {"o": o.detach(), "grads": torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"])}
    if kind == "rank_share":
        with torch.no_grad():
            q_c = ops.pool_tokens(s["q"], 16, 16)
            o_c, idx = ops.flash_attn_topk_func(q_c, s["k_c"], s["v_c"], 32)
            y = ops.sel_attn_merge_chunked(s["q"], s["k"], s["v"], idx, s["gate"], o_c, 16)
        return {"y": y, "idx": idx}
    s["pipe"](*s["host"], s["hy"])
    return s["hy"]


def work(case):
    """Products of the two branches (2.5 times as many again in a backward), and every input read and output
    written once."""
    kind, B, H, T = case["kind"], case["B"], case["H"], case["T"]
    tok = B * H * T * D * 2                                   # one bf16 tensor of the sequence
    if kind == "sel_train":
        b, K = case["block"], case["K"]
        return {"bytes": 8 * tok + 4 * B * H * -(-T // b) * K, "flops": 3.5 * 4 * B * H * T * K * b * D}
    if kind == "rank_share":
        n, nq, nc = T // case["G"], T // case["G"] // 16, T // 16
        return {"bytes": 2 * B * H * D * 2 * (n + T + nc) + 4 * B * H * (n + nq * 32),
                "flops": 4 * B * H * D * (nq * nc + n * 32 * 16)}
    blk, K, Lc, Sc = _settings(case)
    nq, nc = T // blk, (T - Lc) // Sc + 1
    flops = 4 * B * H * D * (nq * nc + T * K * blk)
    gate, idx = B * H * T * 4, B * H * nq * K * 4
    if kind == "op_fwd":
        return {"bytes": 4 * tok + gate + idx, "flops": flops}
    if kind == "op_train":
        return {"bytes": 8 * tok + 2 * gate + idx, "flops": 3.5 * flops}
    if kind == "host":
        return {"bytes": 4 * tok + gate, "flops": flops}
    C = H * D
    x = B * T * C * (4 if case["x"] == "fp32" else 2)
    params, linear = 4 * (4 * C * C + 2 * C * H), 2 * B * T * C * (4 * C + 2 * H)
    if kind == "module_fwd":
        return {"bytes": x + tok + params, "flops": flops + linear}
    return {"bytes": 2 * x + 2 * tok + 2 * params, "flops": 3.5 * flops + 3 * linear}


def tolerance(case):
    """bf16 tensors and bf16 rounding of P and dS inside the kernels.  ``differ``: entries of the table whose
    scores tie within the rounding of fp32 sums.  In the modules q and k are rounded to bf16 twice on the way to the
    table, so that single blocks can be swapped where their scores are close: single rows differ by more."""
    if case["kind"] in ("module_fwd", "module_train"):
        return {"rel": 1.5e-2, "max": 0.6}
    if case["kind"] in ("sel_train", "host"):
        return {"rel": 1e-2}
    return {"rel": 1e-2, "differ": 1e-3}
