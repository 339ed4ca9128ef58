"""Edges of single kernels: sizes and layouts at which a tile, a ring or a dispatch rule changes."""
import pytest
import torch

from _util import assert_bf16_close, assert_idx_match, bf16_round
from oracle import restatement as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def randn(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


def table(seed, B, H, nqb, nkb, K):
    return torch.randint(0, nkb, (B, H, nqb, K), generator=torch.Generator().manual_seed(seed), dtype=torch.int32)


# ------------------------------------------------------------------ selection, blocks of 16
@pytest.mark.parametrize("K", [1, 2, 3, 33, 64])
@pytest.mark.parametrize("layout", ["k below v", "v below k", "k is v"])
def test_sel16_fwd_rings_and_layouts(K, layout):
    """Lists of odd length (the last pair is half empty), one-entry lists, the longest list, a last block cut
    short, and keys and values in either order in memory (one copy brings both) or the same tensor."""
    from speed3r_b200 import ops
    B, H, T = 1, 3, 16 * 21 + 5
    nb = -(-T // 16)
    q, k, v = bf16_round(randn(1, B, H, T, 64), randn(2, B, H, T, 64), randn(3, B, H, T, 64))
    idx = table(4, B, H, nb, nb, K)
    idx[:, :, 2] = -1                                          # a query block without any valid entry
    idx[:, :, 3, 0] = nb - 1                                   # the short block
    buf = torch.empty(2, B, H, T, 64, device=DEV, dtype=torch.bfloat16)
    kd, vd = (buf[0], buf[1]) if layout == "k below v" else (buf[1], buf[0])
    kd.copy_(k)
    if layout == "k is v":
        v, vd = k, kd
    else:
        vd.copy_(v)
    o, lse, _ = ops._sel_fwd(q.to(DEV, torch.bfloat16), kd, vd, idx.to(DEV), None, None, 16, 0.125, True, True, 1)
    ref, lse_ref = R.sel_attn(q, k, v, idx, 16)
    rows = torch.ones(T, dtype=torch.bool)
    rows[32:48] = False
    assert_bf16_close(o[:, :, rows.to(DEV)], ref[:, :, rows], f"sel16 K={K} {layout}")
    assert_bf16_close(lse[:, :, rows.to(DEV)], lse_ref[:, :, rows], "lse", max_abs=5e-3, mean_abs=1e-3, scale_with_ref=False)
    assert (o[:, :, 32:48] == 0).all() and (lse[:, :, 32:48] == -float("inf")).all()


def test_sel16_fwd_offset_follows_growing_scores():
    """Scores that grow along the list past 2^24 times the first pair's move the exponent offset."""
    from speed3r_b200 import ops
    B, H, T, K = 1, 2, 512, 32
    q, k, v = bf16_round(4 * randn(5, B, H, T, 64), randn(6, B, H, T, 64), randn(7, B, H, T, 64))
    k, = bf16_round(k * torch.linspace(0.1, 4.0, T).view(1, 1, T, 1))
    idx = torch.arange(32, dtype=torch.int32).expand(B, H, T // 16, K).contiguous()
    o, lse, _ = ops._sel_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), idx.to(DEV), None, None, 16, 0.125, True, True, 1)
    ref, lse_ref = R.sel_attn(q, k, v, idx, 16)
    assert_bf16_close(o, ref, "growing scores")
    assert ((lse.cpu() - lse_ref).abs() <= 1e-4 * lse_ref.abs() + 1e-3).all()


# ------------------------------------------------------------------ key-centric index
@pytest.mark.parametrize("Nq,Nkb,K", [(768, 700, 32), (769, 700, 32),           # one CTA per head | the five kernels
                                      (100, 8192, 8), (100, 8193, 8), (3000, 40, 32)])
@pytest.mark.parametrize("spread", ["even", "skewed", "one"])
def test_key_csr_segment_classes(Nq, Nkb, K, spread):
    """Segments of every length class on both sides of the one-kernel line, against a stable argsort."""
    from speed3r_b200 import ops
    B, H = 1, 2
    g = torch.Generator().manual_seed(11)
    u = torch.rand(B, H, Nq, K, generator=g)
    idx = {"even": u * Nkb, "skewed": u ** 4 * Nkb, "one": torch.full_like(u, 3)}[spread].int()
    idx[:, :, 1, 0], idx[:, :, 2, 1] = -1, Nkb                  # dropped entries
    off, qids = (t.cpu() for t in ops.build_key_csr(idx.to(DEV), Nkb))
    for h in range(H):
        flat = idx[0, h].flatten().long()
        keep = (flat >= 0) & (flat < Nkb)
        key, q = flat[keep], torch.arange(Nq).repeat_interleave(K)[keep]
        counts = torch.bincount(key, minlength=Nkb)
        assert torch.equal(off[0, h].long(), torch.cat((torch.zeros(1, dtype=torch.long), counts.cumsum(0))))
        order = torch.argsort(key, stable=True)
        assert torch.equal(qids[0, h, :len(key)].long(), q[order])


# ------------------------------------------------------------------ selection backward
@pytest.mark.parametrize("block,K,T", [(16, 1, 16 * 5 + 3), (16, 7, 16 * 40), (32, 3, 32 * 6 + 17), (64, 2, 64 * 3 + 1), (64, 5, 64 * 9)])
def test_sel_bwd_tiles(block, K, T):
    """Odd numbers of tiles, blocks of several tiles, tiles that lie past the end of the sequence, unlisted blocks."""
    from speed3r_b200 import ops
    B, H = 1, 2
    nb = -(-T // block)
    q, k, v, do = bf16_round(*(randn(20 + i, B, H, T, 64) for i in range(4)))
    idx = table(25, B, H, nb, max(1, nb - 1), K)
    idx[:, :, 0, 0] = nb - 1
    qg, kg, vg = (t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v))
    ops.topk_blocksparse_attention(qg, kg, vg, idx.to(DEV), block).backward(do.to(DEV, torch.bfloat16))
    qr, kr, vr = (t.clone().requires_grad_(True) for t in (q, k, v))
    R.sel_attn(qr, kr, vr, idx, block)[0].backward(do)
    for n, a, b in (("dq", qg, qr), ("dk", kg, kr), ("dv", vg, vr)):
        assert_bf16_close(a.grad, b.grad, f"{n} block {block} K {K} T {T}")


# ------------------------------------------------------------------ the op as one autograd node
@pytest.mark.parametrize("block,kernel,stride,topk", [(16, 16, 16, 8), (64, 32, 16, 4), (16, 8, 4, 8), (32, 32, 32, 4)])
def test_op_node_gradients_match_separate_nodes(block, kernel, stride, topk):
    """The pooled branch's gradients added inside the selection kernels (or, for windows that are not multiples of 16,
    by the pooling kernel) against the chain of separate nodes, which rounds each share to bf16 before adding:
    three roundings of 2^-9 relative to a share instead of one."""
    from speed3r_b200 import ops
    B, H, T = 2, 2, 64 * 9
    x = [randn(30 + i, B, H, T, 64).to(DEV, torch.bfloat16) for i in range(3)]
    gate = torch.sigmoid(randn(33, B, H, T, 2)).to(DEV, torch.bfloat16)
    dy = randn(34, B, T, H * 64).to(DEV, torch.bfloat16)
    leaves = lambda: [t.clone().requires_grad_(True) for t in (*x, gate)]
    a = leaves()
    y, idx = ops.sparse_attention_op(*a, block, topk, kernel, stride)
    y.backward(dy)
    b = leaves()
    q_c, k_c, v_c = (ops.pool_tokens(b[0], block, block), ops.pool_tokens(b[1], kernel, stride), ops.pool_tokens(b[2], kernel, stride))
    if kernel == block:
        o_c, idx2 = ops.flash_attn_topk_func(q_c, k_c, v_c, topk)
    else:
        o_c, idx2 = ops.flash_attn_blocktopk_func(q_c, k_c, v_c, topk, block // stride, (block - kernel) // stride + 1)
    y2 = ops.sel_attn_merge(b[0], b[1], b[2], idx2, b[3], o_c, block)
    y2.backward(dy)
    assert torch.equal(y, y2) and torch.equal(idx, idx2)
    assert torch.equal(a[3].grad, b[3].grad)
    for n, s, t in zip("qkv", a, b):
        scale = t.grad.float().abs().max()
        assert (s.grad.float() - t.grad.float()).abs().max() <= 3 * 2 ** -8 * scale, n


# ------------------------------------------------------------------ compression attention and its table
@pytest.mark.parametrize("jump", [1.0, 40.0])
def test_cmp_offset_of_the_first_tile(jump):
    """Rows whose later scores outgrow those of the first 128 keys: within the range of a float (one pass) and far
    beyond it (the CTA's second pass), next to rows that need neither."""
    from speed3r_b200 import ops
    B, H, Nq, Nc = 1, 2, 300, 700
    q, k, v = randn(40, B, H, Nq, 64), randn(41, B, H, Nc, 64), randn(42, B, H, Nc, 64)
    k[:, :, 500:] *= jump
    q[:, :, ::3] *= 0.01
    q, k, v = bf16_round(q, k, v)
    o, lse, idx = ops._cmp_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), 32, 0.125)
    ref, lse_ref, idx_ref = R.cmp_attn_topk(q, k, v, 32)
    S = q @ k.transpose(-1, -2)
    # fp32 sums of 64 products of that size in another order
    assert_idx_match(idx, idx_ref, S, f"jump {jump}", eps=max(1e-3, 64 * 2 ** -24 * S.abs().max().item()))
    assert_bf16_close(o, ref, f"o_c jump {jump}")
    assert ((lse.cpu() - lse_ref).abs() <= 1e-5 * lse_ref.abs() + 1e-3).all()


@pytest.mark.parametrize("Nc", [1, 31, 32, 40, 65, 127, 128, 129, 15 * 128, 15 * 128 + 1, 16 * 128 + 77])
@pytest.mark.parametrize("topk", [1, 7, 32])
def test_cmp_table_sizes(Nc, topk):
    """Fewer keys than table entries, one tile and its neighbours, and both ways of sharing tiles between the two scans."""
    from speed3r_b200 import ops
    B, H, Nq = 1, 2, 257
    q, k, v = bf16_round(randn(50, B, H, Nq, 64), randn(51, B, H, Nc, 64), randn(52, B, H, Nc, 64))
    o, lse, idx = ops._cmp_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), topk, 0.125)
    ref, _, idx_ref = R.cmp_attn_topk(q, k, v, topk)
    assert_idx_match(idx, idx_ref, q @ k.transpose(-1, -2), f"Nc {Nc} topk {topk}")
    assert_bf16_close(o, ref, f"o_c Nc {Nc}")


@pytest.mark.parametrize("heads", [40, 80])
def test_cmp_one_and_two_row_tiles(heads):
    """Both sides of the line between one and two row tiles per CTA, with rows past the end in the second."""
    from speed3r_b200 import ops
    q, k, v = bf16_round(randn(55, 1, heads, 270, 64), randn(56, 1, heads, 200, 64), randn(57, 1, heads, 200, 64))
    o, lse, idx = ops._cmp_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), 32, 0.125)
    ref, _, idx_ref = R.cmp_attn_topk(q, k, v, 32)
    assert_idx_match(idx, idx_ref, q @ k.transpose(-1, -2), f"{heads} heads")
    assert_bf16_close(o, ref, f"o_c {heads} heads")


@pytest.mark.parametrize("period", [1, 16, 64])
def test_cmp_table_when_the_bound_is_loose(period):
    """Keys that repeat with a period: the best logits fall into few of the 64 column groups, so that far more logits than
    a list holds reach the bound and lists are cut; exact repeats are ties, which the smaller column wins."""
    from speed3r_b200 import ops
    B, H, Nq, Nc = 1, 2, 130, 3000
    q, v = bf16_round(randn(60, B, H, Nq, 64), randn(61, B, H, Nc, 64))
    base, = bf16_round(randn(62, B, H, period, 64))
    k = base.repeat(1, 1, -(-Nc // period), 1)[:, :, :Nc].contiguous()
    o, lse, idx = ops._cmp_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), 32, 0.125)
    ref, _, idx_ref = R.cmp_attn_topk(q, k, v, 32)
    assert_idx_match(idx, idx_ref, q @ k.transpose(-1, -2), f"period {period}")
    # equal logits on the device: whole runs of a repeated key, in column order
    first = idx[..., 0:1].cpu().long()
    assert torch.equal(idx.cpu().long(), first + period * torch.arange(32))
    assert_bf16_close(o, ref, "o_c")
