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


class FarMemory:
    """Device memory at addresses at least 2^40 bytes from `near`, as a virtual-memory reservation can have."""

    def __init__(self, near, nbytes):
        from cuda.bindings import driver as cu
        self.cu = cu
        self.prop = cu.CUmemAllocationProp()
        self.prop.type = cu.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
        self.prop.location.type = cu.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
        self.prop.location.id = torch.cuda.current_device()
        grain = self.ok(cu.cuMemGetAllocationGranularity(self.prop, cu.CUmemAllocationGranularity_flags.CU_MEM_ALLOC_GRANULARITY_MINIMUM))
        self.size = -(-nbytes // grain) * grain
        self.handle = self.ok(cu.cuMemCreate(self.size, self.prop, 0))
        self.span = (1 << 42) + self.size                          # addresses only: one of its ends is far enough away
        status, self.start = cu.cuMemAddressReserve(self.span, 0, 0, 0)
        if int(status) != 0:
            self.ok(cu.cuMemRelease(self.handle))
            pytest.skip("no room for a reservation of 4 TB of addresses")
        ends = (int(self.start), int(self.start) + (1 << 42))
        self.ptr = max(ends, key=lambda e: abs(e - near))
        self.ok(cu.cuMemMap(self.ptr, self.size, 0, self.handle, 0))
        access = cu.CUmemAccessDesc()
        access.location = self.prop.location
        access.flags = cu.CUmemAccess_flags.CU_MEM_ACCESS_FLAGS_PROT_READWRITE
        self.ok(cu.cuMemSetAccess(self.ptr, self.size, [access], 1))
        assert abs(self.ptr - near) >= 1 << 40
        self.__cuda_array_interface__ = dict(shape=(nbytes // 2,), typestr="<i2", data=(self.ptr, False), version=3)

    def ok(self, r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) > 1 else None

    def free(self):
        torch.cuda.synchronize()
        self.ok(self.cu.cuMemUnmap(self.ptr, self.size))
        self.ok(self.cu.cuMemRelease(self.handle))
        self.ok(self.cu.cuMemAddressFree(self.start, self.span))


@pytest.mark.parametrize("block", [16, 32])
def test_selection_on_tensors_more_than_a_tensor_map_reaches_apart(block):
    """Values and output gradients 2^41 bytes or more from keys and queries: forward and backward as with tensors side by side."""
    from speed3r_b200 import ops
    B, H, T, K = 1, 2, 16 * 21 + 5, 5
    nb = -(-T // block)
    q, k, v, do = (randn(s, B, H, T, 64).to(DEV, torch.bfloat16) for s in (1, 2, 3, 4))
    idx = table(5, B, H, nb, nb, K).to(DEV)
    def run(v, do):
        o, lse, _ = ops._sel_fwd(q, k, v, idx, None, None, block, 0.125, True, True, 1)
        dlt = ops._ops().delta.default(o, do)
        return (o, lse) + tuple(ops._ops().sel_attn_bwd.default(q, k, v, idx, lse, dlt, do, block, 0.125))
    want = run(v, do)
    far = FarMemory(k.data_ptr(), 2 * v.numel() * 2)
    try:
        both = torch.as_tensor(far, device=DEV).view(torch.bfloat16).view(2, B, H, T, 64)
        both[0].copy_(v)
        both[1].copy_(do)
        got = run(both[0], both[1])
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        del both
    finally:
        far.free()


@pytest.mark.parametrize("block, K", [(16, 32), (32, 32), (64, 16)])
@pytest.mark.parametrize("outgrow", [False, True])
def test_sel_fwd_rounds_no_more_than_its_result(block, K, outgrow):
    """Queries ten times the usual size, so that few keys hold a row's weight, and (outgrow) keys that grow along the list.
    The largest weight has to be exactly 1 in bf16: what is left is the rounding of the result, 1.66e-3 of its 2-norm (rms of
    rounding to 8 bits), and at most 5e-4 from the smaller weights.  Weights relative to an earlier maximum round by
    another 1.55e-3: 2.2e-3 together."""
    from speed3r_b200 import ops
    B, H, T = 1, 2, 4096
    nb = T // block
    ln = lambda x: torch.nn.functional.layer_norm(x, (64,))
    q, k, v = bf16_round(10 * ln(randn(1, B, H, T, 64)), ln(randn(2, B, H, T, 64)), ln(randn(3, B, H, T, 64)))
    if outgrow:
        k = bf16_round(k * torch.linspace(0.2, 1.5, T)[:, None])[0]
    idx = torch.rand(B, H, nb, nb, generator=torch.Generator().manual_seed(4)).topk(K, -1).indices.sort(-1).values.int()
    o, lse, _ = ops._sel_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), idx.to(DEV), None, None, block, 0.125, True, True, 1)
    ref, lse_ref = R.sel_attn(q.double(), k.double(), v.double(), idx, block)
    err = ((o.cpu().double() - ref).norm() / ref.norm()).item()
    assert err <= 1.8e-3, f"blocks of {block}: {err:.3e}"
    assert (lse.cpu() - lse_ref).abs().max() <= 2e-4


@pytest.mark.parametrize("block", [16, 32, 64])
@pytest.mark.parametrize("chunks", [1, 2])
def test_sel_fwd_keeps_non_finite_values_to_the_blocks_that_selected_them(block, chunks):
    """Infinities and NaN in the values of single key blocks, among them the sequence's first, beside query blocks of the
    same row tile with other lists, a shorter list and none at all: rows of the others are the oracle's, and outside those
    row tiles bit for bit what they are without such values; rows of their own have infinities and NaN where the oracle has
    them."""
    from speed3r_b200 import ops
    B, H, T, K = 1, 2, 1024, 4
    nb = T // block
    q, k, v = bf16_round(randn(1, B, H, T, 64), randn(2, B, H, T, 64), randn(3, B, H, T, 64))
    idx = 4 + table(4, B, H, nb, nb - 4, K)                        # blocks 0 to 3 by hand
    idx[:, :, 0, 1], idx[:, :, 5, 2], idx[:, :, 9, 0] = 0, 1, 2
    idx[:, :, 1] = -1                                              # none
    idx[:, :, 4, 1:] = -1                                          # one block
    bad = v.clone()
    bad[:, :, 3, 5], bad[:, :, block + 1, 7], bad[:, :, 2 * block + 2, 60] = float("inf"), float("nan"), float("-inf")
    def run(x):
        t = lambda a: a.to(DEV, torch.bfloat16)
        part = lambda a: t(a).view(B, H, chunks, T // chunks, 64).permute(2, 0, 1, 3, 4).contiguous() if chunks > 1 else t(a)
        return ops._sel_fwd(t(q), part(k), part(x), idx.to(DEV), None, None, block, 0.125, True, True, chunks)[:2]
    (o, lse), (o_clean, lse_clean) = run(bad), run(v)
    hit = torch.zeros(T, dtype=torch.bool)
    for m in (0, 5, 9):
        hit[m * block:(m + 1) * block] = True
    assert torch.equal(lse, lse_clean) and torch.equal(o[:, :, 9 * block + 128:], o_clean[:, :, 9 * block + 128:])
    ref, _ = R.sel_attn(q, k, bad, idx, block)
    ref[:, :, block:2 * block] = 0                                 # the query block without a list
    assert_bf16_close(o.cpu()[:, :, ~hit], ref[:, :, ~hit], f"blocks of {block}, the others")
    got, want = o.cpu().float()[:, :, hit], ref[:, :, hit]
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    fin = want.isfinite()
    assert_bf16_close(got[fin], want[fin], f"blocks of {block}")


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("first", [0, 200])
def test_nan_scores_are_not_lost(first, value):
    """A NaN in one key (or an infinity, whose score is +infinity in half of the rows) makes the rows that see it NaN, wherever in a tile the key stands (head h: key first + h; some
    exponentials are polynomials, whose clamp and exponent arithmetic could make a number of it), and is never ranked."""
    from speed3r_b200 import ops
    B, H, T = 1, 32, 512
    q, k, v = bf16_round(randn(1, B, H, T, 64), randn(2, B, H, T, 64), randn(3, B, H, T, 64))
    for h in range(H):
        k[0, h, first + h, 3] = value
    nan = torch.full((B, H, T), True) if value != value else q[..., 3] > 0        # -infinity: the key has no weight
    t = [x.to(DEV, torch.bfloat16) for x in (q, k, v)]
    o, lse, idx = ops._cmp_fwd(*t, 32, 0.125)
    assert torch.equal(o.isnan().all(-1).cpu(), nan) and torch.equal(o.isnan().any(-1).cpu(), nan)
    assert torch.equal(lse.isnan().cpu(), nan)
    ranked = (idx.cpu() == (first + torch.arange(H))[None, :, None, None]).any(-1)
    assert not ranked.any() if value != value else torch.equal(ranked, nan)
    _, _, blocks = ops._ops().cmp_attn_blocktopk_fwd.default(*t, 16, 0.125, 4, 3)
    if value != value:
        assert (blocks.cpu() != ((first + torch.arange(H)) // 4)[None, :, None, None]).masked_fill(((first + torch.arange(H)) % 4 == 3)[None, :, None, None], True).all()
    for block in (16, 32, 64):
        nb = T // block
        table = torch.arange(nb, dtype=torch.int32).expand(B, H, nb, nb).contiguous().to(DEV)
        o, lse, _ = ops._sel_fwd(*t, table, None, None, block, 0.125, True, True, 1)
        assert torch.equal(o.isnan().all(-1).cpu(), nan) and torch.equal(o.isnan().any(-1).cpu(), nan), f"blocks of {block}"
        assert torch.equal(lse.isnan().cpu(), nan), f"blocks of {block}"


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


@pytest.mark.parametrize("Tq,Tk,K", [(64, 64, 1), (64 * 3 + 1, 64 * 5 + 63, 3), (64 * 7, 64 * 2 + 17, 4), (64 * 40 - 1, 64 * 3, 33), (64 * 2, 64 * 70, 64)])
def test_sel_bwd64_lists(Tq, Tk, K):
    """Blocks of 64: lists of odd and even length, of none and of more entries than a lane holds at once, repeated and skipped
    entries, first, last and cut-short blocks, as many queries as keys or not; values that are not finite stay with the rows
    that use them."""
    from speed3r_b200 import _lib, ops
    B, H = 2, 2
    nq, nk = -(-Tq // 64), -(-Tk // 64)
    assert _lib.load_check().s3r_check_sel_bwd64_pays(B * H, nq, nk, K)
    q, do = bf16_round(randn(90, B, H, Tq, 64), randn(91, B, H, Tq, 64))
    k, v = bf16_round(randn(92, B, H, Tk, 64), randn(93, B, H, Tk, 64))
    idx = table(94, B, H, nq, nk, K)
    idx[:, 1, :, K // 2:] = -1                                           # skipped entries behind the first half
    idx[:, :, 0, 0] = nk - 1                                             # the short block
    idx[1, 1, :, 0] = 0
    if nk > 2:
        idx[0, 0][idx[0, 0] == 1] = 0                                    # a block nobody selects
    ref, idx_ref, do_ref = [t.clone().requires_grad_(True) for t in (q, k, v)], idx.clone(), do.clone()
    if nq > 1:
        idx[1, 0, 1] = -1                                                # a list of none: as if nothing came back to its rows
        idx_ref[1, 0, 1], do_ref[1, 0, 64:128] = 0, 0.0
    R.sel_attn(*ref, idx_ref, 64)[0].backward(do_ref)
    got = [t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v)]
    o = ops.topk_blocksparse_attention(*got, idx.to(DEV), 64)
    grads = torch.autograd.grad(o, got, do.to(DEV, torch.bfloat16), retain_graph=True)
    for n, a, b in zip("qkv", grads, ref):
        assert_bf16_close(a, b.grad, f"d{n} {Tq} {Tk} {K}")
    if nk > 2 and nq > 1:
        bad = do.clone()
        bad[0, 0, 0] = float("nan")                                      # of query block 0: its own keys and its own row
        wrong = torch.autograd.grad(o, got, bad.to(DEV, torch.bfloat16))
        used = torch.zeros(nk, dtype=torch.bool)
        used[idx[0, 0, 0][idx[0, 0, 0] >= 0].long()] = True
        rows = used.repeat_interleave(64)[:Tk]
        for n, a, b in zip("kv", wrong[1:], grads[1:]):
            assert torch.equal(a[0, 0][~rows.to(DEV)], b[0, 0][~rows.to(DEV)]) and torch.equal(a[1], b[1]), n
            assert a[0, 0][rows.to(DEV)].isnan().any(-1).all(), n
        assert wrong[0][0, 0, 0].isnan().all() and torch.equal(wrong[0][0, 0, 1:], grads[0][0, 0, 1:])


@pytest.mark.parametrize("block", [16, 32, 64])
@pytest.mark.parametrize("which", ["q", "k", "v"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_sel_bwd_keeps_non_finite_values_to_the_rows_that_use_them(block, which, value):
    """A query reaches its own row and the keys of its list; a key or value the query blocks that selected it and the keys of their
    lists.  All other gradients are the same bits as without it (from the same forward: that of blocks of 32 and 64 rounds the rows beside
    such rows otherwise)."""
    from speed3r_b200 import ops
    B, H, nb, K, at = 1, 2, 20, 3, 5 * block + 7
    T = block * nb - 5
    x = dict(zip("qkv", bf16_round(*(randn(110 + i, B, H, T, 64) for i in range(3)))))
    do = randn(113, B, H, T, 64).to(DEV, torch.bfloat16)
    idx = table(114, B, H, nb, nb, K)
    idx[:, :, 5], idx[:, :, 6] = torch.tensor([5, 5, nb - 1]), torch.tensor([5, 0, -1])
    users = torch.arange(nb) == 5                                        # query blocks that read the value, and their lists
    if which != "q":
        users = (idx[0, 0] == 5).any(-1)
    listed = torch.zeros(nb, dtype=torch.bool)
    listed[idx[0, 0][users][idx[0, 0][users] >= 0].long()] = True
    rows, keys = (t.repeat_interleave(block)[:T] for t in (users, listed))
    if which == "q":
        rows = torch.arange(T) == at
    idx = idx.to(DEV)
    dev = lambda: [x[n].to(DEV, torch.bfloat16) for n in "qkv"]
    forward = lambda: ops._sel_fwd(*dev(), idx, None, None, block, 0.125, True, True, 1)[:2]
    backward = lambda o, lse: [g.cpu() for g in ops._ops().sel_attn_bwd(*dev(), idx, lse, (o.float() * do.float()).sum(-1), do, block, 0.125)]
    o, lse = forward()
    clean = backward(o, lse)
    x[which] = x[which].clone()
    x[which][0, 0, at, 9] = value
    o_bad, lse_bad = forward()
    o[0, 0, rows], lse[0, 0, rows] = o_bad[0, 0, rows], lse_bad[0, 0, rows]
    bad = backward(o, lse)
    for n, reached, a, b in zip("qkv", (rows, keys, keys), bad, clean):
        assert torch.equal(a[0, 1], b[0, 1]) and torch.equal(a[0, 0][~reached], b[0, 0][~reached]), n
    assert not bad[0][0, 0][rows].isfinite().all() and all(b.isfinite().all() for b in clean)


@pytest.mark.parametrize("Tq,Tk,K", [(64 * 130 - 9, 64 * 130 - 9, 1), (64 * 131, 64 * 130, 2), (64 * 2, 64 * 300 - 1, 16), (64 * 200, 64 * 50, 1)])
def test_sel_bwd_short_lists_of_blocks_of_64(Tq, Tk, K):
    """Lists too short, or too few of them, for the tcgen05 kernel: the kernel of the other block sizes, four tiles per block."""
    from speed3r_b200 import _lib, ops
    B, H, nq, nk = 1, 16, -(-Tq // 64), -(-Tk // 64)
    assert not _lib.load_check().s3r_check_sel_bwd64_pays(H, nq, nk, K)
    q, do = bf16_round(randn(104, B, H, Tq, 64), randn(105, B, H, Tq, 64))
    k, v = bf16_round(randn(106, B, H, Tk, 64), randn(107, B, H, Tk, 64))
    idx = table(108, B, H, nq, nk, K)
    ref = [t.clone().requires_grad_(True) for t in (q, k, v)]
    R.sel_attn(*ref, idx, 64)[0].backward(do)
    got = [t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v)]
    ops.topk_blocksparse_attention(*got, idx.to(DEV), 64).backward(do.to(DEV, torch.bfloat16))
    for n, a, b in zip("qkv", got, ref):
        assert_bf16_close(a.grad, b.grad, f"d{n} {Tq} {Tk} {K}")


@pytest.mark.parametrize("block", [16, 64])
@pytest.mark.parametrize("Tq", [64, 64 * 2, 64 * 3, 64 * 3 - 16, 64 * 6 - 32])
def test_sel_bwd_keys_that_are_minus_infinity(block, Tq):
    """A key whose scores are all minus infinity has no weight: dK and dV there are those of a key far below all others, whether its
    list of query blocks is of odd or even length, and whether or not the last of them is cut short."""
    from speed3r_b200 import ops
    B, H, Tk = 1, 2, 64 * 3
    q, do = bf16_round(randn(100, B, H, Tq, 64), randn(101, B, H, Tq, 64))
    k, v = bf16_round(randn(102, B, H, Tk, 64), randn(103, B, H, Tk, 64))
    q[..., 5] = q[..., 5].abs() + 0.5
    idx = torch.arange(Tk // block, dtype=torch.int32).expand(B, H, -(-Tq // block), -1).contiguous()
    k[:, :, 3, 5] = -1e5
    k[:, :, 77, 5] = -1e5
    ref = [t.clone().requires_grad_(True) for t in (q, k, v)]
    R.sel_attn(*ref, idx, block)[0].backward(do)
    k[k[..., 5] == -1e5, 5] = -float("inf")
    got = [t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v)]
    grads = torch.autograd.grad(ops.topk_blocksparse_attention(*got, idx.to(DEV), block), got, do.to(DEV, torch.bfloat16))
    for n, a, b in zip("kv", grads[1:], ref[1:]):
        assert_bf16_close(a, b.grad, f"d{n}")
        assert (a[:, :, [3, 77]] == 0).all(), f"d{n}"


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


@pytest.mark.parametrize("heads, n", [(2, 130), (16, 128), (16, 1152), (12, 1500), (16, 2400)])
def test_cmp_tables_of_calls_in_a_row(heads, n):
    """A kernel's CTAs start while the one in front is still finishing, within a call and between calls: tables and outputs are
    those of calls that have the GPU to themselves (one row tile per CTA, two, and both kinds in one grid)."""
    from speed3r_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n)
    sets = [[torch.randn(1, heads, n, 64, device=DEV, generator=g).mul_(0.2 + 0.2 * i).bfloat16() for _ in range(3)] for i in range(6)]
    alone = []
    for x in sets:
        torch.cuda.synchronize()
        alone.append([t.clone() for t in ops.flash_attn_topk_func(*x, 32)])
        torch.cuda.synchronize()
    for _ in range(4):
        for x, want in zip(sets, [list(ops.flash_attn_topk_func(*x, 32)) for x in sets]):
            ref = alone[[a is x for a in sets].index(True)]
            assert torch.equal(want[0], ref[0]) and torch.equal(want[1], ref[1])


@pytest.mark.parametrize("take", [0, 3])
@pytest.mark.parametrize("heads, n", [(2, 130), (16, 128), (8, 600), (24, 700), (170, 130)])
def test_cmp_tables_of_operands_just_written_over_stale_tables(heads, n, take):
    """What a call reads is what the kernels directly in front of it wrote, and its bounds are this call's: the operands' buffers get
    other values in front of every call, and the table words that, taken for a bound, would let no key through.  Columns and blocks; one
    row tile per CTA, two, and both kinds in one grid."""
    from speed3r_b200 import _lib
    sets = [bf16_round(*((0.5 + 0.5 * i) * randn(10 * i + j, 1, heads, n, 64) for j in range(3))) for i in range(4)]
    dev = [[t.to(DEV, torch.bfloat16) for t in x] for x in sets]
    q, k, v, o = (torch.empty_like(dev[0][0]) for _ in range(4))
    lse = torch.empty(1, heads, n, device=DEV)
    idx = torch.empty(1, heads, n, 16, device=DEV, dtype=torch.int32)
    got = [[torch.empty_like(idx), torch.empty_like(o)] for _ in sets]
    torch.cuda.synchronize()
    st = torch.cuda.current_stream().cuda_stream
    args = (q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), idx.data_ptr(), 1, heads, n, n, 64, 16, 0.125)
    for i, (x, out) in enumerate(zip(dev, got)):
        idx.fill_((0x7f000000, 0x7f800000)[i % 2])             # 2^127 and +inf as floats
        for a, b in zip((v, k, q), x[::-1]):
            a.copy_(b)
        if take:
            _lib.check(_lib.load().s3r_cmp_attn_blocktopk_fwd(*args, 4, take, st), "s3r_cmp_attn_blocktopk_fwd")
        else:
            _lib.check(_lib.load().s3r_cmp_attn_topk_fwd(*args, st), "s3r_cmp_attn_topk_fwd")
        out[0].copy_(idx)
        out[1].copy_(o)
    assert _lib.device_status() == 0
    for (q_, k_, v_), out in zip(sets, got):
        ref, _, idx_ref = R.cmp_attn_topk(q_, k_, v_, 16, rank_group=(4, take) if take else None)
        S = q_ @ k_.transpose(-1, -2)
        # fp32 sums of 64 products of that size in another order
        eps = max(1e-3, 64 * 2 ** -24 * S.abs().max().item())
        assert_idx_match(out[0], idx_ref, R.block_rank_scores(S, 0.125, 4, take) if take else S, f"{heads} heads {n}", eps=eps)
        assert_bf16_close(out[1], ref, f"o_c {heads} heads {n}")


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


@pytest.mark.parametrize("topk", [1, 6, 32])
@pytest.mark.parametrize("Nc", [50, 130, 1030])
def test_cmp_both_kinds_in_one_grid(topk, Nc):
    """More row tiles than SMs: attention and collection share a grid, twice with the same buffers (the table is filled anew)."""
    from speed3r_b200 import ops
    B, H, Nq = 1, 170, 130
    q, k, v = bf16_round(randn(65, B, H, Nq, 64), randn(66, B, H, Nc, 64), randn(67, B, H, Nc, 64))
    g = [t.to(DEV, torch.bfloat16) for t in (q, k, v)]
    for _ in range(2):
        o, lse, idx = ops._cmp_fwd(*g, topk, 0.125)
    ref, lse_ref, idx_ref = R.cmp_attn_topk(q, k, v, topk)
    assert_idx_match(idx, idx_ref, q @ k.transpose(-1, -2), f"Nc {Nc} topk {topk}")
    assert_bf16_close(o, ref, "o_c")
    assert_bf16_close(lse, lse_ref, "lse", max_abs=5e-3, mean_abs=1e-3, scale_with_ref=False)


@pytest.mark.parametrize("Nc,take,topk,heads", [(3, 3, 4, 2), (128 * 3 + 2, 3, 32, 2), (128 * 4, 1, 16, 2), (128 * 5 - 1, 4, 32, 2),
                                                (128 * 20 + 5, 2, 7, 2), (128 * 3 + 127, 3, 16, 170)])
def test_cmp_block_ranking_tiles(Nc, take, topk, heads):
    """Odd and even numbers of key tiles (two sets of group maxima), a last block that counts only if its columns exist, all
    numbers of counted columns, and both kinds of CTA in one grid."""
    from speed3r_b200 import ops
    B, Nq = 1, 70
    q, k, v = bf16_round(randn(70, B, heads, Nq, 64), randn(71, B, heads, Nc, 64), randn(72, B, heads, Nc, 64))
    o, idx = ops.flash_attn_blocktopk_func(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), topk, 4, take)
    ref, _, idx_ref = R.cmp_attn_topk(q, k, v, topk, rank_group=(4, take))
    scores = R.block_rank_scores(q @ k.transpose(-1, -2), 0.125, 4, take)
    n = scores.shape[-1]
    assert_idx_match(idx[..., :min(topk, n)], idx_ref[..., :min(topk, n)], scores, f"Nc {Nc} take {take}")
    assert (idx[..., n:] == n - 1).all()
    assert_bf16_close(o, ref, "o_c")


@pytest.mark.parametrize("copies", [2, 3, 4, 8, 16, 32])
@pytest.mark.parametrize("Nc", [48, 96, 384, 1536, 3264])
def test_cmp_topk_orders_equal_logits(copies, Nc):
    """Every key there several times, so that each logit is: both lists of a row hold some of the equal ones, for 48 keys the
    bound is negative and its keys are cut.  Powers of two end with the 32nd place, of three copies one is lost: equal logits stand in
    the order of their columns either way, in runs short enough to be put in order as neighbours and in longer ones."""
    from speed3r_b200 import ops
    B, H, Nq, n = 2, 2, 200, Nc // copies
    q, k = bf16_round(randn(95, B, H, Nq, 64), randn(96, B, H, n, 64) / 4)
    k = k.repeat(1, 1, copies, 1)
    v, = bf16_round(randn(97, B, H, n * copies, 64))
    idx = ops._cmp_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), 32, 0.125)[2].cpu()
    S = q.double() @ k[:, :, :n].double().transpose(-1, -2)
    best, cols = S.topk(min(32 // copies + 1, n), dim=-1)
    # rows whose different keys are further apart than fp32 sums of 64 products can differ
    clear = ((best[..., :-1] - best[..., 1:]) > 64 * 2 ** -24 * S.abs().max()).all(-1)
    assert clear.float().mean() > 0.5
    want = (cols[..., None] + torch.arange(copies) * n).flatten(-2)[..., :32]
    assert torch.equal(idx[clear].long(), want[clear])


def test_cmp_topk_of_equal_logits_takes_no_longer():
    """Runs of 32 equal logits, out of order in a row's lists, are sorted once: 64 keys that are all the same take less time than 64
    different ones (0.9 of it; put in order as neighbours, pass by pass, 1.9)."""
    from speed3r_b200 import ops
    q, v = (randn(s, 1, 16, 64, 64).to(DEV, torch.bfloat16) for s in (1, 2))
    k = randn(3, 1, 16, 64, 64).to(DEV, torch.bfloat16)
    def us(k):
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                ops._cmp_fwd(q, k, v, 32, 0.125)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 50)
        return best
    same, different = us(k[:, :, :1].expand(-1, -1, 64, -1).contiguous()), us(k)
    assert same < 1.3 * different, (same, different)


# ------------------------------------------------------------------ selection backward
@pytest.mark.parametrize("block,T,K", [(16, 16 * 500 + 9, 3), (16, 16 * 520, 9), (32, 32 * 270 - 1, 2), (64, 64 * 130 + 1, 5)])
def test_sel_bwd_tasks_handed_over(block, T, K):
    """More tasks than places on the GPU, so that warps take over others' (blocks of 64, whose CTAs do not, beside them): lists of no
    entry, one, and several hundred (a key block that every query block selects), an odd number of tiles, a short last block."""
    from speed3r_b200 import ops
    B, H, nb = 1, 4, -(-T // block)
    q, k, v, do = bf16_round(*(randn(75 + i, B, H, T, 64) for i in range(4)))
    idx = table(79, B, H, nb, nb, K)
    idx[:, 1] = idx[:, 1] // 7 * 7                                       # six of seven blocks unselected
    idx[:, 2, :, 0] = nb // 2                                            # selected by all
    idx[:, 3] = torch.arange(nb, dtype=torch.int32)[:, None]             # every block once per entry
    idx[:, 3, :, 1:] = -1
    ref = [t.clone().requires_grad_(True) for t in (q, k, v)]
    R.sel_attn(*ref, idx, block)[0].backward(do)
    got = [t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v)]
    ops.topk_blocksparse_attention(*got, idx.to(DEV), block).backward(do.to(DEV, torch.bfloat16))
    for n, a, b in zip("qkv", got, ref):
        assert_bf16_close(a.grad, b.grad, f"d{n}")


def test_host_pipeline_default_chunks():
    """The sizes a caller gets who names none: all heads in one group on a short sequence, the last group's queries in quarters."""
    from speed3r_b200 import HostPipeline, ops
    H, T = 6, 16 * 300
    hq, hk, hv = (randn(85 + i, 1, H, T, 64).bfloat16().pin_memory() for i in range(3))
    hgate = torch.sigmoid(randn(88, 1, H, T, 2)).bfloat16().pin_memory()
    q, k, v, gate = (t.to(DEV) for t in (hq, hk, hv, hgate))
    y, _ = ops.sparse_attention_op(q, k, v, gate)
    pipe = HostPipeline(H, T, device=DEV)
    assert pipe.hg == H and pipe.rows_last == 256
    hy = torch.zeros(1, T, H * 64, dtype=torch.bfloat16).pin_memory()
    pipe(hq, hk, hv, hgate, hy)
    torch.cuda.synchronize()
    assert torch.equal(hy, y.cpu())


# ------------------------------------------------------------------ prologue backward, module paths
@pytest.mark.parametrize("B,H,Bs,blocks,norm,rope", [(1, 1, 16, 1, True, True), (2, 16, 16, 7, True, True),
                                                     (1, 17, 16, 3, True, True), (2, 3, 4, 5, True, False),
                                                     (1, 2, 9, 4, False, True), (2, 16, 16, 200, True, True)])
def test_prologue_backward(B, H, Bs, blocks, norm, rope):
    """Gradients of the packed projection and of the norms' parameters against autograd through the fp32 restatement: one
    block, more blocks than CTAs, blocks of odd length, more heads than the small kernel takes, no norms, no rotary embedding."""
    import speed3r_b200
    from speed3r_b200 import ops
    N, d = Bs * blocks, 64
    qkv, = bf16_round(1.5 * randn(70, B, N, 3 * H * d) + 0.3)
    pos = torch.randint(0, 37, (B, N, 2), generator=torch.Generator().manual_seed(71)) if rope else None
    norms = [(1 + 0.2 * randn(72 + i, d), 0.1 * randn(74 + i, d)) for i in range(2)] if norm else None
    shapes = [(B, H, N, d)] * 3 + [(B, H, blocks, d)] * 3
    grads = bf16_round(*(randn(80 + i, *s) for i, s in enumerate(shapes)))
    table = speed3r_b200.RoPE2D(100.0)
    cos, sin = table._cos_sin(d // 2, 37, torch.device(DEV), torch.bfloat16) if rope else (None, None)
    x = qkv.to(DEV, torch.bfloat16).requires_grad_(True)
    leaves = [(w.to(DEV).requires_grad_(True), b.to(DEV).requires_grad_(True), 1e-5) for w, b in norms] if norm else [None, None]
    out = ops._prologue(x, H, Bs, pos.to(DEV) if rope else None, cos, sin, *leaves)
    torch.autograd.backward(out, [g.to(DEV, torch.bfloat16) for g in grads])
    xr = qkv.clone().requires_grad_(True)
    ref_leaves = [(w.clone().requires_grad_(True), b.clone().requires_grad_(True)) for w, b in norms] if norm else [None, None]
    ref = _prologue_fp32(xr, H, Bs, pos, cos, sin, *ref_leaves)
    torch.autograd.backward(ref, grads)
    # one rounding to bf16 (2^-9 of the value), and the mean of the block in the restatement is not rounded to bf16
    scale = xr.grad.abs().max().item()
    assert (x.grad.float().cpu() - xr.grad).abs().max().item() <= 1e-2 * scale
    if norm:
        for (w, b, _), (wr, br) in zip(leaves, ref_leaves):
            for a, r in ((w, wr), (b, br)):
                assert (a.grad.cpu() - r.grad).abs().max() <= 2e-3 * max(1.0, r.grad.abs().max().item())


@pytest.mark.parametrize("Bs, blocks", [(1, 40), (3, 5), (16, 9), (18, 4), (35, 3)])
@pytest.mark.parametrize("norm, rope", [(True, True), (False, True), (True, False)])
def test_prologue_forward_blocks(Bs, blocks, norm, rope):
    """Blocks that are no multiple of the four tokens a row takes side by side, nor of the 16 of a chunk; 21 rows, so that a CTA has some
    that do not exist; tokens and means against fp32."""
    import speed3r_b200
    from speed3r_b200 import ops
    B, H, N = 2, 7, Bs * blocks
    qkv, = bf16_round(1.5 * randn(30, B, N, 3 * H * 64) + 0.3)
    pos = torch.randint(0, 37, (B, N, 2), generator=torch.Generator().manual_seed(2)) if rope else None
    cos, sin = speed3r_b200.RoPE2D(100.0)._cos_sin(32, 37, torch.device(DEV), torch.bfloat16)
    wb = [(1 + 0.2 * randn(31 + i, 64), 0.1 * randn(33 + i, 64)) if norm else None for i in range(2)]
    got = ops.qkv_prologue(qkv.to(DEV, torch.bfloat16), H, Bs, pos.to(DEV) if rope else None, cos if rope else None, sin if rope else None,
                           *[(w[0].to(DEV), w[1].to(DEV), 1e-5) if norm else None for w in wb])
    # positions of the means are truncated, and the means rounded to bf16 in front of the norm: two roundings of 2^-9 of values up to ~6
    for name, a, b in zip(("q", "k", "v", "q_c", "k_c", "v_c"), got, _prologue_fp32(qkv, H, Bs, pos, cos, sin, *wb)):
        assert_bf16_close(a, b, f"{name} {Bs}")


@pytest.mark.parametrize("block", [1, 3, 4, 12, 15, 16, 17, 24, 31, 32, 33, 47, 48])
def test_merge_backward_blocks(block):
    """Blocks of one pass and of several, of 4 tokens and of 16, whole and not, with a last block cut short."""
    from speed3r_b200 import ops
    B, H, T = 2, 3, 5 * block + max(1, block // 3)
    nb = -(-T // block)
    dy, o_s, o_c, gate = bf16_round(randn(1, B, T, H * 64), randn(2, B, H, T, 64), randn(3, B, H, nb, 64), torch.sigmoid(randn(4, B, H, T, 2)))
    do_s, dgate, do_c, delta = ops._ops().merge_bwd(*(t.to(DEV, torch.bfloat16) for t in (dy, gate, o_c, o_s)), block)
    g, of = dy.view(B, T, H, 64).transpose(1, 2), o_c.repeat_interleave(block, 2)[:, :, :T]
    dg = torch.stack(((g * of).sum(-1), (g * o_s).sum(-1)), -1)
    c = torch.zeros(B, H, nb * block, 64)
    c[:, :, :T] = gate[..., :1] * g
    # fp32 sums of 64 products up to 2^4 each, in another order
    assert (dgate.cpu() - dg).abs().max() <= 64 * 2 ** -24 * 64 * 16
    assert (delta.cpu() - gate[..., 1] * dg[..., 1]).abs().max() <= 64 * 2 ** -24 * 64 * 16
    assert_bf16_close(do_s, gate[..., 1:] * g, f"do_s block {block}")
    assert_bf16_close(do_c, c.view(B, H, nb, block, 64).sum(3), f"do_c block {block}")


@pytest.mark.parametrize("Bs, blocks", [(13, 5), (18, 300)])
@pytest.mark.parametrize("norm, rope", [(True, True), (False, True), (True, False)])
def test_prologue_forward_one_by_one(Bs, blocks, norm, rope):
    """Blocks below a chunk, and of a chunk and a bit on a grid beyond the GPU."""
    test_prologue_forward_blocks(Bs, blocks, norm, rope)


@pytest.mark.parametrize("Bs", [6100, 6150, 6300, 6310])
@pytest.mark.parametrize("norm, rope", [(True, True), (False, True), (True, False)])
def test_prologue_forward_long_blocks(Bs, norm, rope):
    """The longest blocks whose rows fit shared memory, beside the tables' and without them, and blocks whose rows do not, or have none:
    tokens as with blocks of ten, bit for bit, means against fp32."""
    import speed3r_b200
    from speed3r_b200 import ops
    B, H, N = 2, 3, Bs
    qkv, = bf16_round(1.5 * randn(30, B, N, 3 * H * 64) + 0.3)
    pos = torch.randint(0, 37, (B, N, 2), generator=torch.Generator().manual_seed(2)) if rope else None
    cos, sin = speed3r_b200.RoPE2D(100.0)._cos_sin(32, 37, torch.device(DEV), torch.bfloat16)
    wb = [(1 + 0.2 * randn(31 + i, 64), 0.1 * randn(33 + i, 64)) if norm else None for i in range(2)]
    args = (pos.to(DEV) if rope else None, cos if rope else None, sin if rope else None,
            *[(w[0].to(DEV), w[1].to(DEV), 1e-5) if norm else None for w in wb])
    got, tens = (ops.qkv_prologue(qkv.to(DEV, torch.bfloat16), H, b, *args) for b in (Bs, 10))
    assert all(torch.equal(a, b) for a, b in zip(got[:3], tens[:3]))
    # The norm divides a block's mean, 0.3 and rounded to bf16 within 2^-11, by its spread of 1.5 / sqrt(Bs) = 0.019: 0.026, times weights
    # up to 1.6 and, rotated, the sum of two; the sum's order may turn a rounding the other way, which doubles it
    for name, a, b in zip(("q_c", "k_c", "v_c"), got[3:], _prologue_fp32(qkv, H, Bs, pos, cos, sin, *wb)[3:]):
        err = (a.float().cpu() - b).abs()
        assert err.max() <= (2 * 2 * 1.6 * 0.026 if norm and name != "v_c" else 2e-2) and err.mean() <= 0.03, f"{name} {Bs}: {err.max()}"


@pytest.mark.parametrize("H, Bs, blocks", [(4, 3, 5), (12, 16, 4), (16, 16, 3), (20, 16, 5), (40, 16, 3), (8, 35, 3), (4, 100, 2), (20, 13, 3), (16, 6300, 1)])
def test_prologue_forward_gates(H, Bs, blocks):
    """The gate's logits: fewer pairs of a block than threads, exactly two per thread, a part of the second and more, in every form of the
    kernel and with a part of the rows that is not whole; the other outputs are those of the projection without them."""
    import speed3r_b200
    from speed3r_b200 import _lib, ops
    B, N, C = 2, Bs * blocks, 3 * H * 64
    proj, = bf16_round(2 * randn(40 + H, B, N, C + 2 * H))
    proj = proj.to(DEV, torch.bfloat16)
    pos = torch.randint(0, 37, (B, N, 2), generator=torch.Generator().manual_seed(2)).to(DEV)
    cos, sin = speed3r_b200.RoPE2D(100.0)._cos_sin(32, 37, torch.device(DEV), torch.bfloat16)
    w = [t.to(DEV) for t in (1 + 0.2 * randn(3, 64), 0.1 * randn(4, 64), 1 + 0.2 * randn(5, 64), 0.1 * randn(6, 64))]
    want = ops.qkv_prologue(proj[..., :C].contiguous(), H, Bs, pos, cos, sin, (w[0], w[1], 1e-5), (w[2], w[3], 1e-5))
    got = [torch.full_like(t, float("nan")) for t in want] + [torch.full((B, H, N, 2), float("nan"), device=DEV, dtype=torch.bfloat16)]
    _lib.check(_lib.load().s3r_qkv_gate_prologue_fwd(
        proj.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), cos.shape[0], *(t.data_ptr() for t in w), 1e-5,
        *(t.data_ptr() for t in got), B, H, N, 64, Bs, torch.cuda.current_stream().cuda_stream), "s3r_qkv_gate_prologue_fwd")
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    gate = torch.sigmoid(proj[..., C:].double()).view(B, N, H, 2).permute(0, 2, 1, 3)
    # one rounding to bf16, whose 8 bits make half a unit of the last 2^-8 of the value at most, of fp32 values good to 2^-18
    assert ((got[6].double() - gate).abs() <= (2 ** -8 + 2 ** -18) * gate).all()


def _prologue_fp32(qkv, H, Bs, pos, cos, sin, qn, kn):
    """Split, LayerNorm, rotary embedding and pooling in fp32 with the given (bf16) rotary tables."""
    B, N, d = qkv.shape[0], qkv.shape[1], 64
    q, k, v = (qkv.view(B, N, 3, H, d)[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    pool = lambda t: t.reshape(B, H, N // Bs, Bs, d).mean(3)
    ln = lambda t, p: t if p is None else torch.nn.functional.layer_norm(t, (d,), *p)
    def rot(t, at):
        if pos is None:
            return t
        halves = []
        for i, h in enumerate(t.chunk(2, -1)):
            c, s = (tab.float().cpu()[at[..., i]][:, None] for tab in (cos, sin))
            a, b = h.chunk(2, -1)
            halves.append(h * c + torch.cat((-b, a), -1) * s)
        return torch.cat(halves, -1)
    at_c = None if pos is None else pos.view(B, N // Bs, Bs, 2).float().mean(2).int().long()
    return (rot(ln(q, qn), pos), rot(ln(k, kn), pos), v, rot(ln(pool(q), qn), at_c), rot(ln(pool(k), kn), at_c), pool(v))


@pytest.mark.parametrize("params,x_dtype,autocast,bias", [(torch.float32, torch.float32, True, True),
                                                          (torch.float32, torch.bfloat16, True, False),
                                                          (torch.bfloat16, torch.bfloat16, False, True)])
def test_module_native_inference_matches_separate_projections(params, x_dtype, autocast, bias):
    """The module as one native call against the same module with a hook on a projection, which keeps the projections in
    PyTorch: same roundings, so equal up to the GEMM's summation order."""
    import speed3r_b200
    torch.manual_seed(0)
    m = speed3r_b200.SparseFlashAttentionRope(256, num_heads=4, qkv_bias=bias, proj_bias=bias, qk_norm=True,
                                              rope=speed3r_b200.RoPE2D(100.0)).to(DEV, params).eval()
    x = torch.randn(2, 512, 256, device=DEV, dtype=x_dtype)
    tok = torch.arange(512, device=DEV) % 256
    xpos = torch.stack((tok // 16, tok % 16), -1)[None].expand(2, -1, -1).contiguous()
    m.record_idx = True
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
        assert m._native_op(x, xpos, 512, 16, 64) is not None
        y = m(x, xpos=xpos)
        idx = m.last_idx
        h = m.proj.register_forward_hook(lambda *a: None)
        assert m._native_op(x, xpos, 512, 16, 64) is None
        y2 = m(x, xpos=xpos)
        h.remove()
    assert y.dtype == y2.dtype and y.shape == y2.shape
    assert (idx != m.last_idx).float().mean() < 2e-2
    assert_bf16_close(y, y2.float(), "native module", max_abs=2e-2, mean_abs=1e-3)


def test_cast_bf16_sizes():
    """Every remainder of a thread's eight elements and of a block's, in one launch with other tensors."""
    import ctypes as C
    from speed3r_b200 import _lib
    sizes = [1, 7, 8, 9, 8191, 8192, 8193, 100003]
    xs = [torch.randn(n, device=DEV) for n in sizes]
    ys = [torch.empty(n, device=DEV, dtype=torch.bfloat16) for n in sizes]
    n = len(sizes)
    _lib.check(_lib.load().s3r_cast_bf16(n, (C.c_void_p * n)(*(t.data_ptr() for t in xs)), (C.c_void_p * n)(*(t.data_ptr() for t in ys)),
                                         (C.c_int64 * n)(*sizes), torch.cuda.current_stream().cuda_stream), "s3r_cast_bf16")
    for x, y in zip(xs, ys):
        assert torch.equal(y, x.bfloat16())


# ------------------------------------------------------------------ selection, blocks of 32 and 64
@pytest.mark.parametrize("block", [32, 64])
@pytest.mark.parametrize("K", [1, 3, 16, 48, 64])
def test_sel_big_fwd_lists(block, K):
    """Row tiles whose lists differ in length (dropped entries), empty lists, a row tile that is not full, a short last
    block, one entry, and lists too long for two CTAs per SM."""
    from speed3r_b200 import ops
    B, H, T = 1, 3, 64 * 7 + 37
    nb = -(-T // block)
    q, k, v = bf16_round(randn(90, B, H, T, 64), randn(91, B, H, T, 64), randn(92, B, H, T, 64))
    idx = table(93, B, H, nb, nb, K)
    idx[:, :, 2] = -1                                          # a query block without any valid entry
    idx[:, :, 3, 0] = nb - 1                                   # the short block
    idx[:, :, 4, K // 2:] = nb + 5                             # half a list dropped
    idx[:, :, 4, 0] = 1
    o, lse, _ = ops._sel_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), idx.to(DEV), None, None, block, 0.125, True, True, 1)
    ref, lse_ref = R.sel_attn(q, k, v, idx, block)
    rows = torch.ones(T, dtype=torch.bool)
    rows[2 * block:3 * block] = False
    assert_bf16_close(o[:, :, rows.to(DEV)], ref[:, :, rows], f"block {block} K {K}")
    assert_bf16_close(lse[:, :, rows.to(DEV)], lse_ref[:, :, rows], "lse", max_abs=5e-3, mean_abs=1e-3, scale_with_ref=False)
    assert (o[:, :, ~rows.to(DEV)] == 0).all() and (lse[:, :, ~rows.to(DEV)] == -float("inf")).all()


@pytest.mark.parametrize("block", [32, 64])
def test_sel_big_fwd_second_pass(block):
    """Scores that outgrow the first key block's by more than 2^64 make a row tile take its keys twice, beside one that does not."""
    from speed3r_b200 import ops
    B, H, T, K = 1, 2, 512, 4
    nb = T // block
    q, k, v = bf16_round(6 * randn(95, B, H, T, 64), randn(96, B, H, T, 64), randn(97, B, H, T, 64))
    k, = bf16_round(k * torch.linspace(0.05, 6.0, T).view(1, 1, T, 1))
    idx = torch.stack([torch.tensor([0, nb // 3, nb // 2, nb - 1])] * nb).int().expand(B, H, nb, K).contiguous()
    idx[:, :, :128 // block] = torch.tensor([nb - 1, 0, 1, 2]).int()
    o, lse, _ = ops._sel_fwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), idx.to(DEV), None, None, block, 0.125, True, True, 1)
    ref, lse_ref = R.sel_attn(q, k, v, idx, block)
    assert_bf16_close(o, ref, "growing scores")
    assert ((lse.cpu() - lse_ref).abs() <= 1e-5 * lse_ref.abs() + 1e-3).all()


@pytest.mark.parametrize("x_dtype,bias,norm,frozen", [(torch.float32, True, True, False), (torch.bfloat16, False, True, False),
                                                      (torch.float32, True, False, True)])
def test_module_native_training_matches_separate_nodes(x_dtype, bias, norm, frozen):
    """The module as one autograd node against the same module with a hook on a projection, which keeps the projections and
    their gradients in PyTorch (bf16 gradients cast to fp32, where the node keeps fp32)."""
    import speed3r_b200
    torch.manual_seed(1)
    B, N, dim = 2, 512, 256
    m = speed3r_b200.SparseFlashAttentionRope(dim, num_heads=4, qkv_bias=bias, proj_bias=bias, qk_norm=norm,
                                              rope=speed3r_b200.RoPE2D(100.0)).to(DEV)
    if not bias:
        m.gate[0].bias = None
    if frozen:
        m.qkv.weight.requires_grad_(False)
    x0 = torch.randn(B, N, dim, device=DEV, dtype=x_dtype)
    dy = 0.1 * torch.randn(B, N, dim, device=DEV)
    tok = torch.arange(N, device=DEV) % 256
    xpos = torch.stack((tok // 16, tok % 16), -1)[None].expand(B, -1, -1).contiguous()
    m.record_idx = True
    res = []
    for native in (True, False):
        h = None if native else m.proj.register_forward_hook(lambda *a: None)
        x = x0.clone().requires_grad_(True)
        m.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert (m._native_op(x, xpos, N, 16, 64) is not None) == native
            y = m(x, xpos=xpos)
        y.backward(dy.to(y.dtype))
        res.append((y.detach(), m.last_idx, x.grad, {k: p.grad for k, p in m.named_parameters()}))
        if h:
            h.remove()
    (y, idx, gx, gp), (y2, idx2, gx2, gp2) = res
    assert y.dtype == y2.dtype and gx.dtype == gx2.dtype
    same = (idx == idx2).all(-1)
    assert same.float().mean() > 0.98
    assert_bf16_close(y, y2.float(), "y", max_abs=2e-2, mean_abs=1e-3)
    rel = lambda a, b: ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-6)).item()
    assert rel(gx, gx2) < 2e-2
    for k in gp:
        assert (gp[k] is None) == (gp2[k] is None), k
        if gp[k] is not None:
            assert gp[k].dtype == gp2[k].dtype and rel(gp[k], gp2[k]) < 2e-2, k


@pytest.mark.parametrize("rows,cols", [(1, 8), (63, 264), (64, 256), (5000, 3104), (200000, 8)])
def test_colsum(rows, cols):
    """One row, slices with a remainder, a last group of columns that is not full."""
    from speed3r_b200 import _lib
    lib = _lib.load()
    x = randn(99, rows, cols).to(DEV, torch.bfloat16)
    out = torch.empty(cols, device=DEV)
    n = lib.s3r_colsum_workspace_bytes(rows, cols)
    ws = torch.empty(n, device=DEV, dtype=torch.uint8)
    _lib.check(lib.s3r_colsum(x.data_ptr(), out.data_ptr(), rows, cols, ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream), "s3r_colsum")
    ref = x.double().sum(0)
    assert ((out.double() - ref).abs() <= 2 ** -24 * rows * x.double().abs().sum(0) / rows * 64 + 1e-6).all()


@pytest.mark.parametrize("Nq, Nc, topk", [(700, 64, 1), (700, 64, 5), (700, 64, 32), (300, 40, 32), (1000, 1024, 1), (1000, 2001, 1), (2500, 8000, 1)])
def test_cmp_topk_keeps_logits_at_the_bound(Nq, Nc, topk):
    """With one entry per row, or one column per group, the bound is itself the last entry's logit: the collection's products
    have to reproduce it bit for bit, or the entry is missing (and the last column in its place)."""
    from speed3r_b200 import ops
    B, H = 1, 16
    ln = lambda x: torch.nn.functional.layer_norm(x, (64,)).to(DEV, torch.bfloat16)
    q, k, v = ln(randn(1, B, H, Nq, 64)), ln(randn(2, B, H, Nc, 64)), ln(randn(3, B, H, Nc, 64))
    _, _, idx = ops._cmp_fwd(q, k, v, topk, 0.125)
    S = q.double() @ k.double().transpose(-1, -2)
    want = S.topk(topk, dim=-1).values
    got = torch.gather(S, -1, idx.long())
    assert (idx.sort(-1).values.diff(dim=-1) > 0).all(), "padding, or a column twice"
    assert (got - want).abs().max() <= 1e-4                        # fp32 sums of 64 products of size 1 to 10


@pytest.mark.parametrize("take", [1, 3, 4])
@pytest.mark.parametrize("size, grow", [(30, 1), (60, 1), (100, 1), (10, 8)])
def test_block_ranking_with_large_logits(take, size, grow):
    """Rows in which fewer than top-k of the column groups lie within the exponentials' range of the row's largest score, and
    (grow) rows whose later keys outgrow the first tile's by more than 2^64, so that the keys are taken a second time."""
    from speed3r_b200 import ops
    B, H, Nq, Nc, K = 1, 2, 200, 1024, 16
    ln = lambda x: torch.nn.functional.layer_norm(x, (64,))
    k = ln(randn(2, B, H, Nc, 64)) * torch.linspace(1, grow, Nc)[:, None]
    q, k, v = bf16_round(size * ln(randn(1, B, H, Nq, 64)), k, ln(randn(3, B, H, Nc, 64)))
    o_ref, _, idx_ref = R.cmp_attn_topk(q, k, v, K, rank_group=(4, take))
    o, idx = ops.flash_attn_blocktopk_func(*(t.to(DEV, torch.bfloat16) for t in (q, k, v)), K, 4, take)
    assert_bf16_close(o, o_ref, "o_c")
    scores = R.block_rank_scores(q @ k.transpose(-1, -2), 0.125, 4, take)
    idx, idx_ref = idx.cpu().long(), idx_ref.long()
    assert (idx.sort(-1).values.diff(dim=-1) > 0).all(), "a block listed twice"
    gap = (torch.gather(scores, -1, idx) - torch.gather(scores, -1, idx_ref)).abs()
    # rounding of scores of this size: a few units of 2^-24 of the largest in both
    assert gap.max() <= 1e-3 + 1e-6 * scores.abs().max(), f"{gap.max():.4g}"


@pytest.mark.parametrize("Nc", [65, 96, 127])
def test_cmp_backward_with_all_logits_far_below_zero(Nc):
    """Logits near -120: a key past the end, whose score is 0, would weigh e^116."""
    from speed3r_b200 import ops
    B, H, Nq = 1, 2, 70
    q, k, v, do = bf16_round(3.875 + 0.1 * randn(1, B, H, Nq, 64), -3.875 + 0.1 * randn(2, B, H, Nc, 64), randn(3, B, H, Nc, 64),
                             randn(4, B, H, Nq, 64))
    ref = [t.clone().requires_grad_(True) for t in (q, k, v)]
    torch.softmax(ref[0] @ ref[1].transpose(-1, -2) * 0.125, -1).matmul(ref[2]).backward(do)
    t = [x.to(DEV, torch.bfloat16).requires_grad_(True) for x in (q, k, v)]
    ops.flash_attn_topk_func(*t, 8)[0].backward(do.to(DEV, torch.bfloat16))
    for name, a, b in zip(("dq", "dk", "dv"), t, ref):
        assert_bf16_close(a.grad, b.grad, name)


@pytest.mark.parametrize("Nq, Nc", [(1, 128), (127, 129), (128, 1), (129, 256), (257, 641), (641, 257), (1409, 130)])
def test_cmp_backward_tiles(Nq, Nc):
    """Tiles of 128 rows on either side: one row, one short or long of a tile, one and several rounds of the ring of five."""
    from speed3r_b200 import ops
    B, H = 1, 2
    q, k, v, do = bf16_round(randn(1, B, H, Nq, 64), randn(2, B, H, Nc, 64), randn(3, B, H, Nc, 64), randn(4, B, H, Nq, 64))
    ref = [t.clone().requires_grad_(True) for t in (q, k, v)]
    torch.softmax(ref[0] @ ref[1].transpose(-1, -2) * 0.125, -1).matmul(ref[2]).backward(do)
    t = [x.to(DEV, torch.bfloat16).requires_grad_(True) for x in (q, k, v)]
    ops.flash_attn_topk_func(*t, 1)[0].backward(do.to(DEV, torch.bfloat16))
    for name, a, b in zip(("dq", "dk", "dv"), t, ref):
        assert_bf16_close(a.grad, b.grad, name)


@pytest.mark.parametrize("scale", [0.0, -0.125, 0.3])
@pytest.mark.parametrize("H, Nq, Nc", [(2, 1, 130), (2, 127, 65), (2, 128, 128), (2, 200, 300), (64, 200, 150)])
def test_cmp_backward_of_any_scale(scale, H, Nq, Nc):
    """The backward takes any softmax scale, 0 and negative ones too, whether the last tile of queries or keys is whole or not."""
    from speed3r_b200 import ops
    B = 1
    q, k, v, do = bf16_round(randn(1, B, H, Nq, 64), randn(2, B, H, Nc, 64), randn(3, B, H, Nc, 64), randn(4, B, H, Nq, 64))
    ref = [t.clone().requires_grad_(True) for t in (q, k, v)]
    S = ref[0] @ ref[1].transpose(-1, -2) * scale
    o = torch.softmax(S, -1) @ ref[2]
    o.backward(do)
    lse = torch.logsumexp(S.detach(), -1).to(DEV)
    got = ops._ops().cmp_attn_bwd(*(t.to(DEV, torch.bfloat16) for t in (q, k, v, o.detach())), lse, do.to(DEV, torch.bfloat16), scale)
    for name, a, b in zip(("dq", "dk", "dv"), got, ref):
        assert_bf16_close(a, b.grad, f"{name} scale {scale}")


@pytest.mark.parametrize("Nq", [64, 70, 128, 200])
def test_cmp_backward_of_a_key_that_is_minus_infinity(Nq):
    """A key that no query gives a weight has no gradient, whether the last tile of queries is whole or not: rows that do not exist
    have no weight.  The other keys' gradients are what they are without it."""
    from speed3r_b200 import ops
    B, H, Nc, at = 1, 2, 96, 5
    q, k, v, do = bf16_round(randn(1, B, H, Nq, 64), randn(2, B, H, Nc, 64), randn(3, B, H, Nc, 64), randn(4, B, H, Nq, 64))
    q[..., 0] = q[..., 0].abs() + 0.5
    k[:, :, at, 0] = float("-inf")
    t = [x.to(DEV, torch.bfloat16).requires_grad_(True) for x in (q, k, v)]
    ops.flash_attn_topk_func(*t, 8)[0].backward(do.to(DEV, torch.bfloat16))
    rest = torch.arange(Nc) != at
    ref = [x.clone().requires_grad_(True) for x in (q, k[:, :, rest], v[:, :, rest])]
    torch.softmax(ref[0] @ ref[1].transpose(-1, -2) * 0.125, -1).matmul(ref[2]).backward(do)
    for name, a, b in zip(("dk", "dv"), t[1:], ref[1:]):
        g = a.grad.cpu()
        assert (g[:, :, at] == 0).all(), name
        assert_bf16_close(g[:, :, rest], b.grad, name)


@pytest.mark.parametrize("H, Nq, Nc", [(64, 129, 256), (64, 256, 130), (64, 200, 200), (40, 150, 255), (32, 257, 384), (32, 500, 449), (48, 640, 577)])
def test_cmp_backward_of_two_row_tiles(H, Nq, Nc):
    """Grids of 256 own rows per CTA: a second row tile of one row, streamed tiles of 64 whole and not, one and several rounds of the ring
    of six; one key that no query gives a weight."""
    from speed3r_b200 import ops
    B, at = 1, Nc - 1
    q, k, v, do = bf16_round(randn(1, B, H, Nq, 64), randn(2, B, H, Nc, 64), randn(3, B, H, Nc, 64), randn(4, B, H, Nq, 64))
    q[..., 0] = q[..., 0].abs() + 0.5
    k[:, :, at, 0] = float("-inf")
    t = [x.to(DEV, torch.bfloat16).requires_grad_(True) for x in (q, k, v)]
    ops.flash_attn_topk_func(*t, 8)[0].backward(do.to(DEV, torch.bfloat16))
    rest = torch.arange(Nc) != at
    ref = [x.clone().requires_grad_(True) for x in (q, k[:, :, rest], v[:, :, rest])]
    torch.softmax(ref[0] @ ref[1].transpose(-1, -2) * 0.125, -1).matmul(ref[2]).backward(do)
    for name, a, b in zip(("dk", "dv"), t[1:], ref[1:]):
        g = a.grad.cpu()
        assert (g[:, :, at] == 0).all(), name
        assert_bf16_close(g[:, :, rest], b.grad, name)
    t = [x.to(DEV, torch.bfloat16).requires_grad_(True) for x in (q, k[:, :, rest].contiguous(), v[:, :, rest].contiguous())]
    ops.flash_attn_topk_func(*t, 8)[0].backward(do.to(DEV, torch.bfloat16))
    for name, a, b in zip(("dq", "dk", "dv"), t, ref):
        assert_bf16_close(a.grad, b.grad, name)


def test_prologue_of_blocks_whose_table_rows_do_not_fit_shared_memory():
    """Blocks of 6400 tokens: token rows as with blocks of 16, bit for bit, means as in fp32, and the backward."""
    import speed3r_b200
    from speed3r_b200 import ops
    B, H, N, Bs = 1, 2, 12800, 6400
    qkv = (1.5 * randn(1, B, N, 3 * H * 64) + 0.3).to(DEV, torch.bfloat16)
    pos = torch.randint(0, 37, (B, N, 2), generator=torch.Generator().manual_seed(2)).to(DEV)
    cos, sin = speed3r_b200.RoPE2D(100.0)._cos_sin(32, 37, torch.device(DEV), torch.bfloat16)
    norm = [(1 + 0.2 * randn(3 + i, 64).to(DEV), 0.1 * randn(5 + i, 64).to(DEV), 1e-5) for i in range(2)]
    long, short = (ops.qkv_prologue(qkv, H, b, pos, cos, sin, *norm) for b in (Bs, 16))
    assert all(torch.equal(a, b) for a, b in zip(long[:3], short[:3]))
    mean = qkv.view(B, N // Bs, Bs, 3, H, 64).float().mean(2).permute(2, 0, 3, 1, 4)
    assert_bf16_close(long[5], mean[2], "v_c")
    test_prologue_backward(B, H, Bs, N // Bs, True, True)


@pytest.mark.parametrize("Tq, Tk, setting", [(512, 1024, (16, 32, 16, 16)), (1040, 336, (16, 8, 16, 16)), (256, 1024, (64, 4, 32, 16))])
def test_op_on_queries_and_keys_of_different_lengths(Tq, Tk, setting):
    """The whole op, forward and backward, where queries attend to another sequence."""
    from speed3r_b200 import ops
    B, H = 1, 2
    block, topk, kernel, stride = setting
    q, k, v = bf16_round(randn(1, B, H, Tq, 64), randn(2, B, H, Tk, 64), randn(3, B, H, Tk, 64))
    gate, = bf16_round(torch.sigmoid(randn(4, B, H, Tq, 2)))
    dy, = bf16_round(randn(5, B, Tq, H * 64))
    t = [x.to(DEV, torch.bfloat16).requires_grad_(True) for x in (q, k, v, gate)]
    y, idx = ops.sparse_attention_op(*t, *setting)
    y.backward(dy.to(DEV, torch.bfloat16))
    with torch.no_grad():
        assert torch.equal(ops.sparse_attention_op(*t, *setting)[0], y)
    r = [x.clone().requires_grad_(True) for x in (q, k, v, gate)]
    pooled = R.pool_tokens(r[0], block, block), R.pool_tokens(r[1], kernel, stride), R.pool_tokens(r[2], kernel, stride)
    o_c = torch.softmax(pooled[0] @ pooled[1].transpose(-1, -2) * 0.125, -1) @ pooled[2]
    y_ref = R.gated_merge(r[3], o_c, R.sel_attn(r[0], r[1], r[2], idx.cpu(), block)[0], block)
    y_ref.backward(dy)
    assert_bf16_close(y, y_ref, "y")
    for name, a, b in zip(("dq", "dk", "dv", "dgate"), t, r):
        assert_bf16_close(a.grad, b.grad, name)


def test_backward_beside_a_capture_of_another_thread():
    """The table's inverse runs on a stream of PyTorch's pool; a capture that another thread has going on one of those is neither
    joined nor broken by it."""
    import threading
    from speed3r_b200 import ops
    B, H, T = 1, 2, 512
    q, k, v = (randn(s, B, H, T, 64).to(DEV, torch.bfloat16).requires_grad_(True) for s in (1, 2, 3))
    gate = torch.sigmoid(randn(4, B, H, T, 2)).to(DEV, torch.bfloat16)
    grads = lambda: torch.autograd.grad(ops.sparse_attention_op(q, k, v, gate)[0].float().sum(), (q, k, v))
    want = grads()
    torch.cuda.synchronize()
    started, finish, failed = threading.Event(), threading.Event(), []
    a = torch.ones(1024, device=DEV)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()

    def capture():
        try:
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                b = a + 1
                started.set()
                assert finish.wait(60)
                b.add_(1)
            graph.replay()
            torch.cuda.synchronize()
            assert (b == 3).all()
        except Exception as e:
            failed.append(e)
            started.set()

    t = threading.Thread(target=capture)
    t.start()
    assert started.wait(60)
    try:
        got = [grads() for _ in range(40)]                         # the pool's 32 streams and more
    finally:
        finish.set()
        t.join()
    assert not failed, failed
    assert all(torch.equal(x, y) for g in got for x, y in zip(g, want))


def test_forward_and_backward_in_a_graph():
    """A captured step of the op, with the second stream inside the capture, replayed on new inputs."""
    from speed3r_b200 import ops
    B, H, T = 2, 2, 1024
    q, k, v = (randn(s, B, H, T, 64).to(DEV, torch.bfloat16).requires_grad_(True) for s in (1, 2, 3))
    gate = torch.sigmoid(randn(4, B, H, T, 2)).to(DEV, torch.bfloat16).requires_grad_(True)
    def step():
        y, idx = ops.sparse_attention_op(q, k, v, gate)
        return (y, idx) + torch.autograd.grad(y, (q, k, v, gate), torch.ones_like(y))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    with torch.no_grad():
        q.copy_(randn(5, B, H, T, 64))
        k.copy_(randn(6, B, H, T, 64))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, step()))


# ------------------------------------------------------------------ the attention module
def module_and_input(seed, B=1, N=512, H=4, dim=None, **kw):
    import speed3r_b200
    dim = H * 64 if dim is None else dim
    torch.manual_seed(seed)
    m = speed3r_b200.SparseFlashAttentionRope(dim, num_heads=H, qkv_bias=True, qk_norm=True, rope=speed3r_b200.RoPE2D(100.0), **kw)
    with torch.no_grad():
        for p in m.parameters():
            p.add_(0.05 * torch.randn_like(p))
    x = torch.randn(B, N, dim)
    pos = torch.stack((torch.arange(N) % 256 // 16, torch.arange(N) % 16), -1)[None].expand(B, -1, -1).contiguous()
    return m.to(DEV), x.to(DEV), pos.to(DEV)


def module_step(m, x, pos, dy=None):
    """(output, gradients) of a training step, or the output alone without gradients."""
    with torch.autocast("cuda", dtype=torch.bfloat16), torch.set_grad_enabled(dy is not None):
        y = m(x, xpos=pos)
    return [y.detach()] + (list(torch.autograd.grad(y, [x] + list(m.parameters()), dy)) if dy is not None else [])


def odd_view(t):
    """The same values in a contiguous view that begins one element behind an aligned address."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    view = flat[1:].view(t.shape)
    view.copy_(t.detach())
    assert view.is_contiguous() and view.data_ptr() % 16
    return view


@pytest.mark.parametrize("which", ["norms", "projections", "input", "gradient"])
@pytest.mark.parametrize("train", [False, True])
def test_module_takes_views_that_begin_anywhere(which, train):
    """Parameters inside a flattened buffer, an input or a gradient that is a slice: as if they were aligned, bit for bit."""
    m, x, pos = module_and_input(0)
    x.requires_grad_(train)
    dy = torch.randn(x.shape, device=DEV).bfloat16() if train else None
    want = module_step(m, x, pos, dy)
    if which == "norms":
        for n in (m.q_norm, m.k_norm):
            n.weight, n.bias = torch.nn.Parameter(odd_view(n.weight)), torch.nn.Parameter(odd_view(n.bias))
    elif which == "projections":
        for lin in (m.qkv, m.proj, m.gate[0]):
            lin.weight, lin.bias = torch.nn.Parameter(odd_view(lin.weight)), torch.nn.Parameter(odd_view(lin.bias))
    elif which == "input":
        x = odd_view(x).requires_grad_(train)
    elif train:
        dy = odd_view(dy)
    got = module_step(m, x, pos, dy)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_ops_take_gradients_that_begin_anywhere():
    from speed3r_b200 import ops
    B, H, T = 1, 2, 512
    q, k, v = (randn(s, B, H, T, 64).to(DEV, torch.bfloat16).requires_grad_(True) for s in (1, 2, 3))
    gate = torch.sigmoid(randn(4, B, H, T, 2)).to(DEV, torch.bfloat16).requires_grad_(True)
    idx = table(5, B, H, T // 16, T // 16, 8).to(DEV)
    o_c = randn(6, B, H, T // 16, 64).to(DEV, torch.bfloat16).requires_grad_(True)
    for what, out, wrt in (
            ("pool", ops.pool_tokens(q), (q,)),
            ("compression", ops.flash_attn_topk_func(q, k, v, 8)[0], (q, k, v)),
            ("selection", ops.topk_blocksparse_attention(q, k, v, idx, 16), (q, k, v)),
            ("merge", ops.sel_attn_merge(q, k, v, idx, gate, o_c, 16), (q, k, v, gate, o_c)),
            ("op", ops.sparse_attention_op(q, k, v, gate)[0], (q, k, v, gate))):
        g = torch.randn(out.shape, device=DEV).bfloat16()
        want = torch.autograd.grad(out, wrt, g, retain_graph=True)
        got = torch.autograd.grad(out, wrt, odd_view(g))
        assert all(torch.equal(a, b) for a, b in zip(got, want)), what


@pytest.mark.parametrize("block,kernel,stride", [(16, 16, 16), (32, 32, 32), (64, 32, 16), (64, 64, 64), (64, 24, 8)])
def test_pooled_gradients_that_begin_anywhere(block, kernel, stride):
    """The pooled branch's gradients, with a short last block and a query block without a list, and as views that begin at any element
    (the operator) or at any multiple of 4 bytes (the library)."""
    from speed3r_b200 import _lib, ops
    B, H, T, K = 1, 2, 64 * 5 + 17, 3
    nb, nw = -(-T // block), (T - kernel) // stride + 1
    q, k, v, do = (randn(s, B, H, T, 64).to(DEV, torch.bfloat16) for s in range(4))
    idx = table(5, B, H, nb, nb, K).to(DEV)
    idx[:, :, 1] = -1
    o, lse, _ = ops._sel_fwd(q, k, v, idx, None, None, block, 0.125, True, True, 1)
    delta = (o.float() * do.float()).sum(-1)
    pooled = [randn(6 + i, B, H, n, 64).to(DEV, torch.bfloat16) for i, n in enumerate((T // block, nw, nw))]
    def moved(t, by):
        m = torch.empty(t.numel() + by, device=DEV, dtype=t.dtype)[by:].view(t.shape)
        return m.copy_(t)
    call = lambda g: ops._ops().sel_attn_bwd_pooled(q, k, v, idx, lse, delta, do, *g, block, kernel, stride, 0.125)
    want = call(pooled)
    alone = ops._ops().sel_attn_bwd(q, k, v, idx, lse, delta, do, block, 0.125)
    for n, got, base, g, size, step in zip("qkv", want, alone, pooled, (block, kernel, kernel), (block, stride, stride)):
        share = torch.zeros_like(base, dtype=torch.float)
        for j in range(g.shape[2]):
            share[:, :, j * step:j * step + size] += g[:, :, j:j + 1].float() / size
        # two roundings to bf16, 2^-9 of what is rounded each, and sums of a few terms in fp32
        assert ((got.float() - base.float() - share).abs() <= 2 ** -8 * (base.float().abs() + got.float().abs()) + 1e-6).all(), n
    assert (alone[0][:, :, block:2 * block] == 0).all()
    for by in (1, 2, 4, 8):
        assert all(torch.equal(a, b) for a, b in zip(call([moved(t, by) for t in pooled]), want)), by
    if kernel % 16 or stride % 16:
        return
    off, qids = ops.build_key_csr(idx, nb)
    for by in (2, 4, 6):
        g, got = [moved(t, by) for t in pooled], [torch.empty_like(t) for t in want]
        _lib.check(_lib.load().s3r_sel_attn_bwd_pooled(*(t.data_ptr() for t in (q, k, v, idx, off, qids, lse, delta, do, *got, *g)), block,
                                                       block, kernel, stride, B, H, T, T, 64, block, K, 0.125,
                                                       torch.cuda.current_stream().cuda_stream), "s3r_sel_attn_bwd_pooled")
        assert all(torch.equal(a, b) for a, b in zip(got, want)), by


def test_module_with_an_output_that_is_not_whole_vectors():
    """A projection to 100 channels: the sum of its bias gradient's rows cannot be read in vectors of eight."""
    m, x, pos = module_and_input(0)
    m.proj = torch.nn.Linear(x.shape[-1], 100).to(DEV)
    x.requires_grad_(True)
    dy = torch.randn(1, x.shape[1], 100, device=DEV).bfloat16()
    grads = dict(zip(["x"] + [n for n, _ in m.named_parameters()], module_step(m, x, pos, dy)[1:]))
    assert_bf16_close(grads["proj.bias"], dy.float().sum((0, 1)), "bias")


def test_module_gradients_with_a_graph_are_the_same_and_final():
    m, x, pos = module_and_input(0)
    x.requires_grad_(True)
    dy = torch.randn(x.shape, device=DEV).bfloat16()
    want = module_step(m, x, pos, dy)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x, xpos=pos)
    got = torch.autograd.grad(y, [x] + list(m.parameters()), dy, create_graph=True)
    assert all(torch.equal(a, b) and a.requires_grad for a, b in zip(got, want[1:]))
    for g in got:
        with pytest.raises(RuntimeError, match="cannot be differentiated again"):
            torch.autograd.grad(g.sum(), x, retain_graph=True)


@pytest.mark.parametrize("wanted", [["proj.weight", "proj.bias"], ["proj.bias"], ["gate.0.bias"], ["k_norm.bias"], ["qkv.weight", "proj.weight"]])
def test_module_backward_of_some_parameters(wanted):
    """The gradients of single parameters are what they are among all; without one before the output projection, none of the
    attention's backward runs (nor is its memory taken)."""
    m, x, pos = module_and_input(0, N=4096)
    dy = torch.randn(x.shape, device=DEV).bfloat16()
    every = dict(zip(["x"] + [n for n, _ in m.named_parameters()], module_step(m, x.requires_grad_(True), pos, dy)[1:]))
    x.requires_grad_(False)
    for n, p in m.named_parameters():
        p.requires_grad_(n in wanted)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x, xpos=pos)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    got = torch.autograd.grad(y, [m.get_parameter(n) for n in wanted], dy)
    peak = torch.cuda.max_memory_allocated() - held
    assert all(torch.equal(a, every[n]) for n, a in zip(wanted, got))
    tokens = x.numel() * 2                                         # bytes of one bf16 tensor of the sequence
    assert (peak < 2 * tokens) == all(n.startswith("proj") for n in wanted), f"{peak / tokens:.1f} tensors of the sequence"


def test_op_backward_of_the_gate_alone():
    from speed3r_b200 import ops
    B, H, T = 1, 2, 1024
    q, k, v = (randn(s, B, H, T, 64).to(DEV, torch.bfloat16).requires_grad_(True) for s in (1, 2, 3))
    gate = torch.sigmoid(randn(4, B, H, T, 2)).to(DEV, torch.bfloat16).requires_grad_(True)
    y, _ = ops.sparse_attention_op(q, k, v, gate)
    dy = torch.randn(y.shape, device=DEV).bfloat16()
    want = torch.autograd.grad(y, gate, dy)[0]
    y, _ = ops.sparse_attention_op(q.detach(), k.detach(), v.detach(), gate)
    assert torch.equal(torch.autograd.grad(y, gate, dy)[0], want)


# ------------------------------------------------------------------ host pipeline
def test_host_pipeline_keeps_dropped_tensors_until_they_are_copied():
    """Pinned memory that the caller gives back while the copies are still enqueued is not handed out again."""
    from speed3r_b200 import HostPipeline
    H, T = 4, 512
    pipe = HostPipeline(H, T, device=torch.device(DEV))
    shapes = [(1, H, T, 64)] * 3 + [(1, H, T, 2), (1, T, H * 64)]
    pinned = lambda: [torch.ones(s, dtype=torch.bfloat16, pin_memory=True) for s in shapes]
    pipe(*pinned())                                                # the pools are filled, the kernels loaded
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)                               # half a second in front of every copy
    tensors = pinned()
    before = {t.data_ptr() for t in tensors}
    pipe(*tensors)
    del tensors
    after = {t.data_ptr() for t in pinned()}
    assert not torch.cuda.current_stream().query(), "the copies were not waiting"
    assert not before & after
