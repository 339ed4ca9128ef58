"""CPU-side checks of the C-ABI boundary: the library loads, exports every function the header
declares, and rejects bad arguments before touching the GPU (no compute is launched here)."""
import ctypes as C
import os
import re

import pytest
import torch

from conftest import ROOT

HEADER = os.path.join(ROOT, "include", "speed3r_b200.h")
CHECK_HEADER = os.path.join(ROOT, "include", "speed3r_b200_check.h")


def declared_functions(header=HEADER):
    src = open(header).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(s3r_[a-z0-9_]+)\s*\(", src)))


def test_header_and_binding_list_agree():
    from speed3r_b200 import _lib
    assert declared_functions() == sorted(_lib.SIGNATURES)
    assert declared_functions(CHECK_HEADER) == sorted(_lib.CHECK_SIGNATURES)


def test_library_exports_every_declared_symbol(lib):
    for name in declared_functions():
        assert hasattr(lib, name), f"{name} is declared in the header but missing from the library"
    assert lib.s3r_version() >= 100
    assert not hasattr(lib, "s3r_check_sel_attn_fwd"), "tests-only kernels must not ship in the product library"


def test_check_library_exports_every_declared_symbol():
    from speed3r_b200 import _lib
    chk = _lib.load_check()
    for name in declared_functions(CHECK_HEADER):
        assert hasattr(chk, name), f"{name} is declared in the check header but missing from the check library"
    import ctypes
    assert chk.s3r_check_wait_gives_up(0, None, None) == -4          # argument errors need no GPU


def test_tiles_of_tensors_far_apart_are_copied_one_by_one():
    """A tensor map's strides are below 2^40 bytes; a distance beyond that takes a map and a copy for each tensor."""
    from speed3r_b200 import _lib
    order, base = _lib.load_check().s3r_check_pair_order, 0x7F0000000000
    assert order(base, base) == 2
    for gap in (16, 1 << 30, (1 << 40) - 16):
        assert order(base, base + gap) == 0 and order(base + gap, base) == 1
    for gap in (1 << 40, (1 << 40) + 16, 1 << 45):
        assert order(base, base + gap) == 4 and order(base + gap, base) == 4


def test_backward_of_short_lists_keeps_the_kernel_that_is_faster_there():
    """Blocks of 64: lists of one or two entries on a full GPU, or of few queries over many keys, are not what tcgen05 pays for."""
    from speed3r_b200 import _lib
    pays = _lib.load_check().s3r_check_sel_bwd64_pays
    for bh, nb, topk, want in ((1, 1, 1, 1), (16, 32, 1, 1), (12, 64, 1, 1), (16, 64, 1, 0), (16, 938, 1, 0), (2, 938, 2, 1), (16, 128, 2, 0),
                               (16, 938, 2, 0), (16, 938, 3, 1), (1, 8, 8, 1), (16, 131, 16, 1), (16, 3938, 16, 1), (16, 1 << 20, 64, 1)):
        assert pays(bh, nb, nb, topk) == want, (bh, nb, topk)
    assert pays(16, 1, 938, 16) == 0 and pays(2, 1, 938, 4) == 0 and pays(2, 1, 938, 32) == 1
    assert pays(16, 938, 16, 1) == 0 and pays(16, 938, 1, 1) == 1                  # one key block that every query block selects


def test_argument_errors_are_reported_without_a_gpu(lib):
    from speed3r_b200 import _lib
    # NULL pointers
    rc = lib.s3r_pool_fwd(None, 0, 0, 0, None, 1, 1, 16, 64, 16, 16, None)
    assert rc == -4 and "NULL" in _lib.last_error()
    buf = (C.c_uint16 * 4096)()
    p = C.addressof(buf)
    p = (p + 255) & ~255
    # head_dim not a multiple of 8
    rc = lib.s3r_pool_fwd(p, 0, 0, 8, p, 1, 1, 16, 60, 16, 16, None)
    assert rc == -2
    # sequence shorter than the pooling window
    rc = lib.s3r_pool_fwd(p, 0, 0, 64, p, 1, 1, 8, 64, 16, 16, None)
    assert rc == -1
    # misaligned pointer
    rc = lib.s3r_pool_fwd(p + 2, 0, 0, 64, p, 1, 1, 16, 64, 16, 16, None)
    assert rc == -3
    # unsupported head_dim / top-k / block
    rc = lib.s3r_cmp_attn_topk_fwd(p, p, p, p, p, p, 1, 1, 16, 16, 128, 32, 0.125, None)
    assert rc == -2 and "head_dim" in _lib.last_error()
    rc = lib.s3r_cmp_attn_topk_fwd(p, p, p, p, p, p, 1, 1, 16, 16, 64, 48, 0.125, None)
    assert rc == -2 and "topk" in _lib.last_error()
    rc = lib.s3r_sel_attn_fwd(p, p, p, 1, 0, p, p, None, None, 0, 0, 0, None, None, 1, 1, 64, 64, 64, 48, 8, 0.125, None)
    assert rc == -2 and "block" in _lib.last_error()
    # prologue: NULL output, ragged sequence, head count, LayerNorm parameters only in part, positions without tables
    pro = lambda **kw: lib.s3r_qkv_prologue_fwd(
        kw.get("qkv", p), kw.get("pos"), kw.get("cos"), kw.get("sin"), kw.get("rows", 0), kw.get("qw"), kw.get("qb"),
        kw.get("kw"), kw.get("kb"), 1e-5, p, p, p, p, p, kw.get("v_c", p), 1, kw.get("H", 4), kw.get("N", 32), 64, 16, None)
    assert pro(v_c=None) == -4
    assert pro(N=40) == -1 and "multiple" in _lib.last_error()
    assert pro(H=43) == -2 and "heads" in _lib.last_error()
    assert pro(qw=p) == -4
    assert pro(pos=p) == -4 and "tables" in _lib.last_error()
    # LayerNorm parameters are loaded in pairs
    for name in ("qw", "qb", "kw", "kb"):
        assert pro(**{n: p + 4 * (n == name) for n in ("qw", "qb", "kw", "kb")}) == -3 and "8-byte" in _lib.last_error()
    for off in ((4, 0), (0, 4)):
        rc = lib.s3r_qkv_prologue_bwd(p, None, None, None, 0, p + off[0], p + off[1], 1e-5, p, p, p, p, p, p, p, p, p, 1 << 30,
                                      1, 4, 32, 64, 16, None)
        assert rc == -3 and "8-byte" in _lib.last_error()
    # 16-byte loads of what a caller hands to a backward
    assert lib.s3r_delta(p, p + 2, p, 16, 64, None) == -3 and lib.s3r_delta(p + 8, p, p, 16, 64, None) == -3
    for i in range(6):
        a = [p + 2 * (i == j) for j in range(6)]                   # dy, gate, o_c, o_s, do_s, do_c
        rc = lib.s3r_merge_bwd(a[0], a[1], 64, 32, 2, a[2], a[3], a[4], p, a[5], p, 1, 1, 16, 64, 16, None)
        assert rc == -3 and "aligned" in _lib.last_error()
    # gradients of the pooled branch are read in words of 4 bytes
    for block in (16, 32, 64):
        for i in range(3):
            rc = lib.s3r_sel_attn_bwd_pooled(*[p] * 12, *[p + 2 * (i == j) for j in range(3)], block, block, 16, 16, 1, 1, 64, 64, 64, block,
                                             1, 0.125, None)
            assert rc == -3 and "pooled" in _lib.last_error()
    # merge arguments must come together
    rc = lib.s3r_sel_attn_fwd(p, p, p, 1, 0, p, p, None, p, 0, 0, 0, None, None, 1, 1, 64, 64, 64, 16, 8, 0.125, None)
    assert rc == -4
    # CSR workspace too small
    need = lib.s3r_csr_workspace_bytes(1, 2, 64, 8, 64)
    assert need > 0
    rc = lib.s3r_build_key_csr(p, p, p, 1, 2, 64, 8, 64, p, need - 1, None)
    assert rc == -6


def test_python_layer_has_no_cpu_fallback():
    import speed3r_b200
    from speed3r_b200 import ops
    q = torch.randn(1, 2, 64, 64, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.flash_attn_topk_func(q, q, q, 8)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.pool_tokens(q, 16, 16)
    m = speed3r_b200.SparseFlashAttentionRope(128, num_heads=2)
    with pytest.raises(RuntimeError):
        m(torch.randn(1, 64, 128))


@pytest.mark.parametrize("op", ["module_infer", "module_train"])
def test_native_module_refuses_shapes_that_do_not_fit(op):
    """The native forms of the module copy its input and weights by size into one allocation: every shape is looked at first
    (before the device, so that this needs no GPU)."""
    from speed3r_b200 import ops
    H, d, N = 4, 64, 32
    C = H * d
    good = dict(x=(1, N, C), w_qkv=(3 * C, C), b_qkv=(3 * C,), w_gate=(2 * H, C), b_gate=(2 * H,), w_proj=(C, C), b_proj=(C,),
                pos=(1, N, 2), cos=(64, d // 2), sin=(64, d // 2), qw=(d,), qb=(d,), kw=(d,), kb=(d,))
    def call(**shapes):
        t = [torch.zeros(s, dtype=torch.int64 if n == "pos" else torch.float32) for n, s in {**good, **shapes}.items()]
        getattr(ops._ops(), op).default(*t, 1e-5, H, 16, 32, 0.125)
    with pytest.raises(RuntimeError, match="CUDA"):                # the shapes fit
        call()
    for name, shape in dict(x=(1, N, C + 1), w_qkv=(3 * C + 8, C), b_qkv=(3 * C + 1,), w_gate=(2 * H + 8, C), b_gate=(2 * H + 8,),
                            w_proj=(C, C + 1), b_proj=(C + 1,), pos=(2, N, 2), cos=(64, d), sin=(63, d // 2), qw=(d - 1,), kb=(1,)).items():
        with pytest.raises(RuntimeError, match="attention module"):
            call(**{name: shape})
    with pytest.raises(RuntimeError, match="attention module"):    # an input of another width than the weights
        call(x=(1, N, 2 * C))
    with pytest.raises(RuntimeError, match="blocks"):
        call(x=(1, N + 1, C), pos=(1, N + 1, 2))


def test_sizes_that_are_divided_by_are_looked_at_first():
    """Zero blocks, windows and strides and empty projections raise (before the device is looked at, so that this needs no
    GPU): divided by in native code, they would end the process."""
    from speed3r_b200 import ops
    o = ops._ops()
    x, f = torch.zeros(1, 2, 64, 64, dtype=torch.bfloat16), torch.zeros(1, 2, 64)
    idx = torch.zeros(1, 2, 4, 8, dtype=torch.int32)
    for call in (lambda: o.pool_fwd.default(x, 0, 16), lambda: o.pool_fwd.default(x, 16, 0), lambda: ops.pool_tokens(x, 16, 0),
                 lambda: o.pool_qkv_fwd.default(x, x, x, 0, 16, 16), lambda: o.pool_qkv_fwd.default(x, x, x, 16, 16, 0),
                 lambda: ops.topk_blocksparse_attention(x, x, x, idx, 0), lambda: ops.sel_attn_merge(x, x, x, idx, x, x, 0),
                 lambda: ops.sel_attn_merge_chunked(x, x[None], x[None], idx, x, x, 0),
                 lambda: o.sel_attn_bwd.default(x, x, x, idx, f, f, x, 0, 0.125),
                 lambda: o.sel_attn_bwd_pooled.default(x, x, x, idx, f, f, x, x, x, x, 16, 16, 0, 0.125),
                 lambda: ops.sparse_attention_op(x, x, x, x, 0, 8, 0, 0)):
        with pytest.raises(RuntimeError, match="must be positive"):
            call()
    for shape in ((0, 16, 384), (1, 0, 384), (1, 16, 0)):
        with pytest.raises(RuntimeError, match="not empty"):
            o.prologue_fwd.default(torch.zeros(shape, dtype=torch.bfloat16), 2, 16, None, None, None, None, None, None, None, 1e-5)


def differentiable_calls(t, gate):
    from speed3r_b200 import ops
    idx = torch.zeros(1, 2, 4, 2, dtype=torch.int32, device=t.device)
    return {"pool": lambda: ops.pool_tokens(t), "compression": lambda: ops.flash_attn_topk_func(t, t, t, 2)[0],
            "blocks": lambda: ops.flash_attn_blocktopk_func(t, t, t, 2, 4, 3)[0],
            "selection": lambda: ops.topk_blocksparse_attention(t, t, t, idx, 16),
            "merge": lambda: ops.sel_attn_merge(t, t, t, idx, gate, t[:, :, :4].contiguous(), 16),
            "op": lambda: ops.sparse_attention_op(t, t, t, gate, 16, 2)[0],
            "prologue": lambda: ops._prologue(t.transpose(1, 2).reshape(1, 64, 128).repeat(1, 1, 3), 2, 16, None, None, None, None, None)[0]}


def meta_inputs():
    return (torch.empty(s, dtype=torch.bfloat16, device="meta") for s in ((1, 2, 64, 64), (1, 2, 64, 2)))


@pytest.mark.parametrize("name", ["pool", "compression", "blocks", "selection", "merge", "op", "prologue"])
@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_is_refused(name, grad):
    """A tangent is not dropped without a word, with reverse-mode gradients or without (meta tensors: no kernel runs)."""
    import torch.autograd.forward_ad as fa
    x, gate = meta_inputs()
    with fa.dual_level():
        t = fa.make_dual(x.requires_grad_(grad), torch.empty_like(x))
        with pytest.raises((NotImplementedError, RuntimeError), match="not implemented"):
            differentiable_calls(t, gate)[name]()


@pytest.mark.parametrize("name", ["pool", "compression", "blocks", "selection", "merge", "op", "prologue"])
def test_second_derivatives_are_refused(name):
    """A gradient taken with create_graph is there; differentiating it raises instead of leaving these operators out."""
    x, gate = meta_inputs()
    x.requires_grad_(True)
    y = differentiable_calls(x, gate)[name]()
    first, = torch.autograd.grad((y.float() * y.float()).sum(), x, create_graph=True)
    assert first.requires_grad
    with pytest.raises(RuntimeError, match="cannot be differentiated again"):
        torch.autograd.grad(first.sum(), x)


def test_op_shapes_for_queries_and_keys_of_different_lengths():
    """Shape functions alone (meta tensors): the table and the output follow the queries."""
    from speed3r_b200 import ops
    q = torch.empty(1, 2, 256, 64, dtype=torch.bfloat16, device="meta")
    k, gate = q.new_empty(1, 2, 512, 64), q.new_empty(1, 2, 256, 2)
    for a, b in ((q, k), (q.requires_grad_(True), k)):
        y, idx = ops.sparse_attention_op(a, b, b, gate, 16, 8)
        assert y.shape == (1, 256, 128) and idx.shape == (1, 2, 16, 8)
    assert [tuple(t.shape) for t in ops._ops().pool_qkv_fwd.default(q, k, k, 16, 16, 16)] == [(1, 2, 16, 64), (1, 2, 32, 64), (1, 2, 32, 64)]


def test_module_keeps_reference_state_dict_keys_and_init():
    """Keys and gate initialisation of pi3/models/layers/sparse_attention.py:62-86."""
    import speed3r_b200
    m = speed3r_b200.SparseFlashAttentionRope(1024, num_heads=16, qkv_bias=True, qk_norm=True)
    keys = set(m.state_dict().keys())
    assert keys == {"qkv.weight", "qkv.bias", "proj.weight", "proj.bias", "q_norm.weight", "q_norm.bias",
                    "k_norm.weight", "k_norm.bias", "gate.0.weight", "gate.0.bias"}
    assert m.gate[0].weight.abs().max() == 0
    assert torch.equal(m.gate[0].bias.data, torch.tensor([-1.0, 1.0]).repeat(16))
    assert m.block_size == 4 and m.topk == 32


def test_rope_matches_oracle_on_cpu():
    import speed3r_b200
    from oracle import restatement as R
    torch.manual_seed(0)
    x = torch.randn(2, 3, 50, 64)
    pos = torch.randint(0, 37, (2, 50, 2))
    assert torch.equal(speed3r_b200.RoPE2D(100.0)(x, pos), R.rope2d(x, pos, 100.0))
    xb = x.bfloat16()
    assert torch.equal(speed3r_b200.RoPE2D(100.0)(xb, pos), R.rope2d(xb, pos, 100.0))


def test_host_pipeline_chunking():
    """Query chunks of the pinned-host pipeline: whole waves of the compression kernel, full cover, in order."""
    from speed3r_b200.host_pipeline import query_chunks, rows_per_chunk_for
    rows = rows_per_chunk_for(16, 148)
    assert rows == 256 * 37 and (16 * (rows // 256)) % 148 == 0
    assert rows_per_chunk_for(12, 148) == 256 * 37 and rows_per_chunk_for(37, 148) == 256 * 4
    ch = query_chunks(63000, rows)
    assert ch[0] == (0, rows) and ch[-1][1] == 63000 and len(ch) == 7
    assert all(a[1] == b[0] for a, b in zip(ch, ch[1:]))
    assert query_chunks(100, rows) == [(0, 100)]
