"""Which way the attention module goes, decided on the host: the native calls are taken only where nobody can tell."""
import pytest
import torch
from torch import nn

import speed3r_b200


class Stub:
    """Stands for a CUDA input in the routing decision; nothing is computed."""
    is_cuda, dtype, requires_grad = True, torch.float32, False

    @staticmethod
    def get_device():
        return -1                                                  # that of CPU parameters


def module(**kw):
    return speed3r_b200.SparseFlashAttentionRope(256, num_heads=4, qkv_bias=True, qk_norm=True, rope=speed3r_b200.RoPE2D(100.0), **kw)


@pytest.fixture
def route(monkeypatch):
    """'infer', 'train' or None for a module; under bf16 autocast with gradients unless told otherwise."""
    import types
    from speed3r_b200 import ops, sparse_attention
    native = types.SimpleNamespace(module_infer=types.SimpleNamespace(default="infer"), module_train=types.SimpleNamespace(default="train"))
    monkeypatch.setattr(ops, "_ops", lambda: native)
    monkeypatch.setattr(sparse_attention, "Tensor", Stub)
    monkeypatch.setattr(torch, "is_autocast_enabled", lambda *_: True)
    monkeypatch.setattr(torch, "get_autocast_dtype", lambda *_: torch.bfloat16)
    def go(m, grad=True, pos=object()):
        with torch.set_grad_enabled(grad):
            return m._native_op(Stub(), pos, 64, 16, 64), m._trains_through_prologue(pos, 64, 16, 64)
    return go


def test_plain_modules_take_the_native_calls(route):
    assert route(module()) == ("train", True)
    assert route(module(), grad=False) == ("infer", True)


@pytest.mark.parametrize("name", ["qkv", "proj", "gate", "gate.0", "gate.1", "q_norm", "k_norm"])
@pytest.mark.parametrize("how", ["forward hook", "backward hook", "own forward"])
def test_watched_modules_are_called(route, name, how):
    m = module()
    sub = m.get_submodule(name)
    if how == "forward hook":
        sub.register_forward_hook(lambda *a: None)
    elif how == "backward hook":
        sub.register_full_backward_hook(lambda *a: None)
    else:
        sub.forward = type(sub).forward.__get__(sub)
    assert route(m)[0] is None and route(m, grad=False)[0] is None
    assert route(m)[1] == (name not in ("q_norm", "k_norm")), "with gradients a watched norm is called"


@pytest.mark.parametrize("what", ["norm", "rope", "rope hook", "rope own forward"])
def test_replaced_norms_and_rotary_modules_are_called_with_gradients(route, what):
    class Norm(nn.LayerNorm):
        def forward(self, x):
            return 2 * super().forward(x)

    class Rope(speed3r_b200.RoPE2D):
        def forward(self, tokens, positions, seq_len=None):
            return tokens

    m = module()
    if what == "norm":
        m.k_norm = Norm(64)
    elif what == "rope":
        m.rope = Rope()
    elif what == "rope hook":
        m.rope.register_forward_hook(lambda *a: None)
    else:
        m.rope.forward = lambda tokens, positions, seq_len=None: tokens
    assert route(m) == (None, False)
    assert what == "norm" or route(m, pos=None) == ("train", True), "without positions the rotary module is not asked"


def test_dispatch_modes_see_the_steps(route):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Count(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    m = module()
    with Count():
        assert route(m)[0] is None and route(m, grad=False)[0] is None
