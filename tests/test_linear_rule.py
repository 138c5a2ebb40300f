"""Which calls `linear` gives to the kernel of few rows (the rule looks at tensors alone, so it runs without a GPU)."""
import pytest
import torch
from torch import nn

from zipage_b200.layers.step_ops import SMALL_ROWS, _small_linear_takes


def _layer(k=64, n=48, bias=False):
    return nn.Linear(k, n, bias=bias, dtype=torch.bfloat16)


def _x(rows=4, k=64):
    return torch.randn(rows, k, dtype=torch.bfloat16)


@torch.no_grad()
def test_the_kernel_takes_plain_calls():
    for rows in (1, SMALL_ROWS):
        assert _small_linear_takes(_layer(), _x(rows)) and _small_linear_takes(_layer(bias=True), _x(rows))
    assert _small_linear_takes(_layer(), _x(4, 128)[:, 64:])


@torch.no_grad()
@pytest.mark.parametrize("k", [32, 63, 65, 96, 128])
def test_an_input_of_another_width_is_the_layers(k):
    """The kernel would read past its rows (or leave a part of them out); the layer refuses."""
    layer = _layer()
    assert not _small_linear_takes(layer, _x(4, k))
    assert not _small_linear_takes(layer, _x(4, 192)[:, :k])
    with pytest.raises(RuntimeError):
        layer(_x(4, k))


@torch.no_grad()
def test_other_sizes_are_the_layers():
    one = _layer(bias=True)
    one.bias = nn.Parameter(torch.ones(1, dtype=torch.bfloat16))      # (is broadcast)
    assert not _small_linear_takes(one, _x())
    assert not _small_linear_takes(_layer(k=0), _x(4, 0))
    assert not _small_linear_takes(_layer(), _x(0)) and not _small_linear_takes(_layer(), _x(SMALL_ROWS + 1))
    assert _small_linear_takes(_layer(k=4096, n=64), _x(4, 4096)) and not _small_linear_takes(_layer(k=4096 + 32, n=64), _x(4, 4096 + 32))
    assert _small_linear_takes(_layer(k=64, n=1 << 15), _x()) and not _small_linear_takes(_layer(k=64, n=(1 << 15) + 16), _x())
    assert not _small_linear_takes(_layer(), _x()[0]) and not _small_linear_takes(_layer(), _x()[None])


@torch.no_grad()
def test_a_call_that_something_looks_at_is_the_layers():
    layer, x = _layer(), _x()
    layer.forward = lambda v: v                                  # (offloading and adapter libraries replace it so)
    assert not _small_linear_takes(layer, x)
    del layer.forward
    assert _small_linear_takes(layer, x)
    for register in (layer.register_forward_hook, layer.register_forward_pre_hook, nn.modules.module.register_module_forward_hook):
        handle = register(lambda *a: None)
        assert not _small_linear_takes(layer, x)
        handle.remove()

    class Function(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))

    class Dispatch(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))

    for context in (Function(), Dispatch(), torch.enable_grad(), torch.autograd.forward_ad.dual_level()):
        with context:
            assert not _small_linear_takes(layer, x)
    seen = []
    torch.vmap(lambda v: seen.append(_small_linear_takes(layer, v)) or v)(x[:, None])
    assert seen == [False]
    with torch.device("cpu"):
        assert _small_linear_takes(layer, x)
    assert _small_linear_takes(layer, x)


@torch.no_grad()
def test_a_patched_class_is_the_layers(monkeypatch):
    monkeypatch.setattr(nn.Linear, "forward", lambda self, v: v)
    assert not _small_linear_takes(_layer(), _x())
