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
    assert not _small_linear_takes(_layer(), _x()[0]) and not _small_linear_takes(_layer(), _x()[None])
