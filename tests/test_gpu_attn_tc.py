"""The shared tcgen05 attention pipeline at the edges of its work items: tiles of two heads and of two row blocks, single rows, rows
without keys, sequences that end inside a tile, several items per block."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = 128


def _cu(lens):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")


def _softmax(q, k, v, scale, seen):
    """fp64 -> result, and the same sum over |v| (what roundings of weights and results are relative to)."""
    G = q.shape[1] // k.shape[1]
    q, k, v = q.double(), k.double().repeat_interleave(G, 1), v.double().repeat_interleave(G, 1)
    s = (torch.einsum("thd,shd->hts", q, k) * scale).masked_fill(~seen[None], float("-inf"))
    w = torch.nan_to_num(torch.softmax(s, -1), 0.0)
    return torch.einsum("hts,shd->thd", w, v), torch.einsum("hts,shd->thd", w, v.abs())


def _no_device_error():
    from zipage_b200 import _lib as L
    torch.cuda.synchronize()
    assert L.device_error(reset=True) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv_heads,lens_q,lens_k", [
    (4, 2, [1], [1]),                                     # two heads, one row, one key
    (2, 2, [1, 127, 128, 129, 300], None),                # a head per key/value head: two row blocks, the second empty or short
    (6, 2, [257, 255, 1, 700], [257, 300, 129, 1100]),    # three heads per key/value head, cached prefixes
    (8, 1, [513, 5, 384], [700, 5, 640]),
    (4, 4, [130, 60], [40, 60]),                          # rows before the first key: zeros
    (64, 8, [1200, 64, 900, 333, 1], None),               # several items per block
])
def test_prefill_edges(dtype, heads, kv_heads, lens_q, lens_k):
    from zipage_b200.layers.attention import varlen_prefill_attention
    lens_k = lens_k or lens_q
    g = torch.Generator(device="cuda").manual_seed(len(lens_q) * heads)
    n = lambda rows, h: torch.randn(rows, h, D, device="cuda", generator=g).to(dtype)
    q, k, v = n(sum(lens_q), heads), n(sum(lens_k), kv_heads), n(sum(lens_k), kv_heads)
    q[:, 0] *= 6                                          # peaked rows, whose reference moves from tile to tile
    out = varlen_prefill_attention(q, k, v, max(lens_q), _cu(lens_q), max(lens_k), _cu(lens_k), impl="tcgen05")
    _no_device_error()
    # the weight and the result are rounded to T once each (half a unit in the last place); the rest is fp32
    unit = (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12) * 2 * 1.1
    a = b = 0
    for x, y in zip(lens_q, lens_k):
        seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
        ref, mag = _softmax(q[a:a + x], k[b:b + y], v[b:b + y], D ** -0.5, seen)
        assert ((out[a:a + x].double() - ref).abs() <= unit * 2 * mag + 1e-6).all()
        a, b = a + x, b + y
