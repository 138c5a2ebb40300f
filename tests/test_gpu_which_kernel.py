"""Which form of a kernel a call takes, at the sizes where that changes, and that the forms give the same bits."""
import re

import pytest
import torch

from test_gpu_attn_tc import _cu, _kernels

pytestmark = pytest.mark.gpu
TYPES = {torch.bfloat16: "__nv_bfloat16", torch.float16: "__half", torch.float32: "float"}


def _form(name, call):
    """Template arguments of the kernel `name` that `call` launches."""
    found = set(re.findall(name + r"<([^()]*(?:\(\w+\)[^()]*)*)>\(", _kernels(call)))
    assert len(found) == 1, found
    return [re.sub(r"\(\w+\)", "", a).strip() for a in found.pop().split(",")]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("heads,kv_heads,n,cached,groups", [(2, 1, 40, 0, 2), (2, 1, 512, 0, 2), (2, 1, 513, 0, 1), (8, 1, 2000, 0, 1), (2, 1, 40, 256, 1),
                                                            (40, 40, 512, 0, 1)])
def test_prompts_of_single_tiles_and_few_keys_have_two_groups(heads, kv_heads, n, cached, groups):
    """Longer chains of key tiles lose by the exchange of every step's maximum."""
    from zipage_b200.layers.attention import varlen_prefill_attention
    g = _gen(n)
    draw = lambda *s: torch.randn(*s, 128, device="cuda", generator=g).to(torch.bfloat16)
    q, cu, cuk = draw(n, heads), _cu([n]), _cu([n + cached])
    if cached:
        pages = (n + cached + 255) // 256
        k, v, table = draw(pages, 256, kv_heads), draw(pages, 256, kv_heads), torch.arange(pages, dtype=torch.int32, device="cuda")[None]
    else:
        k, v, table = draw(n, kv_heads), draw(n, kv_heads), None
    form = _form(r"attn_tc_kernel<zp::PrefillTc", lambda: varlen_prefill_attention(q, k, v, n, cu, n + cached, cuk, block_table=table, impl="tcgen05"))
    assert form[1].rstrip("> ") == str(groups)
