"""The size-dependent forms of the per-step kernels at the sizes where they change over."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv_heads,D", [(32, 8, 128), (5, 1, 128), (18, 6, 64)])
def test_qk_norm_rope_is_the_same_for_few_and_many_tokens(dtype, heads, kv_heads, D):
    """1100 tokens in one call (16 heads a warp) and in halves (four heads a warp): the same arithmetic, the same bits."""
    from zipage_b200.layers import step_ops as P
    g, N, dev = _gen(heads), 1100, "cuda"
    qkv = torch.randn(N, (heads + 2 * kv_heads) * D, device=dev, generator=g).to(dtype)
    pos, cs = torch.randint(0, 4096, (N,), device=dev, generator=g), P.rope_cos_sin_cache(D, 4096, 1e6, dev)
    w = [(1 + 0.1 * torch.randn(D, device=dev, generator=g)).to(dtype) for _ in range(2)]
    slot = torch.randperm(1280, device=dev, generator=g)[:N].to(torch.int32)
    slot[7] = -1
    triples = torch.tensor([[3, 0, 1], [1099, 1, 0], [600, 0, 0]], dtype=torch.int32, device=dev)

    def run(parts):
        kc, vc = (torch.zeros(5, 256, kv_heads, D, dtype=dtype, device=dev) for _ in range(2))
        qc, out = torch.zeros(2, 2, heads, D, dtype=dtype, device=dev), []
        for a, b in parts:
            tr = triples[(triples[:, 0] >= a) & (triples[:, 0] < b)].clone()
            tr[:, 0] -= a
            q, k, _ = P.qk_norm_rope_store(qkv[a:b], pos[a:b], cs, *w, 1e-6, heads, kv_heads, D, kc, vc, slot[a:b], qc, tr.contiguous())
            out.append((q, k))
        return torch.cat([q for q, _ in out]), torch.cat([k for _, k in out]), kc, vc, qc
    for x, y in zip(run([(0, N)]), run([(0, 550), (550, N)])):
        assert torch.equal(x, y)
