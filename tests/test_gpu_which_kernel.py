"""Which form of a kernel a call takes, at the sizes where that changes, and that the forms give the same bits."""
import re

import pytest
import torch

from test_gpu_attn_tc import _cu, _kernels

pytestmark = pytest.mark.gpu
TYPES = {torch.bfloat16: "13__nv_bfloat16", torch.float16: "6__half", torch.float32: "f"}      # (as they are in a symbol)


def _form(name, call):
    """Template arguments of the kernel (or, of a kernel's parameters) `name` that `call` launches."""
    argument = "13__nv_bfloat16|6__half|f|L[ib][0-9]+E"
    found = set(re.findall(f"{len(name)}{name}I((?:{argument})+)E", _kernels(call)))
    assert len(found) == 1, found
    return [re.sub("^L[ib]([0-9]+)E$", r"\1", a) for a in re.findall(argument, found.pop())]


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
    form = _form("PrefillTc", lambda: varlen_prefill_attention(q, k, v, n, cu, n + cached, cuk, block_table=table, impl="tcgen05"))
    assert form == [TYPES[torch.bfloat16], str(groups)]


@pytest.mark.parametrize("E,K,n_out,tiles", [
    (16, 512, 4096, 1), (16, 1024, 1536, 2), (16, 1024, 1024, 1), (16, 2048, 1024, 1),              # 1250 places an expert; 4.4 tiles an SM at 1024 columns, 6.6 at 1536
    (32, 1024, 2048, 1), (32, 1024, 3072, 2), (32, 1536, 1536, 1), (32, 1536, 2048, 2), (32, 2048, 1536, 2), (32, 2048, 1024, 1)])      # 625
def test_gathered_rows_go_in_pairs_where_the_shared_weights_pay(E, K, n_out, tiles):
    from zipage_b200.layers.feed_forward import grouped_gemm
    M = 20000
    x = torch.randn(5000, K, device="cuda", generator=_gen(K)).to(torch.bfloat16)
    w = (torch.randn(E, n_out, K, device="cuda", generator=_gen(n_out)) / K ** 0.5).to(torch.bfloat16)
    rows = torch.randint(0, 5000, (M,), device="cuda", generator=_gen(1)).to(torch.int32)
    off = (torch.arange(E + 1, device="cuda") * (M // E)).to(torch.int32)
    form = _form("grouped_gemm_tc_kernel", lambda: grouped_gemm(x, w, off, M, rows=rows, act="silu_mul"))
    assert form == ["256", "2", "2", str(tiles)]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("taps,bias", [(2, False), (4, False), (4, True)])
def test_convolutions_of_many_blocks_have_fewer_tokens_in_flight(dtype, taps, bias):
    """3072 channels in one call, where four blocks an SM leave fewer waves than three, and in thirds, where they do not; three taps stay as they are."""
    from zipage_b200.layers.short_conv import short_conv
    g, C, lens = _gen(taps), 3072, [2528, 31, 1, 700]
    n = sum(lens)
    x = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    cu, ctx, slots = _cu(lens), torch.tensor(lens, dtype=torch.int32, device="cuda") + 5, torch.arange(4, dtype=torch.int32, device="cuda")
    ring0 = torch.randn(4, taps, C, device="cuda", generator=g).to(dtype)
    w, b = torch.randn(taps, C, device="cuda", generator=g), torch.randn(C, device="cuda", generator=g) if bias else None

    def run(step, taps=taps):
        out, rings = torch.empty_like(x), []
        for c in range(0, C, step):
            s = slice(c, c + step)
            rings.append(ring0[:, :taps, s].contiguous())
            short_conv(x[:, s], w[:taps, s].contiguous(), rings[-1], ctx, slots, cu, max(lens), out[:, s], bias=None if b is None else b[s].contiguous())
        return out, torch.cat(rings, -1)
    many = lambda *a: _form("short_conv_kernel", lambda: run(*a))[-1] == "1"
    assert many(C) and not many(C // 3)
    for whole, parts in zip(run(C), run(C // 3)):
        assert torch.equal(whole, parts)
    if taps == 4:
        assert not many(C, 3)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("width,n,kind,three", [(1024, 1480, "experts", (1, 1, 0)), (1024, 1481, "experts", (0, 0, 0)), (1024, 592, "experts", (1, 1, 1)),
                                                (1536, 2000, "experts", (1, 1, 0)), (2048, 592, "experts", (1, 1, 1)), (4096, 444, "experts", (1, 1, 1)),
                                                (4096, 445, "experts", (0, 0, 0)), (2048, 100, "plain", (0, 0, 0)), (2048, 100, "pair", (0, 0, 0)),
                                                (5120, 8, "experts", (0, 0, 0)), (1030, 8, "experts", (0, 0, 0))])
def test_layer_boundaries_with_registers_for_the_experts_rows(dtype, width, n, kind, three):
    """Rows in one call and in parts of at most 400: the same bits, whichever form they take."""
    from zipage_b200.layers.row_ops import join_norms
    g, top = _gen(width + n), 5
    z = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, a, w1, w2 = z(n, width), z(n, width).to(dtype), z(width), z(width)
    more = {}
    if kind == "experts":
        y, pos, wts = z(n * top, width).to(dtype), torch.randperm(n * top, device="cuda", generator=g).to(torch.int32).view(n, top), z(n, top)
    elif kind == "pair":
        m = [z(n, width).to(dtype) for _ in range(2)]

    def run(step):
        out = []
        for i in range(0, n, step):
            s = slice(i, i + step)
            if kind == "experts":
                more.update(y=y, pos=pos[s], weights=wts[s])
            elif kind == "pair":
                more.update(pair=((m[0][s], w1), (m[1][s], w2)))
            r = x[s].clone()
            out.append([r] + join_norms(r, [(w1, w2), (w2, None)], 1e-5, dtype, a=a[s], **more))
        return [torch.cat(t) for t in zip(*out)]
    for whole, parts in zip(run(n), run(400)):
        assert torch.equal(whole, parts)
    assert (_form("join_norms_kernel", lambda: run(n))[-1] == "3") == bool(three[list(TYPES).index(dtype)])


@pytest.mark.parametrize("dtype,D,n,blocks", [
    (torch.bfloat16, 128, 64, 3), (torch.bfloat16, 128, 6000, 3), (torch.float16, 128, 64, 3), (torch.float16, 128, 1900, 3), (torch.float16, 128, 2000, 0),
    (torch.float16, 128, 1000, 0), (torch.float32, 128, 64, 0), (torch.float32, 128, 1500, 0), (torch.float32, 128, 1600, 3), (torch.float32, 128, 1000, 3),
    (torch.float16, 64, 2000, 3), (torch.float32, 64, 64, 3)])
@pytest.mark.parametrize("packed", [True, False])
def test_registers_of_the_head_norms(dtype, D, n, blocks, packed):
    """One call and parts of 500 rows: the same bits, whichever form they take."""
    from zipage_b200.layers import step_ops as P
    heads, kv_heads, g = 32, 8, _gen(n)
    qkv = torch.randn(n, (heads + 2 * kv_heads) * D, device="cuda", generator=g).to(dtype)
    pos, cs = torch.randint(0, 4096, (n,), device="cuda", generator=g), P.rope_cos_sin_cache(D, 4096, 1e6, "cuda")
    w = [(1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(dtype) for _ in range(2)]
    slot = torch.randperm(n, device="cuda", generator=g).to(torch.int32)

    def run(step):
        cache = [torch.zeros((n + 255) // 256, 256, kv_heads, D, dtype=dtype, device="cuda") for _ in range(2)]
        parts = [P.qk_norm_rope_store(qkv[i:i + step], pos[i:i + step], cs, *w, 1e-6, heads, kv_heads, D, *cache, slot[i:i + step], return_v=packed)
                 for i in range(0, n, step)]
        return [torch.cat(t) for t in zip(*parts)] + cache
    for whole, parts in zip(run(n), run(500)):
        assert torch.equal(whole, parts)
    form = _form("qk_norm_rope_store_kernel", lambda: run(n))
    assert form[:3] == [TYPES[dtype], str(D), str(blocks)] and form[3] == str(int(packed))


def _decoded(B, kp, vp, window=1024, width=35):
    """Arguments of a decoded window of 16 heads on 8, every sequence with all of its keys."""
    g, page = _gen(B + kp), 64
    draw = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    table = torch.randperm(B * width, device="cuda", generator=g).to(torch.int32).view(B, width)
    ctx = torch.full((B,), width * page, dtype=torch.int32, device="cuda")
    return draw(B, 16 * kp), draw(B * width, page, 8, kp), draw(B * width, page, 8, vp), ctx, table, 16, kp, vp, kp ** -0.5, window


@pytest.mark.parametrize("B,kp,vp,merged", [
    (24, 128, 128, True), (28, 128, 128, False), (32, 128, 128, False), (60, 128, 128, True), (40, 64, 64, True), (48, 64, 64, False), (8, 256, 256, True),
    (16, 256, 256, False), (16, 192, 128, True), (32, 192, 128, False), (48, 192, 128, True), (24, 96, 96, True)])
def test_decoded_windows_split_as_the_sms_hold_blocks(B, kp, vp, merged):
    """More than one split leaves a merge behind it; the shared memory of a block counts keys and values by their own sizes."""
    from zipage_b200.layers.attention import window_attention
    args = _decoded(B, kp, vp)
    names = _kernels(lambda: window_attention(*args))
    assert ("window_decode_merge_kernel" in names) == merged
    out, (q, k, v, _, table) = window_attention(*args), args[:5]
    for b in (0, B - 1):
        kk, vv = (t[table[b].long()].flatten(0, 1)[-1024:].double().repeat_interleave(2, 1) for t in (k, v))
        w = torch.softmax(torch.einsum("hd,nhd->hn", q[b].double().view(16, kp), kk) * kp ** -0.5, -1)
        ref, mag = torch.einsum("hn,nhd->hd", w, vv), torch.einsum("hn,nhd->hd", w, vv.abs())
        # weights as two bf16 numbers (2^-16), the result rounded once
        assert ((out[b].view(16, vp).double() - ref).abs() <= (2.0 ** -8 + 2.0 ** -14) * mag + 1e-6).all()


def test_decoded_windows_take_a_workspace_sized_for_a_larger_batch(monkeypatch):
    from zipage_b200 import _lib as L
    from zipage_b200.layers import attention as A
    buf = torch.empty(L.load().zp_window_attention_workspace_bytes(48, 16, 8, 128, 1024), dtype=torch.uint8, device="cuda")
    args = _decoded(24, 128, 128)
    want = A.window_attention(*args)
    monkeypatch.setattr(A, "_workspace", lambda device, nbytes: buf)
    assert buf.numel() and torch.equal(A.window_attention(*args), want)
