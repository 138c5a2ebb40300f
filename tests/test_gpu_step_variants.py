"""The size-dependent forms of the per-step kernels at the sizes where they change over."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv_heads,D", [(32, 8, 128), (5, 1, 128), (18, 6, 64)])
def test_qk_norm_rope_is_the_same_for_few_and_many_tokens(dtype, heads, kv_heads, D):
    """1100 tokens in one call (32 heads a warp) and in halves (four heads a warp): the same arithmetic, the same bits."""
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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N", [1, 37, 1023, 1025])
@pytest.mark.parametrize("kv_heads,D", [(8, 128), (3, 64)])
@pytest.mark.parametrize("stored", [True, False])
def test_values_are_packed_beside_the_keys(dtype, N, kv_heads, D, stored):
    """v is a packed copy of qkv's columns, rows without a cache slot among them, or a view of them: as `return_v` says, or else `return_k`."""
    from zipage_b200.layers import step_ops as P
    g, heads, dev = _gen(N), 4, "cuda"
    wide = torch.randn(N, (heads + 2 * kv_heads) * D + 16, device=dev, generator=g).to(dtype)
    qkv = wide[:, :-16]                                   # (rows further apart than they are long)
    pos, cs = torch.randint(0, 4096, (N,), device=dev, generator=g), P.rope_cos_sin_cache(D, 4096, 1e6, dev)
    w = [torch.ones(D, device=dev, dtype=dtype)] * 2
    cache = {}
    if stored:
        slot = torch.randperm(1280, device=dev, generator=g)[:N].to(torch.int32)
        slot[::5] = -1
        cache = dict(k_cache=torch.zeros(5, 256, kv_heads, D, dtype=dtype, device=dev), v_cache=torch.zeros(5, 256, kv_heads, D, dtype=dtype, device=dev),
                     slot_mapping=slot)
    want = qkv[:, (heads + kv_heads) * D:].unflatten(1, (kv_heads, D))
    _, _, v = P.qk_norm_rope_store(qkv, pos, cs, *w, 1e-6, heads, kv_heads, D, **cache)
    assert v.is_contiguous() and torch.equal(v, want)
    if stored:
        rows = torch.zeros(1280, kv_heads, D, dtype=dtype, device=dev)
        rows[slot[slot >= 0].long()] = want[slot >= 0]
        assert torch.equal(cache["v_cache"].view(1280, kv_heads, D), rows)
    _, k, v = P.qk_norm_rope_store(qkv, pos, cs, *w, 1e-6, heads, kv_heads, D, return_k=False)
    assert k is None and v.data_ptr() == want.data_ptr() and torch.equal(v, want)
    # keys alone, without the copy of the values that their caller does not ask for; and the other way round
    _, keys, v = P.qk_norm_rope_store(qkv, pos, cs, *w, 1e-6, heads, kv_heads, D, return_v=False)
    assert keys.is_contiguous() and v.data_ptr() == want.data_ptr()
    _, k, v = P.qk_norm_rope_store(qkv, pos, cs, *w, 1e-6, heads, kv_heads, D, return_k=False, return_v=True)
    assert k is None and v.is_contiguous() and v.data_ptr() != want.data_ptr() and torch.equal(v, want)


def _draws(seed, rows, V):
    """The Exp(1) draws of the built-in generator (fp64 logarithm of the same uniform numbers)."""
    m = 0xFFFFFFFF

    def mix(x):
        x = x ^ (x >> 16)
        x = (x * 0x7feb352d) & m
        x = x ^ (x >> 15)
        x = (x * 0x846ca68b) & m
        return x ^ (x >> 16)
    r, i = torch.arange(rows, device="cuda")[:, None], torch.arange(V, device="cuda")[None]
    h = mix(((seed & m) ^ ((r * 0x9e3779b9) & m)) + ((i * 0x85ebca6b) & m) & m)
    h = mix(h ^ (seed >> 32) ^ r)
    u = ((h >> 8).float() + 0.5) * (1.0 / 16777216.0)
    return (-torch.log(u.double())).clamp_min(1e-10)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,V", [(1, 1), (3, 7), (5, 8191), (4, 8192), (2, 16385), (3, 50257), (9, 151936)])
@pytest.mark.parametrize("spread", [0.01, 3.0])
def test_sampler_takes_the_best_of_all_draws(dtype, rows, V, spread):
    """Against the race over every draw in fp64: the sampled token's ratio is the largest up to the draws' fp32 rounding (a fast
    logarithm, 2^-21 of its argument's distance from 1, and a few roundings)."""
    from zipage_b200.layers import step_ops as P
    z = (torch.randn(rows, V, device="cuda", generator=_gen(V)) * spread).to(dtype)
    t = 0.5 + torch.rand(rows, device="cuda", generator=_gen(rows))
    seed = (5 << 32) + 12345 + V
    tok = P.sample(z, t, seed=seed)
    q = _draws(seed, rows, V)
    x = z.double() / t.double()[:, None]
    e = torch.exp(x - x.max(-1, keepdim=True).values)
    lower, upper = (e / (q + 1e-6)).max(-1).values, (e / (q - 1e-6).clamp_min(1e-10)).gather(1, tok[:, None])[:, 0]
    assert (upper >= lower * (1 - 1e-5)).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,V", [(1, 70001), (12, 50257), (13, 50257), (27, 25001), (28, 16384), (74, 12288), (75, 70001), (148, 300), (149, 300), (149, 70001), (223, 66000)])
@pytest.mark.parametrize("given", [True, False])
def test_sampler_over_the_numbers_of_rows(dtype, rows, V, given):
    """Where the blocks a row is spread over and their threads change: the sampled token's ratio is the largest up to fp32 roundings."""
    from zipage_b200.layers import step_ops as P
    z = (torch.randn(rows, V, device="cuda", generator=_gen(V)) * 2).to(dtype)
    t = 0.5 + torch.rand(rows, device="cuda", generator=_gen(rows))
    q = torch.empty(rows, V, device="cuda").exponential_(1.0, generator=_gen(rows + V)) if given else None
    tok = P.sample(z, t, noise=q, seed=77)
    q = q.double().clamp_min(1e-10) if given else _draws(77, rows, V)
    x = z.double() / t.double()[:, None]
    e = torch.exp(x - x.max(-1, keepdim=True).values)
    slack = 0.0 if given else 1e-6                        # of the built-in draws, as in the test above
    lower, upper = (e / (q + slack)).max(-1).values, (e / (q - slack).clamp_min(1e-10)).gather(1, tok[:, None])[:, 0]
    assert (upper >= lower * (1 - 1e-5)).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 2, 7, 8])
@pytest.mark.parametrize("n_out,k,bias", [(16, 32, False), (40, 96, True), (1000, 1024, True), (256, 2048 + 32, False)])
def test_small_linear(dtype, rows, n_out, k, bias):
    from zipage_b200.layers.step_ops import linear
    g = _gen(rows + k)
    layer = torch.nn.Linear(k, n_out, bias=bias, device="cuda", dtype=dtype)
    x = torch.randn(rows, 2 * k, device="cuda", generator=g).to(dtype)[:, :k]      # (a column view)
    with torch.no_grad():
        out = linear(layer, x)
        w, b = layer.weight.double(), layer.bias.double() if bias else 0.0
    ref, mag = x.double() @ w.T + b, x.double().abs() @ w.abs().T
    # fp32 sums of k products, then one rounding to 8 or 11 significant bits
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert ((out.double() - ref).abs() <= unit * ref.abs() + 2.0 ** -24 * k * mag + 1e-7).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 5, 8])
@pytest.mark.parametrize("k", [992, 1056, 2016, 2048, 3072, 3104, 4064, 4096])
def test_small_linear_over_the_splits_of_the_inner_dimension(dtype, rows, k):
    """Warps and loads in flight depend on k: whole turns, turns that end early, warps of unequal parts."""
    from zipage_b200.layers.step_ops import linear
    g = _gen(rows + k)
    layer = torch.nn.Linear(k, 72, bias=False, device="cuda", dtype=dtype)
    x = torch.randn(rows, k, device="cuda", generator=g).to(dtype)
    with torch.no_grad():
        out, w = linear(layer, x), layer.weight.double()
    ref, mag = x.double() @ w.T, x.double().abs() @ w.abs().T
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11              # as above
    assert ((out.double() - ref).abs() <= unit * ref.abs() + 2.0 ** -24 * k * mag + 1e-7).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n_out,k", [(40, 256), (40, 512), (40, 768), (40, 1024), (40, 1280), (40, 1536), (40, 1792), (72, 2048), (72, 2304), (2376, 3072), (2368, 3072),
                                     (72, 3328), (2376, 3328), (2368, 3328), (72, 4096)])
def test_small_linear_adds_eight_parts_of_the_inner_dimension(dtype, n_out, k):
    """Whatever the number of loads in flight, the fp32 sums are those of eight consecutive eighths, added in order: 2^24 from the first, 1 + 1 from
    both ends of the second and -2^24 from the last give 2; with the ones added one by one it would be 0."""
    from zipage_b200.layers.step_ops import linear
    layer = torch.nn.Linear(k, n_out, bias=False, device="cuda", dtype=dtype)
    x, e = torch.zeros(3, k, device="cuda", dtype=dtype), k // 8
    x[:, e - 1], x[:, e], x[:, 2 * e - 1], x[:, -1] = 4096, 1, 1, -4096
    with torch.no_grad():
        layer.weight.zero_()
        layer.weight[:, [e - 1, -1]] = 4096
        layer.weight[:, [e, 2 * e - 1]] = 1
        out = linear(layer, x)
    assert torch.equal(out, torch.full_like(out, 2))


def test_linear_leaves_the_rest_to_the_layer():
    from zipage_b200 import kernel as K
    from zipage_b200.layers.step_ops import SMALL_ROWS, linear
    layer = torch.nn.Linear(64, 48, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(SMALL_ROWS + 1, 64, device="cuda", dtype=torch.bfloat16)
    before = K.LAUNCHES
    y = linear(layer, x[:4])                          # gradients wanted
    assert y.requires_grad
    with torch.no_grad():
        assert torch.equal(linear(layer, x), layer(x))
        handle = layer.register_forward_hook(lambda m, i, o: o * 0)
        assert not linear(layer, x[:4]).any()
        handle.remove()
        with torch.autocast("cuda", torch.float16):
            assert linear(layer, x[:4]).dtype == torch.float16
        layer.forward = lambda v: v * 0
        assert not linear(layer, x[:4]).any()
        del layer.forward
        for k in (32, 96):                            # the layer refuses an input of another width
            with pytest.raises(RuntimeError):
                linear(layer, torch.randn(4, k, device="cuda", dtype=torch.bfloat16))
    assert K.LAUNCHES == before


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,heads,kv_heads,width", [(1, 8, 8, 16), (2, 16, 1, 9), (5, 32, 8, 16), (3, 4, 2, 17), (70, 8, 1, 4)])
def test_paged_decode_splits(dtype, B, heads, kv_heads, width):
    """Short tables split within a cluster, longer ones (17 pages) through scratch."""
    from zipage_b200.layers.attention import paged_decode_attention
    g, D = _gen(B), 128
    lens = torch.tensor([1, 63, 64, 65, width * 256][:B] + [128 + 13 * i for i in range(max(0, B - 5))], dtype=torch.int32, device="cuda")
    table = torch.full((B, width), -1, dtype=torch.int32, device="cuda")
    need = ((lens + 255) // 256).tolist()
    ids = torch.randperm(sum(need), device="cuda", generator=g).to(torch.int32)
    for b, part in enumerate(ids.split(need)):
        table[b, :need[b]] = part
    kc, vc = (torch.randn(sum(need), 256, kv_heads, D, device="cuda", generator=g).to(dtype) for _ in range(2))
    q = torch.randn(B, 1, heads, D, device="cuda", generator=g).to(dtype)
    out = paged_decode_attention(q, kc, vc, lens, table)
    unit = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.1      # weights and result are rounded once each
    for b in range(B):
        n = int(lens[b])
        k, v = (c[table[b, :need[b]].long()].flatten(0, 1)[:n].double().repeat_interleave(heads // kv_heads, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,shd->hs", q[b, 0].double(), k) * D ** -0.5, -1)
        ref, mag = torch.einsum("hs,shd->hd", w, v), torch.einsum("hs,shd->hd", w, v.abs())
        assert ((out[b, 0].double() - ref).abs() <= 2 * unit * mag + 1e-6).all()


@pytest.mark.parametrize("B,kv_heads,width", [(55, 8, 3), (56, 8, 3), (444, 1, 2), (445, 1, 2), (75, 8, 2), (3, 2, 1)])
def test_paged_decode_of_as_many_splits_as_fit(B, kv_heads, width):
    """Clusters up to 444 (sequence, key/value head) pairs, two splits with scratch up to 591, none beyond; one page is never split."""
    from zipage_b200.layers.attention import paged_decode_attention
    g, D, heads = _gen(B), 128, 2 * kv_heads
    lens = torch.randint(1, width * 256 + 1, (B,), device="cuda", generator=g, dtype=torch.int32)
    kc, vc = (torch.randn(40, 256, kv_heads, D, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    table = torch.randint(0, 40, (B, width), device="cuda", generator=g, dtype=torch.int32)      # (pages may be shared)
    q = torch.randn(B, 1, heads, D, device="cuda", generator=g).to(torch.bfloat16)
    out = paged_decode_attention(q, kc, vc, lens, table)
    for b in (0, 1, B // 2, B - 1):
        n = int(lens[b])
        k, v = (c[table[b].long()].flatten(0, 1)[:n].double().repeat_interleave(2, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,shd->hs", q[b, 0].double(), k) * D ** -0.5, -1)
        ref, mag = torch.einsum("hs,shd->hd", w, v), torch.einsum("hs,shd->hd", w, v.abs())
        assert ((out[b, 0].double() - ref).abs() <= 2.0 ** -8 * 1.1 * 2 * mag + 1e-6).all()      # as in test_paged_decode_splits


@pytest.mark.parametrize("offset", [0, 4, 8])
def test_paged_decode_takes_scratch_of_exactly_the_needed_size(offset):
    """Wherever floats may lie: all splits run, so that the bits are those of a call with plenty, and nothing is noted."""
    from zipage_b200 import _lib as L
    lib, B, heads, kv_heads, D, width = L.load(), 2, 8, 2, 128, 20
    g = _gen(offset)
    kc, vc = (torch.randn(B * width, 256, kv_heads, D, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    table = torch.arange(B * width, dtype=torch.int32, device="cuda").view(B, width)
    lens, q = torch.tensor([width * 256, 4000], dtype=torch.int32, device="cuda"), torch.randn(B, heads, D, device="cuda", generator=g).to(torch.bfloat16)

    def call(ws, size):
        out = torch.empty_like(q)
        rc = lib.zp_paged_decode(L.ptr(q), L.ptr(kc), L.ptr(vc), L.ptr(lens), L.ptr(table), L.ptr(out), B, width, heads, kv_heads, D, 256, kc.stride(0),
                                 D ** -0.5, L.dtype_code(q), ws, size, L.stream_ptr())
        torch.cuda.synchronize()
        assert rc == 0
        return out
    splits = min(width, 32)                               # (148 * 4 blocks over 2 x 2 would be more)
    exact = B * kv_heads * splits * 4 * (D + 2) * 4       # groups of 4 heads
    plenty = torch.empty(2 * exact, dtype=torch.uint8, device="cuda")
    ws = torch.empty(exact + offset, dtype=torch.uint8, device="cuda")
    want = call(plenty.data_ptr(), plenty.numel())
    call(0, 0)
    unsplit = lib.zp_last_error()
    assert b"unsplit" in unsplit
    assert lib.zp_rms_norm(*[None] * 5, 4, 4096, 4096, 4096, 1e-6, 0, None) != 0       # (another note)
    other = lib.zp_last_error()
    assert torch.equal(call(ws.data_ptr() + offset, exact), want) and lib.zp_last_error() == other
    assert lib.zp_paged_decode_workspace_bytes(B, heads, D, 32) >= exact


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("q_rank,R,rot,heads,dim", [(2048, 1024, 64, 5, 8), (2056, 1024, 64, 1, 128), (8, 8, 8, 33, 64), (1536, 512, 24, 16, 0)])
def test_latent_rows_in_vectors(dtype, q_rank, R, rot, heads, dim):
    from zipage_b200.layers.latent_attention import latent_prepare, latent_rotate_q, rotary_turns
    g, N, KP = _gen(q_rank + rot), 13, (R + rot + 15) // 16 * 16
    n = lambda *s: torch.randn(*s, device="cuda", generator=g)
    y, wq, wk = n(N, q_rank + R + rot).to(dtype), n(q_rank), n(R)
    pos, turns = torch.arange(N, device="cuda") * 4099, rotary_turns(rot, 10000.0, "cuda")
    cache, dense = torch.zeros(1, 16, 1, KP, dtype=dtype, device="cuda"), torch.full((N, KP), 7.0, dtype=dtype, device="cuda")
    slots = torch.arange(N, dtype=torch.int32, device="cuda")
    cq = latent_prepare(y, pos, turns, wq, wk, cache, slots, q_rank, R, rot, 1e-5, dense)
    norm = lambda x, w: x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    angle = pos[:, None].double() * 10000.0 ** (-torch.arange(0, rot, 2, device="cuda").double() / rot)
    c, s = angle.cos(), angle.sin()

    def turn(x):
        a, b = x[..., ::2].double(), x[..., 1::2].double()
        cc, ss = (c, s) if x.dim() == 2 else (c[:, None], s[:, None])
        return torch.stack([a * cc - b * ss, a * ss + b * cc], -1).flatten(-2)

    # one rounding to T (half a unit in the last place) and fp32 arithmetic before it, also where a rotation's two parts cancel
    close = lambda got, want: ((got.double() - want).abs() <= torch.finfo(dtype).eps / 2 * want.abs() + 4e-6).all()
    assert close(cq, norm(y[:, :q_rank], wq))
    want = torch.cat([norm(y[:, q_rank:q_rank + R], wk), turn(y[:, q_rank + R:])], -1)
    assert close(dense[:, :R + rot], want) and (dense[:, R + rot:] == 0).all() and torch.equal(cache.view(16, KP)[:N], dense)
    q = n(N, heads * (dim + rot)).to(dtype)
    want, ql = turn(q.view(N, heads, -1)[..., dim:]), torch.full((N, heads, KP), 7.0, dtype=dtype, device="cuda")
    latent_rotate_q(q, pos, turns, heads, dim, rot, ql, R)
    assert close(ql[..., R:R + rot], want) and (ql[..., R + rot:] == 0).all() and (ql[..., :R] == 7).all()
    before = q.clone()
    latent_rotate_q(q, pos, turns, heads, dim, rot)
    assert close(q.view(N, heads, -1)[..., dim:], want) and torch.equal(q.view(N, heads, -1)[..., :dim], before.view(N, heads, -1)[..., :dim])


@pytest.mark.parametrize("rows,width", [(1, 256), (4, 1024), (8, 2048)])
def test_kernels_that_begin_early_see_what_came_before(rows, width):
    from zipage_b200.layers.step_ops import linear, rms_norm, silu_and_mul
    g = _gen(width)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    x0, r0, norm, ws = n(rows, width), n(rows, width), n(width), [n(2 * width, width) * width ** -0.5 for _ in range(2)]
    layer = torch.nn.Linear(width, 2 * width, bias=False, device="cuda", dtype=torch.bfloat16)
    x, r = x0.clone(), r0.clone()

    @torch.no_grad()
    def chain(after):
        x.copy_(x0), r.copy_(r0)
        for i in range(30):
            layer.weight.copy_(ws[i % 2]), after()          # the weight changes right before it is read
            h, rr = rms_norm(x, norm, 1e-5, r)
            after()
            y = linear(layer, h)
            after()
            x.copy_(silu_and_mul(y)) if i % 3 else x.copy_(rms_norm(silu_and_mul(y), norm, 1e-5))
            r.copy_(rr), after()
        return torch.cat([x, r])

    want = chain(torch.cuda.synchronize).clone()
    assert want.isfinite().all()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(lambda: None)
    for _ in range(5):
        assert torch.equal(chain(lambda: None), want)
        graph.replay()
        assert torch.equal(out, want)


@pytest.mark.parametrize("n,width", [(1, 1), (3, 70), (8, 129), (7, 129), (8, 0)])
def test_decode_inputs(n, width):
    from zipage_b200.layers.step_ops import decode_inputs
    g = _gen(n + width)
    n32 = lambda *s: torch.randint(0, 1000, s, device="cuda", generator=g, dtype=torch.int32)
    ids, num, tab, qid = n32(n).long(), n32(n), n32(n, width + 3)[:, :width], n32(n)
    buffers = (torch.full((8,), 5, dtype=torch.int64, device="cuda"), n32(8), n32(8, 129), n32(8))
    assert decode_inputs(ids, num, tab, qid, buffers)
    want = torch.full((8, 129), -1, dtype=torch.int32, device="cuda")
    want[:n, :width] = tab
    assert torch.equal(buffers[2], want) and torch.equal(buffers[0][:n], ids) and (buffers[0][n:] == 5).all()
    assert torch.equal(buffers[1][:n], num) and (buffers[1][n:] == 0).all() and torch.equal(buffers[3][:n], qid) and (buffers[3][n:] == -1).all()
    assert not decode_inputs(ids, num.long(), tab, qid, buffers) and not decode_inputs(ids, num, tab.cpu(), qid, buffers)
