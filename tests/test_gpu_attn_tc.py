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
    # weights and result are rounded to T once each, to 8 or 11 significant bits; the rest is fp32
    unit = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.1
    a = b = 0
    for x, y in zip(lens_q, lens_k):
        seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
        ref, mag = _softmax(q[a:a + x], k[b:b + y], v[b:b + y], D ** -0.5, seen)
        assert ((out[a:a + x].double() - ref).abs() <= unit * 2 * mag + 1e-6).all()
        a, b = a + x, b + y


def _paged(rows, lens, page, table):
    """rows [sum(lens), ...] on the pages of `table`; everything else holds NaN."""
    cache = torch.full((int(table.max()) + 1, page, *rows.shape[1:]), float("nan"), dtype=rows.dtype, device="cuda")
    at = 0
    for b, n in enumerate(lens):
        for i in range(0, n, page):
            part = rows[at + i:at + min(n, i + page)]
            cache[table[b, i // page], :len(part)] = part
        at += n
    return cache


@pytest.mark.parametrize("many", [False, True])          # launches of few and of many query tiles take different kernels
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 128), (6, 2, 128, 128), (3, 3, 96, 40), (8, 2, 64, 64)])
@pytest.mark.parametrize("window,softcap,keep,biased,chunk", [(0, 0.0, 0, False, 0), (130, 30.0, 0, False, 0), (200, 0.0, 70, True, 0), (0, 50.0, 0, False, 256)])
def test_window_edges(many, heads, kv_heads, dim, vdim, window, softcap, keep, biased, chunk):
    from zipage_b200.layers.attention import window_attention
    copies = 1 + 710 // (10 * heads) if many else 1
    lens_q, lens_k = [1, 129, 400, 250] * copies, [513, 129, 700, 251] * copies
    g = torch.Generator(device="cuda").manual_seed(heads + dim)
    n = lambda rows, h, d: torch.randn(rows, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = n(sum(lens_q), heads, dim), n(sum(lens_k), kv_heads, dim), n(sum(lens_k), kv_heads, vdim)
    pad = lambda t: torch.nn.functional.pad(t, (0, -t.shape[2] % 16))
    need = [(m + 63) // 64 for m in lens_k]
    ids, table = torch.randperm(sum(need), device="cuda", generator=g).to(torch.int32), torch.full((len(need), max(need)), -1, dtype=torch.int32, device="cuda")
    for b, part in enumerate(ids.split(need)):
        table[b, :need[b]] = part
    kc, vc = _paged(pad(k), lens_k, 64, table), _paged(pad(v), lens_k, 64, table)
    slopes = torch.rand(heads, device="cuda", generator=g) * 0.05 if biased else None
    gate, sink = n(sum(lens_q), heads, 1)[..., 0].contiguous(), torch.randn(heads, device="cuda", generator=g)
    out = window_attention(q.flatten(1), kc, vc, torch.tensor(lens_k, dtype=torch.int32, device="cuda"), table, heads, dim, vdim, dim ** -0.5, window,
                           softcap, cu_seqlens_q=_cu(lens_q), max_seqlen_q=max(lens_q), impl="auto" if many else "tcgen05", chunk=chunk, keep=keep, slopes=slopes, sink=sink,
                           gate=gate, gate_mode="head")
    _no_device_error()
    for i, (x, y) in enumerate(zip(lens_q, lens_k)):
        a, b = sum(lens_q[:i]), sum(lens_k[:i])
        if 4 <= i < len(lens_q) - 4:
            continue
        p, j = torch.arange(y - x, y, device="cuda")[:, None], torch.arange(y, device="cuda")[None]
        seen = j <= p
        if window:
            seen &= (p - j < window) | (j < keep)
        if chunk:
            seen &= p // chunk == j // chunk
        G = heads // kv_heads
        kk, vv = k[b:b + y].double().repeat_interleave(G, 1), v[b:b + y].double().repeat_interleave(G, 1)
        s = torch.einsum("thd,shd->hts", q[a:a + x].double(), kk) * dim ** -0.5
        s = softcap * torch.tanh(s / softcap) if softcap else s
        s = s - slopes.double()[:, None, None] * (p - j) if biased else s
        s = torch.cat([s.masked_fill(~seen[None], float("-inf")), sink.double()[:, None, None].expand(-1, x, 1)], -1)
        w = torch.softmax(s, -1)[..., :-1] * torch.sigmoid(gate[a:a + x].double()).T[..., None]
        ref, mag = torch.einsum("hts,shd->thd", w, vv), torch.einsum("hts,shd->thd", w, vv.abs())
        # one rounding of the result to 8 significant bits (at most 2^-8 of it); weights carry 16 bits, their exponents an fp32 rounding
        assert ((out[a:a + x].view(x, heads, vdim).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * mag + 1e-6).all()


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("dim,rot,vdim,rank", [(128, 64, 128, 512), (64, 0, 64, 64), (96, 32, 40, 64), (128, 128, 128, 128)])
def test_latent_prefill_edges(many, dim, rot, vdim, rank):
    from zipage_b200.layers.latent_attention import latent_prefill
    copies = 16 if many else 1
    heads, lens_q, lens_k = 3, [1, 127, 300, 513] * copies, [130, 127, 301, 900] * copies
    g = torch.Generator(device="cuda").manual_seed(dim + rot)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    rows, keys = sum(lens_q), sum(lens_k)
    q, kv, lat = n(rows, heads * (dim + rot)), n(keys, heads * (dim + vdim)), n(keys, rank + rot)
    out = torch.empty(rows, heads * vdim, dtype=torch.bfloat16, device="cuda")
    latent_prefill(q, kv, lat, _cu(lens_q), _cu(lens_k), max(lens_q), out, heads, dim, rot, vdim, rank, (dim + rot) ** -0.5)
    _no_device_error()
    a = b = 0
    for x, y in zip(lens_q, lens_k):
        k = torch.cat([kv[b:b + y, :heads * dim].view(y, heads, dim), lat[b:b + y, None, rank:].expand(-1, heads, -1)], -1)
        seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
        ref, mag = _softmax(q[a:a + x].view(x, heads, dim + rot), k, kv[b:b + y, heads * dim:].view(y, heads, vdim), (dim + rot) ** -0.5, seen)
        assert ((out[a:a + x].view(x, heads, vdim).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * mag + 1e-6).all()
        a, b = a + x, b + y


@pytest.mark.parametrize("scale", [0.0, -0.04])
@pytest.mark.parametrize("kind", ["prompts", "prompts_fp16", "windows_64", "windows_128", "windows_biased", "windows_capped", "latents"])
@pytest.mark.parametrize("copies", [1, 40])              # launches of few and of many query tiles
def test_factors_of_zero_and_below(kind, scale, copies):
    """The mean of the visible values, or weights that fall with the product; masked keys stay unseen."""
    from zipage_b200.layers import attention as A
    from zipage_b200.layers.latent_attention import latent_prefill
    heads, kv_heads, dtype = 4, 2, torch.float16 if kind == "prompts_fp16" else torch.bfloat16
    lens_q, lens_k = [1, 129, 250] * copies, [70, 129, 400] * copies
    g = torch.Generator(device="cuda").manual_seed(copies)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)
    rows, keys, cap, slopes = sum(lens_q), sum(lens_k), 0.0, None
    if kind == "latents":
        kv_heads = heads
        q, kv, lat, out = n(rows, heads * D), n(keys, heads * (64 + 128)), n(keys, 64 + 64), torch.empty(rows, heads * 128, dtype=dtype, device="cuda")
        latent_prefill(q, kv, lat, _cu(lens_q), _cu(lens_k), max(lens_q), out, heads, 64, 64, 128, 64, scale)
        q, v = q.view(rows, heads, D), kv[:, heads * 64:].view(keys, heads, 128)
        k = torch.cat([kv[:, :heads * 64].view(keys, heads, 64), lat[:, None, 64:].expand(-1, heads, -1)], -1)
    elif kind.startswith("prompts"):
        q, k, v = n(rows, heads, D), n(keys, kv_heads, D), n(keys, kv_heads, D)
        out = A.varlen_prefill_attention(q, k, v, max(lens_q), _cu(lens_q), max(lens_k), _cu(lens_k), softmax_scale=scale)
    else:
        d = 64 if kind == "windows_64" else 128
        q, k, v = n(rows, heads, d), n(keys, kv_heads, d), n(keys, kv_heads, d)
        need = [(m + 63) // 64 for m in lens_k]
        table = torch.full((len(need), max(need)), -1, dtype=torch.int32, device="cuda")
        for b, part in enumerate(torch.arange(sum(need), dtype=torch.int32, device="cuda").split(need)):
            table[b, :need[b]] = part
        cap, slopes = 30.0 if kind == "windows_capped" else 0.0, torch.rand(heads, device="cuda", generator=g) * 0.05 if kind == "windows_biased" else None
        out = A.window_attention(q.flatten(1), _paged(k, lens_k, 64, table), _paged(v, lens_k, 64, table), torch.tensor(lens_k, dtype=torch.int32, device="cuda"),
                                 table, heads, d, d, scale, 0, cap, cu_seqlens_q=_cu(lens_q), max_seqlen_q=max(lens_q), slopes=slopes)
    _no_device_error()
    # as in the tests above: weights of prompts are rounded to T, the others carry 16 bits; one rounding of the result
    unit = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.1
    for b in (0, 1, 2, len(lens_q) - 1):
        x, y, r0, k0 = lens_q[b], lens_k[b], sum(lens_q[:b]), sum(lens_k[:b])
        p, j = torch.arange(y - x, y, device="cuda")[:, None], torch.arange(y, device="cuda")[None]
        kk, vv = (t[k0:k0 + y].double().repeat_interleave(heads // kv_heads, 1) for t in (k, v))
        s = torch.einsum("thd,shd->hts", q[r0:r0 + x].double(), kk) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = s if slopes is None else s - slopes.double()[:, None, None] * (p - j)
        w = torch.softmax(s.masked_fill(j > p, float("-inf")), -1)
        ref, mag = torch.einsum("hts,shd->thd", w, vv), torch.einsum("hts,shd->thd", w, vv.abs())
        err = (out[r0:r0 + x].view(x, heads, -1).double() - ref).abs()
        assert (err <= (unit * 2 * mag if kind.startswith("prompts") else 2.0 ** -8 * ref.abs() + 1e-4 * mag) + 1e-6).all()


def _climb(q, k, lens, at):
    """Scores that climb from 128 keys to the next by about 45 powers of two (a steeper step every third time), for the heads whose
    queries look at entry `at`: one head up, one down, the others not.  q, k [rows, heads, d]; scale d^-0.5."""
    step = 45.0 / 1.4427 * q.shape[2] ** 0.5 / 8
    k[:, :, at] = torch.cat([(torch.arange(n, device="cuda") // 128 * 1.0 + torch.arange(n, device="cuda") // 384) * step for n in lens])[:, None].to(k.dtype)
    q[:, :, at] = 0
    q[:, 0, at], q[:, -1, at] = 8, -8


# scores reach some 700 powers of two; the accumulators keep 2^-22 of their raw products, which moves weight and sum by 1.2e-4 each
CLIMB_ERROR = 4e-4


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv_heads", [(4, 2), (3, 1)])
def test_prompts_whose_reference_moves(dtype, heads, kv_heads):
    """The reference moves by more than the lazy bound at almost every key tile, and the accumulator with it."""
    from zipage_b200.layers.attention import varlen_prefill_attention
    lens_q, lens_k = [1000, 130, 700], [1300, 1100, 700]
    g = torch.Generator(device="cuda").manual_seed(heads)
    n = lambda rows, h: torch.randn(rows, h, D, device="cuda", generator=g).to(dtype)
    q, k, v = n(sum(lens_q), heads), n(sum(lens_k), kv_heads), n(sum(lens_k), kv_heads)
    _climb(q, k, lens_k, 5)
    out = varlen_prefill_attention(q, k, v, max(lens_q), _cu(lens_q), max(lens_k), _cu(lens_k))
    _no_device_error()
    unit = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.1      # as in test_prefill_edges
    a = b = 0
    for x, y in zip(lens_q, lens_k):
        seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
        ref, mag = _softmax(q[a:a + x], k[b:b + y], v[b:b + y], D ** -0.5, seen)
        assert ((out[a:a + x].double() - ref).abs() <= (unit * 2 + CLIMB_ERROR) * mag + 1e-6).all()
        a, b = a + x, b + y


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("key", [0, 31, 63, 64, 100, 127])
@pytest.mark.parametrize("heads,n", [(2, 512), (2, 600), (40, 600)])      # a tile an SM, two groups of warps that share a row or one; pairs of tiles
def test_prompts_whose_reference_moves_in_one_half_of_a_row(dtype, key, heads, n):
    """One key of the third and of the fourth tile is far above all others: the half of the row without it has to follow."""
    from zipage_b200.layers.attention import varlen_prefill_attention
    g = torch.Generator(device="cuda").manual_seed(key)
    q, k, v = (torch.randn(n, heads, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    q[..., 0], k[..., 0] = 24.0, 0.0
    k[256 + key, :, 0], k[384 + key, :, 0] = 24.0, 64.0   # 73 and 196 powers of two
    out = varlen_prefill_attention(q, k, v, n, _cu([n]), n, _cu([n]), impl="tcgen05")
    _no_device_error()
    seen = torch.arange(n, device="cuda")[None] <= torch.arange(n, device="cuda")[:, None]
    ref, mag = _softmax(q, k, v, D ** -0.5, seen)
    unit = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.1      # as in test_prefill_edges
    assert ((out.double() - ref).abs() <= (unit * 2 + CLIMB_ERROR) * mag + 1e-6).all()


@pytest.mark.parametrize("many", [False, True])          # launches of few and of many query tiles
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(8, 4, 128, 128), (6, 2, 48, 16), (3, 3, 72, 104)])
@pytest.mark.parametrize("softcap,steep,window", [(30.0, False, 300), (0.0, True, 0), (0.0, True, 300)])
@pytest.mark.parametrize("gated", ["entry", None])
def test_windows_of_views(many, heads, kv_heads, dim, vdim, softcap, steep, window, gated):
    """Columns of wider rows for queries, gates and results, a gate per entry, a factor, climbing scores, several items per block."""
    from zipage_b200.layers.attention import window_attention
    copies = 1 + 2000 // (10 * heads) if many else 1
    lens_q, lens_k = [1, 129, 400, 250] * copies, [513, 129, 700, 1000] * copies
    g = torch.Generator(device="cuda").manual_seed(heads + dim)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    rows, keys = sum(lens_q), sum(lens_k)
    q, k, v = n(rows, heads, dim), n(keys, kv_heads, dim), n(keys, kv_heads, vdim)
    if steep:
        _climb(q, k, lens_k, 5)
    wide, gate = n(rows, heads * dim + 24), n(rows, 8 + heads * vdim + 16)[:, 8:8 + heads * vdim]
    wide[:, 16:-8] = q.flatten(1)
    pad = lambda t: torch.nn.functional.pad(t, (0, -t.shape[2] % 16))
    need = [(m + 63) // 64 for m in lens_k]
    ids, table = torch.randperm(sum(need), device="cuda", generator=g).to(torch.int32), torch.full((len(need), max(need)), -1, dtype=torch.int32, device="cuda")
    for b, part in enumerate(ids.split(need)):
        table[b, :need[b]] = part
    results = torch.full((rows, heads * vdim + 16), 3.0, dtype=torch.bfloat16, device="cuda")
    window_attention(wide[:, 16:-8], _paged(pad(k), lens_k, 64, table), _paged(pad(v), lens_k, 64, table), torch.tensor(lens_k, dtype=torch.int32, device="cuda"),
                     table, heads, dim, vdim, dim ** -0.5, window, softcap, cu_seqlens_q=_cu(lens_q), max_seqlen_q=max(lens_q), out=results[:, 8:-8],
                     impl="tcgen05", gate=gate if gated else None, gate_mode=gated, out_scale=0.7)
    _no_device_error()
    assert (results[:, :8] == 3).all() and (results[:, -8:] == 3).all()
    for i in [*range(4), *range(len(lens_q) - 4, len(lens_q))]:
        x, y, a, b = lens_q[i], lens_k[i], sum(lens_q[:i]), sum(lens_k[:i])
        p, j = torch.arange(y - x, y, device="cuda")[:, None], torch.arange(y, device="cuda")[None]
        seen = (j <= p) & (p - j < window) if window else j <= p
        kk, vv = (t[b:b + y].double().repeat_interleave(heads // kv_heads, 1) for t in (k, v))
        s = torch.einsum("thd,shd->hts", q[a:a + x].double(), kk) * dim ** -0.5
        s = softcap * torch.tanh(s / softcap) if softcap else s
        w = torch.softmax(s.masked_fill(~seen[None], float("-inf")), -1) * 0.7
        f = torch.sigmoid(gate[a:a + x].double()).view(x, heads, vdim) if gated else 1.0
        ref, mag = torch.einsum("hts,shd->thd", w, vv) * f, torch.einsum("hts,shd->thd", w, vv.abs()) * f
        # as in test_window_edges
        assert ((results[a:a + x, 8:-8].view(x, heads, vdim).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (CLIMB_ERROR if steep else 1e-4) * mag + 1e-6).all()


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("dim,rot", [(128, 64), (64, 0)])
def test_latents_whose_reference_moves(many, dim, rot):
    from zipage_b200.layers.latent_attention import latent_prefill
    copies = 60 if many else 1
    heads, vdim, rank, lens_q, lens_k = 3, 128, 64, [1, 300, 513] * copies, [900, 301, 1300] * copies
    g = torch.Generator(device="cuda").manual_seed(dim + rot)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    rows, keys = sum(lens_q), sum(lens_k)
    q, k, v, lat = n(rows, heads, dim + rot), n(keys, heads, dim), n(keys, heads, vdim), n(keys, rank + rot)
    _climb(q, k, lens_k, 5)
    kv, out = torch.cat([k.flatten(1), v.flatten(1)], -1), torch.empty(rows, heads * vdim, dtype=torch.bfloat16, device="cuda")
    latent_prefill(q.flatten(1), kv, lat, _cu(lens_q), _cu(lens_k), max(lens_q), out, heads, dim, rot, vdim, rank, (dim + rot) ** -0.5)
    _no_device_error()
    for i in [*range(3), *range(len(lens_q) - 3, len(lens_q))]:
        x, y, a, b = lens_q[i], lens_k[i], sum(lens_q[:i]), sum(lens_k[:i])
        kk = torch.cat([k[b:b + y], lat[b:b + y, None, rank:].expand(-1, heads, -1)], -1)
        seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
        ref, mag = _softmax(q[a:a + x], kk, v[b:b + y], (dim + rot) ** -0.5, seen)
        assert ((out[a:a + x].view(x, heads, vdim).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + CLIMB_ERROR * mag + 1e-6).all()


def _kernels(call):
    """Names of the kernels that `call` launches, as they are in a graph captured from it (a profiler's recording comes back without some of them now
    and then)."""
    driver = pytest.importorskip("cuda.bindings.driver")
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()

    def done(answer):
        assert answer[0] == driver.CUresult.CUDA_SUCCESS, answer[0]
        return answer[1]
    handle = driver.CUgraph(graph.raw_cuda_graph())
    nodes = done(driver.cuGraphGetNodes(handle, driver.cuGraphGetNodes(handle)[2]))
    kernels = [n for n in nodes if done(driver.cuGraphNodeGetType(n)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]
    return " ".join(done(driver.cuFuncGetName(done(driver.cuGraphKernelNodeGetParams(n)).func)).decode() for n in kernels)


@pytest.mark.parametrize("rows,context,short", [(128, 512, True), (100, 400, True), (128, 500, False), (129, 2000, False), (128, 0, False)])
def test_latents_of_single_tiles(rows, context, short):
    """Portions of one tile behind a context of at least four times their length leave the pairs of the shared pipeline half empty."""
    from zipage_b200.layers.latent_attention import latent_prefill
    heads, B, dim, rot, vdim, rank = 8, 40, 64, 64, 128, 64
    lens_q, lens_k = [rows] * B, [rows + context] * B
    g = torch.Generator(device="cuda").manual_seed(rows)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    q, kv, lat = n(rows * B, heads * (dim + rot)), n((rows + context) * B, heads * (dim + vdim)), n((rows + context) * B, rank + rot)
    out, cq, ck = torch.empty(rows * B, heads * vdim, dtype=torch.bfloat16, device="cuda"), _cu(lens_q), _cu(lens_k)
    names = _kernels(lambda: latent_prefill(q, kv, lat, cq, ck, rows, out, heads, dim, rot, vdim, rank, D ** -0.5))
    _no_device_error()
    assert ("short" in names) == short
    for b in (0, B - 1):
        a, x, y = b * rows, rows, rows + context
        part = kv[b * y:b * y + y]
        k = torch.cat([part[:, :heads * dim].view(y, heads, dim), lat[b * y:b * y + y, None, rank:].expand(-1, heads, -1)], -1)
        seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
        ref, mag = _softmax(q[a:a + x].view(x, heads, D), k, part[:, heads * dim:].view(y, heads, vdim), D ** -0.5, seen)
        assert ((out[a:a + x].view(x, heads, vdim).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * mag + 1e-6).all()


def _plain_windows(heads, kv_heads, d, lens, context, window, softcap):
    """Windows over random portions behind `context` keys: the names of the kernels, and the check of the first and last portion."""
    from zipage_b200.layers.attention import window_attention
    lens_k = [n + context for n in lens]
    g = torch.Generator(device="cuda").manual_seed(len(lens) + d)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = n(sum(lens), heads, d), n(sum(lens_k), kv_heads, d), n(sum(lens_k), kv_heads, d)
    need = [(m + 63) // 64 for m in lens_k]
    table = torch.full((len(need), max(need)), -1, dtype=torch.int32, device="cuda")
    for b, part in enumerate(torch.arange(sum(need), dtype=torch.int32, device="cuda").split(need)):
        table[b, :need[b]] = part
    args = (q.flatten(1), _paged(k, lens_k, 64, table), _paged(v, lens_k, 64, table), torch.tensor(lens_k, dtype=torch.int32, device="cuda"), table, heads, d, d,
            d ** -0.5, window, softcap)
    cu = _cu(lens)
    out = window_attention(*args, cu_seqlens_q=cu, max_seqlen_q=max(lens))
    names = _kernels(lambda: window_attention(*args, cu_seqlens_q=cu, max_seqlen_q=max(lens)))
    _no_device_error()
    for i in (0, len(lens) - 1):
        x, y, a, b = lens[i], lens_k[i], sum(lens[:i]), sum(lens_k[:i])
        p, j = torch.arange(y - x, y, device="cuda")[:, None], torch.arange(y, device="cuda")[None]
        seen = (j <= p) & (p - j < window) if window else j <= p
        kk, vv = (t[b:b + y].double().repeat_interleave(heads // kv_heads, 1) for t in (k, v))
        s = torch.einsum("thd,shd->hts", q[a:a + x].double(), kk) * d ** -0.5
        s = softcap * torch.tanh(s / softcap) if softcap else s
        w = torch.softmax(s.masked_fill(~seen[None], float("-inf")), -1)
        ref, mag = torch.einsum("hts,shd->thd", w, vv), torch.einsum("hts,shd->thd", w, vv.abs())
        assert ((out[a:a + x].view(x, heads, d).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * mag + 1e-6).all()
    return "short" if "tc_short" in names else "pairs" if "attn_tc" in names else "mma" if "window_prefill_mma" in names else names


@pytest.mark.parametrize("heads,kv_heads,lens,context,window,softcap,kernel", [
    (32, 8, [128] * 13, 0, 0, 0.0, "short"), (32, 8, [128] * 14, 0, 0, 0.0, "pairs"),                  # 416 and 448 tiles
    (32, 8, [200] * 11, 1100, 0, 30.0, "short"), (32, 8, [200] * 12, 1100, 0, 30.0, "pairs"),          # 704 and 768, far, capped
    (32, 8, [200] * 11, 700, 0, 30.0, "pairs"), (32, 8, [200] * 11, 1100, 0, 0.0, "pairs"), (32, 8, [200] * 11, 1100, 512, 30.0, "short"),
    (8, 8, [128] * 60, 0, 0, 0.0, "pairs"), (8, 8, [128] * 60, 64, 0, 0.0, "short"), (8, 8, [128] * 60, 0, 100, 0.0, "short"),
])
def test_which_windows_go_in_pairs(heads, kv_heads, lens, context, window, softcap, kernel):
    assert _plain_windows(heads, kv_heads, 128, lens, context, window, softcap) == kernel


@pytest.mark.parametrize("lens,context,kernel", [
    ([96] + [64] * 30, 0, "mma"), ([300] + [40] * 30, 500, "mma"), ([96] + [80] * 30, 0, "pairs"), ([300] + [110] * 30, 0, "pairs"), ([96] + [64] * 3, 0, "short"),
    ([96] * 11, 0, "mma"), ([96] * 11, 600, "short"), ([96] * 28, 0, "pairs"), ([140] * 11, 0, "short"),
])
def test_which_windows_of_small_heads_take_tcgen05(lens, context, kernel):
    assert _plain_windows(16, 4, 64, lens, context, 0, 0.0) == kernel


@pytest.mark.parametrize("B", [4, 5])                    # 128 tiles, of an SM each; 160 in pairs of heads
def test_prompts_of_about_as_many_tiles_as_sms(B):
    from zipage_b200.layers.attention import varlen_prefill_attention
    heads, kv_heads, x, y = 32, 8, 33, 700
    g = torch.Generator(device="cuda").manual_seed(B)
    n = lambda rows, h: torch.randn(rows, h, D, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = n(x * B, heads), n(y * B, kv_heads), n(y * B, kv_heads)
    out = varlen_prefill_attention(q, k, v, x, _cu([x] * B), y, _cu([y] * B))
    _no_device_error()
    seen = torch.arange(y, device="cuda")[None] <= torch.arange(x, device="cuda")[:, None] + y - x
    for b in range(B):
        ref, mag = _softmax(q[b * x:b * x + x], k[b * y:b * y + y], v[b * y:b * y + y], D ** -0.5, seen)
        assert ((out[b * x:b * x + x].double() - ref).abs() <= 2.0 ** -8 * 1.1 * 2 * mag + 1e-6).all()      # as in test_prefill_edges


@pytest.mark.parametrize("B,kv_heads,dim", [(1, 8, 128), (18, 8, 128), (19, 8, 128), (27, 8, 128), (28, 8, 128), (56, 8, 128), (37, 8, 64), (20, 8, 96)])
@pytest.mark.parametrize("width,window,keep", [(24, 0, 0), (25, 0, 0), (40, 512, 0), (40, 512, 64)])
def test_decoded_windows_over_the_numbers_of_splits(B, kv_heads, dim, width, window, keep):
    """Sequences and keys in sight around which the splits of a sequence change, and the workspace with them."""
    from zipage_b200.layers.attention import window_attention
    heads, page = 2 * kv_heads, 64
    g = torch.Generator(device="cuda").manual_seed(B)
    lens = [1 + (b * 37) % (width * page) for b in range(B)]
    lens[0] = width * page
    pages = B * width
    table = torch.randperm(pages, device="cuda", generator=g).to(torch.int32).view(B, width)
    k, v = (torch.randn(pages, page, kv_heads, dim, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(B, heads * dim, device="cuda", generator=g).to(torch.bfloat16)
    out = torch.empty_like(q)
    window_attention(q, k, v, torch.tensor(lens, dtype=torch.int32, device="cuda"), table, heads, dim, dim, dim ** -0.5, window, 0.0, out=out, keep=keep)
    _no_device_error()
    for b in list(range(0, B, 9)) + [B - 1]:
        n = lens[b]
        j = torch.arange(n, device="cuda")
        seen = ((j > n - 1 - window) | (j < keep))[None] if window else torch.ones(1, n, dtype=torch.bool, device="cuda")
        kk, vv = (t[table[b, :(n + page - 1) // page].long()].flatten(0, 1)[:n] for t in (k, v))
        ref, mag = _softmax(q[b].view(1, heads, dim), kk, vv, dim ** -0.5, seen)
        # weights as two bf16 numbers (2^-16), the result rounded once
        assert ((out[b].view(1, heads, dim).double() - ref).abs() <= (2.0 ** -8 + 2.0 ** -14) * mag + 1e-6).all()
