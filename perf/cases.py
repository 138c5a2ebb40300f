"""The work whose time is measured: calls of the framework's public entry points as a serving program makes them.

A case is a dict of plain values; `kind` names the path:

  decode_step  one decode step of Qwen3 blocks as a replayed CUDA graph (`DecodeGraphRunner`)
  decode       attention of one decoding layer: bookkeeping, q/k norm + rotation + stores, paged attention
  prefill      attention of one layer over prompts: q/k norm + rotation + stores, varlen attention (over the pages with a
               cached prefix)
  compress     `Compressor.compress_tables`, host lists in and out
  row_ops      the launches between the matrix products of a block on a batch of prompt tokens
  sample       a step's tokens from its logits
  window       one layer's windowed attention in a portion step (decoded tokens beside portions of prompts)
  latent       one layer's latent attention in a portion step, without its matrix products
  experts      a mixture of gated experts and the layer boundary that joins it
  recurrent    one layer's delta rule or linear attention in a portion step, with its convolution and norm

Weights are random, token counts are spread over the stated range by the case alone, so that `work` knows them.
"""
from __future__ import annotations

import math
import random
from types import SimpleNamespace

import numpy as np
import torch

from zipage_b200.compress import CompressConfig
from zipage_b200.engine.compressor import Compressor
from zipage_b200.engine.decode_graph import DecodeGraphRunner
from zipage_b200.layers import attention as A
from zipage_b200.layers import feed_forward as F
from zipage_b200.layers import gated_delta as G
from zipage_b200.layers import latent_attention as LA
from zipage_b200.layers import linear_state as LS
from zipage_b200.layers import row_ops as R
from zipage_b200.layers import step_ops as P
from zipage_b200.layers.qwen3_block import Qwen3Model
from zipage_b200.layers.short_conv import short_conv

DEV = "cuda"
D = 128                 # head size of the compressed-cache path
PAGE = 256              # its page size; the portion-served models use pages of 64
PORTION_PAGE = 64
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
EPS = 1e-6
f64 = torch.float64


# -- the cases -----------------------------------------------------------------------------------------
def listed():
    heads = {"heads": 32, "kv_heads": 8}
    return [
        # a chat with few users: every launch of a step counts
        {"name": "decode_step_4", "kind": "decode_step", "seqs": 4, "layers": 4, "hidden": 1024, "heads": 16, "kv_heads": 8,
         "inter": 3072, "min_tokens": 700, "max_tokens": 2304},
        # a full server after compression: every sequence holds its budget of 8 pages and a part of the ninth
        {"name": "decode_192", "kind": "decode", "seqs": 192, **heads, "min_tokens": 2049, "max_tokens": 2304, "dtype": "bf16"},
        # prompts of a mixed load, some much shorter than others
        {"name": "prefill_ragged", "kind": "prefill", "prompts": 12, **heads, "min_tokens": 60, "max_tokens": 1500, "cached_pages": 0,
         "dtype": "bf16"},
        # one long document
        {"name": "prefill_16k", "kind": "prefill", "prompts": 1, **heads, "min_tokens": 16384, "max_tokens": 16384, "cached_pages": 0,
         "dtype": "bf16"},
        # the sequences that fill their ninth page in one step of a busy server
        {"name": "compress_lightning", "kind": "compress", "seqs": 32, "layers": 8, **heads, "min_pages": 9, "max_pages": 9, "window": 32,
         "redundancy": "lightning", "global_score": False, "dtype": "bf16"},
        # long prompts compressed for the first time, with the exact similarity and the global score
        {"name": "compress_exact_long", "kind": "compress", "seqs": 4, "layers": 8, **heads, "min_pages": 10, "max_pages": 28, "window": 32,
         "redundancy": "exact", "global_score": True, "dtype": "bf16"},
        # a prompt batch between the matrix products of a block of an 8B-class model
        {"name": "row_ops_8192", "kind": "row_ops", "tokens": 8192, "hidden": 4096, "inter": 12288, "dtype": "bf16"},
        # sampling for a full server
        {"name": "sample_256", "kind": "sample", "rows": 256, "vocab": 151936, "dtype": "bf16"},
        # sliding windows with a soft cap, decoded tokens beside portions of prompts
        {"name": "window_portions", "kind": "window", "decode": 32, "portions": 4, **heads, "dim": 128, "min_tokens": 500, "max_tokens": 3000,
         "context": 2200, "window": 1024, "softcap": 30.0, "biased": False},
        # latent attention, decoded tokens (direct form) beside portions (expanded form)
        {"name": "latent_portions", "kind": "latent", "decode": 48, "portions": 3, "heads": 32, "dim": 128, "rot": 64, "vdim": 128,
         "q_rank": 1536, "kv_rank": 512, "min_tokens": 600, "max_tokens": 3000, "context": 2200},
        # experts of a prompt batch
        {"name": "experts_4096", "kind": "experts", "tokens": 4096, "width": 2048, "experts": 64, "top": 6, "ff": 1024},
        # recurrent heads, decoded tokens beside portions
        {"name": "delta_portions", "kind": "recurrent", "rule": "delta", "decode": 32, "portions": 4, "heads": 32, "kv_heads": 16, "dim": 128,
         "vdim": 128, "min_tokens": 300, "max_tokens": 2500},
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    pick = rng.choice
    span = lambda hi: {"min_tokens": max(1, int(hi * rng.uniform(0.05, 1.0))), "max_tokens": hi}
    dtype = {"dtype": pick(["bf16", "bf16", "fp16"])}
    heads = pick([{"heads": 32, "kv_heads": 8}, {"heads": 16, "kv_heads": 8}, {"heads": 8, "kv_heads": 1}, {"heads": 64, "kv_heads": 8}])
    kind = pick(["decode_step", "decode", "prefill", "prefill", "compress", "compress", "row_ops", "sample", "window", "latent", "experts",
                 "recurrent"])
    if kind == "decode_step":
        return {"kind": kind, "seqs": log(1, 32), "layers": rng.randint(2, 4), "hidden": 1024, "heads": 16, "kv_heads": 8, "inter": 3072,
                **span(log(64, 2304))}
    if kind == "decode":
        return {"kind": kind, "seqs": log(1, 192), **heads, **span(log(16, 2304)), **dtype}
    if kind == "prefill":
        n = log(1, 16)
        return {"kind": kind, "prompts": n, **heads, **span(log(32, min(12000, 32000 // n))), "cached_pages": pick([0, 0, 0, 1, 4]), **dtype}
    if kind == "compress":
        h = pick([{"heads": 32, "kv_heads": 8}, {"heads": 16, "kv_heads": 8}, {"heads": 8, "kv_heads": 1}])
        most = rng.randint(9, 28)
        return {"kind": kind, "seqs": log(1, 288 // most), "layers": pick([1, 2, 4, 8]), **h, "min_pages": rng.randint(9, most), "max_pages": most,
                "window": 16 if h["kv_heads"] == 1 else pick([16, 32]), "redundancy": pick(["none", "lightning", "lightning", "exact"]),
                "global_score": pick([False, False, True]), **dtype}
    if kind == "row_ops":
        hidden, inter = pick([(1024, 3072), (2048, 6144), (2560, 9728), (4096, 12288)])
        return {"kind": kind, "tokens": log(1, 8192), "hidden": hidden, "inter": inter, **dtype}
    if kind == "sample":
        return {"kind": kind, "rows": log(1, 256), "vocab": pick([32000, 32768, 50257, 151936]), **dtype}
    if kind == "window":
        h = pick([{"heads": 32, "kv_heads": 8}, {"heads": 16, "kv_heads": 8}, {"heads": 16, "kv_heads": 4}])
        biased = pick([False, False, True])
        return {"kind": kind, "decode": rng.randint(0, 48), "portions": rng.randint(1, 6), **h, "dim": pick([64, 96, 128, 128]), **span(log(40, 3000)),
                "context": log(50, 2300), "window": pick([0, 512, 1024]), "softcap": 0.0 if biased else pick([0.0, 30.0, 50.0]), "biased": biased}
    if kind == "latent":
        return {"kind": kind, "decode": rng.randint(1, 64), "portions": rng.randint(1, 4), "heads": pick([16, 32]), "dim": 128, "rot": 64, "vdim": 128,
                "q_rank": 1536, "kv_rank": 512, **span(log(64, 3000)), "context": log(50, 2300)}
    if kind == "experts":
        return {"kind": kind, "tokens": log(1, 4096), "width": pick([1024, 2048]), "experts": pick([32, 64]), "top": pick([2, 4, 6]),
                "ff": pick([512, 768, 1024])}
    rule = pick(["delta", "forget", "power", "scalar"])
    h = {"delta": (32, 16, 128, 128), "scalar": (32, 2, 128, 128)}.get(rule, (16, 16, 128, 256))
    return {"kind": kind, "rule": rule, "decode": rng.randint(0, 48), "portions": rng.randint(1, 6), "heads": h[0], "kv_heads": h[1], "dim": h[2],
            "vdim": h[3], **span(log(64, 2500))}


# -- shared parts --------------------------------------------------------------------------------------
def lengths(n, lo, hi):
    """n whole numbers spread over lo .. hi, the largest among them."""
    r = random.Random(1000003 * n + 1009 * lo + hi)
    return [hi] + [r.randint(lo, hi) for _ in range(n - 1)] if n else []


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


class Draws:
    """Seeded tensors on the GPU, and page tables."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, dtype=torch.bfloat16, std=1.0):
        return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=self.gen)

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.gen, device=DEV)

    def tables(self, pages):
        """Scattered pages: -> (total, table [B, widest] int32 with -1 padding)."""
        total = sum(pages)
        ids = torch.randperm(total, generator=self.gen, device=DEV).to(torch.int32)
        table = torch.full((len(pages), max(pages)), -1, dtype=torch.int32, device=DEV)
        at = 0
        for b, n in enumerate(pages):
            table[b, :n] = ids[at:at + n]
            at += n
        return total, table


def pages_of(tokens, page):
    return [(n + page - 1) // page for n in tokens]


def slots_of(table, first, count, page):
    """Cache slots of the positions first .. first + count - 1 of each sequence, one after the other."""
    out = []
    for b, (f, n) in enumerate(zip(first, count)):
        p = torch.arange(f, f + n, device=DEV)
        out.append(table[b, p // page].long() * page + p % page)
    return torch.cat(out).to(torch.int32)


def positions_of(first, count):
    return torch.cat([torch.arange(f, f + n, device=DEV) for f, n in zip(first, count)])


def running(counts):
    return i32([0] + np.cumsum(counts).tolist())


def pairs_of(first, count, window=0):
    """Visible (query, key) pairs of causal attention, with a window where there is one."""
    total = 0
    for f, n in zip(first, count):
        p = np.arange(f, f + n) + 1
        total += int(np.minimum(p, window).sum() if window else p.sum())
    return total


def paged_rows(cache, table, b, n):
    """The first n rows of sequence b of a paged cache in 64 bits."""
    page = cache.shape[1]
    ids = table[b, :(n + page - 1) // page].long()
    return cache[ids].flatten(0, 1)[:n].to(f64)


def rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def softmax_attention(q, k, v, scale, first, window=0, softcap=0.0, keep=0, slopes=None):
    """q [n, H, d] at positions first .. over k, v [m, G, d] in 64 bits, one head at a time."""
    n, H, m, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=f64, device=DEV)
    p, j = torch.arange(first, first + n, device=DEV)[:, None], torch.arange(m, device=DEV)[None]
    seen = j <= p
    if window:
        seen &= (p - j < window) | (j < keep)
    for h in range(H):
        g = h * G // H
        s = q[:, h] @ k[:, g].T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if slopes is not None:
            s = s - slopes[h].to(f64) * (p - j)
        out[:, h] = torch.softmax(s.masked_fill(~seen, -math.inf), dim=-1) @ v[:, g]
    return out


def rope_half(x, cos_sin):
    """x [n, H, d] with the pairs (t, t + d / 2) turned by a row of [cos | sin] each."""
    c, s = cos_sin.to(f64)[:, None].chunk(2, dim=-1)
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def qk_exact(rows, qkv, heads, kv_heads, cos_sin, wq, wk):
    q, k, v = qkv.to(f64).view(qkv.shape[0], -1, D).split([heads, kv_heads, kv_heads], dim=1)
    cs = cos_sin[rows]
    return rope_half(rms(q, EPS) * wq.to(f64), cs), rope_half(rms(k, EPS) * wk.to(f64), cs), v


# -- decode step of whole blocks -----------------------------------------------------------------------
WINDOW = 32             # observation window of the compressed-cache path


class DecodeStep:
    @staticmethod
    def inputs(c, seed):
        d = Draws(seed)
        n = lengths(c["seqs"], c["min_tokens"], c["max_tokens"])
        total, table = d.tables(pages_of(n, PAGE))
        H, kv, hid, inter = c["heads"], c["kv_heads"], c["hidden"], c["inter"]
        shapes = {"self_attn.qkv_proj": ((H + 2 * kv) * D, hid), "self_attn.o_proj": (hid, H * D), "mlp.gate_up_proj": (2 * inter, hid),
                  "mlp.down_proj": (hid, inter)}
        w = {f"layers.{i}.{k}.weight": d.normal(*s, std=s[1] ** -0.5) for i in range(c["layers"]) for k, s in shapes.items()}
        w["embed_tokens.weight"] = d.normal(4096, hid)
        return dict(w=w, num_tokens=i32(n), table=table, ids=torch.randint(0, 4096, (c["seqs"],), generator=d.gen, device=DEV),
                    query_ids=i32(list(range(c["seqs"]))), kv=d.normal(2, c["layers"], total, PAGE, kv, D),
                    query=torch.zeros(c["layers"], c["seqs"], WINDOW, H, D, dtype=torch.bfloat16, device=DEV))

    @classmethod
    def prepare(cls, c, seed):
        t = cls.inputs(c, seed)
        cfg = SimpleNamespace(hidden_size=c["hidden"], num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"], head_dim=D,
                              max_position_embeddings=4096, rms_norm_eps=EPS, rope_theta=1e6, intermediate_size=c["inter"], hidden_act="silu",
                              num_hidden_layers=c["layers"], vocab_size=4096)
        before = torch.get_default_dtype()
        torch.set_default_dtype(torch.bfloat16)
        try:
            with torch.device(DEV):
                model = Qwen3Model(cfg).eval()
        finally:
            torch.set_default_dtype(before)
        model.load_state_dict(t.pop("w"), strict=False)      # (norm weights are ones)
        model.bind_caches(t["kv"], t["query"])
        t["runner"] = DecodeGraphRunner(model, c["hidden"], max_bs=c["seqs"], max_num_blocks=t["table"].shape[1], query_cache_len=WINDOW,
                                        graph_bs=[c["seqs"]])
        t["runner"].capture()
        return t

    @staticmethod
    def run(s):
        return s["runner"].run(s["ids"], s["num_tokens"], s["table"], s["query_ids"]), s["kv"], s["query"]

    @classmethod
    def exact(cls, c, seed):
        t = cls.inputs(c, seed)
        n = t["num_tokens"].tolist()
        pos = [x - 1 for x in n]
        cs = cos_sin_table(max(n))[pos]
        w, kv, query = {k: v.to(f64) for k, v in t["w"].items()}, t["kv"].to(f64), t["query"].to(f64)
        one = torch.ones((), dtype=f64, device=DEV)
        slot = slots_of(t["table"], pos, [1] * len(n), PAGE).long()
        x, H, G = w["embed_tokens.weight"][t["ids"]], c["heads"], c["kv_heads"]
        for i in range(c["layers"]):
            p = f"layers.{i}."
            q, k, v = qk_exact(slice(None), rms(x, EPS) @ w[p + "self_attn.qkv_proj.weight"].T, H, G, cs, one, one)
            kv[0, i].view(-1, G, D)[slot], kv[1, i].view(-1, G, D)[slot] = k, v
            store_window(query[i], q, n)
            o = torch.cat([softmax_attention(q[b:b + 1], paged_rows(kv[0, i], t["table"], b, m), paged_rows(kv[1, i], t["table"], b, m), D ** -0.5, m - 1)
                           for b, m in enumerate(n)])
            x = x + o.flatten(1) @ w[p + "self_attn.o_proj.weight"].T
            g, u = (rms(x, EPS) @ w[p + "mlp.gate_up_proj.weight"].T).chunk(2, dim=-1)
            x = x + (torch.nn.functional.silu(g) * u) @ w[p + "mlp.down_proj.weight"].T
        return rms(x, EPS), kv, query

    @staticmethod
    def work(c):
        n, H, G, hid = lengths(c["seqs"], c["min_tokens"], c["max_tokens"]), c["heads"], c["kv_heads"], c["hidden"]
        weights = (2 * H + 2 * G) * D * hid + 3 * c["inter"] * hid
        return {"bytes": c["layers"] * (2.0 * weights + sum(n) * G * D * 4.0) + 4.0 * c["seqs"] * hid,
                "flops": c["layers"] * (2.0 * c["seqs"] * weights + 4.0 * D * H * sum(n))}

    @staticmethod
    def tolerance(c):
        return {"rel": 2.5e-2, "max": 0.3}   # bf16 activations through up to four blocks


def cos_sin_table(n):
    """cos | sin of the angles of positions below n, base 1e6, as the fp32 table of the layers holds them."""
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, dtype=torch.float) / D))
    f = torch.einsum("i,j -> ij", torch.arange(n, dtype=torch.float), inv)
    return torch.cat((f.cos(), f.sin()), dim=-1).to(DEV)


def store_window(cache, q, n):
    """Queries whose position lies among the last WINDOW slots of a page go to the window buffer."""
    for b, m in enumerate(n):
        at = (m - 1) % PAGE - (PAGE - WINDOW)
        if at >= 0:
            cache[b, at] = q[b]


# -- attention of one decoding layer -------------------------------------------------------------------
class Decode:
    @staticmethod
    def prepare(c, seed):
        d, dt = Draws(seed), DTYPES[c["dtype"]]
        n = lengths(c["seqs"], c["min_tokens"], c["max_tokens"])
        total, table = d.tables(pages_of(n, PAGE))
        H, G = c["heads"], c["kv_heads"]
        return dict(H=H, G=G, table=table, num_tokens=i32(n), query_ids=i32(list(range(c["seqs"]))), cos_sin=cos_sin_table(max(n)),
                    qkv=d.normal(c["seqs"], (H + 2 * G) * D, dtype=dt), wq=(1 + d.normal(D, std=0.1)).to(dt), wk=(1 + d.normal(D, std=0.1)).to(dt),
                    k=d.normal(total, PAGE, G, D, dtype=dt), v=d.normal(total, PAGE, G, D, dtype=dt),
                    query=torch.zeros(c["seqs"], WINDOW, H, D, dtype=dt, device=DEV))

    @staticmethod
    def run(s):
        pos, ctx, slot, triples, count = P.prepare_decode(s["num_tokens"], s["table"], s["query_ids"], WINDOW, PAGE)
        q, _, _ = P.qk_norm_rope_store(s["qkv"], pos, s["cos_sin"], s["wq"], s["wk"], EPS, s["H"], s["G"], D, s["k"], s["v"], slot, s["query"], triples,
                                       return_k=False, query_slot_count=count)
        return A.paged_decode_attention(q.unsqueeze(1), s["k"], s["v"], ctx, s["table"]), s["k"], s["v"], s["query"]

    @classmethod
    def exact(cls, c, seed):
        s = cls.prepare(c, seed)
        n = s["num_tokens"].tolist()
        pos = [x - 1 for x in n]
        q, k, v = qk_exact(pos, s["qkv"], s["H"], s["G"], s["cos_sin"], s["wq"], s["wk"])
        slot = slots_of(s["table"], pos, [1] * len(n), PAGE).long()
        kc, vc, query = s["k"].to(f64), s["v"].to(f64), s["query"].to(f64)
        kc.view(-1, s["G"], D)[slot], vc.view(-1, s["G"], D)[slot] = k, v
        store_window(query, q, n)
        o = [softmax_attention(q[b:b + 1], paged_rows(kc, s["table"], b, m), paged_rows(vc, s["table"], b, m), D ** -0.5, m - 1) for b, m in enumerate(n)]
        return torch.stack(o), kc, vc, query

    @staticmethod
    def work(c):
        n, H, G = lengths(c["seqs"], c["min_tokens"], c["max_tokens"]), c["heads"], c["kv_heads"]
        return {"bytes": 4.0 * D * G * sum(n) + 2.0 * D * c["seqs"] * (2 * H + 4 * G), "flops": 4.0 * D * H * sum(n)}

    @staticmethod
    def tolerance(c):
        return {"rel": 1e-2 if c["dtype"] == "bf16" else 2e-3, "max": 0.1}


# -- attention of one layer over prompts ---------------------------------------------------------------
class Prefill:
    @staticmethod
    def prepare(c, seed):
        d, dt = Draws(seed), DTYPES[c["dtype"]]
        n = lengths(c["prompts"], c["min_tokens"], c["max_tokens"])
        first = [c["cached_pages"] * PAGE] * len(n)
        ends = [f + m for f, m in zip(first, n)]
        total, table = d.tables(pages_of(ends, PAGE))
        H, G = c["heads"], c["kv_heads"]
        # window queries: those of each prompt's tokens in the last WINDOW slots of a page it fills
        at = np.cumsum([0] + n)
        triples = [(int(at[b]) + p - first[b], b, p % PAGE - (PAGE - WINDOW)) for b in range(len(n))
                   for p in range(max(first[b], ends[b] // PAGE * PAGE - WINDOW), ends[b] // PAGE * PAGE)]
        return dict(H=H, G=G, n=n, first=first, most=max(n), most_k=max(ends), paged=c["cached_pages"] > 0, table=table, cos_sin=cos_sin_table(max(ends)),
                    cu=running(n), cu_k=running(ends), positions=positions_of(first, n), slot=slots_of(table, first, n, PAGE),
                    triples=i32(triples) if triples else None, qkv=d.normal(sum(n), (H + 2 * G) * D, dtype=dt),
                    wq=(1 + d.normal(D, std=0.1)).to(dt), wk=(1 + d.normal(D, std=0.1)).to(dt), k=d.normal(total, PAGE, G, D, dtype=dt),
                    v=d.normal(total, PAGE, G, D, dtype=dt), query=torch.zeros(len(n), WINDOW, H, D, dtype=dt, device=DEV))

    @staticmethod
    def run(s):
        q, k, v = P.qk_norm_rope_store(s["qkv"], s["positions"], s["cos_sin"], s["wq"], s["wk"], EPS, s["H"], s["G"], D, s["k"], s["v"], s["slot"],
                                       s["query"] if s["triples"] is not None else None, s["triples"], return_k=not s["paged"])
        if s["paged"]:
            o = A.varlen_prefill_attention(q, s["k"], s["v"], s["most"], s["cu"], s["most_k"], s["cu_k"], block_table=s["table"])
        else:
            o = A.varlen_prefill_attention(q, k, v.contiguous(), s["most"], s["cu"], s["most_k"], s["cu_k"])
        return o, s["k"], s["v"], s["query"]

    @classmethod
    def exact(cls, c, seed):
        s = cls.prepare(c, seed)
        q, k, v = qk_exact(s["positions"], s["qkv"], s["H"], s["G"], s["cos_sin"], s["wq"], s["wk"])
        kc, vc, query = s["k"].to(f64), s["v"].to(f64), s["query"].to(f64)
        slot = s["slot"].long()
        kc.view(-1, s["G"], D)[slot], vc.view(-1, s["G"], D)[slot] = k, v
        if s["triples"] is not None:
            r, b, w = s["triples"].long().T
            query[b, w] = q[r]
        out, at = [], 0
        for b, (f, n) in enumerate(zip(s["first"], s["n"])):
            out.append(softmax_attention(q[at:at + n], paged_rows(kc, s["table"], b, f + n), paged_rows(vc, s["table"], b, f + n), D ** -0.5, f))
            at += n
        return torch.cat(out), kc, vc, query

    @staticmethod
    def work(c):
        n, H, G, f = lengths(c["prompts"], c["min_tokens"], c["max_tokens"]), c["heads"], c["kv_heads"], c["cached_pages"] * PAGE
        return {"bytes": 2.0 * D * (sum(n) * (2 * H + 4 * G) + 2 * G * f * len(n)), "flops": 4.0 * D * H * pairs_of([f] * len(n), n)}

    @staticmethod
    def tolerance(c):
        return {"rel": 1e-2 if c["dtype"] == "bf16" else 2e-3, "max": 0.15}


# -- compression ---------------------------------------------------------------------------------------
BUDGET = 8


class Compress:
    @staticmethod
    def prepare(c, seed):
        d, dt = Draws(seed), DTYPES[c["dtype"]]
        pages = lengths(c["seqs"], c["min_pages"], c["max_pages"])
        total, table = d.tables(pages)
        tables = [row[:n] for row, n in zip(table.tolist(), pages)]
        L, H, G = c["layers"], c["heads"], c["kv_heads"]
        cfg = CompressConfig(budget_blocks=BUDGET, query_cache_len=c["window"], use_global_score=c["global_score"], use_redudancy=c["redundancy"] != "none",
                             lightning_redudancy=c["redundancy"] == "lightning", redudancy_lambda=0.5, enable_pooling=True, pooling_size=7)
        kv = torch.empty((2, L, total, PAGE, G, D), dtype=dt, device=DEV)
        for t in kv.flatten(0, 1):
            t.normal_(generator=d.gen)
        scores = (d.uniform(L, total, PAGE, G) / (max(pages) * PAGE)).to(dt) if c["global_score"] else None
        return dict(kv=kv, scores=scores, tables=tables, targets=[t[:BUDGET + 1] for t in tables], query_ids=list(range(len(pages))),
                    compressed=[n == BUDGET + 1 for n in pages],
                    op=Compressor(kv, d.normal(L, len(pages), c["window"], H, D, dtype=dt), scores, cfg))

    @staticmethod
    def run(s):
        tables, ctx = s["op"].compress_tables(s["tables"], s["targets"], s["query_ids"], s["compressed"])
        return s["kv"], s["scores"], np.asarray(tables), np.asarray(ctx)

    @staticmethod
    def exact(c, seed):
        return None                          # bytes are moved; which ones is decided by scores of 16 bits

    @staticmethod
    def work(c):
        pages, G, H = lengths(c["seqs"], c["min_pages"], c["max_pages"]), c["kv_heads"], c["heads"]
        units = [c["layers"] * G * n * PAGE for n in pages]          # keys
        kept = c["layers"] * G * BUDGET * PAGE * len(pages)
        pair = {"none": 0.0, "lightning": float(PAGE), "exact": None}[c["redundancy"]]
        similar = sum(2.0 * D * u * (n * PAGE if pair is None else pair) / 2 for u, n in zip(units, pages))
        return {"bytes": sum(units) * D * 2.0 + 2 * kept * D * 2.0 * 2 + c["layers"] * len(pages) * c["window"] * H * D * 2.0,
                "flops": sum(units) * 2.0 * D * c["window"] * H / G + similar}

    @staticmethod
    def tolerance(c):
        return "exact"                       # one key kept instead of another would move all rows behind it


# -- row ops -------------------------------------------------------------------------------------------
class RowOps:
    @staticmethod
    def prepare(c, seed):
        d, dt = Draws(seed), DTYPES[c["dtype"]]
        N, W = c["tokens"], c["hidden"]
        return dict(x=d.normal(N, W, dtype=dt), residual=d.normal(N, W, dtype=dt, std=2.0), w1=(1 + d.normal(W, std=0.1)).to(dt), y=d.normal(N, W, dtype=dt),
                    w2=(1 + d.normal(W, std=0.1)).to(dt), gate_up=d.normal(N, 2 * c["inter"], dtype=dt))

    @staticmethod
    def run(s):
        a, res = P.rms_norm(s["x"], s["w1"], EPS, s["residual"])         # (what attention and the block before left)
        b, res2 = P.rms_norm(s["y"], s["w2"], EPS, res)
        return a, b, res2, P.silu_and_mul(s["gate_up"])

    @classmethod
    def exact(cls, c, seed):
        s = {k: t.to(f64) for k, t in cls.prepare(c, seed).items()}
        r1 = s["x"] + s["residual"]
        r2 = r1 + s["y"]
        g, u = s["gate_up"].chunk(2, dim=-1)
        return rms(r1, EPS) * s["w1"], rms(r2, EPS) * s["w2"], r2, torch.nn.functional.silu(g) * u

    @staticmethod
    def work(c):
        N = float(c["tokens"])
        return {"bytes": 2.0 * N * (8 * c["hidden"] + 3 * c["inter"]), "flops": N * (16.0 * c["hidden"] + 8 * c["inter"])}

    @staticmethod
    def tolerance(c):
        return {"rel": 1e-2 if c["dtype"] == "bf16" else 1.5e-3, "max": 0.05}


# -- sampling ------------------------------------------------------------------------------------------
class Sample:
    @staticmethod
    def prepare(c, seed):
        d = Draws(seed)
        # logits of a language model: most tokens far below a few likely ones
        z = d.normal(c["rows"], c["vocab"], dtype=torch.float32, std=2.0)
        z.scatter_add_(1, torch.randint(0, c["vocab"], (c["rows"], 40), generator=d.gen, device=DEV), 8 + d.normal(c["rows"], 40, dtype=torch.float32, std=3.0))
        return dict(logits=z.to(DTYPES[c["dtype"]]), temperatures=0.6 + 0.4 * d.uniform(c["rows"]), seed=seed)

    @staticmethod
    def run(s):
        return P.sample(s["logits"], s["temperatures"], seed=s["seed"])

    @staticmethod
    def exact(c, seed):
        return None                          # tokens

    @staticmethod
    def work(c):
        n = float(c["rows"]) * c["vocab"]
        return {"bytes": 2.0 * n, "flops": 20.0 * n}

    @staticmethod
    def tolerance(c):
        return "exact"


# -- windowed attention in a portion step --------------------------------------------------------------
KEEP = 64


class Window:
    @staticmethod
    def shape(c):
        """-> (first position, count) of every sequence's rows: decoded tokens first, then portions; every other portion continues a prompt."""
        done = lengths(c["decode"], max(1, c["context"] // 2), c["context"])
        new = lengths(c["portions"], c["min_tokens"], c["max_tokens"])
        return [n - 1 for n in done] + [(b % 2) * min(c["context"], 1000) for b in range(len(new))], [1] * len(done) + new

    @classmethod
    def prepare(cls, c, seed):
        d = Draws(seed)
        first, count = cls.shape(c)
        ends = [f + n for f, n in zip(first, count)]
        total, table = d.tables(pages_of(ends, PORTION_PAGE))
        H, G, n = c["heads"], c["kv_heads"], c["dim"]
        z = lambda: d.normal(total, PORTION_PAGE, G, n)
        return dict(c=c, x=d.normal(sum(count), (H + 2 * G) * n), k=z(), v=z(), slot=slots_of(table, first, count, PORTION_PAGE), cu=running(count),
                    ctx=i32(ends), table=table, most=max(count), first=first, count=count,
                    slopes=torch.tensor(A.distance_slopes(H), device=DEV) if c["biased"] else None)

    @staticmethod
    def run(s):
        c = s["c"]
        H, G, n, nd = c["heads"], c["kv_heads"], c["dim"], c["decode"]
        q, k, v = s["x"].split([H * n, G * n, G * n], dim=1)
        A.store_kv_padded(k, v, s["k"], s["v"], s["slot"], n, n)
        out = torch.empty_like(q, memory_format=torch.contiguous_format)
        shape = (H, n, n, n ** -0.5, c["window"], c["softcap"])
        kw = dict(out=out, keep=KEEP if c["biased"] else 0, slopes=s["slopes"])
        if nd:
            A.window_attention(q, s["k"], s["v"], s["ctx"][:nd], s["table"][:nd], *shape, **kw)
        A.window_attention(q, s["k"], s["v"], s["ctx"][nd:], s["table"][nd:], *shape, cu_seqlens_q=s["cu"][nd:], max_seqlen_q=s["most"], **kw)
        return out, s["k"], s["v"]

    @classmethod
    def exact(cls, c, seed):
        s = cls.prepare(c, seed)
        H, G, n = c["heads"], c["kv_heads"], c["dim"]
        q, k, v = (t.to(f64).unflatten(1, (-1, n)) for t in s["x"].split([H * n, G * n, G * n], dim=1))
        kc, vc = s["k"].to(f64), s["v"].to(f64)
        slot = s["slot"].long()
        kc.view(-1, G, n)[slot], vc.view(-1, G, n)[slot] = k, v
        out, at = [], 0
        for b, (f, m) in enumerate(zip(s["first"], s["count"])):
            out.append(softmax_attention(q[at:at + m], paged_rows(kc, s["table"], b, f + m), paged_rows(vc, s["table"], b, f + m), n ** -0.5, f, c["window"],
                                         c["softcap"], KEEP if c["biased"] else 0, s["slopes"]))
            at += m
        return torch.cat(out).flatten(1), kc, vc

    @classmethod
    def work(cls, c):
        first, count = cls.shape(c)
        H, G, n, rows = c["heads"], c["kv_heads"], c["dim"], sum(count)
        reach = lambda f, m: f + m if not c["window"] else min(f + m, c["window"] + m - 1 + (KEEP if c["biased"] else 0))
        return {"bytes": 2.0 * n * (rows * (2 * H + 4 * G) + 2 * G * sum(reach(f, m) - m for f, m in zip(first, count))),
                "flops": 4.0 * n * H * pairs_of(first, count, c["window"])}

    @staticmethod
    def tolerance(c):
        return {"rel": 7e-3, "max": 0.1}


# -- latent attention in a portion step ----------------------------------------------------------------
class Latent:
    shape = staticmethod(Window.shape)

    @classmethod
    def prepare(cls, c, seed):
        d = Draws(seed)
        first, count = cls.shape(c)
        ends = [f + n for f, n in zip(first, count)]
        total, table = d.tables(pages_of(ends, PORTION_PAGE))
        H, QR, KR, nd, rows = c["heads"], c["q_rank"], c["kv_rank"], c["decode"], sum(count)
        KP, keys = KR + c["rot"], sum(ends[nd:])
        return dict(c=c, y=d.normal(rows, QR + KP), positions=positions_of(first, count), turns=LA.rotary_turns(c["rot"], 1e6, DEV),
                    wq=1 + d.normal(QR, dtype=torch.float32, std=0.1), wk=1 + d.normal(KR, dtype=torch.float32, std=0.1),
                    cache=d.normal(total, PORTION_PAGE, 1, KP), slot=slots_of(table, first, count, PORTION_PAGE), ctx=i32(ends), table=table,
                    cu=running(count[nd:]), cu_k=running(ends[nd:]), keys=keys, most=max(count), first=first, count=count,
                    # what the matrix products around these launches leave: queries, the decoded tokens' key-side queries, expanded keys and values
                    q=d.normal(rows, H * (c["dim"] + c["rot"])), q_lat=d.normal(nd, H, KP, std=0.3), kv=d.normal(keys, H * (c["dim"] + c["vdim"])))

    @staticmethod
    def run(s):
        c = s["c"]
        H, dim, rot, vdim, KR, nd = c["heads"], c["dim"], c["rot"], c["vdim"], c["kv_rank"], c["decode"]
        scale, pos = (dim + rot) ** -0.5, s["positions"]
        cq = LA.latent_prepare(s["y"], pos, s["turns"], s["wq"], s["wk"], s["cache"], s["slot"], c["q_rank"], KR, rot, 1e-5)
        LA.latent_rotate_q(s["q"][:nd], pos[:nd], s["turns"], H, dim, rot, s["q_lat"], KR)
        low = LA.latent_attention(s["q_lat"], s["cache"], s["ctx"][:nd], s["table"][:nd], KR, scale)
        rows = LA.gather_rows(s["cache"], s["table"][nd:], s["cu_k"], s["keys"])
        q = s["q"][nd:].clone()              # (the rotation is in place and a pass can be repeated)
        LA.latent_rotate_q(q, pos[nd:], s["turns"], H, dim, rot)
        out = torch.empty(q.shape[0], H * vdim, dtype=q.dtype, device=q.device)
        LA.latent_prefill(q, s["kv"], rows, s["cu"], s["cu_k"], s["most"], out, H, dim, rot, vdim, KR, scale)
        return cq, low, out, rows, s["cache"]

    @classmethod
    def exact(cls, c, seed):
        s = cls.prepare(c, seed)
        H, dim, rot, vdim, QR, KR, nd = c["heads"], c["dim"], c["rot"], c["vdim"], c["q_rank"], c["kv_rank"], c["decode"]
        angle = s["positions"].to(f64)[:, None] * (s["turns"] * 2 * math.pi)

        def turned(x):                       # [rows, heads, rot], pairs (2t, 2t + 1)
            a, b = x[..., 0::2], x[..., 1::2]
            co, si = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
            return torch.stack([a * co - b * si, b * co + a * si], dim=-1).flatten(-2)

        y = s["y"].to(f64)
        cache = s["cache"].to(f64)
        cache.view(-1, KR + rot)[s["slot"].long()] = torch.cat([rms(y[:, QR:QR + KR], 1e-5) * s["wk"].to(f64), turned(y[:, None, QR + KR:])[:, 0]], dim=1)
        q = s["q"].to(f64).view(-1, H, dim + rot)
        q = torch.cat([q[..., :dim], turned(q[..., dim:])], dim=-1)
        scale, low, out, rows, at, at_k = (dim + rot) ** -0.5, [], [], [], nd, 0
        for b, (f, n) in enumerate(zip(s["first"], s["count"])):
            lat = paged_rows(cache, s["table"], b, f + n)
            if b < nd:
                ql = torch.cat([s["q_lat"][b:b + 1, :, :KR].to(f64), q[b:b + 1, :, dim:]], dim=-1)
                low.append(softmax_attention(ql, lat, lat[..., :KR], scale, f))
                continue
            kv = s["kv"][at_k:at_k + f + n].to(f64)
            k = torch.cat([kv[:, :H * dim].unflatten(1, (H, dim)), lat[:, :, KR:].expand(-1, H, -1)], dim=-1)
            out.append(softmax_attention(q[at:at + n], k, kv[:, H * dim:].unflatten(1, (H, vdim)), scale, f).flatten(1))
            rows.append(lat[:, 0])
            at, at_k = at + n, at_k + f + n
        return rms(y[:, :QR], 1e-5) * s["wq"].to(f64), torch.cat(low), torch.cat(out), torch.cat(rows), cache

    @classmethod
    def work(cls, c):
        first, count = cls.shape(c)
        H, dim, rot, vdim, QR, KR, nd = c["heads"], c["dim"], c["rot"], c["vdim"], c["q_rank"], c["kv_rank"], c["decode"]
        KP, rows, keys = KR + rot, sum(count[nd:]), sum(f + n for f, n in zip(first[nd:], count[nd:]))
        done = sum(f + 1 for f in first[:nd])
        return {"bytes": 2.0 * (2 * (rows + nd) * (QR + KP) + done * KP + nd * H * (KP + KR) + 2 * keys * KP + rows * H * (dim + rot + vdim)
                                + keys * H * (dim + vdim)),
                "flops": 2.0 * H * (done * (KP + KR) + pairs_of(first[nd:], count[nd:]) * (dim + rot + vdim))}

    @staticmethod
    def tolerance(c):
        return {"rel": 8e-3, "max": 0.1}


# -- experts -------------------------------------------------------------------------------------------
class Experts:
    @staticmethod
    def prepare(c, seed):
        d, f = Draws(seed), torch.float32
        N, W, E, ff = c["tokens"], c["width"], c["experts"], c["ff"]
        return dict(c=c, h=d.normal(N, W), logits=d.normal(N, E, dtype=f, std=1.5), gate_up=d.normal(E, 2 * ff, W, std=W ** -0.5),
                    down=d.normal(E, W, ff, std=ff ** -0.5), x=d.normal(N, W, dtype=f), a=d.normal(N, W), w1=1 + d.normal(W, dtype=f, std=0.1),
                    b1=d.normal(W, dtype=f, std=0.1), w2=1 + d.normal(W, dtype=f, std=0.1), b2=d.normal(W, dtype=f, std=0.1))

    @staticmethod
    def run(s):
        c, h = s["c"], s["h"]
        places = h.shape[0] * c["top"]
        w, experts, pos, rows, offsets = F.moe_route(s["logits"], c["experts"], c["top"], "softmax_top")
        mid = F.grouped_gemm(h, s["gate_up"], offsets, places, rows=rows, act="silu_mul")
        y = F.grouped_gemm(mid, s["down"], offsets, places)
        x = s["x"].clone()                   # (the residual stream is updated in place and a pass can be repeated)
        n1, n2 = R.join_norms(x, [(s["w1"], s["b1"]), (s["w2"], s["b2"])], 1e-5, h.dtype, a=s["a"], y=y, pos=pos, weights=w)
        return x, n1, n2, w, experts

    @classmethod
    def exact(cls, c, seed):
        s = cls.prepare(c, seed)
        z, i = s["logits"].to(f64).topk(c["top"], dim=-1)
        w = torch.softmax(z, dim=-1)
        h, x, ff = s["h"].to(f64), s["x"].to(f64) + s["a"].to(f64), c["ff"]
        for e in range(c["experts"]):
            t, k = (i == e).nonzero(as_tuple=True)
            if len(t):
                gu = (h[t] @ s["gate_up"][e].to(f64).T).view(len(t), ff // 16, 2, 16)
                m = (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).flatten(1)
                x.index_add_(0, t, (m @ s["down"][e].to(f64).T) * w[t, k][:, None])
        u = x - x.mean(-1, keepdim=True)
        u = rms(u, 1e-5)
        return x, u * s["w1"].to(f64) + s["b1"].to(f64), u * s["w2"].to(f64) + s["b2"].to(f64), w, None

    @staticmethod
    def work(c):
        N, W, ff, M = c["tokens"], c["width"], c["ff"], c["tokens"] * c["top"]
        used = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** N)       # experts that a token reaches, on average
        return {"bytes": used * 3 * ff * W * 2.0 + N * W * (2.0 + 2.0 + 8.0 + 4.0) + N * (c["experts"] + 2 * c["top"]) * 4.0, "flops": 6.0 * M * W * ff}

    @staticmethod
    def tolerance(c):
        return {"rel": 7e-3, "max": 0.1, "differ": 1e-4}


# -- recurrent heads in a portion step -----------------------------------------------------------------
TAPS = 4


class Recurrent:
    @staticmethod
    def shape(c):
        """Decoded tokens, then portions of new prompts."""
        return [99] * c["decode"] + [0] * c["portions"], [1] * c["decode"] + lengths(c["portions"], c["min_tokens"], c["max_tokens"])

    @staticmethod
    def columns(c):
        """Columns of q, k, v, the gate and the fp32 gates."""
        H, G, dk, dv, rule = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["rule"]
        fp32 = {"delta": 2 * H, "scalar": H}.get(rule, H * dk)
        return G * dk, 0 if rule == "forget" else G * dk, H * dv, 0 if rule == "forget" else H * dv, fp32

    @classmethod
    def prepare(cls, c, seed):
        d, f = Draws(seed), torch.float32
        first, count = cls.shape(c)
        H, dk, dv, rule, rows, B = c["heads"], c["dim"], c["vdim"], c["rule"], sum(count), len(count)
        nq, nk, nv, ng, nz = cls.columns(c)
        s = dict(c=c, x=d.normal(rows, nq + nk + nv), gate=d.normal(rows, ng) if ng else None, z=d.normal(rows, nz, dtype=f), cu=running(count),
                 ctx=i32([a + n for a, n in zip(first, count)]), slots=torch.randperm(B, generator=d.gen, device=DEV).to(torch.int32), most=max(count),
                 state=d.normal(B, H, dk, dv, dtype=f, std=0.1), first=first, count=count)
        if rule in ("delta", "scalar"):      # these have a convolution
            s.update(conv=d.normal(TAPS, nq + nk + nv, dtype=f, std=0.5), ring=d.normal(B, TAPS, nq + nk + nv))
        if rule == "delta":
            s.update(A_log=d.normal(H, dtype=f, std=0.3), dt_bias=d.normal(H, dtype=f, std=0.3) - 2, norm=1 + d.normal(dv, dtype=f, std=0.1))
        elif rule == "scalar":
            s.update(conv_bias=d.normal(nq + nk + nv, dtype=f, std=0.1), A_log=d.normal(H, dtype=f, std=0.3), D=1 + d.normal(H, dtype=f, std=0.1),
                     bias=d.normal(H, dtype=f, std=0.3) - 2, norm=1 + d.normal(H * dv, dtype=f, std=0.1))
        else:
            s.update(bias=1 + d.normal(H * dk, dtype=f, std=0.3), lower=0.5 * d.uniform(H * dk) if rule == "forget" else None,
                     norm=1 + d.normal(dv, dtype=f, std=0.1))
        return s

    @staticmethod
    def run(s):
        c, x = s["c"], s["x"]
        H, G_, dk, dv, rule, nd = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["rule"], c["decode"]
        out = torch.empty(x.shape[0], H * dv, dtype=x.dtype, device=x.device)
        seqs = lambda part: (s["ctx"][part], s["slots"][part])
        done, new, cu = slice(0, nd), slice(nd, None), s["cu"][nd:]
        conv = rule in ("delta", "scalar")
        decoded = dict(conv_weight=s["conv"], ring=s["ring"]) if conv else {}
        if conv:
            y = torch.empty_like(x)
        if rule == "delta":
            call = lambda u, part, **kw: G.gated_delta(u, s["gate"], s["z"], s["A_log"], s["dt_bias"], s["norm"], s["state"], out, *seqs(part), H, G_, dk,
                                                       dv, 1e-5, **kw)
        else:
            if rule == "scalar":
                decoded["conv_bias"] = s["conv_bias"]
                more = dict(A_log=s["A_log"], D=s["D"])
            else:
                more = dict(lower=s["lower"]) if rule == "forget" else dict(rtau=1 / 16, qscale=dk ** -0.5)

            def call(u, part, **kw):
                nv, nk = H * dv, G_ * dk
                q, k, v = (u[:, nv + nk:], u[:, nv:nv + nk], u[:, :nv]) if rule == "scalar" else \
                    (u[:, :nk], None, u[:, nk:]) if rule == "forget" else (u[:, :nk], u[:, nk:2 * nk], u[:, 2 * nk:])
                LS.linear_state(rule, q, k, v, s["z"], s["bias"], s["state"], out, *seqs(part), H, G_, dk, dv, **more, **kw)
        if nd:
            call(x, done, **decoded)
        if conv:
            short_conv(x, s["conv"], s["ring"], *seqs(new), cu, s["most"], y, bias=s.get("conv_bias"))
        call(y if conv else x, new, cu_seqlens_q=cu)
        if rule != "delta":                  # (the delta rule norms its own outputs)
            parts, pre, post = (G_, s["gate"], None) if rule == "scalar" else (H, None, s["gate"])
            LS.group_norm_gate(out, s["norm"], parts, 1e-5, pre_gate=pre, post_gate=post, out=out)
        return (out, s["state"], s["ring"]) if conv else (out, s["state"])

    @classmethod
    def exact(cls, c, seed):
        s = cls.prepare(c, seed)
        H, G_, dk, dv, rule = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["rule"]
        first, count = cls.shape(c)
        B, most, silu, sp = len(count), max(count), torch.nn.functional.silu, torch.nn.functional.softplus
        x, z = s["x"].to(f64), s["z"].to(f64)
        state, slots = s["state"].to(f64), s["slots"].tolist()
        at = np.cumsum([0] + count)
        ring = None
        if "conv" in s:
            w, ring, y = s["conv"].to(f64), s["ring"].to(f64), torch.empty_like(x)
            for b, (f, n) in enumerate(zip(first, count)):
                before = [ring[slots[b], (f - j) % TAPS] if f - j >= 0 else torch.zeros_like(x[0]) for j in range(TAPS - 1, 0, -1)]
                u = torch.cat([torch.stack(before), x[at[b]:at[b + 1]]])
                y[at[b]:at[b + 1]] = silu(sum(w[j] * u[j:j + n] for j in range(TAPS)) + (s["conv_bias"].to(f64) if "conv_bias" in s else 0.0))
                for p in range(max(f, f + n - TAPS), f + n):
                    ring[slots[b], p % TAPS] = x[at[b] + p - f]
            x = y
        heads = lambda t, h, n: t.view(-1, h, n).repeat_interleave(H // h, dim=1)
        nq, nk, nv = G_ * dk, G_ * dk, H * dv
        if rule == "scalar":
            v, k, q = x[:, :nv].view(-1, H, dv), heads(x[:, nv:nv + nk], G_, dk), heads(x[:, nv + nk:], G_, dk)
            dt = sp(z + s["bias"].to(f64))
            a, k = torch.exp(-torch.exp(s["A_log"].to(f64)) * dt)[..., None].expand(-1, H, dk), k * dt[..., None]
        elif rule == "delta":
            unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
            q, k, v = unit(heads(x[:, :nq], G_, dk)) * dk ** -0.5, unit(heads(x[:, nq:nq + nk], G_, dk)), x[:, nq + nk:].view(-1, H, dv)
            g = torch.exp(-torch.exp(s["A_log"].to(f64)) * sp(z[:, :H] + s["dt_bias"].to(f64)))
            a, beta = g[..., None].expand(-1, H, dk), torch.sigmoid(z[:, H:])
        else:
            sig = torch.sigmoid(z + s["bias"].to(f64)).view(-1, H, dk)
            q = x[:, :nq].view(-1, H, dk)
            if rule == "forget":
                low = s["lower"].to(f64).view(H, dk)
                a = low + (1 - low) * sig
                q, k, v = silu(q), 1 - a, x[:, nq:].view(-1, H, dv)
            else:
                a, q, k, v = sig ** (1 / 16), q * dk ** -0.5, x[:, nq:2 * nq].view(-1, H, dk), x[:, 2 * nq:].view(-1, H, dv)
        # all sequences side by side, token after token
        S = torch.stack([state[i] if f else torch.zeros_like(state[i]) for i, f in zip(slots, first)])
        o = torch.empty(x.shape[0], H, dv, dtype=f64, device=DEV)
        for t in range(most):
            live = [b for b in range(B) if t < count[b]]
            r = torch.tensor([int(at[b]) + t for b in live], device=DEV)
            live = torch.tensor(live, device=DEV)
            now = S[live] * a[r][..., None]
            u = v[r]
            if rule == "delta":
                u = beta[r][..., None] * (u - torch.einsum("bhkv,bhk->bhv", now, k[r]))
            now += k[r][..., None] * u[:, :, None]
            S[live] = now
            o[r] = torch.einsum("bhkv,bhk->bhv", now, q[r])
        state[torch.tensor(slots, device=DEV)] = S
        gate = silu(s["gate"].to(f64)) if s["gate"] is not None else 1.0
        norm = s["norm"].to(f64)
        if rule == "scalar":
            o = (o + s["D"].to(f64)[:, None] * v).flatten(1) * gate
            out = rms(o.unflatten(1, (G_, -1)), 1e-5).flatten(1) * norm
        else:
            out = (rms(o, 1e-5) * norm).flatten(1) * gate
        return (out, state, ring) if ring is not None else (out, state)

    @classmethod
    def work(cls, c):
        first, count = cls.shape(c)
        cols, rows, H, dk, dv, B = cls.columns(c), sum(count), c["heads"], c["dim"], c["vdim"], len(count)
        return {"bytes": rows * (2.0 * sum(cols[:4]) + 4.0 * cols[4] + 2.0 * H * dv) + 4.0 * H * dk * dv * (B + c["decode"]),
                "flops": rows * 2.0 * H * (64 * (dk + dv) + 3 * dk * dv if c["rule"] == "delta" else 32 * (dk + dv) + 2 * dk * dv)}

    @staticmethod
    def tolerance(c):
        return {"rel": 1e-2, "max": 0.4}     # bf16 operands; a norm follows that magnifies the heads' small outputs


KINDS = {"decode_step": DecodeStep, "decode": Decode, "prefill": Prefill, "compress": Compress, "row_ops": RowOps, "sample": Sample, "window": Window,
         "latent": Latent, "experts": Experts, "recurrent": Recurrent}


def prepare(case, seed):
    return {"kind": case["kind"], "state": KINDS[case["kind"]].prepare(case, seed)}


def run(state):
    return KINDS[state["kind"]].run(state["state"])


def exact(case, seed):
    return KINDS[case["kind"]].exact(case, seed)


def work(case):
    return KINDS[case["kind"]].work(case)


def tolerance(case):
    return KINDS[case["kind"]].tolerance(case)
