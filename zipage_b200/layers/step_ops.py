"""The per-step ops around the attention path on libzipage_b200 kernels.

Same names and call contracts as the reference modules they replace:
`RMSNorm` (third_party/nanovllm/layers/layernorm.py), `SiluAndMul`
(third_party/nanovllm/layers/activation.py), `Sampler` (zipage/layers/sampler.py);
`qk_norm_rope_store` replaces the q/k normalisation + rotation of `Qwen3Attention.forward`
(third_party/nanovllm/models/qwen3.py:75-79) together with the two cache writes at the head of
`Attention.forward` (zipage/layers/attention.py:72-77); `prepare_decode` replaces the host loop of
`ModelRunner.prepare_decode` (zipage/engine/model_runner.py:633-675) from device-resident state.
There is no CPU path: non-CUDA tensors are rejected.
"""
from __future__ import annotations

import torch
from torch import nn
from torch.autograd import forward_ad
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

from .. import _lib as L
from ..kernel import _count


def rms_norm(x, weight, eps, residual=None):
    """x [..., H]; returns out, or (out, new_residual) when a residual is given."""
    L.require_cuda(x, weight, residual)
    H = x.shape[-1]
    x2 = x.reshape(-1, H)
    assert x2.stride(-1) == 1 and weight.is_contiguous() and weight.dtype == x.dtype
    out = torch.empty((x2.shape[0], H), dtype=x.dtype, device=x.device)
    res_out = None
    if residual is not None:
        residual = residual.reshape(-1, H)
        assert residual.is_contiguous() and residual.dtype == x.dtype
        res_out = torch.empty_like(residual)
    L.check(L.load().zp_rms_norm(L.ptr(x2), L.ptr(residual), L.ptr(weight), L.ptr(out), L.ptr(res_out),
                                 x2.shape[0], H, x2.stride(0), out.stride(0), float(eps),
                                 L.dtype_code(x), L.stream_ptr()), "rms_norm")
    _count(1)
    out = out.view(x.shape)
    return out if residual is None else (out, res_out.view(x.shape))


class RMSNorm(nn.Module):
    """layernorm.py:5-50."""

    def __init__(self, hidden_size: int, eps: float = 1e-6) -> None:
        super().__init__()
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(hidden_size))

    def forward(self, x, residual=None):
        return rms_norm(x, self.weight, self.eps, residual)


# Rows, entries and sides of the weight up to which `linear` takes this library's kernel.  At 8 rows it takes 0.4 to 0.7 of cuBLAS's time
# for weights of up to 2^23 entries (2048 x 1024: 2.2 us for 5.1; 6144 x 1024: 3.6 for 5.3; 1024 x 3072: 3.8 for 8.8; 256 x 4096: 4.0 for 7.7); larger
# ones go either way (4096 x 4096: 7.4 for 12.1; 5120 x 2048: 6.0 for 6.6; 8192 x 2048: 7.9 for 8.1; 12288 x 4096: 20.4 for 18.2).  A block walks 16 whole
# rows of the weight, so very long ones leave SMs idle (256 x 8192: 7.0 for 12.6, but 32 x 65536: 33 for 13), and very many short ones are blocks of
# little work (32768 x 256: 5.6 for 5.4).
SMALL_ROWS, SMALL_WEIGHT, SMALL_K, SMALL_N = 8, 1 << 23, 4096, 1 << 15


_linear_forward = nn.Linear.forward


def _plain_call(layer):
    """Whether layer(x) is nn.Linear's product and nothing around it looks at the call: no hooks, no forward or compiled call of the layer's
    own, no function or dispatch mode (a default device is one, but leaves products alone), no transform (vmap, forward-mode
    derivatives), no gradients, autocast, tracing or compilation."""
    modes = _get_current_function_mode_stack() if torch._C._len_torch_function_stack() else ()
    return (type(layer) is nn.Linear and nn.Linear.forward is _linear_forward and "forward" not in layer.__dict__
            and layer._compiled_call_impl is None
            and not (layer._forward_hooks or layer._forward_pre_hooks or nn.modules.module._has_any_global_hook())
            and all(type(m) is DeviceContext for m in modes) and not torch._C._len_torch_dispatch_stack()
            and torch._C._functorch.peek_interpreter_stack() is None and forward_ad._current_level < 0
            and not torch.is_grad_enabled() and not torch.is_autocast_enabled("cuda")
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling())


def _small_linear_takes(layer, x):
    """Whether `zp_small_linear` computes layer(x), for x on the current CUDA device.  The kernel takes its sizes from the weight, so
    they are compared here."""
    if x.dim() != 2 or x.shape[0] > SMALL_ROWS or not _plain_call(layer):      # (what tells most other calls apart comes first)
        return False
    w, b = layer.weight, layer.bias
    return (type(w) is nn.Parameter and x.layout is w.layout is torch.strided and w.dim() == 2 and x.shape[0] > 0
            and 0 < x.shape[1] == w.shape[1] <= SMALL_K and w.shape[0] <= SMALL_N and w.numel() <= SMALL_WEIGHT and x.dtype in (torch.bfloat16, torch.float16) and w.dtype == x.dtype
            and w.device == x.device and w.is_contiguous() and x.stride(1) == 1 and x.stride(0) % 8 == 0 and w.shape[1] % 32 == 0
            and (w.data_ptr() | x.data_ptr()) % 16 == 0
            and (b is None or b.shape == w.shape[:1] and b.dtype == x.dtype and b.device == x.device and b.is_contiguous()))


def linear(layer, x):
    """layer(x) for an nn.Linear: the few rows of a small decode step through `zp_small_linear`, everything else
    (more rows, fp32, odd sizes, sizes that do not fit, gradients, subclasses, hooks, modes) through the layer itself."""
    if type(x) is torch.Tensor and x.is_cuda and x.device.index == torch.cuda.current_device() and _small_linear_takes(layer, x):
        w, b = layer.weight, layer.bias
        out = torch.empty((x.shape[0], w.shape[0]), dtype=x.dtype, device=x.device)
        L.check(L.load().zp_small_linear(L.ptr(x), x.stride(0), L.ptr(w), L.ptr(b), L.ptr(out), x.shape[0], w.shape[0], w.shape[1],
                                         L.dtype_code(x), L.stream_ptr()), "small_linear")
        _count(1)
        return out
    return layer(x)


def silu_and_mul(x):
    L.require_cuda(x)
    two_i = x.shape[-1]
    x2 = x.reshape(-1, two_i)
    assert x2.is_contiguous() and two_i % 2 == 0
    out = torch.empty((x2.shape[0], two_i // 2), dtype=x.dtype, device=x.device)
    L.check(L.load().zp_silu_and_mul(L.ptr(x2), L.ptr(out), x2.shape[0], two_i // 2, L.dtype_code(x),
                                     L.stream_ptr()), "silu_and_mul")
    _count(1)
    return out.view(*x.shape[:-1], two_i // 2)


class SiluAndMul(nn.Module):
    """activation.py:6-14."""

    def forward(self, x):
        return silu_and_mul(x)


def rope_cos_sin_cache(head_dim, max_position, base, device):
    """RotaryEmbedding.cos_sin_cache (rotary_embedding.py:84-89, default rope type) as
    [max_position, head_dim] fp32."""
    inv_freq = 1.0 / (base ** (torch.arange(0, head_dim, 2, dtype=torch.float) / head_dim))
    t = torch.arange(max_position, dtype=torch.float)
    freqs = torch.einsum("i,j -> ij", t, inv_freq)
    return torch.cat((freqs.cos(), freqs.sin()), dim=-1).to(device)


def qk_norm_rope_store(qkv, positions, cos_sin, q_weight, k_weight, eps, num_heads, num_kv_heads,
                       head_dim, k_cache=None, v_cache=None, slot_mapping=None, query_cache=None,
                       query_slot_mapping=None, return_k=True, query_slot_count=None, return_v=None):
    """qkv [N, (Hq+2Hkv)*D] -> q [N,Hq,D] (normalised, rotated), k [N,Hkv,D] (or None), and, when
    given, K/V rows written to the paged caches at slot_mapping and window queries written to
    query_cache at the (row, query_id, index) triples — one launch.  `query_slot_count`: a device
    int32 tensor with the number of valid rows of `query_slot_mapping` (as `prepare_decode` returns
    it); without it every row is taken.  v [N,Hkv,D]: a packed copy with `return_v` (None: as `return_k`, whose callers
    mostly attend over the rows themselves), else a view of qkv."""
    L.require_cuda(qkv, positions, cos_sin, q_weight, k_weight, k_cache, v_cache, slot_mapping,
                   query_cache, query_slot_mapping, query_slot_count)
    N = qkv.shape[0]
    Hq, Hkv, D = num_heads, num_kv_heads, head_dim
    assert qkv.shape[1] == (Hq + 2 * Hkv) * D and qkv.stride(1) == 1
    assert positions.dtype == torch.int64 and cos_sin.dtype == torch.float32 and cos_sin.is_contiguous()
    q = torch.empty((N, Hq, D), dtype=qkv.dtype, device=qkv.device)
    k, v = (torch.empty((N, Hkv, D), dtype=qkv.dtype, device=qkv.device) if wanted else None
            for wanted in (return_k, return_k if return_v is None else return_v))
    ntrip = 0 if query_slot_mapping is None else query_slot_mapping.shape[0]
    cs_seq = query_cache.stride(0) if query_cache is not None else 0
    cs_slot = query_cache.stride(1) if query_cache is not None else 0
    if k_cache is not None:
        assert k_cache.is_contiguous() and v_cache.is_contiguous()
    L.check(L.load().zp_qk_norm_rope_store_v(
        L.ptr(qkv), L.ptr(positions), L.ptr(cos_sin), L.ptr(q_weight), L.ptr(k_weight), float(eps),
        L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(k_cache), L.ptr(v_cache), L.ptr(slot_mapping), L.ptr(query_cache),
        L.ptr(query_slot_mapping), ntrip, L.ptr(query_slot_count), N, Hq, Hkv, D, qkv.stride(0), cs_seq, cs_slot,
        L.dtype_code(qkv), L.stream_ptr()), "qk_norm_rope_store")
    _count(1)
    if v is None:
        v = qkv[:, (Hq + Hkv) * D:].view(N, Hkv, D)
    return q, k, v


def sample(logits, temperatures, noise=None, seed=0):
    """tokens [B] int64; `noise` = the Exp(1) draws ([B, V] fp32) or None for the built-in
    counter-based generator keyed by `seed`."""
    L.require_cuda(logits, temperatures, noise)
    B, V = logits.shape
    assert logits.is_contiguous() and temperatures.dtype == torch.float32
    if noise is not None:
        assert noise.dtype == torch.float32 and noise.is_contiguous() and noise.shape == logits.shape
    out = torch.empty(B, dtype=torch.int64, device=logits.device)
    L.check(L.load().zp_sample(L.ptr(logits), L.ptr(temperatures), L.ptr(noise), L.ptr(out), B, V,
                               int(seed), L.dtype_code(logits), L.stream_ptr()), "sample")
    _count(1)
    return out


class Sampler(nn.Module):
    """zipage/layers/sampler.py:6-48 without the repetition penalty (a transformers logits
    processor the reference applies before this op).  Each call advances the seed."""

    def __init__(self, seed: int = 0):
        super().__init__()
        self.seed = seed

    def forward(self, logits, temperatures, noise=None):
        self.seed += 1
        return sample(logits, temperatures, noise, self.seed)


def decode_inputs(input_ids, num_tokens, block_tables, query_ids, buffers):
    """The inputs of a decode step into the runner's buffers (ids, counts, tables, query ids), the rest cleared: one launch, or False
    where the tensors are not such that the kernel can read them."""
    ids, num, tab, qid = buffers
    given = ((input_ids, ids), (num_tokens, num), (block_tables, tab), (query_ids, qid))
    if not all(type(x) is torch.Tensor and x.device == y.device and x.dtype == y.dtype and x.dim() == y.dim() and (x.shape[-1] <= 1 or x.stride(-1) == 1)
               for x, y in given) or not tab.is_cuda or not len(input_ids) == len(num_tokens) == len(block_tables) == len(query_ids):
        return False
    L.check(L.load().zp_decode_inputs(L.ptr(input_ids), L.ptr(num_tokens), L.ptr(block_tables), block_tables.stride(0), L.ptr(query_ids),
                                      len(input_ids), block_tables.shape[1], L.ptr(ids), L.ptr(num), L.ptr(tab), L.ptr(qid),
                                      len(ids), tab.shape[1], L.stream_ptr()), "decode_inputs")
    _count(1)
    return True


def prepare_decode(num_tokens, block_tables, query_ids, query_cache_len, block_size=256):
    """Device tensors in, device tensors out: positions [B] i64, context_lens [B] i32,
    slot_mapping [B] i32, triples [B,3] i32 with n_triples [1] i32 valid rows."""
    L.require_cuda(num_tokens, block_tables, query_ids)
    B, W = block_tables.shape
    dev = block_tables.device
    pos = torch.empty(B, dtype=torch.int64, device=dev)
    ctx = torch.empty(B, dtype=torch.int32, device=dev)
    slot = torch.empty(B, dtype=torch.int32, device=dev)
    trip = torch.empty((B, 3), dtype=torch.int32, device=dev)
    ntrip = torch.empty(1, dtype=torch.int32, device=dev)
    assert num_tokens.dtype == torch.int32 and block_tables.dtype == torch.int32 and block_tables.is_contiguous()
    L.check(L.load().zp_prepare_decode(L.ptr(num_tokens), L.ptr(block_tables), L.ptr(query_ids), B, W,
                                       query_cache_len, block_size, L.ptr(pos), L.ptr(ctx), L.ptr(slot),
                                       L.ptr(trip), L.ptr(ntrip), L.stream_ptr()), "prepare_decode")
    _count(1)
    return pos, ctx, slot, trip, ntrip
