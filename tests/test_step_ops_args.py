"""Argument checking of the per-step entry points: every rejection happens before any CUDA call,
so it can be exercised without a GPU (no kernel is launched by these tests)."""
import ctypes as C
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))

from zipage_b200 import _lib as L  # noqa: E402

INVALID = -1


def _err(lib):
    return lib.zp_last_error().decode()


def test_rms_norm_rejects_bad_arguments():
    lib = L.load()
    assert lib.zp_rms_norm(None, None, None, None, None, 0, 4096, 4096, 4096, 1e-6, 0, None) == 0  # empty batch
    assert lib.zp_rms_norm(None, None, None, None, None, 4, 4096, 4096, 4096, 1e-6, 0, None) == INVALID
    assert "null pointer" in _err(lib)
    p = C.c_void_p(4096)
    assert lib.zp_rms_norm(p, None, p, p, p, 4, 4096, 4096, 4096, 1e-6, 0, None) == INVALID   # residual_out without residual
    assert lib.zp_rms_norm(p, None, p, p, None, 4, 4100, 4100, 4100, 1e-6, 0, None) == INVALID  # not a multiple of 8 elements
    assert lib.zp_rms_norm(C.c_void_p(4098), None, p, p, None, 4, 4096, 4096, 4096, 1e-6, 0, None) == INVALID
    assert "aligned" in _err(lib)
    assert lib.zp_rms_norm(p, None, p, p, None, 4, 1 << 20, 1 << 20, 1 << 20, 1e-6, 0, None) == INVALID
    assert "too large" in _err(lib)
    assert lib.zp_rms_norm(p, None, p, p, None, 4, 4096, 4096, 4096, 1e-6, 7, None) == INVALID   # dtype code


def test_other_step_ops_reject_bad_arguments():
    lib = L.load()
    p = C.c_void_p(4096)
    assert lib.zp_silu_and_mul(None, None, 0, 128, 0, None) == 0
    assert lib.zp_silu_and_mul(None, p, 3, 128, 0, None) == INVALID
    assert lib.zp_silu_and_mul(p, p, 3, 100, 0, None) == INVALID          # 100 bf16 is not whole vectors
    args = lambda **kw: [kw.get("qkv", p), p, p, p, p, 1e-6, kw.get("q_out", p), None, kw.get("kc"), kw.get("vc"),
                         kw.get("slots"), kw.get("qc"), kw.get("trip"), kw.get("ntrip", 0), None, kw.get("n", 5), 8, 2,
                         kw.get("D", 128), 1536, 0, 0, 0, None]
    assert lib.zp_qk_norm_rope_store(*args(n=0)) == 0
    assert lib.zp_qk_norm_rope_store(*args(q_out=None)) == INVALID
    assert lib.zp_qk_norm_rope_store(*args(slots=p)) == INVALID             # slot mapping without caches
    assert lib.zp_qk_norm_rope_store(*args(ntrip=2)) == INVALID             # triples without a window buffer
    assert lib.zp_qk_norm_rope_store(*args(D=96)) == INVALID
    assert "head_dim" in _err(lib)
    assert lib.zp_qk_norm_rope_store(*args(qkv=C.c_void_p(4100))) == INVALID
    # the form that packs the values too checks the same and one pointer more, which may be missing
    packed = lambda v_out, **kw: (lambda a: lib.zp_qk_norm_rope_store_v(*a[:8], v_out, *a[8:]))(args(**kw))
    assert packed(p, n=0) == packed(None, n=0) == 0
    assert packed(C.c_void_p(4100)) == INVALID and "aligned" in _err(lib)
    assert packed(p, q_out=None) == packed(p, slots=p) == packed(p, D=96) == packed(p, qkv=C.c_void_p(4100)) == INVALID
    assert lib.zp_sample(None, None, None, None, 0, 1000, 0, 0, None) == 0
    assert lib.zp_sample(p, None, None, p, 2, 1000, 0, 0, None) == INVALID
    assert lib.zp_sample(p, p, None, p, 2, 0, 0, 0, None) == INVALID
    assert lib.zp_prepare_decode(p, p, p, 3, 9, 32, 256, p, p, p, p, None, None) == INVALID
    assert lib.zp_prepare_decode(None, p, p, 3, 9, 32, 256, p, p, p, p, p, None) == INVALID
    assert lib.zp_prepare_decode(p, p, p, 3, 9, 300, 256, p, p, p, p, p, None) == INVALID  # window longer than a page


def test_latent_rows_reject_unknown_types():
    lib, p = L.load(), C.c_void_p(4096)
    for dtype in (3, 7, -1):
        assert lib.zp_latent_prepare(p, 640, p, p, p, p, p, p, None, p, 5, 64, 512, 64, 576, 100, 1e-6, dtype, None) == INVALID
        assert "dtype" in _err(lib)
        assert lib.zp_latent_rotate_q(p, 640, p, p, None, 5, 4, 96, 64, 0, 0, dtype, None) == INVALID


def test_small_linear_rejects_bad_arguments():
    lib, p = L.load(), C.c_void_p(4096)
    call = lambda x=p, stride=64, w=p, out=p, rows=4, n=48, k=64, dtype=0: lib.zp_small_linear(x, stride, w, None, out, rows, n, k, dtype, None)
    assert call(rows=0) == 0 and call(n=0) == 0
    for bad in (dict(x=None), dict(w=None), dict(out=None), dict(rows=9), dict(rows=-1), dict(n=-1), dict(k=0), dict(k=48), dict(stride=65),
                dict(x=C.c_void_p(4100)), dict(w=C.c_void_p(4100)), dict(k=1 << 27), dict(n=2 ** 31 - 1)):
        assert call(**bad) == INVALID, bad
    assert call(dtype=7) != 0


def test_window_workspace_covers_every_split_that_a_decode_step_may_take():
    """Four blocks an SM and at least two tiles of 64 keys each, whatever the head sizes: a caller may size its buffer once, for its largest batch."""
    lib = L.load()
    for B in (1, 8, 20, 24, 37, 48, 74, 100):
        for kv_heads in (1, 8):
            for dim in (64, 96, 128, 256):
                for span in (64, 200, 1024, 1536, 1537, 4096):
                    splits = max(1, min(-(-592 // (B * kv_heads)), ((span + 63) // 64 + 1) // 2, 32))
                    want = B * 16 * splits * (dim + 2) * 4 if splits > 1 else 0
                    assert lib.zp_window_attention_workspace_bytes(B, 16, kv_heads, dim, span) == want
