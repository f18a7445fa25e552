"""Python face of the whole-stack decode kernel (csrc/decode_stack.cu)."""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._lib import c_float, c_int, c_ll, c_void_p


def _words(rows: int, hidden: int, ffn: int, heads: int, kv_heads: int) -> int:
    fn = _lib.load().snu1_decode_stack_takes
    fn.restype = c_ll
    return fn(c_int(rows), c_int(hidden), c_int(ffn), c_int(heads), c_int(kv_heads))


MAX_KEYS = 3072      # longer documents: attention as a launch of its own is faster (both sides in csrc/decode_stack.cu)


def takes(rows: int, hidden: int, ffn: int, heads: int, kv_heads: int, keys: int) -> bool:
    """Whether the kernel is built for these sizes, and the better choice."""
    return 0 < keys <= MAX_KEYS and _words(rows, hidden, ffn, heads, kv_heads) > 0


class Scratch:
    """What the CTAs of a launch exchange, for one engine; launches that share it must follow one another on the device."""

    def __init__(self, device):
        ctas = torch.cuda.get_device_properties(device).multi_processor_count
        self.count = torch.zeros(ctas + 1, dtype=torch.int32, device=device)       # launches, by CTA; given up
        self.words = torch.zeros(0, dtype=torch.int64, device=device)

    def fit(self, words: int):
        if self.words.numel() < words:
            self.words = torch.zeros(words, dtype=torch.int64, device=self.count.device)


def decode_stack(x, layers, out, scratch: Scratch, heads: int, kv_heads: int, ffn: int, plan, kv_rows, pos3, kv_len: int,
                 inv_t, inv_hw, eps: float, scale: float):
    """``x`` [rows, H], one new token per document, through all ``layers`` (tuples wqkv, wo, w13, w2, attn_norm, qk_norm,
    ffn_norm, k cache, v cache) into ``out`` [rows, H]; the new keys and values go to cache rows ``kv_rows`` (int64)."""
    rows, H = x.shape
    table = (c_ll * (9 * len(layers)))()
    cache = layers[0][7]
    shapes = [((heads + 2 * kv_heads) * 128, H), (H, heads * 128), (2 * ffn, H), (H, ffn), (H,), (4, 64), (H,)] + [tuple(cache.shape)] * 2
    for l, tensors in enumerate(layers):
        for i, (t, want) in enumerate(zip(tensors, shapes)):
            if t.dtype != torch.bfloat16 or tuple(t.shape) != want or not t.is_contiguous():
                raise ValueError(f"layer {l}, operand {i}: expected contiguous bf16 {want}, got {t.dtype} {tuple(t.shape)}")
            table[9 * l + i] = t.data_ptr()
    if not (x.is_contiguous() and out.is_contiguous() and pos3.is_contiguous() and x.dtype == out.dtype == torch.bfloat16
            and out.shape == x.shape and pos3.dtype == torch.int32 and pos3.shape == (3, rows)
            and kv_rows.dtype == torch.int64 and kv_rows.numel() == rows and cache.shape[1:] == (kv_heads, 128)
            and plan.first.dtype == torch.int32 and plan.first.numel() == rows and plan.meta_q.shape == (rows, 4)
            and plan.meta_k.shape == (kv_len, 4) and kv_len <= cache.shape[0] and x.data_ptr() != out.data_ptr()):
        raise ValueError("decode_stack: operands of other shapes or types")
    scratch.fit(_words(rows, H, ffn, heads, kv_heads))
    P = lambda t: c_void_p(t.data_ptr())
    _lib.call("decode_stack", ctypes.cast(table, c_void_p), c_int(len(layers)), c_int(rows), c_int(H), c_int(ffn), c_int(heads),
              c_int(kv_heads), c_int(kv_len), c_ll(cache.shape[0]), P(x), P(out), P(scratch.words), c_ll(scratch.words.numel()),
              P(scratch.count), P(plan.meta_q), P(plan.meta_k), P(plan.first), P(kv_rows), P(pos3), P(inv_t), P(inv_hw),
              c_int(plan.max_keys), c_float(eps), c_float(scale), c_void_p(_lib.stream()))
    return out
