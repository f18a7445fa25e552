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


# by rows; longer documents: attention as a launch of its own is faster (both sides in csrc/decode_stack.cu)
MAX_KEYS = {1: 3072, 2: 1792}


def takes(rows: int, hidden: int, ffn: int, heads: int, kv_heads: int, keys: int) -> bool:
    """Whether the kernel is built for these sizes, and the better choice."""
    return 0 < keys <= MAX_KEYS.get(rows, 0) and _words(rows, hidden, ffn, heads, kv_heads) > 0


# A launch has 384 phase numbers of 32 bits: they come round after 11 million launches, and a word that has not been written since
# (of a second row, of more parts) could then be taken for a new one.  Scratch is replaced between requests well before that; a
# request adds at most a launch per 48 layers and key.
MAX_LAUNCHES = 1 << 23


class Scratch:
    """What the CTAs of a launch exchange, for one engine; launches that share it must follow one another on the device.
    ``count[-1]`` is not zero once a launch has run out of time: phase numbers may differ from then on, and every later launch
    on this scratch returns at once."""

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


# ---- between the LM head and the layers (csrc/decode_step.cu) -----------------------------------------------------
def argmax_rows(x):
    """``x.argmax(-1)`` of fp32 rows: NaN counts as largest, of equal elements the first."""
    rows, V = x.shape
    if x.dtype != torch.float32 or x.stride(1) != 1 or (rows > 1 and x.stride(0) < V):
        raise ValueError("argmax_rows takes fp32 rows")
    out = torch.empty(rows, dtype=torch.long, device=x.device)
    _lib.call("argmax_rows", c_void_p(x.data_ptr()), c_ll(max(x.stride(0), V)), c_int(rows), c_int(V), c_void_p(out.data_ptr()),
              c_void_p(_lib.stream()))
    return out


class Rows:
    """Device state of a decode: what the step in progress reads (``x``, ``pos3``, ``meta_q``, ``kv_rows``) and what
    :meth:`advance` needs to make it from the next tokens."""

    def __init__(self, pos, kv_rows, hidden: int, new: int):
        """``pos`` (int32) / ``kv_rows`` (int64): position and cache row of every document's first new token."""
        n, dev = pos.numel(), pos.device
        if pos.dtype != torch.int32 or kv_rows.dtype != torch.int64 or kv_rows.numel() != n:
            raise ValueError("positions are int32 and cache rows int64, one per document")
        self.pos0, self.row0 = pos.contiguous(), kv_rows.contiguous()
        self.out = torch.full((n, new), -1, dtype=torch.long, device=dev)
        self.done = torch.zeros(n, dtype=torch.int32, device=dev)
        self.x = torch.empty(n, hidden, dtype=torch.bfloat16, device=dev)
        self.pos3 = torch.empty(3, n, dtype=torch.int32, device=dev)
        self.meta_q = torch.empty(n, 4, dtype=torch.int32, device=dev)
        self.kv_rows = torch.empty(n, dtype=torch.int64, device=dev)

    def advance(self, tokens, embed, meta_k):
        """Tokens (int64 [docs]) are stored; their embeddings, positions, cache rows and metadata become the step's."""
        n, H = self.x.shape
        if (tokens.dtype != torch.int64 or tokens.numel() != n or not tokens.is_contiguous() or embed.dtype != torch.bfloat16
                or embed.shape[1] != H or not embed.is_contiguous() or meta_k.dtype != torch.int32 or meta_k.shape[1] != 4
                or not meta_k.is_contiguous()):
            raise ValueError("advance: tokens int64 [docs], embedding [vocab, hidden], metadata int32 [rows, 4]")
        P = lambda t: c_void_p(t.data_ptr())
        _lib.call("decode_advance", P(tokens), P(embed), c_int(embed.shape[0]), c_int(H), c_int(n), c_int(meta_k.shape[0]), P(self.done),
                  P(self.pos0), P(self.row0), P(self.out), c_int(self.out.shape[1]), P(self.x), P(self.pos3), P(self.meta_q),
                  P(meta_k), P(self.kv_rows), c_void_p(_lib.stream()))
