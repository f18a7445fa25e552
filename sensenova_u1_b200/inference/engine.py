"""CUDA inference engine of the NEO-unify MoT model: prefix (understanding branch)
forward with KV cache, flow-matching image denoising through the generation branch,
and greedy text decoding — all on the sm_100a kernels of this package.

Differences from the reference's generation loops
(src/sensenova_u1/models/neo_unify/modeling_neo_chat.py:1691-1860, modeling_qwen3.py:583-745):
the conditional and unconditional branches run as two documents of ONE packed forward
(one GEMM launch per projection instead of two passes), the prefix attention uses the
tile-classified tensor-core kernel instead of eager fp32 softmax, K/V of the prefix stay
in place in a per-layer buffer and only the image rows are rewritten each step, and the
CFG combine + Euler step + re-patchify are one kernel.
"""
from __future__ import annotations

import math
from dataclasses import dataclass
from typing import List, Optional, Sequence

import torch

from ..config import ModelConfig
from ..data.batch import apply_time_schedule
from ..models import oracle
from ..models.engine import Workspace
from ..models.params import GEN, UND, ParamStore
from ..ops import _lib, attention as attn_ops, decode_stack, fused, gemm, moe
from ..ops._lib import c_float, c_int, c_void_p

CFG_NORMS = {"none": 0, "global": 1, "channel": 2, "cfg_zero_star": 3}


def _pad128(n):
    return (n + 127) // 128 * 128


def upload(device, *tensors):
    """Host tensors on the device, in one copy from pinned memory that nothing waits for.  (A copy from pageable memory
    waits for all work of the stream: with ten of them per request, the device idled 2 - 8 ms while the host prepared
    indexes, launches and the decode graph.)  Tensors that are on a device already are only moved if needed."""
    device = torch.device(device)
    host = [t for t in tensors if not t.is_cuda]
    if device.type != "cuda" or not host:
        return [t.to(device) for t in tensors]
    offsets, n = [], 0
    for t in host:
        offsets.append(n)
        n += (t.numel() * t.element_size() + 15) // 16 * 16
    buf = torch.empty(max(n, 16), dtype=torch.uint8, pin_memory=True)
    at = lambda b, t, o: b[o:o + t.numel() * t.element_size()].view(t.dtype).view(t.shape)
    for t, o in zip(host, offsets):
        at(buf, t, o).copy_(t)
    dev = buf.to(device, non_blocking=True)
    it = iter([at(dev, t, o) for t, o in zip(host, offsets)])
    return [t.to(device) if t.is_cuda else next(it) for t in tensors]


@dataclass
class DocLayout:
    """Row ranges of one document inside the per-layer KV buffer."""
    kv_start: int      # first KV row of the document
    prefix_len: int    # text / understanding rows already cached
    img_start: int     # first row reserved for the image being generated
    next_pos: int      # t index the next token / image takes


@dataclass
class DecodeRows:
    """One query row per document, each reading its own document's cache rows up to its own: stands in for a
    ``TilePlan`` in :meth:`InferenceEngine.layers`."""
    meta_q: torch.Tensor
    meta_k: torch.Tensor
    first: torch.Tensor    # int32 [docs] first cache row of the document
    max_keys: int          # longest range of the request


class InferenceEngine:
    def __init__(self, cfg: ModelConfig, store: ParamStore, offload=None):
        """``offload``: a ``utils.offload.LayerOffloader``; the decoder-layer weights then come from it
        (streamed from pinned host memory one layer ahead) and ``store`` only needs the other tensors."""
        if cfg.head_dim != 128:
            raise ValueError("the sm_100a attention kernels need head_dim 128")
        self.cfg, self.store, self.p = cfg, store, store.p
        self.offload = offload
        self.dev = store.device
        self.ws = Workspace(self.dev)
        inv_t, inv_hw = oracle.rope_inv_freq(cfg, self.dev)
        self.inv_t, self.inv_hw = inv_t.contiguous(), inv_hw.contiguous()
        half = cfg.vision_hidden // 2
        self.inv_v = (1.0 / (cfg.rope_theta_vision ** (
            torch.arange(0, half, 2, dtype=torch.float32, device=self.dev) / half))).contiguous()
        self.scale = cfg.head_dim ** -0.5
        self.kc: List[torch.Tensor] = []
        self.vc: List[torch.Tensor] = []
        self.stats = torch.zeros(4 + 4 * 592, dtype=torch.float32, device=self.dev)   # sums + per-block partials
        self._graph = self._capture_stream = None     # last captured decode step, for its memory (see _capture)
        self._graph_bytes = 0
        self.sp = None      # sequence-parallel sampling state (enable_sequence_parallel)
        self._stack = None  # scratch of the whole-stack decode kernel

    def enable_sequence_parallel(self, group) -> None:
        """Splits the image tokens of :meth:`denoise` over the ranks of ``group`` (all of which run the same
        call with the same arguments).  The per-layer K/V caches move to symmetric memory: every rank writes
        the keys / values of its token slice into all peers' caches with peer stores, a device-side flag
        barrier per layer orders the writes before the attention reads.  Call before the first prefill."""
        import torch.distributed as dist
        from ..parallel.symm import FlagBarrier
        self.sp = {"group": group, "world": dist.get_world_size(group), "rank": dist.get_rank(group),
                   "bar": FlagBarrier(group, self.dev), "k": None, "v": None}
        self.kc, self.vc = [], []

    # ------------------------------------------------------------ building blocks
    def vision_embed(self, br: str, patches, px, py):
        cfg, p = self.cfg, self.p
        m2 = cfg.merge_size ** 2
        a1 = gemm.gemm_nt(patches, p[f"vision_{br}.patch_w"], residual=p[f"vision_{br}.patch_b"], w_static=True)
        fused.gelu_fwd(a1, a1)
        r1 = fused.rope2d(a1, torch.empty_like(a1), px, py, self.inv_v)
        return gemm.gemm_nt(r1.view(r1.shape[0] // m2, m2 * cfg.vision_hidden), p[f"vision_{br}.merge_w"],
                            residual=p[f"vision_{br}.merge_b"], w_static=True)

    def scalar_embed(self, name, t):
        p = self.p
        s = oracle.sinusoid(t, self.cfg.timestep_freq_dim).to(torch.bfloat16)
        h = torch.nn.functional.silu(gemm.gemm_nt(s, p[name + ".w1"], residual=p[name + ".b1"]))
        return gemm.gemm_nt(h, p[name + ".w2"], residual=p[name + ".b2"])

    def alloc_cache(self, kv_rows: int):
        cfg = self.cfg
        if self.kc and self.kc[0].shape[0] >= kv_rows:
            return
        if self.sp is not None:
            from ..parallel.symm import SymmetricBuffer
            n = cfg.num_layers * kv_rows * cfg.kv_dim
            self.sp["k"] = SymmetricBuffer(n, torch.bfloat16, self.dev, self.sp["group"])
            self.sp["v"] = SymmetricBuffer(n, torch.bfloat16, self.dev, self.sp["group"])
            self.sp["rows"] = kv_rows
            shape = (cfg.num_layers, kv_rows, cfg.num_kv_heads, 128)
            self.kc = list(self.sp["k"].tensor.view(shape).unbind(0))
            self.vc = list(self.sp["v"].tensor.view(shape).unbind(0))
            return
        self.kc = [torch.zeros(kv_rows, cfg.num_kv_heads, 128, dtype=torch.bfloat16, device=self.dev)
                   for _ in range(cfg.num_layers)]
        self.vc = [torch.zeros(kv_rows, cfg.num_kv_heads, 128, dtype=torch.bfloat16, device=self.dev)
                   for _ in range(cfg.num_layers)]

    def layers(self, x, branch: int, pos3, plan, kv_rows, kv_len: int, publish=None):
        """Runs the decoder stack on rows ``x`` [R,H] with one branch's weights.  The rows'
        K/V are written to cache rows ``kv_rows`` (int64 [R]); attention reads cache rows
        [0, kv_len).  Returns the final hidden state (before the final norm).

        ``publish`` (sequence-parallel sampling): runs of rows [(first row of x, count, first cache row)]
        whose K/V go to every rank of the sequence-parallel group instead of the local cache only."""
        cfg, p, ws = self.cfg, self.p, self.ws
        R, H = x.shape
        qd, kd = cfg.q_dim, cfg.kv_dim
        if self.offload is not None:
            self.offload.set_phase("prefix" if branch == UND else "denoise")
        static = self.offload is None           # offloaded weights arrive from a copy stream between the kernels
        if isinstance(plan, DecodeRows) and self._one_launch(R, plan.max_keys):
            return self._decode_layers(x, branch, pos3, plan, kv_rows, kv_len)
        h1, h2, x1 = (ws.get(n, (R, H)) for n in ("i.h1", "i.h2", "i.x1"))
        xo = [ws.get(f"i.x{i}", (R, H)) for i in range(2)]
        qkv, qk = ws.get("i.qkv", (R, qd + 2 * kd)), ws.get("i.qk", (R, qd + kd))
        qf = qk[:, :qd]
        q = qf.unflatten(1, (cfg.num_heads, 128))
        o = ws.get("i.o", (R, cfg.num_heads, 128))
        of = o.view(R, qd)
        decode = isinstance(plan, DecodeRows)
        act = None
        if not cfg.is_moe:
            act = ws.get("i.act", (R, cfg.ffn_size))
        normed = False
        for l in range(cfg.num_layers):
            s = f"layers.{l}."
            if self.offload is not None:
                lw = self.offload.layer_weights(l)          # this branch's tensors, on the device
                W = WE = lambda n: lw[n]
            else:
                W = lambda n: p[s + n][branch]
                WE = lambda n: p[s + n]                     # expert mixtures are whole tensors of one branch
            if not normed:
                fused.rmsnorm_fwd(x, W("attn_norm"), None, h1, None, cfg.rms_eps)
            normed = False
            gemm.gemm_nt(h1, W("wqkv"), out=qkv, w_static=static, in_parts=True)
            if publish is None:
                fused.qknorm_rope_cache(qkv, qf, self.kc[l], self.vc[l], kv_rows, W("qk_norm"), pos3, self.inv_t,
                                        self.inv_hw, cfg.num_heads, cfg.num_kv_heads, cfg.rms_eps)
            else:
                from ..parallel.symm import peer_put
                fused.qknorm_rope_fwd(qkv, qk, W("qk_norm"), None, pos3, self.inv_t, self.inv_hw,
                                      cfg.num_heads, cfg.num_kv_heads, cfg.rms_eps)
                kt, vt = ws.get("i.kt", (R, kd)), ws.get("i.vt", (R, kd))
                kt.copy_(qk[:, qd:])
                vt.copy_(qkv[:, qd + kd:])
                base = l * self.sp["rows"]
                for a, n, c in publish:
                    peer_put(kt[a:a + n], self.sp["k"], (base + c) * kd)
                    peer_put(vt[a:a + n], self.sp["v"], (base + c) * kd)
                # every peer's slice of this layer is in my cache after the barrier; a peer can only come
                # back to this layer (next step) after the barriers of all later layers, i.e. after I read
                self.sp["bar"].barrier()
            k, v = self.kc[l][:kv_len], self.vc[l][:kv_len]
            if decode:
                attn_ops.attention_decode(q, k, v, plan.meta_q, plan.meta_k, plan.first, kv_rows, plan.max_keys,
                                          self.scale, o)
            else:
                attn_ops.attention_fwd(q, k, v, plan, self.scale, out=o, want_lse=False)
            gemm.gemm_nt(of, W("wo"), out=x1, residual=x, w_static=static, in_parts=True)
            fused.rmsnorm_fwd(x1, W("ffn_norm"), None, h2, None, cfg.rms_eps)
            if not cfg.is_moe:
                gemm.linear_swiglu(h2, W("w13"), out=act, w_static=static)
                x = gemm.gemm_nt(act, W("w2"), out=xo[l & 1], residual=x1, w_static=static, in_parts=True)
            else:
                # the next layer's norm rides on the experts' combination when few rows are routed
                gain = p[f"layers.{l + 1}.attn_norm"][branch] if static and R <= moe.FEW_ROWS and l + 1 < cfg.num_layers else None
                x, normed = self._moe_ffn(WE, h2, x1, branch, xo[l & 1], gain, h1), gain is not None
        return x

    def _one_launch(self, rows: int, keys: int) -> bool:
        """Whether a decode step of ``rows`` documents of up to ``keys`` keys is one launch for all layers."""
        cfg = self.cfg
        return (self.offload is None and not cfg.is_moe
                and decode_stack.takes(rows, cfg.hidden_size, cfg.ffn_size, cfg.num_heads, cfg.num_kv_heads, keys))

    def _decode_layers(self, x, branch, pos3, plan, kv_rows, kv_len):
        """:meth:`layers` for one new token of a few documents: one launch for the whole stack."""
        cfg, p = self.cfg, self.p
        if self._stack is None:
            self._stack = decode_stack.Scratch(self.dev)
        names = [f"layers.{l}.{{}}" for l in range(cfg.num_layers)]
        table = [tuple(p[n.format(w)][branch] for w in ("wqkv", "wo", "w13", "w2", "attn_norm", "qk_norm", "ffn_norm"))
                 + (self.kc[l], self.vc[l]) for l, n in enumerate(names)]
        return decode_stack.decode_stack(x, table, self.ws.get("i.x0", tuple(x.shape)), self._stack, cfg.num_heads,
                                         cfg.num_kv_heads, cfg.ffn_size, plan, kv_rows, pos3, kv_len, self.inv_t, self.inv_hw,
                                         cfg.rms_eps, self.scale)

    def _moe_ffn(self, W, h2, x1, branch, out, gain=None, h=None):
        """Dropless top-k expert FFN of one branch: device-side routing, tokens gathered into expert
        segments, one grouped GEMM per projection, weighted combine + residual (the reference loops
        over experts in Python: src/sensenova_u1/models/neo_unify/modeling_qwen3_moe.py:51-119).  With ``gain`` the norm of
        the result goes to ``h`` as well."""
        cfg, p, ws = self.cfg, self.p, self.ws
        br = "und" if branch == UND else "gen"
        K = cfg.num_experts_per_tok if branch == UND else cfg.gen_num_experts_per_tok
        R, H = h2.shape
        Fe = cfg.moe_intermediate_size
        gate = W(f"moe_{br}.gate")
        logits = gemm.gemm_nt(h2, gate, out=ws.get("i.moe.logits", (R, gate.shape[0]), torch.float32),
                              out_mode=gemm.OUT_F32_STORE, w_static=self.offload is None, in_parts=True)
        if R <= moe.FEW_ROWS:
            # Decoding: the experts' weights are streamed like those of any short product, only the experts in use.
            # One token (8 of 128 experts, 768 x 2048), whole block: 99 -> 45 us.
            r = moe.route_few(logits, K, cfg.norm_topk_prob, ws)
            # one row: every expert in use reads it where it is
            xp = h2 if R == 1 else moe.gather(h2, r, ws.get("i.moe.xp", (r.max_rows, H)))
            act = gemm.gemm_experts(xp, W(f"moe_{br}.w13"), ws.get("i.moe.act", (r.max_rows, Fe)), r.tile_group, R, swiglu=True)
            yp = gemm.gemm_experts(act, W(f"moe_{br}.w2"), ws.get("i.moe.yp", (r.max_rows, H)), r.tile_group, R)
            if gain is not None and H <= 8192:
                return moe.combine_norm(yp, r, x1, out, gain, h, cfg.rms_eps)
        else:
            r = moe.route(logits, K, cfg.norm_topk_prob)
            # rows between the experts' segments are never read: nothing is cleared
            xp = ws.get("i.moe.xp", (r.max_rows, H))
            moe.gather(h2, r, xp)
            act = gemm.linear_swiglu(xp, W(f"moe_{br}.w13"), out=ws.get("i.moe.act", (r.max_rows, Fe)),
                                     tile_group=r.tile_group)
            yp = gemm.gemm_nt(act, W(f"moe_{br}.w2"), out=ws.get("i.moe.yp", (r.max_rows, H)), tile_group=r.tile_group)
        moe.combine(yp, r, x1, out)
        if gain is not None:
            fused.rmsnorm_fwd(out, gain, None, h, None, cfg.rms_eps)
        return out

    def final_norm(self, x, branch):
        return fused.rmsnorm_fwd(x, self.p["final_norm"][branch], None, torch.empty_like(x), None, self.cfg.rms_eps)

    # ------------------------------------------------------------------- prefix
    def prefill(self, docs_ids: Sequence[torch.Tensor], reserve_image_tokens: int,
                docs_embeds: Optional[Sequence[torch.Tensor]] = None,
                docs_pos3: Optional[Sequence[torch.Tensor]] = None):
        """Understanding-branch forward of several prompts packed as documents; fills the KV
        cache.  Returns (layouts, last hidden rows [n_docs,H]).  ``docs_embeds`` / ``docs_pos3``
        override token embeddings / (t,h,w) indexes (prompts that contain images)."""
        cfg = self.cfg
        n_docs = len(docs_ids)
        lens = [int(d.numel()) for d in docs_ids]
        layouts, kv_pos = [], 0
        for n in lens:
            layouts.append(DocLayout(kv_pos, n, kv_pos + n, n))
            kv_pos += n + reserve_image_tokens
        self.alloc_cache(_pad128(kv_pos))
        # indexes and metadata are made on the host (they come from it) and go up together
        doc = torch.repeat_interleave(torch.arange(n_docs, dtype=torch.int32), torch.tensor(lens))
        if docs_pos3 is None:
            pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in lens])
            pos3 = torch.stack([pos, torch.zeros_like(pos), torch.zeros_like(pos)])
            img = None
        else:
            pos3 = torch.cat([p.cpu() for p in docs_pos3], dim=1).int().contiguous()
            pos = pos3[0]
            # tokens that share a t index with a neighbour belong to one image: bidirectional
            img = ((pos3[1] > 0) | (pos3[2] > 0) | (torch.roll(pos, 1) == pos) | (torch.roll(pos, -1) == pos)).int() * (pos + 1)
        kv_rows = torch.cat([torch.arange(lay.kv_start, lay.kv_start + n) for lay, n in zip(layouts, lens)])
        # keys: cache rows [0, kv_pos); rows not written yet are blocked
        mk = torch.zeros(kv_pos, 4, dtype=torch.int32)
        mk[:, 0] = -7
        mk[:, 3] = attn_ops.FLAG_BLOCKED
        mq = attn_ops.make_meta(doc, pos, img)
        mk[kv_rows] = mq
        self._meta_host = mk                         # as the prefill left it: decoding advances the device's copy
        ends = torch.tensor(lens).cumsum(0) - 1
        for lay, t in zip(layouts, pos[ends].tolist()):
            lay.next_pos = t + 1
        ids = None
        if docs_embeds is None:
            ids = torch.cat([d.to(docs_ids[0].device) for d in docs_ids]).long()
        pos3, kv_rows, mk, mq, last, *ids = upload(self.dev, pos3, kv_rows, mk, mq, ends, *([] if ids is None else [ids]))
        x = self.p["embed_tokens"].index_select(0, ids[0]) if docs_embeds is None else torch.cat(list(docs_embeds))
        plan = attn_ops.build_plan(mq, mk)
        x = self.layers(x.contiguous(), UND, pos3, plan, kv_rows, kv_pos)
        self._meta_k = mk
        self._doc_starts = [lay.kv_start for lay in layouts]
        return layouts, x.index_select(0, last)

    # ------------------------------------------------------------ text decoding
    def decode_greedy(self, layouts: List[DocLayout], last_hidden, max_new_tokens: int,
                      stop_ids: Sequence[int] = (), use_graph: bool = True, check_every: int = 8):
        """Greedy continuation: :meth:`decode` without sampling."""
        return self.decode(layouts, last_hidden, max_new_tokens, stop_ids, use_graph, check_every, sampling=None)

    @staticmethod
    def _pick_token(logits, sampling, seen=None):
        """Next token per row from fp32 logits.  ``sampling`` None: argmax.  Otherwise, in the order of transformers'
        logits processors: repetition penalty on the tokens marked in ``seen`` ([rows, vocab] bool: prompt and
        generated tokens; positive logits divided by the penalty, negative ones multiplied), then, with ``do_sample``,
        temperature, top-k and nucleus (top-p) filtering and a draw by the exponential-race form of categorical
        sampling (argmax of p / Exp(1)), which stays on the device and is capturable in a CUDA graph."""
        best = lambda x: (decode_stack.argmax_rows(x) if x.is_cuda and x.dtype == torch.float32 and x.dim() == 2 and x.stride(1) == 1
                          and x.stride(0) >= x.shape[1] and 0 < x.shape[0] < 65536 and x.shape[1] > 0 else x.argmax(-1))
        if not sampling:
            return best(logits)
        lg = logits.float()
        rp = float(sampling.get("repetition_penalty", 1.0) or 1.0)
        if seen is not None and rp != 1.0:
            lg = torch.where(seen, torch.where(lg > 0, lg / rp, lg * rp), lg)
        if not sampling.get("do_sample", False):
            return best(lg)
        t = float(sampling.get("temperature", 1.0) or 1.0)
        k = int(sampling.get("top_k", 0) or 0)
        p_ = float(sampling.get("top_p", 1.0) or 1.0)
        if (lg.is_cuda and lg.dim() == 2 and 0 < lg.shape[0] < 65536 and 0 < k < lg.shape[-1] and k <= fused.SAMPLER_MAX_K
                and lg.shape[-1] <= fused.SAMPLER_MAX_VOCAB):
            # the same draw in one launch: top-k first bounds what has to be sorted
            noise = torch.empty(lg.shape, dtype=lg.dtype, device=lg.device).exponential_(1.0)    # in row order for any strides
            return fused.sample_top_k_top_p(lg, noise, t, k, p_)
        if t != 1.0:
            lg = lg / t
        if 0 < k < lg.shape[-1]:
            kth = torch.topk(lg, k, dim=-1).values[..., -1:]
            lg = lg.masked_fill(lg < kth, float("-inf"))
        if p_ < 1.0:
            srt, idx = torch.sort(lg, dim=-1, descending=True)
            cum = torch.softmax(srt, dim=-1).cumsum(-1)
            drop = (cum - torch.softmax(srt, dim=-1)) > p_          # keep the token that crosses the threshold
            srt = srt.masked_fill(drop, float("-inf"))
            lg = torch.full_like(lg, float("-inf")).scatter(-1, idx, srt)
        probs = torch.softmax(lg, dim=-1)
        return (probs / torch.empty_like(probs).exponential_(1.0)).argmax(-1)

    def decode(self, layouts: List[DocLayout], last_hidden, max_new_tokens: int, stop_ids: Sequence[int] = (),
               use_graph: bool = True, check_every: int = 8, sampling: Optional[dict] = None,
               prompt_ids: Optional[Sequence[torch.Tensor]] = None):
        """Continuation of every document (understanding branch), one token per step: greedy, or sampled with
        ``sampling = {do_sample, temperature, top_k, top_p, repetition_penalty, seed}`` (the knobs of the reference's
        ``generate``, src/sensenova_u1/models/neo_unify/modeling_neo_chat.py:1916-1975, examples/vqa/inference.py:29-112).
        ``prompt_ids`` (one id tensor per document) lets the repetition penalty see the prompt as well.
        The reserved image rows of the cache are used for the new tokens; a request that runs past the end of the cache raises.

        One decode step is the final norm, the LM head, the token, what follows from it, and the layers: one launch
        for all of them where ``_one_launch`` says so, seven to ten short ones per layer otherwise.  The host takes longer to
        launch those than they run, so after one eager step the step is captured
        in a CUDA graph and replayed; all of its state (token, position, cache row, output slot)
        lives in device tensors that the graph itself advances.  The host only looks at the tokens
        every ``check_every`` steps to see whether every document has stopped."""
        n_docs = len(layouts)
        if max_new_tokens <= 0:
            return [[] for _ in range(n_docs)]
        dev = self.dev
        pos, kv_rows, first = upload(
            dev, torch.tensor([lay.next_pos for lay in layouts], dtype=torch.int32), torch.tensor([lay.img_start for lay in layouts]),
            torch.tensor(self._doc_starts[:n_docs], dtype=torch.int32))
        rows = decode_stack.Rows(pos, kv_rows, self.cfg.hidden_size, max_new_tokens)
        st = {"h": last_hidden.contiguous().clone()}
        kv_len = self._meta_k.shape[0]
        # Documents are numbered by their place in the last prefill: when the layouts are those documents in order, row
        # d reads cache rows [kv_start, its own] and nothing else can be visible to it, so its keys are split over CTAs.
        # Any other selection of layouts takes the tile plan, which looks at every cache row.
        if [lay.kv_start for lay in layouts] != self._doc_starts[:n_docs]:
            first = None
        else:
            max_keys = max(lay.img_start - lay.kv_start for lay in layouts) + max_new_tokens
        if sampling and float(sampling.get("repetition_penalty", 1.0) or 1.0) != 1.0:
            vocab = self.p["lm_head"].shape[0]
            st["seen"] = torch.zeros(n_docs, vocab, dtype=torch.bool, device=dev)      # advanced inside the graph
            for d, ids in enumerate(prompt_ids or ()):
                st["seen"][d, ids.to(dev).long().clamp_(0, vocab - 1)] = True

        def step_fn():
            logits = gemm.gemm_nt(self.final_norm(st["h"], UND), self.p["lm_head"], out_mode=gemm.OUT_F32_STORE)
            nxt = self._pick_token(logits, sampling, st.get("seen"))
            if "seen" in st:
                st["seen"].scatter_(1, nxt.view(-1, 1), True)
            rows.advance(nxt, self.p["embed_tokens"], self._meta_k)
            plan = (DecodeRows(rows.meta_q, self._meta_k, first, max_keys) if first is not None
                    else attn_ops.build_plan(rows.meta_q, self._meta_k))
            # the same buffer after every step: the captured step reads what it (or the eager one) has left there
            st["h"] = self.layers(rows.x, UND, rows.pos3, plan, rows.kv_rows, kv_len)

        done = 0
        graph = None
        stops = set(int(t) for t in stop_ids)
        room = kv_len - max(lay.img_start for lay in layouts)       # steps that the prefill left cache rows for
        if room <= 0:
            raise ValueError("decode: the prefill reserved no cache rows behind the last document")

        one_launch = first is not None and self._one_launch(n_docs, max_keys)

        def tokens():
            """The tokens so far.  A whole-stack launch that ran out of time (or follows one that did) leaves its output as it
            was: the request fails, and the next one gets fresh scratch."""
            new = rows.out[:, :done]
            if not one_launch:
                return new.tolist()
            count = self._stack.count
            *flat, st["launches"], gave_up = torch.cat([new.reshape(-1), count[:1], count[-1:]]).tolist()     # one read for all
            if gave_up:
                self._stack = None
                _lib.check_status()
                raise _lib.NativeLibraryError("decode: a launch of the whole-stack kernel ran out of time")
            return [flat[d * done:(d + 1) * done] for d in range(n_docs)]

        def finished():
            toks = tokens() if stops else []
            return all(any(t in stops for t in row) for row in toks) if stops else False

        if sampling and sampling.get("do_sample", False) and sampling.get("seed") is not None and dev.type == "cuda":
            torch.cuda.manual_seed(int(sampling["seed"]))
        step_fn()                                   # eager: also warms every lazy initialisation
        done = 1
        if use_graph and max_new_tokens > 2:
            graph = self._capture(step_fn)
        while done < max_new_tokens:
            if (done % check_every == 0 or done >= room) and finished():
                break
            if done >= room:
                raise ValueError(f"decode: the prefill reserved {room} cache rows, and not every document has stopped after as many tokens")
            if graph is not None:
                graph.replay()
            else:
                step_fn()
            done += 1
        out = []
        for row in tokens():
            cut = len(row)
            for i, t in enumerate(row):
                if t in stops:
                    cut = i + 1
                    break
            out.append(row[:cut])
        if st.get("launches", 0) > decode_stack.MAX_LAUNCHES:
            self._stack = None                      # the next request starts with fresh scratch
        for lay in layouts:                         # every executed step consumed one cache row
            lay.img_start += done
            lay.prefix_len += done
            lay.next_pos += done
        self.last_decode_steps, self.last_decode_graph = done, graph is not None
        return out

    GRAPH_POOL_LIMIT = 256 << 20     # bytes that a decode graph may keep from one request to the next

    def _capture(self, fn):
        """CUDA graph of ``fn()``.  Its temporaries come from the memory pool of the graph before it, which is kept (and
        never replayed again) for that purpose: ``torch.cuda.graph`` empties the allocator's cache first, and every request
        then paid for returning that memory to the driver and asking for it again (5 - 400 ms on a shared host).  A pool that
        has grown past ``GRAPH_POOL_LIMIT`` is not kept: it goes back to the allocator with its request's graph."""
        with torch.cuda.device(self.dev):
            cur, old = torch.cuda.current_stream(), self._graph
            if self._capture_stream is None:         # always the same one: the pool's free blocks belong to a stream
                self._capture_stream = torch.cuda.Stream(self.dev)
            self._capture_stream.wait_stream(cur)
            before = self._reserved()
            graph = torch.cuda.CUDAGraph()
            try:
                self._record(graph, old, fn)
            except torch.cuda.OutOfMemoryError:      # the cache holds what the pool needs: let torch empty it first
                graph = None
            if graph is None:                        # here the error no longer holds on to the broken capture's memory
                self.release_decode_memory()
                old = None
                torch.cuda.synchronize()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=self._capture_stream):
                    before = self._reserved()
                    fn()
            cur.wait_stream(self._capture_stream)
            self._graph_bytes += max(0, self._reserved() - before)
            self._graph = graph
            if self._graph_bytes > self.GRAPH_POOL_LIMIT:
                self.release_decode_memory()
        return graph

    def _reserved(self) -> int:
        # memory_reserved() without its flat copy of all counters
        return torch.cuda.memory_stats_as_nested_dict(self.dev)["reserved_bytes"]["all"]["current"]

    def _record(self, graph, old, fn):
        with torch.cuda.stream(self._capture_stream):
            graph.capture_begin(pool=None if old is None else old.pool())
            try:
                fn()
            except BaseException:
                try:
                    graph.capture_end()
                except RuntimeError:                 # a broken capture: what broke it is the error to report
                    pass
                raise
            graph.capture_end()

    def release_decode_memory(self) -> None:
        """Gives the memory that the last decode graph keeps for the next one back to the allocator."""
        self._graph, self._graph_bytes = None, 0

    # --------------------------------------------------------------- generation
    @torch.no_grad()
    def t2i(self, cond_ids: torch.Tensor, uncond_ids: Optional[torch.Tensor], image_size=(256, 256),
            num_steps: int = 50, cfg_scale: float = 4.0, timestep_shift: float = 3.0,
            cfg_norm: str = "none", cfg_interval=(0.0, 1.0), t_eps: float = 0.02, seed: int = 0,
            batch_size: int = 1, noise: Optional[torch.Tensor] = None, cfg_group=None, par_group=None):
        """Text-to-image: returns pixels [B,3,H,W] float32 in [-1,1].  ``image_size`` = (W,H).
        ``cfg_group``: two ranks, one per guidance branch; ``par_group``: all ranks of a guidance-parallel x
        sequence-parallel run (see :meth:`denoise`)."""
        use_cfg = cfg_scale > 1 and uncond_ids is not None
        branches = [(cond_ids, None, None)] + ([(uncond_ids, None, None)] if use_cfg else [])
        return self.denoise([branches] * batch_size, image_size, num_steps, cfg_scale, 0.0, timestep_shift,
                            cfg_norm, cfg_interval, t_eps, seed, noise, cfg_group=cfg_group if use_cfg else None,
                            par_group=par_group)

    def _cfg_parallel(self, group, nb: int, numel: int, par_group=None):
        """Exchange state of parallel sampling: two symmetric prediction buffers ([branches][B*T][token_dim])
        and a flag barrier over ``par_group``, the ranks that exchange predictions (default: ``group``)."""
        import torch.distributed as dist
        from ..parallel.symm import FlagBarrier, SymmetricBuffer
        if group is not None and dist.get_world_size(group) != nb:
            raise ValueError(f"guidance-parallel sampling needs one rank per branch ({nb}), "
                             f"group has {dist.get_world_size(group)}")
        par_group = par_group if par_group is not None else group
        st = getattr(self, "_cfgpar", None)
        if st is None or st["numel"] < numel or st["nb"] != nb or st["group"] is not par_group:
            st = {"numel": numel, "nb": nb, "rank": dist.get_rank(group) if group is not None else None,
                  "group": par_group, "bar": FlagBarrier(par_group, self.dev),
                  "x": [SymmetricBuffer(nb * numel, torch.bfloat16, self.dev, par_group) for _ in range(2)]}
            self._cfgpar = st
        return st

    @torch.no_grad()
    def denoise(self, samples, image_size=(256, 256), num_steps: int = 50, cfg_scale: float = 4.0,
                img_cfg_scale: float = 1.0, timestep_shift: float = 3.0, cfg_norm: str = "none",
                cfg_interval=(0.0, 1.0), t_eps: float = 0.02, seed: int = 0, noise: Optional[torch.Tensor] = None,
                cfg_group=None, par_group=None):
        """Flow-matching Euler sampling of one image per sample.

        Sequence-parallel sampling (after :meth:`enable_sequence_parallel`): every rank of the group runs the
        decoder on its contiguous slice of each image's tokens; keys / values are exchanged per layer, the
        predictions per step, through peer memory.  Combines with ``cfg_group`` (ranks = branches x slices;
        ``par_group`` is then the group of all of them, default the world group).

        ``cfg_group``: guidance-parallel sampling.  A process group with one rank per guidance branch
        (2 for text-to-image, 3 for editing): rank r runs branch r only, stores its prediction into
        every rank's symmetric buffer with peer stores, and after a device-side flag barrier every
        rank applies the same fused guidance + Euler step, so the latents stay bit-identical without a
        broadcast.  The reference has no multi-GPU sampler (docs/inference_infra.md:20-21 points to
        an external engine for CFG/SP parallelism).

        ``samples[b]`` lists the guidance branches of sample b as (ids, embeds or None, pos3 or None):
        branch 0 the full condition, branch 1 the unconditional prompt, branch 2 (editing /
        interleaved generation) the image-only condition; v = v_u + s_t (v_c - v_i) + s_i (v_i - v_u)
        (modeling_neo_chat.py:1606-1663).  Every branch of every sample is one document of the same
        packed forward.  Returns pixels [B,3,H,W] in [-1,1]."""
        cfg = self.cfg
        W, Hh = image_size
        tp = cfg.token_pixels
        th, tw = Hh // tp, W // tp
        T = th * tw
        batch_size = len(samples)
        nb = len(samples[0])
        par = None
        sp = self.sp
        if sp is not None and (T % (128 * sp["world"]) != 0):
            raise ValueError(f"sequence-parallel sampling needs the image token count ({T}) to be a multiple of "
                             f"128 x {sp['world']} ranks")
        use_cfg_par = cfg_group is not None and nb > 1
        if use_cfg_par or sp is not None:
            import torch.distributed as dist
            if use_cfg_par and sp is not None and par_group is None:
                par_group = dist.group.WORLD
            par = self._cfg_parallel(cfg_group if use_cfg_par else None, nb, batch_size * T * cfg.token_dim,
                                     par_group if par_group is not None else (cfg_group if use_cfg_par else sp["group"]))
            if use_cfg_par:
                samples = [[smp[par["rank"]]] for smp in samples]       # my guidance branch only
        nb_all, nb = nb, len(samples[0])
        Tl = T // sp["world"] if sp is not None else T                   # image tokens of one document on this rank
        s0 = sp["rank"] * Tl if sp is not None else 0
        prompts = [br for smp in samples for br in smp]
        has_emb = any(e is not None for _, e, _ in prompts)
        layouts, _ = self.prefill([p[0] for p in prompts], reserve_image_tokens=T,
                                  docs_embeds=[p[1] if p[1] is not None else self.p["embed_tokens"].index_select(
                                      0, p[0].to(self.dev).long()) for p in prompts] if has_emb else None,
                                  docs_pos3=[p[2] if p[2] is not None else torch.stack(
                                      [torch.arange(p[0].numel()), torch.zeros(p[0].numel(), dtype=torch.long),
                                       torch.zeros(p[0].numel(), dtype=torch.long)]) for p in prompts] if has_emb else None)
        n_docs = len(prompts)
        hh = torch.arange(th, dtype=torch.int32).view(th, 1).expand(th, tw).reshape(-1)
        ww = torch.arange(tw, dtype=torch.int32).view(1, tw).expand(th, tw).reshape(-1)
        # rows are grouped by branch: [all conditional images | all unconditional | all image-only]
        order = [i for k in range(nb) for i in range(n_docs) if i % nb == k]
        pos3 = torch.cat([torch.stack([torch.full((T,), layouts[i].next_pos, dtype=torch.int32), hh, ww]) for i in order], dim=1)
        kv_rows = torch.cat([torch.arange(layouts[i].img_start, layouts[i].img_start + T) for i in order])
        doc = torch.cat([torch.full((T,), i, dtype=torch.int32) for i in order])
        mk = self._meta_host.clone()
        mk[kv_rows] = attn_ops.make_meta(doc, torch.zeros_like(doc))
        m, ps = cfg.merge_size, cfg.patch_size
        ty = hh.view(-1, 1, 1) * m + torch.arange(m, dtype=torch.int32).view(1, m, 1)
        tx = ww.view(-1, 1, 1) * m + torch.arange(m, dtype=torch.int32).view(1, 1, m)
        py = ty.expand(T, m, m).reshape(-1).repeat(batch_size)
        px = tx.expand(T, m, m).reshape(-1).repeat(batch_size)
        pos3, kv_rows, mq, mk, px, py = upload(self.dev, pos3, kv_rows, attn_ops.make_meta(doc, torch.full_like(doc, 1 << 28)), mk,
                                               px, py)
        publish = None
        if sp is not None:
            # my rows: the slice [s0, s0 + Tl) of every document, in the same document order
            loc = torch.cat([torch.arange(j * T + s0, j * T + s0 + Tl) for j in range(len(order))]).to(self.dev)
            pos3 = pos3.index_select(1, loc).contiguous()
            kv_rows = kv_rows.index_select(0, loc)
            mq = mq.index_select(0, loc).contiguous()
            publish = [(j * Tl, Tl, layouts[i].img_start + s0) for j, i in enumerate(order)]
        plan = attn_ops.build_plan(mq, mk)
        kv_len = mk.shape[0]
        ns = min(math.sqrt(T / float(cfg.noise_scale_base_image_seq_len)) * cfg.noise_scale
                 if cfg.noise_scale_mode in ("resolution", "dynamic", "dynamic_sqrt") else cfg.noise_scale,
                 cfg.noise_scale_max_value)
        if noise is None:
            g = torch.Generator(device=self.dev).manual_seed(seed)
            noise = torch.randn(batch_size, 3, Hh, W, device=self.dev, generator=g)
        img = ns * noise.float()
        z = img.reshape(batch_size, 3, th, tp, tw, tp).permute(0, 2, 4, 3, 5, 1).reshape(batch_size * T, cfg.token_dim).contiguous()
        patches = z.reshape(batch_size * T, m, ps, m, ps, 3).permute(0, 1, 3, 5, 2, 4).reshape(
            batch_size * T * m * m, cfg.patch_dim).to(torch.bfloat16).contiguous()
        ts = torch.linspace(0.0, 1.0, num_steps + 1)
        ts = apply_time_schedule(ts, T, cfg, timestep_shift=timestep_shift).tolist()
        ns_emb = None
        if cfg.add_noise_scale_embedding:
            ns_emb = self.scalar_embed("noise_scale_embedder", torch.full((1,), ns / cfg.noise_scale_max_value, device=self.dev))
        BT = batch_size * T
        BTl = batch_size * Tl
        m2 = m * m
        if sp is not None:
            prow = torch.cat([torch.arange((b * T + s0) * m2, (b * T + s0 + Tl) * m2) for b in range(batch_size)]).to(self.dev)
            px_l, py_l = px.index_select(0, prow).contiguous(), py.index_select(0, prow).contiguous()
        plan_c = None
        for step in range(num_steps):
            t, t_next = ts[step], ts[step + 1]
            if sp is not None:
                emb = self.vision_embed("gen", patches.index_select(0, prow), px_l, py_l)
            else:
                emb = self.vision_embed("gen", patches, px, py)
            e_t = self.scalar_embed("timestep_embedder", torch.full((1,), t, device=self.dev))
            emb = emb + (e_t + ns_emb if ns_emb is not None else e_t)
            in_interval = cfg_interval[0] <= t <= cfg_interval[1]
            branches = nb if (nb > 1 and in_interval) else 1
            if use_cfg_par:
                branches = nb_all if in_interval else 1
            if branches == nb or use_cfg_par:
                x = emb if nb == 1 else torch.cat([emb] * nb, 0)
                h = self.layers(x.contiguous(), GEN, pos3, plan, kv_rows, kv_len, publish)
            else:  # outside the guidance interval only the conditional documents run
                sub = slice(0, BTl)
                if plan_c is None:
                    plan_c = attn_ops.build_plan(mq[sub].contiguous(), mk)
                h = self.layers(emb.contiguous(), GEN, pos3[:, sub].contiguous(), plan_c, kv_rows[sub], kv_len,
                                publish[:batch_size] if publish is not None else None)
            hf = self.final_norm(h, GEN)
            if cfg.use_pixel_head:
                # convolutional decoder: cuDNN convolutions on the token grids (not a tcgen05 path)
                x_pred = oracle.pixel_head(self.p, hf, [(th, tw)] * (hf.shape[0] // T), cfg).to(torch.bfloat16).contiguous()
            else:
                a1 = gemm.gemm_nt(hf, self.p["fm_head.w1"], residual=self.p["fm_head.b1"], w_static=True)
                fused.gelu_fwd(a1, a1)
                x_pred = gemm.gemm_nt(a1, self.p["fm_head.w2"], residual=self.p["fm_head.b2"], w_static=True)
            if par is not None:
                from ..parallel.symm import peer_put
                buf = par["x"][step & 1]                     # two buffers: a slow peer may still read the other
                if sp is None:
                    peer_put(x_pred, buf, par["rank"] * BT * cfg.token_dim)
                else:
                    # my token slice of every (branch, sample) goes to its place in every rank's buffer
                    for k in range(x_pred.shape[0] // BTl):
                        kb = par["rank"] if use_cfg_par else k
                        for b in range(batch_size):
                            peer_put(x_pred[(k * batch_size + b) * Tl:(k * batch_size + b + 1) * Tl], buf,
                                     ((kb * batch_size + b) * T + s0) * cfg.token_dim)
                par["bar"].barrier()
                x_pred = buf.tensor
            _lib.call("sampler_step", c_void_p(x_pred.data_ptr()), c_void_p(z.data_ptr()),
                      c_void_p(patches.data_ptr()), c_void_p(self.stats.data_ptr()), c_int(BT),
                      c_int(cfg.token_dim), c_int(branches), c_int(ps), c_int(m), c_float(t), c_float(t_next),
                      c_float(t_eps), c_float(cfg_scale), c_float(img_cfg_scale), c_int(1 if branches > 1 else 0),
                      c_int(CFG_NORMS[cfg_norm]), c_int(1 if step == 0 else 0), c_void_p(_lib.stream()))
        self.last_layouts = layouts
        return z.reshape(batch_size, th, tw, tp, tp, 3).permute(0, 5, 1, 3, 2, 4).reshape(batch_size, 3, Hh, W)
