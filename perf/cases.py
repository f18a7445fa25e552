"""Representative workloads of the framework, each one call sequence of its public entry points.

Four kinds of work, over the sizes they are used at:

* ``t2i`` / ``edit``: flow-matching image sampling (``InferenceEngine.t2i``, ``NEOChatModel.it2i_generate``): prompt
  prefill, then a few Euler steps with classifier-free guidance.  A released image takes 50 steps; the cost of a
  pass is linear in them.
* ``chat``: a text request, one conversation or a batch of them: prefill with a K/V cache, then decoding
  (``InferenceEngine.prefill`` / ``decode``; with a picture ``NEOChatModel.generate``).
* ``prefill``: one long prompt read into the cache.
* ``train``: one optimizer step of packed multimodal fine-tuning from pinned host batches (``Trainer.train_step``):
  forward, backward, AdamW.

All layers of a model have the same shape, so the presets run at full width with fewer layers: 12 of the 8B-MoT's 42
for inference, 2 or 3 for training, 8 or 2 of the A3B-MoT's 48.
"""
from __future__ import annotations

import gc
import math

import torch

from sensenova_u1_b200.config import get_config
from sensenova_u1_b200.data.synthetic import interleaved_batch, synthetic_batch
from sensenova_u1_b200.inference.api import ByteTokenizer, NEOChatModel
from sensenova_u1_b200.models.params import ParamStore
from sensenova_u1_b200.train.freeze import frozen_ranges
from sensenova_u1_b200.train.optimizer import AdamConfig
from sensenova_u1_b200.train.trainer import Trainer

EOS = 5                     # a reserved id that the greedy chains below never reach: requests run to their length
NO_IMAGE = 0
CFG_SCALE = 4.0


def listed():
    return [
        # a thumbnail / preview: 64 image tokens per guidance branch, bound by launches and weight reads
        dict(name="t2i_256", kind="t2i", layers=12, width=256, height=256, prompt=40, batch=1, steps=5, norm="none"),
        # the common preview resolution, two images of one prompt, guidance renormalised per sample
        dict(name="t2i_1024", kind="t2i", layers=12, width=1024, height=1024, prompt=120, batch=2, steps=3, norm="global"),
        # the headline resolution: 4096 image tokens per branch
        dict(name="t2i_2048", kind="t2i", layers=12, width=2048, height=2048, prompt=256, batch=1, steps=2, norm="none"),
        # editing a photograph of odd proportions (29 x 37 tokens): three guidance branches, one with the picture only
        dict(name="edit_odd", kind="edit", layers=12, width=1184, height=928, prompt=60, batch=1, steps=3, norm="none"),
        # a short chat turn: one sequence, latency of a token
        dict(name="chat_short", kind="chat", model="8b-mot", layers=12, docs=1, prompt=37, new=32, width=NO_IMAGE,
             height=NO_IMAGE, sample=False),
        # a question about a picture (24 x 32 tokens), answered with nucleus sampling
        dict(name="chat_picture", kind="chat", model="8b-mot", layers=12, docs=1, prompt=71, new=24, width=1024, height=768,
             sample=True),
        # a batch of conversations of ragged length decoded together
        dict(name="chat_batch", kind="chat", model="8b-mot", layers=12, docs=24, prompt=1500, new=24, width=NO_IMAGE,
             height=NO_IMAGE, sample=False),
        # the mixture-of-experts model answering a short turn
        dict(name="chat_moe", kind="chat", model="a3b-mot", layers=8, docs=1, prompt=90, new=24, width=NO_IMAGE, height=NO_IMAGE,
             sample=False),
        # a document at the documented context length (32 K), not a multiple of any tile
        dict(name="prefill_long", kind="prefill", layers=12, prompt=32001),
        # generation pre-training with the convolutional pixel head, understanding branch frozen, short packed sequence
        dict(name="train_pixel_head", kind="train", model="8b-mot", layers=2, seq=4096, data="packed", head=True, policy="none"),
        # the headline fine-tuning step: 16384 packed tokens, every layer recomputed in backward as on one GPU
        dict(name="train_16k", kind="train", model="8b-mot", layers=3, seq=16384, data="packed", head=False, policy="full"),
        # mixture-of-experts fine-tuning at its packed length
        dict(name="train_moe", kind="train", model="a3b-mot", layers=2, seq=8192, data="packed", head=False, policy="full"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["t2i", "t2i", "edit", "chat", "chat", "chat", "prefill", "train", "train"])
    if kind in ("t2i", "edit"):
        tokens = _log(rng, 64, 4096 if kind == "t2i" else 1073)
        cols = max(4, min(int(round(math.sqrt(tokens) * math.exp(rng.uniform(-0.4, 0.4)))), tokens // 4))
        rows = max(4, tokens // cols)
        batch = 1 if rows * cols > 1024 else rng.choice([1, 1, 2])
        steps = 2 if rows * cols > 1024 else 3
        return dict(kind=kind, layers=12, width=32 * cols, height=32 * rows, prompt=_log(rng, 10, 256),
                    batch=1 if kind == "edit" else batch, steps=steps, norm=rng.choice(["none", "none", "global", "channel"]))
    if kind == "chat":
        model = rng.choice(["8b-mot", "8b-mot", "a3b-mot"])
        docs = rng.choice([1, 1, 1, _log(rng, 2, 24)])
        picture = docs == 1 and rng.random() < 0.3
        return dict(kind="chat", model=model, layers=12 if model == "8b-mot" else 8, docs=docs,
                    prompt=_log(rng, 12, 1500), new=rng.randint(12, 32 if docs == 1 else 24), width=32 * rng.randint(8, 32) if picture else NO_IMAGE,
                    height=32 * rng.randint(8, 32) if picture else NO_IMAGE, sample=rng.random() < 0.3)
    if kind == "prefill":
        return dict(kind="prefill", layers=12, prompt=_log(rng, 200, 32001))
    if rng.random() < 0.3:
        return dict(kind="train", model="a3b-mot", layers=2, seq=128 * rng.randint(8, 64), data="packed", head=False,
                    policy="full")
    head = rng.random() < 0.3
    seq = 128 * (_log(rng, 16, 48) if head else _log(rng, 16, 128))
    data = "interleaved" if seq >= 4096 and not head and rng.random() < 0.4 else "packed"
    return dict(kind="train", model="8b-mot", layers=2, seq=seq, data=data, head=head,
                policy=rng.choice(["full", "attention", "none"]))


# ------------------------------------------------------------------------------------------------- preparation
def _as_trained(store, seed):
    """What a trained model's heads have and random ones lack.  It is sure of most tokens, where random weights choose
    between nearly equal ones by their rounding: the embeddings get unit scale and the LM head answers id + 1.  Its
    picture predictions with and without the prompt agree for the larger part, so that guidance does not blow up
    rounding: the generation head gets a common picture and a twelfth of the random part."""
    p = store.p
    p["embed_tokens"].mul_(50.0)
    p["lm_head"].copy_(torch.roll(p["embed_tokens"], 1, 0).mul_(0.02))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    p["fm_head.b2"].copy_(torch.rand(p["fm_head.b2"].shape, device="cuda", generator=gen) * 2 - 1)
    p["fm_head.w2"].mul_(1 / 12)


def _model(case, seed):
    cfg = get_config(case.get("model", "8b-mot"), num_layers=case["layers"])
    store = ParamStore(cfg, device="cuda", with_grads=False)
    store.init_weights(seed)
    _as_trained(store, seed)
    return cfg, NEOChatModel(cfg, store)


def _ids(cfg, n, gen):
    return torch.randint(8, cfg.vocab_size // 2, (n,), generator=gen)


def _lengths(case):
    """Ragged prompt lengths of a batch of conversations: from a few tokens up to the longest."""
    n, top = case["docs"], case["prompt"]
    return [max(9, top * (i * 7919 % n + 1) // n) for i in range(n)]


def prepare(case, seed):
    gen = torch.Generator().manual_seed(seed)
    kind = case["kind"]
    if kind == "train":
        return _prepare_training(case, seed)
    cfg, model = _model(case, seed)
    st = dict(case=case, cfg=cfg, model=model, seed=seed)
    if kind == "t2i":
        st["cond"] = _ids(cfg, case["prompt"], gen).pin_memory()
        st["uncond"] = _ids(cfg, 8, gen).pin_memory()
    elif kind == "edit":
        st["tokenizer"] = ByteTokenizer(cfg.vocab_size)
        st["text"] = "".join(chr(97 + int(i)) for i in torch.randint(0, 26, (case["prompt"],), generator=gen))
        # a decoded picture in host memory, ImageNet-normalised, as the image loader returns it
        st["image"] = torch.rand(3, case["height"], case["width"], generator=gen) * 4 - 2
    elif kind == "prefill":
        st["docs"] = [_ids(cfg, case["prompt"], gen)]
    elif case["width"]:
        # prompt with the picture's placeholder run in front, patches as the picture processor emits them
        m = cfg.merge_size
        gh, gw = case["height"] // cfg.patch_size, case["width"] // cfg.patch_size
        ctx = 1
        model.img_context_token_id = ctx
        n = (gh // m) * (gw // m)
        st["ids"] = torch.cat([torch.full((n,), ctx), _ids(cfg, case["prompt"], gen)])[None]
        st["patches"] = torch.randn(gh * gw, cfg.patch_dim, generator=gen)
        st["grid"] = torch.tensor([[gh, gw]])
    else:
        st["docs"] = [_ids(cfg, n, gen) for n in _lengths(case)]
    return st


def _prepare_training(case, seed):
    gc.collect()            # a trainer and its engine refer to each other: a dropped one is freed by the collector
    kw = dict(num_layers=case["layers"])
    if case["head"]:
        kw.update(use_pixel_head=True, ce_loss_weight=0.0)
    cfg = get_config(case["model"], **kw)
    store = ParamStore(cfg, device="cuda")
    store.init_weights(seed)
    adam = AdamConfig(lr=2e-4, beta2=0.95, clip_grad_norm=1.0, state_dtype="fp32")
    if case["head"]:
        adam.frozen = frozen_ranges(store, freeze_llm=True, freeze_backbone=True, unfreeze_mot_gen=True)
    trainer = Trainer(cfg, store, adam, max_tokens=case["seq"])
    trainer.engine.recompute = case["policy"]
    if case["head"]:
        trainer.engine.skip_wgrad_groups = (0,)
    if case["data"] == "interleaved":
        batch = interleaved_batch(cfg, case["seq"], seed=seed)
    else:                                   # the pixel head trains on text-to-image samples only
        batch = synthetic_batch(cfg, case["seq"], seed=seed, gen_frac=1.0 if case["head"] else 0.5)
    return dict(case=case, store=store, trainer=trainer, batch=batch.pin())


# ---------------------------------------------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "train":
        out = st["trainer"].train_step([st["batch"]])
        store = st["store"]
        got = {"weights": store.arena["mat"], "gains": store.arena["vec"], "losses": [out["loss"], out["ce"], out["fm"]]}
        if not store.cfg.is_moe:
            # the gradient of every matrix but the two of the vocabulary, where a few rows of frequent ids hold nearly all
            # of it (the embedding's are summed by bf16 atomics, in an order that changes from run to run); their updates
            # are in the weights.  Expert gradients move by a token when a router tie breaks the other way, so the
            # mixture model returns its updated weights only.
            got["grads"] = {s.name: store.g[s.name] for s in store.specs
                            if s.arena == "mat" and s.name not in ("embed_tokens", "lm_head")}
        return got
    model = st["model"]
    eng = model.engine
    if kind == "t2i":
        return eng.t2i(st["cond"], st["uncond"], image_size=(case["width"], case["height"]), num_steps=case["steps"],
                       cfg_scale=CFG_SCALE, timestep_shift=3.0, cfg_norm=case["norm"], seed=st["seed"], batch_size=case["batch"])
    if kind == "edit":
        return model.it2i_generate(st["tokenizer"], st["text"], [st["image"]], cfg_scale=CFG_SCALE, img_cfg_scale=1.0,
                                   cfg_norm=case["norm"], num_steps=case["steps"], batch_size=case["batch"], seed=st["seed"])
    if kind == "prefill":
        with torch.no_grad():
            _, hidden = eng.prefill(st["docs"], reserve_image_tokens=128)
        return {"hidden": hidden, "keys": eng.kc, "values": eng.vc}
    sampling = dict(do_sample=True, temperature=0.7, top_p=0.9, top_k=50, seed=st["seed"]) if case["sample"] else {}
    if case["width"]:
        tokens = model.generate(pixel_values=st["patches"], input_ids=st["ids"], grid_hw=st["grid"], max_new_tokens=case["new"],
                                eos_token_id=EOS, **sampling)
        return {"tokens": tokens, "keys": eng.kc, "values": eng.vc}
    with torch.no_grad():
        layouts, hidden = eng.prefill(st["docs"], reserve_image_tokens=case["new"])
        tokens = eng.decode(layouts, hidden, case["new"], stop_ids=(EOS,), sampling=sampling or None)
    return {"tokens": torch.tensor(tokens), "hidden": hidden, "keys": eng.kc, "values": eng.vc}


# --------------------------------------------------------------------------------------------- work and tolerance
def _layer(cfg):
    """(parameters read, multiply-adds per token) of one decoder layer of one branch."""
    attn = cfg.hidden_size * (2 * cfg.q_dim + 2 * cfg.kv_dim)
    if cfg.is_moe:
        one = 3 * cfg.hidden_size * cfg.moe_intermediate_size
        return attn, attn + cfg.num_experts_per_tok * one, one
    ffn = 3 * cfg.hidden_size * cfg.ffn_size
    return attn + ffn, attn + ffn, 0


def _layer_bytes(cfg, tokens, experts):
    dense, _, one = _layer(cfg)
    used = experts * (1 - (1 - 1 / experts) ** (tokens * cfg.num_experts_per_tok)) if cfg.is_moe else 0
    return 2 * (dense + used * one)


def _attention(cfg, pairs):
    return 4 * cfg.q_dim * pairs


def _prefill(cfg, lens):
    n, L = sum(lens), cfg.num_layers
    flops = 2 * n * _layer(cfg)[1] * L + _attention(cfg, sum(x * (x + 1) / 2 for x in lens)) * L
    nbytes = _layer_bytes(cfg, n, cfg.num_experts or 1) * L + n * (2 * cfg.hidden_size + 4 * cfg.kv_dim * L)
    return nbytes, flops


def work(case):
    cfg = get_config(case.get("model", "8b-mot"), num_layers=case["layers"])
    L, H, V = cfg.num_layers, cfg.hidden_size, cfg.vocab_size
    kind = case["kind"]
    if kind == "train":
        # forward + backward without recomputation: three products per weight and token; about half of the tokens carry a
        # label (LM head).  A document is about 2000 tokens.  AdamW: weights, master remainder, two moments and gradient.
        S = case["seq"]
        half = 2 if case["head"] else 3                              # frozen branch: no weight gradients there
        doc = S if case["data"] == "interleaved" else min(S, 2000)
        flops = 2 * half * S * _layer(cfg)[1] * L + 3.5 * _attention(cfg, S * doc / 2) * L
        flops += 0 if case["head"] else 2 * 3 * (S // 3) * H * V
        n = cfg.num_params()
        touched = n if not case["head"] else n - (V * H * 2 + L * _layer(cfg)[0])
        return {"bytes": 2 * 2 * (n - V * H) + 24.0 * touched, "flops": flops}
    if kind == "prefill":
        b, f = _prefill(cfg, [case["prompt"]])
        return {"bytes": b, "flops": f}
    if kind in ("t2i", "edit"):
        T = (case["width"] // 32) * (case["height"] // 32)
        tail = 260                                                   # template and system prompt around an edit request
        prompts = [case["prompt"], 8] if kind == "t2i" else [T + tail + case["prompt"], 20, T + tail]
        b, f = _prefill(cfg, prompts * case["batch"])
        rows = T * case["batch"] * len(prompts)
        per_step = 2 * rows * _layer(cfg)[1] * L + 2 * T * case["batch"] * 4 * cfg.vision_hidden * (cfg.patch_dim + H)
        per_step += 2 * rows * cfg.fm_head_dim * (H + cfg.token_dim)
        per_step += sum(_attention(cfg, T * (T + p)) for p in prompts) * case["batch"] * L
        step_bytes = _layer_bytes(cfg, rows, cfg.gen_num_experts or 1) * L + 2 * cfg.fm_head_dim * (H + cfg.token_dim)
        step_bytes += sum(4 * cfg.kv_dim * (T + p) for p in prompts) * case["batch"] * L + 8 * T * case["batch"] * cfg.token_dim
        return {"bytes": b + case["steps"] * step_bytes, "flops": f + case["steps"] * per_step}
    lens = [case["prompt"] + (case["width"] // 32) * (case["height"] // 32)] if case["width"] else _lengths(case)
    b, f = _prefill(cfg, lens)
    n = len(lens)
    for i in range(case["new"]):
        b += _layer_bytes(cfg, n, cfg.num_experts or 1) * L + 2 * V * H + 4 * cfg.kv_dim * L * (sum(lens) + n * i)
        f += 2 * n * (_layer(cfg)[1] * L + V * H) + _attention(cfg, sum(lens) + n * i) * L
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Measured by rounding the decoder's input the other way (up to one unit in the last place of bf16), which moves the
    hidden state and the cached keys and values by up to 2.2e-2, sampled pictures by up to 2.4e-2, matrix gradients by up
    to 2e-2 (the pixel front-end, the others 1e-2), and the updated weights of a mixture model by 1.3e-3."""
    if case["kind"] == "train" and case["model"] == "a3b-mot":
        return {"rel": 0.005, "max": 0.2}
    return {"rel": 0.03, "max": 0.6}
