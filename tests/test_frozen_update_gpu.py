"""Frozen ranges of an optimizer step: left alone while their moments are zero, decayed as before when they are not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _trainer(moe=False, skip=False):
    from sensenova_u1_b200.config import tiny_mot
    from sensenova_u1_b200.models.params import ParamStore
    from sensenova_u1_b200.train.freeze import frozen_ranges
    from sensenova_u1_b200.train.optimizer import AdamConfig
    from sensenova_u1_b200.train.trainer import Trainer
    kw = dict(num_experts=8, num_experts_per_tok=2, gen_num_experts=8, gen_num_experts_per_tok=2, moe_intermediate_size=128) if moe else {}
    cfg = tiny_mot(head_dim=128, patch_size=16, num_layers=2, **kw)
    store = ParamStore(cfg, device="cuda")
    store.init_weights(0, std=0.05)
    fr = frozen_ranges(store, freeze_llm=True, freeze_backbone=True, unfreeze_mot_gen=True)
    tr = Trainer(cfg, store, AdamConfig(lr=1e-2, frozen=fr, state_dtype="fp32", clip_grad_norm=1.0, weight_decay=0.1))
    if skip:
        tr.engine.skip_wgrad_groups = (0,)
    return cfg, store, fr, tr


def _steps(cfg, tr, n=2, micro=2):
    from sensenova_u1_b200.data.synthetic import tiny_batch
    for step in range(n):
        batches = [tiny_batch(cfg, seed=10 * step + i, n_text=200, image_px=8 * 32).to("cuda") for i in range(micro)]
        g = torch.Generator(device="cuda").manual_seed(step)
        tr.step_on_device(batches, noise=[torch.randn(b.gen_x16.shape, device="cuda", generator=g) for b in batches])


def _frozen(x, ranges):
    return torch.cat([x[s:e].float() for s, e in ranges])


@pytest.mark.parametrize("moe,skip", [(False, False), (False, True), (True, False)])
def test_frozen_ranges_are_left_alone(moe, skip):
    cfg, store, fr, tr = _trainer(moe, skip)
    before = {a: t.clone() for a, t in store.arena.items()}
    for a in store.grad_arena:                                   # whatever an earlier program left there
        for s, e in fr[a]:
            store.grad_arena[a][s:e].fill_(float("nan"))
    _steps(cfg, tr)
    for a in store.sizes:
        assert torch.equal(_frozen(store.arena[a], fr[a]), _frozen(before[a], fr[a]))
        assert not _frozen(store.grad_arena[a], fr[a]).any()
        assert not _frozen(tr.optim.state[a]["m"], fr[a]).any() and not _frozen(tr.optim.state[a]["v"], fr[a]).any()
        assert torch.isfinite(store.arena[a].float()).all()
    assert not torch.equal(store.arena["mat"], before["mat"])
    # the whole update, frozen ranges included, gives the same weights; the gradient norm is summed by atomics, so a few of them
    # land on the other side of a rounding to bf16 (2^-8 of themselves)
    cfg2, store2, _, tr2 = _trainer(moe, skip)
    tr2.optim._frozen_moments_zero = False
    _steps(cfg2, tr2)
    rel = (store.arena["mat"].float() - store2.arena["mat"].float()).norm() / store2.arena["mat"].float().norm()
    assert rel < 2e-3
    assert int(tr.optim.skipped) == 0


def test_moments_of_a_loaded_state_decay():
    cfg, store, fr, tr = _trainer()
    sd = tr.optim.state_dict()
    s, e = fr["mat"][0]
    sd["state"]["mat"]["m"][s:e] = 1.0
    tr.optim.load_state_dict(sd)
    _steps(cfg, tr, n=1, micro=1)
    assert torch.allclose(tr.optim.state["mat"]["m"][s:e], torch.full((e - s,), 0.9, device="cuda"))
    sd["state"]["mat"]["m"][s:e] = 0.0
    tr.optim.load_state_dict(sd)
    assert tr.optim._frozen_moments_zero


def test_a_norm_that_is_not_finite_is_noticed():
    cfg, store, fr, tr = _trainer()
    before = store.arena["mat"].clone()
    store.p["fm_head.w2"].fill_(float("inf"))
    _steps(cfg, tr, n=1, micro=1)
    assert int(tr.optim.skipped) == 1
    for s, e in fr["mat"]:
        assert torch.equal(store.arena["mat"][s:e], before[s:e])
