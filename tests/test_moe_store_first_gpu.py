"""Mixture-of-experts training without cleared buffers: only the rows that pad the experts' segments are zeroed, and the
first micro-batch stores the expert gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 130, 1000])
def test_zero_pads_clears_the_padding_rows_only(R):
    from sensenova_u1_b200.ops import moe
    E, K, H = 9, 2, 64
    g = torch.Generator(device="cuda").manual_seed(R)
    logits = torch.randn(R, E, device="cuda", generator=g)
    logits[:, 4] = -30.0                                      # an expert without rows
    r = moe.route(logits, K, True)
    a = moe.zero_pads(torch.full((r.max_rows, H), 5.0, device="cuda", dtype=torch.bfloat16), r)
    want = torch.full_like(a, 5.0)
    for s, e, c in zip(r.seg_start.tolist(), r.seg_end.tolist(), r.counts.tolist()):
        want[s + c:e] = 0
    assert torch.equal(a, want)


@pytest.mark.parametrize("image", [True, False])              # without a picture the generation mixture has no rows
def test_first_micro_batch_stores_expert_gradients(image):
    from sensenova_u1_b200.config import tiny_mot
    from sensenova_u1_b200.data.synthetic import Sample, Segment, build_packed_batch, tiny_batch
    from sensenova_u1_b200.models.params import ParamStore
    from sensenova_u1_b200.ops import _lib
    from sensenova_u1_b200.train.optimizer import AdamConfig
    from sensenova_u1_b200.train.trainer import Trainer
    cfg = tiny_mot(head_dim=128, patch_size=16, num_layers=2, num_experts=8, num_experts_per_tok=2, gen_num_experts=8,
                   gen_num_experts_per_tok=2, moe_intermediate_size=128, router_aux_loss_coef=0.01)

    def batch(seed):
        if image:
            return tiny_batch(cfg, seed=seed, n_text=200, image_px=8 * 32).to("cuda")
        ids = torch.randint(8, cfg.vocab_size, (200,), generator=torch.Generator().manual_seed(seed))
        segs = [Segment("text", ids=ids[:90], loss=False), Segment("text", ids=ids[90:], loss=True)]
        return build_packed_batch([Sample(segs, task=3)], cfg, seed=seed).to("cuda")
    grads = []
    for fast in (True, False):
        store = ParamStore(cfg, device="cuda")
        store.init_weights(0, std=0.05)
        tr = Trainer(cfg, store, AdamConfig(lr=1e-2, state_dtype="fp32", clip_grad_norm=0.0))
        tr.store_first_enabled = fast
        if fast:
            store.grad_arena["mat"].fill_(float("nan"))
        batches = [batch(i) for i in range(2)]
        g = torch.Generator(device="cuda").manual_seed(1)
        noise = [torch.randn(b.gen_x16.shape, device="cuda", generator=g) for b in batches]
        tr.step_on_device(batches, lr=1e-2, noise=noise)
        _lib.check_status()
        grads.append({n: store.g[n].float().clone() for n in store.g if n.startswith("layers.") and store.g[n].dim() > 1})
    for n, a in grads[0].items():
        b = grads[1][n]
        assert torch.isfinite(a).all(), n
        # bf16 gradients of two micro-batches; the router's atomically summed statistics move them by rounding
        assert (a - b).norm() <= 2e-2 * b.norm() + 1e-6, n
