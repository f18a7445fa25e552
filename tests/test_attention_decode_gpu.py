"""Decode attention (csrc/attn_decode.cu) against the fp32 dense reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1, 3, 16])
@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (4, 2), (8, 2), (16, 2)])       # 1, 2, 4 and 8 query heads per K/V head
@pytest.mark.parametrize("lens", [[1], [63, 64, 65], [1, 700, 2, 129, 300]])   # rows of a step: 64
def test_ragged_documents(lens, Hq, Hkv, split):
    from sensenova_u1_b200.ops import attention as A
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(sum(lens) + Hq)
    spare = 5                                                   # rows of a document that nothing has written yet
    starts, n = [], 0
    for x in lens:
        starts.append(n)
        n += x + spare
    q = torch.randn(len(lens), Hq, 128, device=dev, generator=g).to(torch.bfloat16)
    # keys and values as slices of wider rows, as a cache row holds all heads
    k = torch.randn(n, Hkv, 128, device=dev, generator=g).to(torch.bfloat16)
    v = torch.randn(n, Hkv, 128, device=dev, generator=g).to(torch.bfloat16)
    meta_k = torch.zeros(n, 4, dtype=torch.int32, device=dev)
    meta_k[:, 0], meta_k[:, 3] = -7, A.FLAG_BLOCKED
    for d, (s, x) in enumerate(zip(starts, lens)):
        meta_k[s:s + x] = A.make_meta(torch.full((x,), d, device=dev), torch.arange(x, device=dev))
    if lens[0] > 2:
        meta_k[1, 3] = A.FLAG_BLOCKED                           # a hole inside the range
    pos = torch.tensor(lens, dtype=torch.int32, device=dev) - 1
    if len(lens) > 3:
        pos[3] = 40                                             # a query that may not read the later keys
    meta_q = A.make_meta(torch.arange(len(lens), device=dev), pos)
    first = torch.tensor(starts, dtype=torch.int32, device=dev)
    last = torch.tensor([s + x - 1 for s, x in zip(starts, lens)], dtype=torch.long, device=dev)
    out = torch.full_like(q, float("nan"))
    A.attention_decode(q, k, v, meta_q, meta_k, first, last, max(lens), 128 ** -0.5, out, split=split)
    ref = A.reference_attention(q, k, v, meta_q, meta_k, 128 ** -0.5)
    # one rounding to bf16 at the end: half of the last of 8 bits, 2^-8 of the value; before it fp32 sums of up to 700
    # products with |v| < 4.5 on both sides, 700 * 4.5 * 2^-24 = 2e-4 (the approximate exponentials are good to 2^-22)
    assert ((out.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 2e-4).all()


def test_row_without_keys_is_zero():
    from sensenova_u1_b200.ops import attention as A
    q = torch.ones(1, 4, 128, device="cuda", dtype=torch.bfloat16)
    k = torch.ones(70, 1, 128, device="cuda", dtype=torch.bfloat16)
    mk = A.make_meta(torch.full((70,), 3, device="cuda"), torch.arange(70, device="cuda"))
    mq = A.make_meta(torch.zeros(1, device="cuda", dtype=torch.int32), torch.full((1,), 99, device="cuda"))
    for hi in (-1, 69):
        out = torch.full_like(q, float("nan"))
        A.attention_decode(q, k, k, mq, mk, torch.zeros(1, dtype=torch.int32, device="cuda"),
                           torch.full((1,), hi, dtype=torch.long, device="cuda"), 70, 0.1, out)
        assert (out == 0).all()


@pytest.mark.parametrize("order", [[0, 1, 2], [2, 0]])
def test_decoding_splits_keys_only_for_the_prefilled_documents(order, monkeypatch):
    """Any other selection of layouts keeps the tile plan; both give the same tokens for the documents in order."""
    from sensenova_u1_b200.config import tiny_mot
    from sensenova_u1_b200.inference import engine as E
    from sensenova_u1_b200.models.params import ParamStore
    cfg = tiny_mot(head_dim=128, patch_size=16)
    store = ParamStore(cfg, device="cuda:0", with_grads=False)
    store.init_weights(3)
    eng = E.InferenceEngine(cfg, store)
    docs = [torch.arange(5, 5 + n) for n in (9, 70, 3)]
    real, used = E.attn_ops.attention_decode, []
    monkeypatch.setattr(E.attn_ops, "attention_decode", lambda *a, **k: (used.append(1), real(*a, **k))[1])
    lay, h = eng.prefill(docs, reserve_image_tokens=8)
    got = eng.decode([lay[i] for i in order], h[order], 5)
    assert bool(used) == (order == [0, 1, 2])
    if order == [0, 1, 2]:
        lay, h = eng.prefill(docs, reserve_image_tokens=8)
        eng._doc_starts = []                                    # as if the documents were others: the tile plan
        assert eng.decode(lay, h, 5) == got
