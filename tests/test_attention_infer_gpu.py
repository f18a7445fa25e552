"""Attention forward without a log-sum-exp (csrc/attn_infer_sm100.cu) against dense fp32 softmax."""
import pytest
import torch

from test_attention_gpu import _meta, _rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("slots", [None, 0, 3])                       # mask bits of all, none and a few partial tiles
@pytest.mark.parametrize("S,Hq,Hkv,kind", [(1, 2, 1, "causal"), (100, 1, 1, "full"), (128, 1, 1, "full"), (129, 2, 2, "causal"),
                                           (257, 4, 1, "mixed"), (1000, 8, 2, "docs"), (1500, 4, 1, "mixed"),
                                           (2048, 8, 2, "causal")])   # one and two query tiles, tiles that only one needs
def test_matches_dense_softmax(S, Hq, Hkv, kind, slots):
    from sensenova_u1_b200.ops import _lib, attention as A
    g = torch.Generator(device=DEV).manual_seed(S)
    q, k, v = (torch.randn(S, h, 128, device=DEV, generator=g).to(torch.bfloat16) for h in (Hq, Hkv, Hkv))
    q = q * 3                                                         # maxima that move: O is rescaled
    meta = _meta(S, kind)
    out = torch.full((S + 1, Hq, 128), 7.0, device=DEV, dtype=torch.bfloat16)
    o, lse = A.attention_fwd(q, k, v, A.build_plan(meta, mask_slots=slots), 128 ** -0.5, out=out[:S], want_lse=False)
    _lib.check_status()
    assert lse is None and (out[S] == 7).all()
    ref = A.reference_attention(q, k, v, meta, meta, 128 ** -0.5)
    # P and the output are rounded to bf16: 2^-9 of a probability, 2^-9 of the value (the limits of the other kernel)
    assert _rel(o, ref) < 6e-3 and (o.float() - ref).abs().max() < 2e-2 * ref.abs().max()


def test_other_keys_than_queries_and_rows_without_keys():
    from sensenova_u1_b200.ops import _lib, attention as A
    g = torch.Generator(device=DEV).manual_seed(0)
    q = torch.randn(300, 4, 128, device=DEV, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(900, 2, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    mk = _meta(900, "docs")                                           # documents 0 .. 4 of 200 keys
    doc = torch.arange(300, device=DEV) // 40                         # 5, 6, 7: nothing to read, a whole query tile and more
    mq = A.make_meta(doc, torch.full_like(doc, 5000))
    o, _ = A.attention_fwd(q, k, v, A.build_plan(mq, mk), 128 ** -0.5, want_lse=False)
    _lib.check_status()
    ref = A.reference_attention(q, k, v, mq, mk, 128 ** -0.5)
    assert _rel(o, ref) < 6e-3 and (o[doc >= 5] == 0).all()
