"""Decoding ends where the cache rows that the prefill reserved end (csrc/decode_step.cu only drops what does not fit)."""
import types

import pytest
import torch

from sensenova_u1_b200.inference import engine as E

STOP = 3


def _engine(monkeypatch, kv_len, stop_after):
    """An engine whose step is a fake: the token after ``stop_after`` steps is STOP, before that 1."""
    steps = []

    class Rows:
        def __init__(self, pos, kv_rows, hidden, new):
            self.out = torch.full((pos.numel(), new), -1, dtype=torch.long)
            self.row0, self.x, self.pos3, self.meta_q, self.kv_rows = kv_rows, None, None, None, None

        def advance(self, tokens, embed, meta_k):
            assert int(self.row0.max()) + len(steps) < meta_k.shape[0]       # csrc/decode_step.cu: no metadata for this row
            self.out[:, len(steps)] = tokens
            steps.append(1)

    monkeypatch.setattr(E.decode_stack, "Rows", Rows)
    monkeypatch.setattr(E.gemm, "gemm_nt", lambda *a, **k: None)
    eng = E.InferenceEngine.__new__(E.InferenceEngine)
    eng.dev, eng.cfg = torch.device("cpu"), types.SimpleNamespace(hidden_size=8)
    eng.p = {"lm_head": None, "embed_tokens": None}
    eng._meta_k, eng._doc_starts = torch.zeros(kv_len, 4, dtype=torch.int32), [0, 10]
    eng.final_norm = lambda h, br: h
    eng.layers = lambda *a: torch.zeros(2, 8)
    eng._one_launch = lambda rows, keys: False
    eng._pick_token = lambda logits, sampling, seen: torch.full((2,), STOP if len(steps) >= stop_after else 1)
    lays = [E.DocLayout(0, 4, 4, 4), E.DocLayout(10, 5, 15, 5)]
    return eng, lays, steps


@pytest.mark.parametrize("room, new, stop_after, stops, ok", [
    (6, 6, 99, (), True),                 # exactly the reserved rows
    (6, 7, 99, (), False),
    (6, 4096, 99, (STOP,), False),        # a budget that nothing ends in time
    (6, 4096, 2, (STOP,), True),          # a budget beyond the reserved rows, all documents stopped within them
    (6, 4096, 5, (STOP,), True),          # with the last of them
    (6, 4096, 6, (STOP,), False),
    (0, 1, 99, (), False)])
def test_decode_stays_within_the_reserved_rows(monkeypatch, room, new, stop_after, stops, ok):
    eng, lays, steps = _engine(monkeypatch, 15 + room, stop_after)
    run = lambda: eng.decode(lays, torch.zeros(2, 8), new, stop_ids=stops, use_graph=False, check_every=4)
    if ok:
        n = min(new, stop_after + 1)
        assert [len(t) for t in run()] == [n, n]
    else:
        with pytest.raises(ValueError, match="reserved"):
            run()
    assert len(steps) <= room
