"""The kernels between the LM head and the layers of a decode step (csrc/decode_step.cu)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 7, 8, 513, 4096, 151936])          # fewer elements than CTAs, ragged parts, a vocabulary
@pytest.mark.parametrize("rows", [1, 3, 24])
def test_argmax_is_the_first_of_the_largest(V, rows):
    from sensenova_u1_b200.ops.decode_stack import argmax_rows
    g = torch.Generator(device="cuda").manual_seed(V + rows)
    x = torch.randn(rows, V + 5, device="cuda", generator=g)[:, :V]                        # rows of a wider buffer
    got = argmax_rows(x)
    assert torch.equal(got, x.argmax(-1))
    tied = (x * 2).round()                                                                 # many equal elements
    first = (tied == tied.max(-1, keepdim=True).values).int().argmax(-1)
    assert torch.equal(argmax_rows(tied), first)
    for fill in (float("-inf"), float("inf"), torch.finfo(torch.float32).min, float("nan")):
        assert argmax_rows(torch.full((rows, V), fill, device="cuda")).eq(0).all()
    y = x.clone()
    y[:, V // 2] = float("inf")
    assert argmax_rows(y).eq(V // 2).all()
    y[:, V - 1] = float("nan")
    assert argmax_rows(y).eq(V - 1).all()


@pytest.mark.parametrize("n,H", [(1, 8), (2, 4096), (24, 264)])
def test_advance_makes_what_a_token_implies(n, H):
    from sensenova_u1_b200.ops import _lib, attention as A
    from sensenova_u1_b200.ops.decode_stack import Rows
    g = torch.Generator(device="cuda").manual_seed(n)
    V, Sk, new = 50, 40 * n, 5
    embed = torch.randn(V, H, device="cuda", generator=g).to(torch.bfloat16)
    meta = torch.full((Sk, 4), -7, dtype=torch.int32, device="cuda")
    pos = torch.arange(3, 3 + n, dtype=torch.int32, device="cuda")
    row = torch.arange(n, device="cuda") * 40 + 7
    st, want = Rows(pos, row, H, new), meta.clone()
    for step in range(new):
        t = torch.randint(0, V, (n,), device="cuda", generator=g)
        st.advance(t, embed, meta)
        m = A.make_meta(torch.arange(n, dtype=torch.int32, device="cuda"), pos + step)
        want.index_copy_(0, row + step, m)
        assert torch.equal(st.out[:, step], t) and (st.out[:, step + 1:] == -1).all()
        assert torch.equal(st.x, embed[t]) and torch.equal(st.kv_rows, row + step) and torch.equal(st.meta_q, m)
        assert torch.equal(st.pos3, torch.stack([pos + step, pos * 0, pos * 0])) and torch.equal(meta, want)
    _lib.check_status()


def test_advance_reports_what_does_not_fit():
    from sensenova_u1_b200.ops import _lib
    from sensenova_u1_b200.ops.decode_stack import Rows
    embed = torch.ones(4, 8, device="cuda", dtype=torch.bfloat16)
    one = lambda v, dt=torch.int64: torch.tensor([v], dtype=dt, device="cuda")
    for token, row, steps in ((4, 0, 1), (-1, 0, 1), (0, 9, 1), (0, -1, 1), (0, 0, 3)):       # token, cache row, output slot
        meta = torch.full((9, 4), -7, dtype=torch.int32, device="cuda")
        st = Rows(one(0, torch.int32), one(row), 8, 2)
        for _ in range(steps):
            st.advance(one(token), embed, meta)
        with pytest.raises(_lib.NativeLibraryError):
            _lib.check_status()
        if not 0 <= row < 9:
            assert (meta == -7).all()
    for bad in (dict(tokens=one(0).int()), dict(embed=embed.float()), dict(meta_k=meta[:, :3])):
        kw = dict(tokens=one(0), embed=embed, meta_k=meta)
        kw.update(bad)
        with pytest.raises(ValueError):
            st.advance(**kw)
