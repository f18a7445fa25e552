"""Top-k / top-p sampling in one launch (csrc/token_sampler.cu) against the same rule as separate torch operations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(lg, sampling, seed, monkeypatch):
    from sensenova_u1_b200.inference.engine import InferenceEngine
    from sensenova_u1_b200.ops import fused
    out = []
    for limit in (1024, 0):                                  # 0: the torch operations
        monkeypatch.setattr(fused, "SAMPLER_MAX_K", limit)
        torch.cuda.manual_seed(seed)
        out.append(InferenceEngine._pick_token(lg, sampling))
    return out


@pytest.mark.parametrize("V", [9, 77, 513, 4096, 151936])    # less than one element per thread up to a released vocabulary
@pytest.mark.parametrize("k", [1, 2, 50, 511, 1024])
@pytest.mark.parametrize("p", [1e-6, 0.3, 0.9, 1.0])
def test_same_draws_as_the_separate_operations(V, k, p, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(V + k)
    lg = torch.randn(24, V, device="cuda", generator=g) * 3
    for seed in range(5):
        a, b = _both(lg, dict(do_sample=True, temperature=0.7, top_k=k, top_p=p), seed, monkeypatch)
        # A token whose cumulative probability meets top_p to the last bits may stay on one side only (the prefix sums are
        # rounded in another order); it decides a draw with about its probability, far below one row in 24.
        assert a.dtype == b.dtype and int((a != b).sum()) <= (0 if p in (1e-6, 1.0) else 1)


def test_rows_of_a_wider_buffer_and_one_row(monkeypatch):
    lg = torch.randn(4, 1000, device="cuda")[:, :900]
    for rows in (lg, lg[2:3]):
        a, b = _both(rows, dict(do_sample=True, temperature=1.3, top_k=7), 3, monkeypatch)
        assert torch.equal(a, b)


def test_ties_signed_zeros_and_infinities(monkeypatch):
    from sensenova_u1_b200.ops import fused
    g = torch.Generator(device="cuda").manual_seed(1)
    quant = torch.randint(-2, 3, (16, 5000), device="cuda", generator=g).float()      # a thousand ties of the largest
    quant[:, ::7] *= -1.0                                                             # some zeros negative
    masked = torch.full((16, 5000), float("-inf"), device="cuda")
    masked[:, 11::900] = torch.randn(16, 6, device="cuda", generator=g)               # fewer finite values than k
    lowest = torch.full((16, 300), torch.finfo(torch.float32).min, device="cuda")
    lowest[:, 17] = 1.0
    for lg in (quant, masked, lowest):
        a, b = _both(lg, dict(do_sample=True, top_k=50), 7, monkeypatch)
        assert torch.equal(a, b)
    # ties cut by top_p: the lowest indexes stay
    flat = torch.zeros(3, 1000, device="cuda")
    noise = torch.rand(3, 1000, device="cuda", generator=g) + 0.1
    got = fused.sample_top_k_top_p(flat, noise, 1.0, 10, 0.25)                        # 0 .. 250 have at most 0.25 before them
    assert torch.equal(got, (1 / noise[:, :251]).argmax(1)) or torch.equal(got, (1 / noise[:, :250]).argmax(1))
    bad = torch.full((2, 64), float("nan"), device="cuda")
    assert ((0 <= fused.sample_top_k_top_p(bad, noise[:2, :64].contiguous(), 1.0, 5, 0.9))).all()


@pytest.mark.parametrize("k", [2, 50, 1024])
@pytest.mark.parametrize("p", [1e-9, 1e-30, 0.0])      # below any rounding of a sum of probabilities
def test_tiny_top_p_is_greedy(k, p, monkeypatch):
    """Nothing comes before the most likely token, so it stays whatever ``top_p`` is."""
    g = torch.Generator(device="cuda").manual_seed(k)
    lg = torch.randn(64, 5000, device="cuda", generator=g)
    got, ref = _both(lg, dict(do_sample=True, top_k=k, top_p=p or 1e-300), 1, monkeypatch)
    assert torch.equal(got, lg.argmax(-1)) and torch.equal(ref, got)


def test_logits_of_any_strides(monkeypatch):
    """Columns first, every other column, one row repeated: the same draws as the separate operations."""
    g = torch.Generator(device="cuda").manual_seed(2)
    base = torch.randn(4000, 6, device="cuda", generator=g)
    for lg in (base.t(), base.t().contiguous()[:, ::2], base[:, 0].expand(5, 4000)):
        a, b = _both(lg, dict(do_sample=True, temperature=0.9, top_k=40, top_p=0.95), 4, monkeypatch)
        assert torch.equal(a, b)
