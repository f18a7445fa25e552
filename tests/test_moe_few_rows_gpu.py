"""Expert FFN of a few rows (decoding): one-CTA routing and expert products against the general path and fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Bufs:
    def get(self, name, shape, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device="cuda")


@pytest.mark.parametrize("R", [1, 2, 31, 32])
@pytest.mark.parametrize("E,K", [(3, 2), (32, 1), (33, 5), (128, 8), (256, 16)])
@pytest.mark.parametrize("norm", [True, False])
def test_route_few_lays_out_like_route(R, E, K, norm):
    from sensenova_u1_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(R * E)
    logits = torch.randn(R, E, device="cuda", generator=g) * 2
    a, b = moe.route_few(logits, K, norm, _Bufs()), moe.route(logits, K, norm)
    assert torch.equal(a.top_idx, b.top_idx) and torch.equal(a.top_w, b.top_w) and torch.equal(a.dest, b.dest)
    n = a.tile_group.numel()
    assert n == min(R * K, E)
    want = torch.full_like(a.tile_group, -1)
    m = min(n, b.tile_group.numel())
    want[:m] = b.tile_group[:m]
    assert torch.equal(a.tile_group, want)


@pytest.mark.parametrize("rows", [1, 16, 17, 32])                       # row tiles of 16 and 32
@pytest.mark.parametrize("N,K", [(24, 72), (200, 520), (768, 2048)])    # ragged and whole weight tiles
@pytest.mark.parametrize("swiglu", [False, True])
def test_expert_products(rows, N, K, swiglu):
    from sensenova_u1_b200.ops import _lib, gemm
    g = torch.Generator(device="cuda").manual_seed(rows + N)
    E, tg = 5, torch.tensor([4, 0, 2, -1], dtype=torch.int32, device="cuda")
    x = torch.randn(4 * 128, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(E, N * (2 if swiglu else 1), K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    out = gemm.gemm_experts(x, w, torch.full((4 * 128, N), 7.0, device="cuda", dtype=torch.bfloat16), tg, rows, swiglu=swiglu)
    _lib.check_status()
    for t, e in enumerate(tg.tolist()):
        got = out[t * 128:t * 128 + rows].double()
        if e < 0:
            assert (out[t * 128:(t + 1) * 128] == 7).all()
            continue
        ref = x[t * 128:t * 128 + rows].double() @ w[e].double().t()
        # fp32 sums, one rounding (2^-8 of the value); silu: both factors rounded first and the hardware tanh (2^-11)
        if swiglu:
            gate, up = ref[:, :N].to(torch.bfloat16).double(), ref[:, N:].to(torch.bfloat16).double()
            ref = torch.nn.functional.silu(gate) * up
            tol = ref.abs() * 2.0 ** -6 + (gate * up).abs() * 2.0 ** -10 + 1e-2
        else:
            tol = ref.abs() * 2.0 ** -8 + 1e-4
        assert ((got - ref).abs() <= tol).all()


def test_one_cta_path_equals_the_general_path(monkeypatch):
    from sensenova_u1_b200.config import get_config
    from sensenova_u1_b200.inference.engine import InferenceEngine
    from sensenova_u1_b200.models.params import UND, ParamStore
    from sensenova_u1_b200.ops import moe
    cfg = get_config("a3b-mot", num_layers=1, num_experts=16, gen_num_experts=16)
    store = ParamStore(cfg, device="cuda:0", with_grads=False)
    store.init_weights(1)
    eng = InferenceEngine(cfg, store)
    x = torch.randn(32, cfg.hidden_size, device="cuda").to(torch.bfloat16)
    W = lambda n: store.p["layers.0." + n]
    outs = []
    for few in (32, 0):
        monkeypatch.setattr(moe, "FEW_ROWS", few)
        outs.append(eng._moe_ffn(W, x, x, UND, torch.empty_like(x)).float())
    # two bf16 roundings of the experts' outputs may differ by an ulp each
    assert ((outs[0] - outs[1]).abs() <= outs[1].abs() * 2.0 ** -7 + 2e-2).all()


@pytest.mark.parametrize("R,E,K,bad", [(32, 32, 8, 17), (32, 128, 8, 20), (32, 256, 16, 31), (5, 3, 2, 5), (200, 128, 8, 60)])
@pytest.mark.parametrize("what", [float("nan"), float("inf"), float("-inf")])
def test_rows_without_a_finite_score(R, E, K, bad, what):
    """A row of NaN (or whose softmax is NaN) still takes K different experts: no expert gets more rows than there are, and
    every slot lies inside the permuted buffer.  The other rows are not affected."""
    from sensenova_u1_b200.ops import _lib, moe
    g = torch.Generator(device="cuda").manual_seed(R + E)
    good = torch.randn(R, E, device="cuda", generator=g)
    logits = good.clone()
    logits[:bad] = what
    logits[0, 1:] = good[0, 1:]                                            # one row with a single bad score
    for route in ([moe.route] if R > 32 else [moe.route, lambda x, k, n: moe.route_few(x, k, n, _Bufs())]):
        r, ref = route(logits, K, True), route(good, K, True)
        _lib.check_status()
        idx, dest = r.top_idx.cpu(), r.dest.cpu()
        assert ((0 <= idx) & (idx < E)).all() and all(len(set(row)) == K for row in idx.tolist())
        assert (dest >= 0).all() and (dest < r.max_rows).all() and dest.unique().numel() == R * K
        tiles = r.tile_group.cpu()
        assert torch.equal(tiles[(dest // 128).view(-1).long()], idx.view(-1))     # every slot in a tile of its expert
        assert torch.equal(r.top_idx[bad:], ref.top_idx[bad:]) and torch.equal(r.top_w[bad:], ref.top_w[bad:])
        assert torch.isnan(r.top_w[1:bad]).all()                            # what the row held goes on into its output


@pytest.mark.parametrize("R,K,H", [(1, 1, 8), (3, 8, 2048), (32, 5, 8192), (2, 6, 2056)])
def test_combination_and_norm(R, K, H):
    from sensenova_u1_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    yp, res, gain = rnd(R * K * 128, H), rnd(R, H), rnd(H)
    r = moe.route_few(torch.randn(R, 16, device="cuda", generator=g), K, True, _Bufs())
    y, h = torch.empty_like(res), torch.empty_like(res)
    moe.combine_norm(yp, r, res, y, gain, h, 1e-6)
    want = moe.combine(yp, r, res, torch.empty_like(res))
    assert torch.equal(y, want)
    ref = want.double() * (want.double().pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * gain.double()
    # fp32 arithmetic, one rounding to bf16: half a unit in the last place, 2^-8 of the value
    assert ((h.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-6).all()


@pytest.mark.parametrize("rows", [1, 17])
def test_experts_that_share_their_rows(rows):
    from sensenova_u1_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(rows)
    tg = torch.tensor([3, 0, -1, 4], dtype=torch.int32, device="cuda")
    x = torch.randn(rows, 520, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(5, 400, 520, device="cuda", generator=g).to(torch.bfloat16)
    each = torch.zeros(4 * 128, 520, device="cuda", dtype=torch.bfloat16)
    each.view(4, 128, 520)[:, :rows] = x
    for swiglu, n in ((False, 400), (True, 200)):
        a, b = (gemm.gemm_experts(t, w, torch.full((4 * 128, n), 7.0, device="cuda", dtype=torch.bfloat16), tg, rows, swiglu=swiglu)
                for t in (x, each))
        used = torch.zeros(4 * 128, dtype=torch.bool, device="cuda")
        used.view(4, 128)[:, :rows] = True
        assert torch.equal(a[used], b[used]) and (a.view(4, 128, n)[2] == 7).all()
