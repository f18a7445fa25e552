"""The weight-streaming product for a few rows (csrc/gemm_small_sm100.cu) against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1, 3, 8])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128, 129])      # edges of the row tiles 16 / 32 / 64 / 128
@pytest.mark.parametrize("N,K", [(24, 520), (1000, 1096), (4096, 2048)])   # ragged weight rows and reduction
def test_small_rows(M, N, K, split):
    from sensenova_u1_b200.ops import _lib
    from sensenova_u1_b200.ops._lib import c_float, c_int, c_ll, c_void_p
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    x, w, r = rnd(M, K), rnd(N, K), rnd(M, N)
    ref = x.double() @ w.double().t()
    P = lambda t: c_void_p(None if t is None else t.data_ptr())

    def product(out, residual, f32):
        _lib.call("gemm_small", P(x), P(w), P(out), c_int(M), c_int(N), c_int(K), c_ll(K), c_ll(K), c_ll(N), c_int(f32),
                  P(residual), c_ll(0 if residual is None or residual.dim() == 1 else N), c_float(1.0), c_int(split),
                  c_void_p(_lib.stream()))
        return out.double()
    f = product(torch.empty(M, N, device="cuda"), None, 1)
    b = product(torch.empty(M, N, device="cuda", dtype=torch.bfloat16), r, 0)
    bias = product(torch.empty(M, N, device="cuda", dtype=torch.bfloat16), r[0].contiguous(), 0)
    _lib.check_status()
    # fp32 sums of K / 16 tensor-core steps, each off by at most one unit in the last place of a partial sum
    assert (f - ref).norm() / ref.norm() < K / 16 * 2.0 ** -23 + 1e-6
    # one rounding to bf16: at most half a unit in the last place, 2^-8 of the value
    for got, want in ((b, ref + r.double()), (bias, ref + r[0].double())):
        assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 1e-2).all()


def _streamed(x, w, out, split=0, f32=1, residual=None, **wrong):
    """The exported entry point; ``wrong``: arguments in place of the operands' own."""
    from sensenova_u1_b200.ops import _lib
    from sensenova_u1_b200.ops._lib import c_float, c_int, c_ll, c_void_p
    P = lambda t: c_void_p(None if t is None else t.data_ptr())
    v = dict(N=w.shape[0], K=x.shape[1], ldx=x.stride(0), ldw=w.stride(0), ldc=out.stride(0), ldr=0 if residual is None else residual.stride(0))
    v.update(wrong)
    _lib.call("gemm_small", P(x), P(w), P(out), c_int(x.shape[0]), c_int(v["N"]), c_int(v["K"]), c_ll(v["ldx"]), c_ll(v["ldw"]),
              c_ll(v["ldc"]), c_int(f32), P(residual), c_ll(v["ldr"]), c_float(1.0), c_int(split), c_void_p(_lib.stream()))
    return out


@pytest.mark.parametrize("M", [1, 16, 32, 33, 128])
def test_few_rows_take_the_weight_streaming_kernel(M):
    """``gemm_nt`` up to 128 rows has this kernel's bits (a reduction in several parts), at 129 rows the pair kernel's."""
    from sensenova_u1_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(129, 4096, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(4096, 4096, device="cuda", generator=g).to(torch.bfloat16)
    few, many = (gemm.gemm_nt(t, w, out_mode=gemm.OUT_F32_STORE) for t in (x[:M], x))
    assert torch.equal(few, _streamed(x[:M], w, torch.empty_like(few)))
    assert not torch.equal(few, many[:M])                      # so that equal bits mean the same kernel
    # the same products in another order: K / 16 steps of fp32 sums on both sides
    assert (few - many[:M]).norm() / many[:M].norm() < 2 * 4096 / 16 * 2.0 ** -23


@pytest.mark.parametrize("K", [8, 64, 72, 200])               # 1, 1, 2 and 4 pieces of 64 for up to 8 CTAs
@pytest.mark.parametrize("split", [2, 5, 8, 16, 100])
def test_split_of_a_short_reduction(K, split):
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).to(torch.bfloat16) for n in (20, 256))
    out = _streamed(x, w, torch.full((20, 256), float("nan"), device="cuda"), split)
    ref = x.double() @ w.double().t()
    # fp32 sums of at most 13 tensor-core steps, each off by at most one unit in the last place of a partial sum
    assert (out - ref).norm() / ref.norm() < 13 * 2.0 ** -23


def test_entry_point_refuses_what_the_kernel_cannot_address():
    x, w = (torch.zeros(n, 64, device="cuda", dtype=torch.bfloat16) for n in (20, 256))
    bf, f = torch.zeros(20 * 256 + 16, device="cuda", dtype=torch.bfloat16), torch.zeros(20 * 256 + 8, device="cuda")
    for kw in (dict(N=250), dict(K=60), dict(ldx=60), dict(ldw=60), dict(ldc=258), dict(K=0), dict(N=0),
               dict(out=f[1:1 + 20 * 256]), dict(out=bf[4:4 + 20 * 256], f32=0), dict(residual=bf[:20 * 256]),
               dict(f32=0, out=bf[:20 * 256], residual=bf[4:4 + 20 * 256]),
               dict(f32=0, out=bf[:20 * 256], residual=bf[:20 * 256], ldr=252)):
        kw = {k: v.view(20, 256) if torch.is_tensor(v) else v for k, v in kw.items()}
        with pytest.raises(RuntimeError):
            _streamed(x, w, kw.pop("out", f[:20 * 256].view(20, 256)), **kw)


@pytest.mark.parametrize("M", [1, 17, 64, 128, 129, 300, 1000])        # weight-streaming kernel up to 128 rows, pair kernel beyond
@pytest.mark.parametrize("F,K", [(24, 72), (64, 512), (200, 1096), (768, 2048), (3072, 1024)])   # ragged and whole column tiles
@pytest.mark.parametrize("static", [False, True])
def test_linear_swiglu_equals_product_and_activation(M, F, K, static):
    from sensenova_u1_b200.ops import fused, gemm
    g = torch.Generator(device="cuda").manual_seed(M + F)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    guard = torch.full((M + 1, F), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.linear_swiglu(x, w, out=guard[:M], w_static=static)
    gu = gemm.gemm_nt(x, w)
    ref = fused.swiglu_fwd(gu, torch.empty(M, F, device="cuda", dtype=torch.bfloat16))
    # the same sums in the same order, the same roundings
    assert torch.equal(guard[:M], ref) and (guard[M] == 7).all()
    want = torch.nn.functional.silu(gu[:, :F].double()) * gu[:, F:].double()
    # hardware tanh: absolute error 2^-11 of sigmoid, then one rounding
    assert ((ref.double() - want).abs() <= want.abs() * 2.0 ** -8 + (gu[:, :F] * gu[:, F:]).double().abs() * 2.0 ** -11 + 1e-6).all()


def test_linear_swiglu_grouped():
    from sensenova_u1_b200.ops import fused, gemm
    g = torch.Generator(device="cuda").manual_seed(5)
    F, K, tg = 384, 256, torch.tensor([1, 1, 0, -1, 2, 0, 2], dtype=torch.int32, device="cuda")
    x = torch.randn(7 * 128, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(3, 2 * F, K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    out = gemm.linear_swiglu(x, w, out=torch.full((7 * 128, F), 7.0, device="cuda", dtype=torch.bfloat16), tile_group=tg)
    gu = gemm.gemm_nt(x, w, out=torch.zeros(7 * 128, 2 * F, device="cuda", dtype=torch.bfloat16), tile_group=tg)
    ref = fused.swiglu_fwd(gu, torch.empty(7 * 128, F, device="cuda", dtype=torch.bfloat16))
    keep = (tg >= 0).repeat_interleave(128)
    assert torch.equal(out[keep], ref[keep]) and (out[~keep] == 7).all()


def test_static_weights_written_just_before_a_request():
    """A weight declared static may be read before the kernel in front of the product has finished: new values that were
    written right before a prompt and a decode step are the ones they use."""
    from sensenova_u1_b200.config import tiny_mot
    from sensenova_u1_b200.inference.engine import InferenceEngine
    from sensenova_u1_b200.models.params import ParamStore
    cfg = tiny_mot(head_dim=128, patch_size=16)
    store = ParamStore(cfg, device="cuda:0", with_grads=False)
    store.init_weights(3)
    eng = InferenceEngine(cfg, store)
    names = [n for n, t in store.p.items() if n.startswith("layers.0.") and t.dim() == 3]
    first = {n: store.p[n].clone() for n in names}
    second = {n: torch.randn_like(store.p[n]) * 0.05 for n in names}
    want = []
    for wait in (True, False):
        for rep in range(1 if wait else 10):
            for values in (first, second):
                for n in names:
                    store.p[n].copy_(values[n])
                if wait:
                    torch.cuda.synchronize()
                lay, h = eng.prefill([torch.arange(5, 25)], reserve_image_tokens=8)
                got = (h.clone(), eng.decode(lay, h, 1), eng.kc[0].clone(), eng.kc[1].clone())
                if wait:
                    want.append(got)
                else:
                    ref = want[0 if values is first else 1]
                    assert torch.equal(got[0], ref[0]) and got[1] == ref[1]
                    assert torch.equal(got[2], ref[2]) and torch.equal(got[3], ref[3])
    assert not torch.equal(want[0][0], want[1][0])


@pytest.mark.parametrize("N,K,M,streams", [(4096, 1096, 512, True), (4096, 1096, 513, False), (2048, 1096, 1024, True),
                                           (2048, 1096, 1025, False), (128, 520, 1000, True), (6144, 520, 384, True),
                                           (6144, 520, 385, False), (18944, 200, 128, True), (18944, 200, 129, False)])
def test_one_wave_of_tiles_takes_the_weight_streaming_kernel(N, K, M, streams):
    """An engine's weights up to 1024 rows, while 128 x 128 tiles are one wave (148 SMs)."""
    from sensenova_u1_b200.ops import _lib, gemm
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line is drawn by the number of SMs")
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w, r = (torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16) for n, k in ((M, K), (N, K), (M, N)))
    y = gemm.gemm_nt(x, w, residual=r, w_static=True)
    f = gemm.gemm_nt(x, w, out_mode=gemm.OUT_F32_STORE, w_static=True)
    one = _streamed(x, w, torch.empty_like(f))
    _lib.check_status()
    ref = x.double() @ w.double().t()
    # fp32 sums of K / 16 tensor-core steps, each off by at most one unit in the last place of a partial sum
    assert (f - ref).norm() / ref.norm() < K / 16 * 2.0 ** -23 + 1e-6
    assert ((y.double() - ref - r.double()).abs() <= (ref + r.double()).abs() * 2.0 ** -8 + 1e-2).all()
    assert torch.equal(f, one) or not streams


@pytest.mark.parametrize("split", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("M", [1, 24, 33, 64, 100, 128, 130])          # no, one and several steps of two per thread, ragged
@pytest.mark.parametrize("N,K", [(136, 1096), (4096, 520)])
def test_residual_joins_the_same_sums(M, N, K, split):
    g = torch.Generator(device="cuda").manual_seed(M + split)
    x, w, r = (torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16) for s in ((M, K), (N, K), (M, N)))
    sums = _streamed(x, w, torch.full((M, N), float("nan"), device="cuda"), split)
    guard = torch.full((M + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)
    guard[:M] = r                                                       # in place, as a layer may have it
    _streamed(x, w, guard[:M], split, f32=0, residual=guard[:M])
    # one fp32 addition and one rounding behind the sums of the same parts in the same order
    assert torch.equal(guard[:M], (sums + r.float()).to(torch.bfloat16)) and (guard[M] == 7).all()
    exact = x.double() @ w.double().t()
    assert (sums.double() - exact).abs().max() <= K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t()).max()
