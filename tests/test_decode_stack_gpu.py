"""The whole-stack decode kernel (csrc/decode_stack.cu) against the kernels it stands in for and against the layers in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(seed=3, **kw):
    from sensenova_u1_b200.config import tiny_mot
    from sensenova_u1_b200.inference import engine as E
    from sensenova_u1_b200.models.params import ParamStore
    cfg = tiny_mot(head_dim=128, patch_size=16, **kw)
    store = ParamStore(cfg, device="cuda:0", with_grads=False)
    store.init_weights(seed)
    return E, cfg, E.InferenceEngine(cfg, store)


# rings of 5 and 6 stages, one to many tiles per CTA, CTAs without rows, one to many parts per document
SIZES = [dict(hidden_size=1024, num_heads=8, num_kv_heads=2, ffn_size=1024, num_layers=1),
         dict(hidden_size=2048, num_heads=8, num_kv_heads=2, ffn_size=3072, num_layers=3),
         dict(hidden_size=1024, num_heads=16, num_kv_heads=2, ffn_size=12288, num_layers=2)]


@pytest.mark.parametrize("size", range(len(SIZES)))
@pytest.mark.parametrize("lens", [(1,), (64,), (700,), (3000,), (9, 70), (300, 1)])
def test_stack_equals_the_layers_one_by_one(size, lens, monkeypatch):
    E, cfg, eng = _engine(**SIZES[size])
    docs = [torch.arange(5, 5 + n) % cfg.vocab_size for n in lens]

    def step(stack):
        monkeypatch.setattr(E.decode_stack, "takes", lambda *a: stack)
        lay, h = eng.prefill(docs, reserve_image_tokens=4)
        dev = eng.dev
        pos = torch.tensor([x.next_pos for x in lay], dtype=torch.int32, device=dev)
        rows = torch.tensor([x.img_start for x in lay], device=dev)
        mq = E.attn_ops.make_meta(torch.arange(len(lay), dtype=torch.int32, device=dev), pos)
        eng._meta_k.index_copy_(0, rows, mq)
        plan = E.DecodeRows(mq, eng._meta_k, torch.tensor([x.kv_start for x in lay], dtype=torch.int32, device=dev), max(lens) + 4)
        x = eng.p["embed_tokens"][7:7 + len(lay)].contiguous()
        out = eng.layers(x, E.UND, torch.stack([pos, pos * 0, pos * 0]), plan, rows, eng._meta_k.shape[0]).clone()
        E._lib.check_status()
        return out, [t.clone() for t in eng.kc + eng.vc], rows
    want, cache, rows = step(False)
    for _ in range(2):                                          # words of an earlier launch are not taken for this one's
        got, cache2, _ = step(True)
        # the same roundings to bf16 at the same places (half a unit in the last place each), on sums in another order: a
        # rounding that falls the other way is one unit, 2^-7, of one element; a handful of stages per layer compound
        assert (got.double() - want.double()).norm() <= 2.0 ** -7 * cfg.num_layers * want.double().norm()
        for a, b in zip(cache2, cache):
            other = torch.ones(a.shape[0], dtype=torch.bool, device="cuda")
            other[rows] = False
            assert torch.equal(a[other], b[other])              # nothing else in the cache is touched
            assert (a[rows].double() - b[rows].double()).norm() <= 2.0 ** -7 * cfg.num_layers * b[rows].double().norm()
    monkeypatch.undo()


def _exact(eng, cfg, x, pos3, first, rows, caches):
    """The layers in fp64 for one new token per document: weights, x and the cache rows before the step as they are stored, angles
    as fp32 products."""
    p, D, Hq, Hk, eps = eng.p, 128, cfg.num_heads, cfg.num_kv_heads, cfg.rms_eps
    norm = lambda v, g: v * (v.pow(2).mean(-1, keepdim=True) + eps).rsqrt() * g.double()
    lin = lambda v, w: v @ w.double().t()
    ang = [torch.cat([a, a], -1)[:, None].double() for a in (pos3[i].float()[:, None] * inv for i, inv in
                                                              enumerate((eng.inv_t, eng.inv_hw, eng.inv_hw)))]

    def rope(v, gains):
        parts = torch.cat([norm(v[..., :64], gains[0]), norm(v[..., 64:], gains[1])], -1).split([64, 32, 32], -1)
        turn = lambda t: torch.cat([-t[..., t.shape[-1] // 2:], t[..., :t.shape[-1] // 2]], -1)
        return torch.cat([t * a.cos() + turn(t) * a.sin() for t, a in zip(parts, ang)], -1)
    x = x.double()
    for l in range(cfg.num_layers):
        W = lambda n: p[f"layers.{l}.{n}"][0]
        q, k, v = lin(norm(x, W("attn_norm")), W("wqkv")).split([Hq * D, Hk * D, Hk * D], -1)
        q, k, v = rope(q.unflatten(-1, (Hq, D)), W("qk_norm")[:2]), rope(k.unflatten(-1, (Hk, D)), W("qk_norm")[2:]), v.unflatten(-1, (Hk, D))
        o = torch.empty_like(q)
        for d, (lo, hi) in enumerate(zip(first, rows)):
            kd, vd = (torch.cat([c[lo:hi].double(), new[d:d + 1]]).repeat_interleave(Hq // Hk, 1)
                      for c, new in ((caches[0][l], k), (caches[1][l], v)))
            a = torch.softmax(torch.einsum("hd,khd->hk", q[d], kd) * D ** -0.5, -1)
            o[d] = torch.einsum("hk,khd->hd", a, vd)
        x = x + lin(o.flatten(1), W("wo"))
        gate, up = lin(norm(x, W("ffn_norm")), W("w13")).chunk(2, -1)
        x = x + lin(torch.nn.functional.silu(gate) * up, W("w2"))
    return x


WIDE = dict(hidden_size=4096, num_heads=32, num_kv_heads=8, ffn_size=12288, num_layers=2)      # the 8B model's widths
DEEP = dict(hidden_size=1024, num_heads=8, num_kv_heads=2, ffn_size=1024, num_layers=49)       # two launches


@pytest.mark.parametrize("size,lens", [(WIDE, n) for n in [(1,), (64,), (65,), (3000,), (1, 1), (64, 65), (1700, 3)]]
                         + [(DEEP, (70,)), (DEEP, (9, 200))])
def test_stack_against_the_layers_in_fp64(size, lens, monkeypatch):
    E, cfg, eng = _engine(**size)
    dev, n = eng.dev, len(lens)
    g = torch.Generator(device=dev).manual_seed(sum(lens))
    lay, _ = eng.prefill([torch.arange(5, 5 + k) % cfg.vocab_size for k in lens], reserve_image_tokens=4)
    for c in eng.kc + eng.vc:                                   # keys and values of the size of the new ones
        c.copy_(torch.randn(c.shape, device=dev, generator=g))
    pos = torch.tensor([x.next_pos for x in lay], dtype=torch.int32, device=dev)
    rows, first = torch.tensor([x.img_start for x in lay], device=dev), [x.kv_start for x in lay]
    mq = E.attn_ops.make_meta(torch.arange(n, dtype=torch.int32, device=dev), pos)
    eng._meta_k.index_copy_(0, rows, mq)
    plan = E.DecodeRows(mq, eng._meta_k, torch.tensor(first, dtype=torch.int32, device=dev), max(lens) + 4)
    x = torch.randn(n, cfg.hidden_size, device=dev, generator=g).to(torch.bfloat16)
    pos3 = torch.stack([pos, pos * 0 + 3, pos * 0 + 5])
    before = [[t.clone() for t in c] for c in (eng.kc, eng.vc)]

    def step(stack):
        monkeypatch.setattr(E.decode_stack, "takes", lambda *a: stack)
        for new, old in zip(eng.kc + eng.vc, before[0] + before[1]):
            new[rows] = old[rows]
        out = eng.layers(x, E.UND, pos3, plan, rows, eng._meta_k.shape[0]).clone()
        return out, torch.cat([t[rows].flatten() for t in eng.kc + eng.vc])
    ref = _exact(eng, cfg, x, pos3, first, rows.tolist(), before)
    err = {}
    for stack in (False, True):
        got = step(stack)
        # ten roundings to bf16 per layer (half a unit in the last place, 2^-9 of the value): independent, each carried on at
        # most at its own size.  One element: six deviations, and its own last rounding
        err[stack], size = (got[0].double() - ref).abs(), ref.pow(2).mean().sqrt()
        dev_ = 2.0 ** -9 * (10 * cfg.num_layers) ** 0.5 * size
        print(f"stack={stack} {lens} rms {float(err[stack].pow(2).mean().sqrt() / size):.2e} (bound {float(dev_ / size):.2e}) "
              f"max {float(err[stack].max() / size):.2e}")
        assert err[stack].pow(2).mean().sqrt() <= dev_
        assert (err[stack] <= 6 * dev_ + ref.abs() * 2.0 ** -8).all()
    # no further away than the chain, whose roundings lie at the same places (the two differ by chance)
    assert err[True].norm() <= 1.2 * err[False].norm()
    for _ in range(60):                                         # sums have a fixed order: always the same bits
        again = step(True)
        assert torch.equal(again[0], got[0]) and torch.equal(again[1], got[1])
    E._lib.check_status()


@pytest.mark.parametrize("spoil", ["type", "shape", "stride"])
def test_operands_of_other_forms_are_refused(spoil):
    E, cfg, eng = _engine(**SIZES[0])
    lay, h = eng.prefill([torch.arange(5, 9)], reserve_image_tokens=4)
    dev = eng.dev
    one = torch.tensor([4], dtype=torch.int32, device=dev)
    plan = E.DecodeRows(E.attn_ops.make_meta(one * 0, one), eng._meta_k, one * 0, 8)
    pos3 = torch.stack([one, one * 0, one * 0])
    x = eng.p["embed_tokens"][7:8].contiguous()
    if spoil == "type":
        x = x.float()
    elif spoil == "shape":
        pos3 = pos3[:2].contiguous()
    else:
        pos3 = pos3.repeat(1, 2)[:, ::2]
    with pytest.raises(ValueError):
        eng._decode_layers(x, E.UND, pos3, plan, torch.tensor([4], device=dev), eng._meta_k.shape[0])


def test_takes_refuses_what_the_kernel_is_not_built_for():
    from sensenova_u1_b200.ops.decode_stack import takes
    assert takes(1, 4096, 12288, 32, 8, 3072) and takes(2, 4096, 12288, 32, 8, 1) and takes(2, 1024, 1024, 8, 2, 9)
    for bad in ((0, 1024, 1024, 8, 2, 9), (3, 1024, 1024, 8, 2, 9), (1, 1024, 32768, 8, 2, 9), (2, 16384, 4096, 32, 8, 9),
                (1, 512, 1024, 8, 2, 9), (1, 1024, 1536, 8, 2, 9), (1, 1024, 0, 8, 2, 9), (1, 1024, 1024, 8, 4, 9),
                (1, 1024, 1024, 4, 1, 9), (1, 1024, 1024, 8, 3, 9), (1, 4096, 12288, 32, 8, 3073)):
        assert not takes(*bad)


def test_two_long_documents_keep_the_chain():
    from sensenova_u1_b200.ops.decode_stack import takes
    at = lambda rows, keys: takes(rows, 4096, 12288, 32, 8, keys)
    assert at(1, 3072) and not at(1, 3073) and at(2, 1792) and not at(2, 1793) and not at(3, 1)


def test_two_engines_on_two_streams():
    """Whole-chip cooperative launches of two engines in two threads: each runs alone on the device, whichever comes first."""
    import threading
    E, cfg, one = _engine(**SIZES[1])
    two = E.InferenceEngine(cfg, one.store)
    docs = [torch.arange(5, 5 + n) % cfg.vocab_size for n in (60, 200)]

    def request(eng, doc):
        lay, h = eng.prefill([doc], reserve_image_tokens=24)
        return eng.decode(lay, h, 24)
    want = [request(e, d) for e, d in zip((one, two), docs)]
    got, errors = [[], []], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()), torch.no_grad():
                for _ in range(4):
                    # eager steps: a capture would not let the other thread allocate meanwhile
                    lay, h = (one, two)[i].prefill([docs[i]], reserve_image_tokens=24)
                    got[i].append((one, two)[i].decode(lay, h, 24, use_graph=False))
        except Exception as e:                            # noqa: BLE001 - reported below
            errors.append(e)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    E._lib.check_status()
    assert not errors and got == [[want[0]] * 4, [want[1]] * 4]


@pytest.mark.parametrize("stop_ids", [(), (3,)])
def test_a_launch_that_gave_up_fails_its_request_only(stop_ids):
    E, cfg, eng = _engine(**SIZES[0])
    doc = [torch.arange(5, 25)]

    def request(new=12):
        lay, h = eng.prefill(doc, reserve_image_tokens=new)
        return eng.decode(lay, h, new, stop_ids=stop_ids, check_every=4)
    want = request()
    eng._stack.count[-1] = 1                                    # as a launch leaves it that has waited for too long
    with pytest.raises(E._lib.NativeLibraryError):
        request()
    E._lib.check_status()                                       # the error has been reported: nothing is left for the next one
    assert request() == want
    eng.prefill(doc * 4, reserve_image_tokens=4)                # a chain of launches does not look at the scratch
    eng._stack.count[-1] = 1
    lay, h = eng.prefill(doc * 4, reserve_image_tokens=4)
    assert len(eng.decode(lay, h, 4)) == 4
    E._lib.check_status()


def test_scratch_is_replaced_before_its_phase_numbers_come_round():
    E, cfg, eng = _engine(**SIZES[0])

    def request(new=6):
        lay, h = eng.prefill([torch.arange(5, 25)], reserve_image_tokens=new)
        return eng.decode(lay, h, new)
    want = request()
    old = eng._stack
    assert request() == want and eng._stack is old              # kept from one request to the next
    numbers = 2 ** 32 // (48 * 8)
    assert E.decode_stack.MAX_LAUNCHES + max(E.decode_stack.MAX_KEYS.values()) * 16 < numbers      # up to 768 layers
    old.count[:-1] = E.decode_stack.MAX_LAUNCHES
    assert request() == want and eng._stack is None
    assert request() == want and int(eng._stack.count[0]) == 6
    E._lib.check_status()
