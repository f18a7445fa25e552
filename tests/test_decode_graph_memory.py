"""Memory of the captured decode step (``InferenceEngine._capture``): kept from one request to the next, bounded, given back."""
import contextlib
import gc

import pytest
import torch

from sensenova_u1_b200.inference.engine import InferenceEngine


class _Cuda:
    """Stand-in for ``torch.cuda`` that records what a capture does."""
    OutOfMemoryError = torch.cuda.OutOfMemoryError

    def __init__(self, end_raises=False):
        self.log, self.reserved, self.end_raises = [], 0, end_raises
        outer = self

        class Stream:
            def __init__(self, device=None):
                self.device = device

            def wait_stream(self, other):
                pass

        class CUDAGraph:
            def capture_begin(self, pool=None):
                self.stream = outer.log[-1][1]
                self._pool = pool or object()
                outer.log.append(("begin", pool))

            def capture_end(self):
                outer.log.append(("end",))
                if outer.end_raises:
                    raise RuntimeError("invalid capture")

            def pool(self):
                return self._pool

        @contextlib.contextmanager
        def graph(g, pool=None, stream=None):
            outer.log.append(("graph", stream))
            g._pool = pool or object()
            yield

        self.Stream, self.CUDAGraph, self.graph = Stream, CUDAGraph, graph
        self.cur = Stream()

    def current_stream(self, device=None):
        return self.cur

    @contextlib.contextmanager
    def stream(self, s):
        self.log.append(("stream", s))
        yield

    @contextlib.contextmanager
    def device(self, d):
        self.log.append(("device", d))
        yield

    def memory_stats_as_nested_dict(self, device=None):
        return {"reserved_bytes": {"all": {"current": self.reserved}}}

    def synchronize(self, device=None):
        pass


@pytest.fixture
def engine(monkeypatch):
    eng = InferenceEngine.__new__(InferenceEngine)
    eng.dev = torch.device("cuda", 3)
    eng._graph = eng._capture_stream = None
    eng._graph_bytes = 0

    def cuda(**kw):
        c = _Cuda(**kw)
        for n in ("Stream", "CUDAGraph", "graph", "current_stream", "stream", "device", "memory_stats_as_nested_dict", "synchronize"):
            monkeypatch.setattr(torch.cuda, n, getattr(c, n))
        return c
    return eng, cuda


def _raise_once():
    calls = []

    def fn():
        calls.append(1)
        if len(calls) == 1:
            raise torch.cuda.OutOfMemoryError("no memory")
    return fn, calls


@pytest.mark.parametrize("end_raises", [False, True])
def test_out_of_memory_falls_back_on_the_same_stream(engine, end_raises):
    eng, cuda = engine
    c = cuda(end_raises=end_raises)
    fn, calls = _raise_once()
    g = eng._capture(fn)
    assert len(calls) == 2 and eng._graph is g
    assert [x for x in c.log if x[0] == "graph"] == [("graph", eng._capture_stream)]
    assert eng._capture_stream.device == eng.dev                # also when another device is the current one


def test_other_errors_are_not_hidden_by_the_end_of_the_capture(engine):
    eng, cuda = engine
    cuda(end_raises=True)

    def fn():
        raise KeyError("first")
    with pytest.raises(KeyError):
        eng._capture(fn)


def test_pool_is_reused_bounded_and_given_back(engine):
    eng, cuda = engine
    c = cuda()

    def fn(n):
        def grow():
            c.reserved += n
        return grow
    first = eng._capture(fn(1 << 20))
    eng._capture(fn(1 << 20))
    assert [x[1] for x in c.log if x[0] == "begin"] == [None, first.pool()]
    assert eng._graph_bytes == 2 << 20
    big = eng._capture(fn(eng.GRAPH_POOL_LIMIT))
    assert big is not None and eng._graph is None and eng._graph_bytes == 0        # dies with its request
    eng._capture(fn(1 << 20))
    assert c.log[-2] == ("begin", None) and eng._graph is not None
    eng.release_decode_memory()
    assert eng._graph is None and eng._graph_bytes == 0


def _engine():
    from sensenova_u1_b200.config import tiny_mot
    from sensenova_u1_b200.models.params import ParamStore
    cfg = tiny_mot(head_dim=128, patch_size=16)
    store = ParamStore(cfg, device="cuda:0", with_grads=False)
    store.init_weights(3)
    return InferenceEngine(cfg, store)


@pytest.mark.gpu
def test_requests_of_other_sizes_on_one_engine():
    """One document, many, one again, other lengths: the steps captured into the same pool give what eager steps give."""
    eng = _engine()
    for rep in range(2):
        for lens, new, kw in (((9,), 5, {}), ((30, 1, 64, 7, 130), 9, {}), ((200,), 12, dict(sampling=dict(do_sample=True, top_k=9, seed=1))),
                              ((3, 4), 4, dict(sampling=dict(do_sample=True, seed=2, repetition_penalty=1.3)))):
            docs = [torch.arange(5, 5 + n) for n in lens]
            out = []
            for graph in (True, False):
                lay, h = eng.prefill(docs, reserve_image_tokens=new)
                out.append(eng.decode(lay, h, new, use_graph=graph, **kw))
            assert out[0] == out[1] and eng.last_decode_steps == new


@pytest.mark.gpu
def test_fallback_and_release_on_the_device():
    eng = _engine()
    x = torch.zeros(1000, device="cuda")
    fn, calls = _raise_once()

    def step():
        fn()
        x.add_(torch.ones(1000, device="cuda"))
    g = eng._capture(step)
    g.replay()
    g2 = eng._capture(lambda: x.add_(torch.full((500000,), 2.0, device="cuda")[:1000]))     # into the pool of the fallback's graph
    del g
    g2.replay()
    assert (x == 3).all()
    lay, h = eng.prefill([torch.arange(5, 30)], reserve_image_tokens=6)
    want = eng.decode(lay, h, 6)
    del g2
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_reserved()
    eng.release_decode_memory()
    torch.cuda.empty_cache()
    assert torch.cuda.memory_reserved() < before                # the pool went back to the driver
    lay, h = eng.prefill([torch.arange(5, 30)], reserve_image_tokens=6)
    assert eng.decode(lay, h, 6) == want
