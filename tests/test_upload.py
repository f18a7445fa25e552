"""Host tensors of a request on the device in one copy (``inference.engine.upload``)."""
import pytest
import torch

from sensenova_u1_b200.inference.engine import upload


def _tensors():
    return [torch.arange(7, dtype=torch.int32), torch.arange(12).view(3, 4).t(), torch.zeros(0, dtype=torch.int64),
            torch.tensor([1.5, -2.0], dtype=torch.float64), torch.tensor(3, dtype=torch.uint8)]


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_upload_keeps_values_types_and_shapes(device):
    want = _tensors()
    for _ in range(3):                                   # the pinned memory of an earlier call is used again
        got = upload(device, *_tensors())
        for g, w in zip(got, want):
            assert g.device.type == device and g.dtype == w.dtype and g.shape == w.shape and torch.equal(g.cpu(), w)
            assert device == "cpu" or g.data_ptr() % 16 == 0


@pytest.mark.gpu
def test_upload_takes_tensors_of_both_kinds_in_order():
    a = torch.arange(5, device="cuda")
    x, y, z = upload("cuda", torch.ones(3), a, torch.zeros(2))
    assert y is a or torch.equal(y, a)
    assert x.tolist() == [1, 1, 1] and z.tolist() == [0, 0]
    assert upload("cuda", a)[0].data_ptr() == a.data_ptr()


def test_stand_in_tokenizer_prefers_special_tokens_from_the_left():
    from sensenova_u1_b200.inference.api import ByteTokenizer
    t = ByteTokenizer(2000)
    a, b = list(t.specials)[:2]
    assert t.encode("é" + a + "x" + b + a + "<") == list("é".encode()) + [t.specials[a], ord("x"), t.specials[b], t.specials[a], ord("<")]
    assert t.encode("") == [] and t.decode(t.encode("p" + a + "é")) == "p" + a + "é"
