"""Shapes that a read takes: what ``read(name).view(*shape)`` takes.  The library call is left
out, so that it runs on the CPU."""
import pytest
import torch

from neuzip_b200 import backend


@pytest.fixture
def be(monkeypatch):
    monkeypatch.setattr(backend, "_CUDA", torch.device("cpu"))
    be = backend._cuda.Manager_f7_n0()
    be._decode = lambda entry, out: out.fill_(1.0)
    be._cache["w"] = backend._Entry(24, torch.bfloat16, 256, 0, torch.zeros(64, dtype=torch.uint8),
                                    torch.zeros(24, dtype=torch.uint8))
    return be


@pytest.mark.parametrize("shape", ((24,), (4, 6), (-1, 6), (4, -1), (2, -1, 3), torch.Size((6, 4)), [3, 8]))
def test_shapes_that_fit(be, shape):
    got = be.read_shaped("w", shape)
    assert got.shape == torch.empty(24).view(*shape).shape and bool((got == 1).all())
    assert got.is_contiguous()


@pytest.mark.parametrize("shape", ((25,), (5, 5), (-1, 5), (-1, -1), (-4, -6), (1 << 20, 1 << 20), ()))
def test_shapes_that_do_not(be, shape):
    with pytest.raises(RuntimeError) as wanted:
        torch.empty(24).view(tuple(shape))
    with pytest.raises(RuntimeError) as got:
        be.read_shaped("w", shape)
    if not shape or min(shape) >= -1:
        assert str(got.value) == str(wanted.value)


@pytest.mark.parametrize("bias", (None, torch.zeros(4, dtype=torch.bfloat16)))
def test_linear_with_one_size_left_open(be, bias):
    x = torch.ones(2, 6, dtype=torch.bfloat16)
    y = (be.linear_without_bias("w", x, (-1, 6)) if bias is None else be.linear("w", x, (-1, 6), bias))
    assert torch.equal(y, torch.full((2, 4), 6.0, dtype=torch.bfloat16))
