"""The gradient buffer of an embedding is zeroed where a tracer or a dispatch mode can see it."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.utils._python_dispatch import TorchDispatchMode

from tensorplay_b200.ops import decode


@pytest.fixture
def memsets(monkeypatch):
    """CPU tensors would be zeroed by the memset; returns the calls."""
    took = []

    class Lib:
        def tpb_zero(self, *a):
            took.append(a)
            return 0

    monkeypatch.setattr(decode, "use_native", lambda *t: True)
    monkeypatch.setattr(decode, "lib", Lib)
    monkeypatch.setattr(decode, "stream_ptr", lambda: 0)
    return took


def test_plain_buffer(memsets):
    decode._zero_(torch.empty(4, 8))
    assert memsets[0][1] == 4 * 8 * 4


def test_fake_buffer(memsets):
    with FakeTensorMode():
        t = torch.empty(4, 8)
        decode._zero_(t)
    decode._zero_(t)
    assert not memsets


def test_mode_sees_the_zeroing(memsets):
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    t = torch.ones(4, 8)
    with Mode():
        decode._zero_(t)
    assert torch.ops.aten.zero_.default in seen and not t.any() and not memsets


def test_functional_transform(memsets):
    out = torch.func.vmap(lambda t: decode._zero_(t.clone()))(torch.ones(3, 4))
    assert not out.any() and not memsets
