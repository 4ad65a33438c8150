"""The bias gradient of a linear layer where something follows the backward pass: a second differentiation, a batch of
gradients, a dispatch mode. The kernel that sums the columns is out of their sight."""
import importlib

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import tensorplay_b200.ops as O
from tensorplay_b200.ops import _ckpt

gemm_module = importlib.import_module("tensorplay_b200.ops.gemm")   # the package shows the function of that name


@pytest.fixture
def bias_kernel(monkeypatch):
    """CPU tensors would take the kernel for the bias gradient (and only there); returns the calls that did."""
    took = []

    class Lib:
        def tpb_bias_grad_chunks(self, rows, N):
            return 1

        def tpb_bias_grad(self, x, part, out, *a):
            took.append(1)
            return 0

    monkeypatch.setattr(gemm_module, "use_native", lambda *t: len(t) == 1)
    monkeypatch.setattr(gemm_module, "lib", Lib)
    monkeypatch.setattr(gemm_module, "stream_ptr", lambda: 0)
    return took


def _layer():
    torch.manual_seed(0)
    b = torch.zeros(16, dtype=torch.bfloat16, requires_grad=True)
    with _ckpt.record():   # the autograd function of the layer, on the CPU
        y = O.linear(torch.randn(6, 8).bfloat16(), torch.randn(16, 8).bfloat16(), b)
    return y, b, torch.randn(6, 16).bfloat16()


def test_plain_gradient_takes_the_kernel(bias_kernel):
    y, b, dy = _layer()
    torch.autograd.grad(y, b, dy)
    assert bias_kernel


def test_differentiated_again(bias_kernel):
    y, b, dy = _layer()
    dy.requires_grad_()
    (db,) = torch.autograd.grad(y, b, dy, create_graph=True)
    (g,) = torch.autograd.grad(db.float().square().sum(), dy)
    assert torch.equal(g, (2 * dy.detach().float().sum(0).bfloat16().float()).bfloat16().expand(6, 16)) and not bias_kernel


def test_batch_of_gradients(bias_kernel):
    y, b, dy = _layer()
    many = torch.stack([dy, 2 * dy])
    (db,) = torch.autograd.grad(y, b, many, is_grads_batched=True)
    assert torch.equal(db, many.float().sum(1).bfloat16()) and not bias_kernel


def test_dispatch_mode_sees_the_sum(bias_kernel):
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    y, b, dy = _layer()
    with Mode():
        torch.autograd.grad(y, b, dy)
    assert torch.ops.aten.sum.dim_IntList in seen and not bias_kernel
