"""Multi-tensor AdamW: chunk edges, tails, more tensors than one launch holds, addresses that rule out vector accesses."""
import pytest
import torch

from tensorplay_b200 import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("with_model", [True, False])
def test_chunks_and_alignment(grad_dtype, with_model):
    torch.manual_seed(0)
    sizes = [1, 3, 8191, 8192, 8193, 3 * 8192 + 5, 70001] + [17] * 60
    off = [i % 3 for i in range(len(sizes))]

    def make(dtype):
        return [(torch.rand(n + o, device="cuda") - 0.5).to(dtype)[o:] for n, o in zip(sizes, off)]

    master, m, v, grad = make(torch.float32), make(torch.float32), make(torch.float32), make(grad_dtype)
    v = [x.abs() for x in v]
    model = make(torch.bfloat16) if with_model else None
    ref = []
    for p, a, b, g in zip(master, m, v, grad):
        p, a, b, g = (x.double() for x in (p, a, b, g))
        a, b = 0.9 * a + 0.1 * g, 0.99 * b + 0.01 * g * g
        ref.append((p * (1 - 1e-2 * 0.1), 1e-2 / (1 - 0.9 ** 3) * a / ((b / (1 - 0.99 ** 3)).sqrt() + 1e-8), a, b))
    O.adamw_multi_(master, m, v, grad, model, lr=1e-2, beta1=0.9, beta2=0.99, eps=1e-8, weight_decay=0.1, step=3)
    for i, (p, upd, a, b) in enumerate(ref):
        # fp32 arithmetic on values of at most 1: a few ulp; the bias corrections 1 - beta^3 (0.03 at least) carry
        # 2^-24 / 0.03 into the update
        assert ((master[i].double() - (p - upd)).abs() <= 8e-6 * upd.abs() + 3e-7).all(), i
        assert (m[i].double() - a).abs().max() < 3e-7 and (v[i].double() - b).abs().max() < 3e-7
        if model is not None:
            assert torch.equal(model[i], master[i].bfloat16())


def test_blocks_that_take_several_chunks():
    """More chunks than blocks: a block's second and third chunk lie several tensors further on, or in the same large one."""
    chunks = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    torch.manual_seed(1)
    sizes = [5, 8193, 17, (chunks + 3) * 8192 + 1234, 9, 3 * 8192, 1, chunks * 4096 + 8, 40, 8192]
    assert sum(-(-n // 8192) for n in sizes) > chunks + chunks // 2
    master, m = ([torch.rand(n, device="cuda") - 0.5 for n in sizes] for _ in range(2))
    v = [torch.rand(n, device="cuda") for n in sizes]
    grad = [(torch.rand(n, device="cuda") - 0.5).bfloat16() for n in sizes]
    model = [torch.empty(n, device="cuda", dtype=torch.bfloat16) for n in sizes]
    ref = []
    for p, a, b, g in zip(master, m, v, grad):
        a, b = 0.9 * a.double() + 0.1 * g.double(), 0.99 * b.double() + 0.01 * g.double() ** 2
        ref.append((p.double() * (1 - 1e-2 * 0.1), 1e-2 / (1 - 0.9 ** 3) * a / ((b / (1 - 0.99 ** 3)).sqrt() + 1e-8), a, b))
    O.adamw_multi_(master, m, v, grad, model, lr=1e-2, beta1=0.9, beta2=0.99, eps=1e-8, weight_decay=0.1, step=3)
    for i, (p, upd, a, b) in enumerate(ref):   # bounds as above
        assert ((master[i].double() - (p - upd)).abs() <= 8e-6 * upd.abs() + 3e-7).all(), i
        assert (m[i].double() - a).abs().max() < 3e-7 and (v[i].double() - b).abs().max() < 3e-7
        assert torch.equal(model[i], master[i].bfloat16())
