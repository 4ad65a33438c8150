"""Row kernels of the norms at the widths where the threads per row change, with few and odd numbers of rows."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H", [8, 128, 136, 256, 264, 768, 1000, 1024, 1032, 2048, 2056])
@pytest.mark.parametrize("rows", [1, 9, 1231])
def test_forward_and_gradients(H, rows):
    torch.manual_seed(H + rows)
    x, r = (torch.randn(rows, H, device=DEV).bfloat16().requires_grad_() for _ in range(2))
    w, b = (torch.randn(H, device=DEV).bfloat16().requires_grad_() for _ in range(2))
    dy, ds = (torch.randn(rows, H, device=DEV).bfloat16() for _ in range(2))
    xd, rd, wd, bd = (t.detach().double().requires_grad_() for t in (x, r, w, b))

    y = O.layer_norm(x, w, b)
    yr = torch.nn.functional.layer_norm(xd, (H,), wd, bd, 1e-5)
    got, ref = torch.autograd.grad(y, (x, w, b), dy), torch.autograd.grad(yr, (xd, wd, bd), dy.double())
    y2, s = O.rms_norm(x, w, 1e-5, residual=r)
    sd = (xd + rd) + ((xd + rd).to(torch.bfloat16).double() - (xd + rd)).detach()   # the sum is kept in bf16
    y2r = sd * torch.rsqrt(sd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    got2 = torch.autograd.grad((y2, s), (x, w), (dy, ds))
    ref2 = torch.autograd.grad((y2r, sd), (xd, wd), (dy.double(), ds.double()))
    for g, f in zip((y, *got, y2, *got2), (yr, *ref, y2r, *ref2)):
        # one rounding to bf16 and fp32 sums of at most `rows` or `H` terms
        assert ((g.double() - f).abs() <= 2.0 ** -8 * f.abs() + 1e-5 * max(rows, H) ** 0.5).all()
