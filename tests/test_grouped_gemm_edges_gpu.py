"""Grouped GEMM: output widths off the 64-column stores, experts without rows, accumulation and fp32 output."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.parallel.moe import grouped_gemm

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,K", [(64, 64), (96, 200), (264, 320), (520, 136)])
@pytest.mark.parametrize("counts", [(128, 0, 5, 300), (0, 0, 1, 0)])
@pytest.mark.parametrize("out_dtype,acc", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False)])
def test_modes(N, K, counts, out_dtype, acc):
    torch.manual_seed(N + K)
    o = [0]
    for c in counts:
        o.append(o[-1] + (c + 127) // 128 * 128)
    G, rows = len(counts), o[-1]
    offs = torch.tensor(o, dtype=torch.int32, device=DEV)
    live = torch.zeros(rows, 1, device=DEV)
    for e, c in enumerate(counts):
        live[o[e]:o[e] + c] = 1
    x = (torch.randn(rows, K, device=DEV) * live).bfloat16()
    dy = (torch.randn(rows, N, device=DEV) * live).bfloat16()
    w = torch.randn(G, N, K, device=DEV).bfloat16()

    def run(a, b, shape, **kw):
        out = torch.randn(shape, device=DEV).to(out_dtype) if acc else torch.empty(shape, device=DEV, dtype=out_dtype)
        base = out.double() if acc else 0.0
        return grouped_gemm(a, b, offs, out=out, accumulate=acc, **kw).double() - 0.0, base

    def close(got, ref, red):
        # fp32 accumulation of `red` unit-variance products, one rounding to the output
        tol = 2.0 ** -8 * ref.abs() * (out_dtype == torch.bfloat16) + (red / 16 + 1) * 2.0 ** -22 * max(1, red) ** 0.5 + 1e-6
        assert ((got - ref).abs() <= tol).all()

    seg = [slice(o[e], o[e + 1]) for e in range(G)]
    y, base = run(x, w, (rows, N))
    close(y, torch.cat([x[s].double() @ w[e].double().t() for e, s in enumerate(seg)]) + base, K)
    dx, base = run(dy, w, (rows, K), b_mn=True)
    close(dx, torch.cat([dy[s].double() @ w[e].double() for e, s in enumerate(seg)]) + base, N)
    dw, base = run(dy, x, (G, N, K), mode=1)
    close(dw, torch.stack([dy[s].double().t() @ x[s].double() for s in seg]) + base, max(counts))
    O.check_status()
