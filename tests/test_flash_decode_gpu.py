"""Attention of a few query rows over a long cache: key splits, row tiles, masks, strided caches."""
import pytest
import torch

from tensorplay_b200 import ops as O
from tensorplay_b200.ops.attention import _few_rows, flash_fwd

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _reference(q, k, v, causal, window):
    """64-bit formula; ``(o, lse)``, rows without a key give zeros and -inf."""
    B, Tq, Hq, D = q.shape
    Tk, g = k.shape[1], Hq // k.shape[2]
    qf = q.double().permute(0, 2, 1, 3)
    kf, vf = (t.double().permute(0, 2, 1, 3).repeat_interleave(g, 1) for t in (k, v))
    s = qf @ kf.transpose(-1, -2) / D ** 0.5
    i = torch.arange(Tq, device=q.device).view(-1, 1) + Tk - Tq
    j = torch.arange(Tk, device=q.device).view(1, -1)
    hide = torch.zeros(Tq, Tk, dtype=torch.bool, device=q.device)
    if causal:
        hide |= j > i
    if window:
        hide |= j < i - window + 1
    s = s.masked_fill(hide, float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - torch.where(lse == float("-inf"), torch.zeros_like(lse), lse).unsqueeze(-1))
    return (p @ vf).permute(0, 2, 1, 3), lse


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,causal,window", [
    (1, 1, 1, 8, 8, True, 0),            # one key
    (2, 1, 63, 8, 2, True, 0),           # no split, ragged step
    (1, 1, 4097, 32, 8, True, 0),        # a full cluster of splits, one ragged key
    (1, 1, 700, 16, 2, True, 0),         # a cluster, few keys each
    (1, 2, 20001, 8, 2, True, 0),        # splits merged by a second launch
    (1, 3, 30000, 8, 2, True, 5000),     # the same with a window: most splits have no key
    (3, 1, 1000, 16, 1, True, 0),        # a full 16-row tile
    (2, 3, 517, 24, 4, True, 0),         # 18 rows: two tiles, the second nearly empty
    (1, 8, 2051, 64, 8, True, 0),        # 64 rows
    (1, 16, 300, 4, 4, False, 0),        # unmasked
    (2, 5, 3, 8, 4, True, 0),            # more queries than keys: rows without any key
    (2, 1, 5000, 8, 2, True, 300),       # window: whole splits lie outside
    (1, 4, 640, 8, 4, True, 17),
])
def test_few_query_rows(D, B, Tq, Tk, Hq, Hkv, causal, window):
    torch.manual_seed(Tk + Tq)
    q = torch.randn(B, Tq, Hq, D, device=DEV, dtype=torch.bfloat16) * 1.5
    cache = torch.full((2, B, Hkv, Tk + 37, D), float("nan"), device=DEV, dtype=torch.bfloat16)   # room past the end
    cache[:, :, :, :Tk] = torch.randn(2, B, Hkv, Tk, D, device=DEV)
    k, v = (c[:, :, :Tk].transpose(1, 2) for c in cache)
    assert _few_rows(q, k, v)
    o, lse = flash_fwd(q, k, v, causal, D ** -0.5, window=window)
    O.check_status()
    ref, rlse = _reference(q, k, v, causal, window)
    # probabilities rounded to bf16 (2^-9 each, against an output of weights summing to one and |v| < 6) and the output
    assert (o.double() - ref).abs().max().item() < 6 * 2.0 ** -8
    assert ((o.double() - ref).norm() / ref.norm().clamp_min(1e-30)).item() < 4e-3
    got = lse[:, :, :Tq].double()
    assert torch.equal(got == float("-inf"), rlse == float("-inf"))
    fin = rlse != float("-inf")
    assert (got[fin] - rlse[fin]).abs().max().item() < 2e-5 * max(1.0, rlse[fin].abs().max().item())


def test_token_major_views_and_backward():
    """q, k, v as slices of one packed projection, and the gradient through a few rows."""
    torch.manual_seed(3)
    B, T, H, D = 2, 9, 4, 64
    packed = torch.randn(B, T, 3, H, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    o = O.flash_attention(packed[:, :, 0], packed[:, :, 1], packed[:, :, 2], causal=True)
    do = torch.randn_like(o)
    (g,) = torch.autograd.grad(o, packed, do)
    ref_in = packed.detach().float().requires_grad_()
    r = O.attention_reference(ref_in[:, :, 0], ref_in[:, :, 1], ref_in[:, :, 2])
    (rg,) = torch.autograd.grad(r, ref_in, do.float())
    assert ((o.float() - r).norm() / r.norm()).item() < 6e-3
    assert ((g.float() - rg).norm() / rg.norm()).item() < 1.5e-2


@pytest.mark.parametrize("Tk", [100, 4097, 20001])   # one split, a cluster of them, two launches
@pytest.mark.parametrize("case", ["query", "key", "many keys", "value", "overflow"])
def test_nan_and_infinity_reach_the_output(Tk, case):
    """A NaN query row, one NaN key, whole splits of them, a NaN value, scores of +inf; rows without a key stay zero."""
    torch.manual_seed(Tk)
    B, Tq, Hq, Hkv, D = 2, 4, 8, 4, 64
    q, k, v = (torch.randn(B, T, H, D, device=DEV).bfloat16() for T, H in ((Tq, Hq), (Tk, Hkv), (Tk, Hkv)))
    if case == "query":
        q[1, 2, 3] = float("nan")
    elif case == "key":
        k[0, 7, 1, 5] = float("nan")
    elif case == "many keys":
        k[0, : Tk - 50, 2] = float("nan")
    elif case == "value":
        v[0, 7, 1] = float("nan")
    else:
        q[0, 1, 0], k[0, 9, 0] = 1e25, 1e25
    assert _few_rows(q, k, v)
    o, lse = flash_fwd(q, k, v, True, D ** -0.5)
    ref = O.attention_reference(q.float(), k.float(), v.float(), True)
    assert torch.equal(o.isnan(), ref.isnan()) and ref.isnan().any()
    fin = ~ref.isnan()
    assert (o.float() - ref)[fin].abs().max().item() < 6 * 2.0 ** -8
    rows = ~ref.isnan().all(-1).transpose(1, 2)
    assert lse[:, :, :Tq][rows].isfinite().all()
    none, _ = flash_fwd(q, k[:, :2], v[:, :2], True, D ** -0.5)   # the first two queries have no key
    assert (none[:, :2] == 0).all()



@pytest.mark.parametrize("n", range(1, 9))
@pytest.mark.parametrize("D,Tk", [(64, 517), (128, 1030)])
def test_every_cluster_size(n, D, Tk):
    """Two row tiles, the second ragged, merged by clusters of any size, the last split short or empty."""
    from tensorplay_b200.ops._common import lib, stream_ptr
    torch.manual_seed(n)
    B, Tq, Hq, Hkv = 2, 3, 12, 2
    q, k, v = (torch.randn(B, T, H, D, device=DEV).bfloat16() for T, H in ((Tq, Hq), (Tk, Hkv), (Tk, Hkv)))
    o, lse = torch.empty_like(q), torch.empty(B, Hq, 128, device=DEV)
    strides = [t.stride(i) for t in (q, k, v, o) for i in (1, 2, 0)]
    assert lib().tpb_flash_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), None, None, B, Tq,
                                  Tk, Hq, Hkv, D, *strides, 128, 1, D ** -0.5, 0, n, stream_ptr()) == 0
    ref, rlse = _reference(q, k, v, True, 0)
    assert (o.double() - ref).abs().max().item() < 6 * 2.0 ** -8
    assert (lse[:, :, :Tq].double() - rlse).abs().max().item() < 2e-5 * rlse.abs().max().item()
