"""Operands whose sizes do not belong together are refused on the host, before a kernel is given their addresses."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.models.llama import LlamaBlock, LlamaConfig
from tensorplay_b200.ops import attention, decode, norm, rope


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16)


@pytest.fixture
def as_native(monkeypatch):
    """CPU tensors take the native branch of the norms; a launch would fail the test."""
    def no_launch(*a):
        raise AssertionError("a kernel would have been launched")

    monkeypatch.setattr(norm, "_native_ok", lambda x, w: True)
    monkeypatch.setattr(norm, "use_native", lambda *t: True)
    monkeypatch.setattr(norm, "lib", no_launch)


@pytest.mark.parametrize("width", [0, 8, 32])
def test_norm_weight_of_another_width(as_native, width):
    x = _bf16(2, 3, 16)
    with pytest.raises(ValueError):
        O.rms_norm(x, _bf16(width))
    with pytest.raises(ValueError):
        O.layer_norm(x, _bf16(width), None)
    with pytest.raises(ValueError):
        O.layer_norm(x, _bf16(16), _bf16(width))


@pytest.mark.parametrize("shape", [(1, 3, 16), (2, 3, 8), (2, 6, 16)])
def test_norm_residual_of_another_shape(as_native, shape):
    with pytest.raises(ValueError):
        O.rms_norm(_bf16(2, 3, 16), _bf16(16), residual=_bf16(*shape))


@pytest.mark.parametrize("name,shape", [
    (None, None), ("attn_norm", (0,)), ("wqkv", (0,)), ("ffn_norm", (72,)), ("wqkv", (5 * 16, 64)), ("wo", (64, 80)),
    ("w_gate_up", (2 * 88, 64)), ("w_gate_up", (2 * 104, 64)), ("w_down", (64, 88)), ("x", (1, 4, 72)), ("x", (4, 64)),
    ("cos", (32, 16)), ("sin", (31, 8))])
def test_block_shapes(name, shape):
    """Only a block whose every operand has the configured shape may go to the native halves."""
    cfg = LlamaConfig.tiny(hidden_size=64, num_heads=4, num_kv_heads=2, head_dim=16, ffn_size=96)
    block = LlamaBlock(cfg, dtype=torch.bfloat16)
    ops = dict(x=_bf16(1, 4, 64), cos=torch.zeros(32, 8), sin=torch.zeros(32, 8))
    if name in ops:
        ops[name] = torch.zeros(shape, dtype=ops[name].dtype)
    elif name:
        getattr(block, name).data = _bf16(*shape)
    assert block._shapes_as_configured(**ops) == (name is None)


def test_own_cached_attention_is_kept(monkeypatch):
    """A subclass or an instance with its own cached attention never goes to the native halves."""
    class Block(LlamaBlock):
        def _attend_cached(self, *a):
            return super()._attend_cached(*a)

    cfg = LlamaConfig.tiny(hidden_size=64, num_heads=4, num_kv_heads=2, head_dim=16, ffn_size=96)
    replaced = LlamaBlock(cfg, dtype=torch.bfloat16)
    replaced._attend_cached = lambda *a: None
    x, cos = _bf16(1, 4, 64), torch.zeros(32, 8)
    asked = []
    monkeypatch.setattr(torch, "is_grad_enabled", lambda: asked.append(1) or True)   # the first question after the method
    for block, goes_on in ((LlamaBlock(cfg, dtype=torch.bfloat16), True), (Block(cfg, dtype=torch.bfloat16), False),
                           (replaced, False)):
        asked.clear()
        assert not block._plain_inference(x, cos, cos)
        assert bool(asked) == goes_on


@pytest.mark.parametrize("pos", [torch.arange(6).view(1, 6), torch.arange(13), torch.zeros(2, 6, device="meta", dtype=torch.long)])
def test_positions_that_do_not_fit(monkeypatch, pos):
    """One position per token, on the tokens' device: the kernels read as many as there are tokens."""
    def no_launch(*a):
        raise AssertionError("a kernel would have been launched")

    class OnGpu(torch.Tensor):   # a CPU tensor that takes the native branches
        is_cuda = True

    for module in (attention, rope):
        monkeypatch.setattr(module, "use_native", lambda *t: True)
        monkeypatch.setattr(module, "lib", no_launch)
    cos = torch.zeros(32, 32)
    with pytest.raises(ValueError):
        O.apply_rope(_bf16(2, 6, 4, 64).as_subclass(OnGpu), cos, cos, pos)
    with pytest.raises(ValueError):
        O.qkv_attention(_bf16(2, 6, 4 * 64).as_subclass(OnGpu), cos, cos, pos, 2, 1, 64)


@pytest.mark.parametrize("shape,pos", [((3, 2, 1, 16), 0), ((2, 3, 1, 16), 0), ((2, 2, 3, 16), 6), ((2, 2, 1, 16), 8),
                                       ((2, 2, 1, 24), 0), ((2, 2, 1, 16), -1)])
def test_append_outside_of_a_cache(monkeypatch, shape, pos):
    def no_launch(*a):
        raise AssertionError("a kernel would have been launched")

    monkeypatch.setattr(decode, "use_native", lambda *t: True)
    monkeypatch.setattr(decode, "lib", no_launch)
    cache, new = _bf16(2, 2, 8, 16), _bf16(*shape)
    with pytest.raises(ValueError):
        O.kv_append(cache, new, pos)
    with pytest.raises(ValueError):
        decode.kv_append_pair(cache, cache.clone(), new, new, pos)
