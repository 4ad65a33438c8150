"""Llama-family decoder (RMSNorm, RoPE, grouped-query attention, SwiGLU) with packed QKV and
gate/up projections, so that a layer is four GEMMs plus row kernels.

Shapes follow the named configurations: Llama-3-8B (32 layers, hidden 4096, 32/8 heads of 128,
FFN 14336, vocab 128256, theta 5e5) and Llama-3-70B (80 layers, hidden 8192, 64/8 heads,
FFN 28672). The reference composes the same math from ``nn.GroupedQueryAttention`` /
``nn.SwiGLUMLP`` / ``nn.RMSNorm`` (tensorplay/nn/modules/causal_attention.py:30-187,
modern_block.py:29-103).
"""
from __future__ import annotations

import math
from array import array
from dataclasses import dataclass
from typing import Optional

import torch
from torch import Tensor, nn

from torch.nn.modules import module as _nn_module

from .. import _native, ops
from ..nn.cache import DynamicCache, StaticCache
from ..ops._common import lib, status_word, stream_ptr, use_native, watched
from ..ops.attention import few_rows_sizes
from ..ops.rope import flat_positions


@dataclass
class LlamaConfig:
    vocab_size: int = 128256
    hidden_size: int = 4096
    num_layers: int = 32
    num_heads: int = 32
    num_kv_heads: int = 8
    head_dim: int = 128
    ffn_size: int = 14336
    rms_eps: float = 1e-5
    rope_theta: float = 500000.0
    max_seq_len: int = 4096
    tie_embeddings: bool = False
    init_std: float = 0.02

    @staticmethod
    def llama3_8b(**kw) -> "LlamaConfig":
        return LlamaConfig(**kw)

    @staticmethod
    def llama3_70b(**kw) -> "LlamaConfig":
        return LlamaConfig(hidden_size=8192, num_layers=80, num_heads=64, num_kv_heads=8,
                           ffn_size=28672, **kw)

    @staticmethod
    def tiny(**kw) -> "LlamaConfig":
        base = dict(vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, num_kv_heads=2,
                    head_dim=64, ffn_size=512, max_seq_len=256)
        base.update(kw)
        return LlamaConfig(**base)

    def num_params(self) -> int:
        per_layer = (self.hidden_size * (self.num_heads + 2 * self.num_kv_heads) * self.head_dim
                     + self.num_heads * self.head_dim * self.hidden_size
                     + 3 * self.hidden_size * self.ffn_size + 2 * self.hidden_size)
        emb = self.vocab_size * self.hidden_size
        return self.num_layers * per_layer + emb * (1 if self.tie_embeddings else 2) + self.hidden_size

    def flops_per_token(self, seq_len: int, backward: bool = True, recompute: bool = False) -> float:
        """Model FLOPs per token: 2 * matmul params (+ causal attention), x3 with backward."""
        mm = self.num_params() - self.vocab_size * self.hidden_size * (0 if self.tie_embeddings else 1) \
            - self.hidden_size * (2 * self.num_layers + 1)
        fwd = 2.0 * mm + 2.0 * 2 * self.num_layers * self.num_heads * self.head_dim * seq_len / 2
        mult = 1.0 + (2.0 if backward else 0.0) + (1.0 if recompute else 0.0)
        return fwd * mult


def _plain(w, shape, dev) -> bool:
    """A bf16 parameter that a kernel may read by its address."""
    return type(w) is nn.Parameter and w.dtype is torch.bfloat16 and w.device == dev and w.shape == shape \
        and w.is_contiguous() and not w.data_ptr() % 16


class LlamaBlock(nn.Module):
    def __init__(self, cfg: LlamaConfig, layer_idx: int = 0, device=None, dtype=None) -> None:
        super().__init__()
        kw = {"device": device, "dtype": dtype}
        H, D = cfg.hidden_size, cfg.head_dim
        self.cfg = cfg
        self.layer_idx = layer_idx
        self.attn_norm = nn.Parameter(torch.ones(H, **kw))
        self.wqkv = nn.Parameter(torch.empty((cfg.num_heads + 2 * cfg.num_kv_heads) * D, H, **kw))
        self.wo = nn.Parameter(torch.empty(H, cfg.num_heads * D, **kw))
        self.ffn_norm = nn.Parameter(torch.ones(H, **kw))
        self.w_gate_up = nn.Parameter(torch.empty(2 * cfg.ffn_size, H, **kw))
        self.w_down = nn.Parameter(torch.empty(H, cfg.ffn_size, **kw))

    def reset_parameters(self, generator=None) -> None:
        for w in (self.wqkv, self.wo, self.w_gate_up, self.w_down):
            nn.init.normal_(w, mean=0.0, std=self.cfg.init_std, generator=generator)
        nn.init.ones_(self.attn_norm)
        nn.init.ones_(self.ffn_norm)

    def forward(self, x: Tensor, cos: Tensor, sin: Tensor, position_ids: Optional[Tensor] = None,
                past_key_values=None) -> Tensor:
        cfg = self.cfg
        if past_key_values is not None and self._plain_inference(x, cos, sin):
            return self._infer_cached(x, cos, sin, position_ids, past_key_values)
        h = ops.rms_norm(x, self.attn_norm, cfg.rms_eps)
        qkv = ops.linear(h, self.wqkv)
        if past_key_values is None:
            a = ops.qkv_attention(qkv, cos, sin, position_ids, cfg.num_heads, cfg.num_kv_heads,
                                  cfg.head_dim, causal=True)
        else:
            a = self._attend_cached(qkv, cos, sin, position_ids, past_key_values)
        a = ops.linear(a, self.wo)
        h, x = ops.rms_norm(a, self.ffn_norm, cfg.rms_eps, residual=x)
        gu = ops.linear(h, self.w_gate_up)
        return x + ops.linear(ops.swiglu_packed(gu), self.w_down)

    def _weights(self):
        return self.attn_norm, self.ffn_norm, self.wqkv, self.wo, self.w_gate_up, self.w_down

    def _shapes_as_configured(self, x: Tensor, cos: Tensor, sin: Tensor, weights=None) -> bool:
        """Whether every operand has the shape that the native halves of the block read it with. They take all sizes from
        ``cfg``; a pruned or widened weight, the empty placeholder of a sharded one or an input of another width goes
        operator by operator, where sizes come from the tensors and a mismatch raises."""
        cfg = self.cfg
        H, I, D = cfg.hidden_size, cfg.ffn_size, cfg.head_dim
        A, table = cfg.num_heads * D, cos.shape
        attn_norm, ffn_norm, wqkv, wo, w_gate_up, w_down = weights or self._weights()
        return (x.dim() == 3 and x.shape[2] == H and attn_norm.shape == (H,) and ffn_norm.shape == (H,)
                and wqkv.shape == (A + 2 * cfg.num_kv_heads * D, H) and wo.shape == (H, A)
                and w_gate_up.shape == (2 * I, H) and w_down.shape == (H, I)
                and len(table) == 2 and table[1] == D // 2 and sin.shape == table)

    def _plain_inference(self, x: Tensor, cos: Tensor, sin: Tensor) -> bool:
        """Whether a forward pass with a cache may go to the native halves of the block: plain CUDA bf16 tensors of the
        configured shapes, no gradient, and nothing that watches, transforms or replaces single steps."""
        if getattr(self._attend_cached, "__func__", None) is not LlamaBlock._attend_cached:
            return False   # a subclass or an instance brings its own cached attention
        if torch.is_grad_enabled() or type(x) is not Tensor or not x.is_cuda or x.dtype != torch.bfloat16 \
                or not x.is_contiguous() or x.data_ptr() % 16 or x.numel() == 0 or self.cfg.head_dim not in (64, 128) \
                or self.cfg.hidden_size % 8 or self.cfg.ffn_size % 8:
            return False
        if watched():
            return False
        dev = x.device
        weights = self._weights()
        for w in weights:
            if type(w) is not nn.Parameter or w.dtype != torch.bfloat16 or w.device != dev or not w.is_contiguous() \
                    or w.data_ptr() % 16:
                return False
        for t in (cos, sin):
            if type(t) is not Tensor or t.dtype != torch.float32 or t.device != dev or not t.is_contiguous() \
                    or t.data_ptr() % 16:
                return False
        return self._shapes_as_configured(x, cos, sin, weights) and dev.index == torch._C._cuda_getDevice() and use_native(x)

    def _infer_cached(self, x: Tensor, cos: Tensor, sin: Tensor, position_ids: Optional[Tensor], cache) -> Tensor:
        """The block as two native calls around the cache and the attention. Of at most 128 rows the last product is
        accumulated into the residual stream."""
        cfg = self.cfg
        B, T, H = x.shape
        Hq, Hkv, D, I = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim, cfg.ffn_size
        off = cache.get_seq_length(self.layer_idx)
        pos = flat_positions(position_ids, B * T, x.device)
        if pos is None and off + T > cos.shape[0]:
            raise IndexError(f"rotary tables of {cos.shape[0]} positions are too short for position {off + T - 1}")
        rows, tot, L = B * T, Hq + 2 * Hkv, lib()
        st, stream = status_word(x.device).data_ptr(), stream_ptr()
        qkv, qk = x.new_empty(B, T, tot, D), x.new_empty(B, T, Hq + Hkv, D)
        scratch = x.new_empty(rows * (2 * H + 3 * I))
        h = scratch.data_ptr()
        o, gu = h + 2 * rows * H, h + 4 * rows * H
        act = gu + 4 * rows * I
        _native.check(L.tpb_block_pre(
            x.data_ptr(), self.attn_norm.data_ptr(), cfg.rms_eps, self.wqkv.data_ptr(), h, qkv.data_ptr(), qk.data_ptr(),
            cos.data_ptr(), sin.data_ptr(), None if pos is None else pos.data_ptr(), off, rows, T, H, Hq, Hkv, D, st,
            stream), "tpb_block_pre")
        k, v = cache.update(qk[:, :, Hq:].transpose(1, 2), qkv[:, :, Hq + Hkv:].transpose(1, 2), self.layer_idx)
        a = ops.flash_attention(qk[:, :, :Hq], k.transpose(1, 2), v.transpose(1, 2), causal=True)
        if not a.is_contiguous():
            a = a.contiguous()
        x2 = torch.empty_like(x)
        y = x2 if rows <= 128 else torch.empty_like(x)
        _native.check(L.tpb_block_post(
            a.data_ptr(), self.wo.data_ptr(), o, x.data_ptr(), self.ffn_norm.data_ptr(), cfg.rms_eps, x2.data_ptr(), h,
            self.w_gate_up.data_ptr(), gu, act, self.w_down.data_ptr(), y.data_ptr(), int(y is x2), rows, H, Hq * D, I, st,
            stream), "tpb_block_post")
        return x2 if y is x2 else x2 + y

    def _attend_cached(self, qkv, cos, sin, position_ids, cache):
        cfg = self.cfg
        B, T, _ = qkv.shape
        Hq, Hkv, D = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim
        packed = qkv.view(B, T, Hq + 2 * Hkv, D)
        off = cache.get_seq_length(self.layer_idx)
        pos = position_ids
        if pos is None and off:
            pos = torch.arange(off, off + T, device=qkv.device).expand(B, T)
        qk = ops.apply_rope(packed[:, :, : Hq + Hkv], cos, sin, pos)
        k, v = cache.update(qk[:, :, Hq:].transpose(1, 2), packed[:, :, Hq + Hkv:].transpose(1, 2),
                            self.layer_idx)
        o = ops.flash_attention(qk[:, :, :Hq], k.transpose(1, 2), v.transpose(1, 2), causal=True)
        return o.reshape(B, T, Hq * D)


class Llama(nn.Module):
    """Decoder-only LM. ``forward(tokens, targets=None)`` returns logits, or the mean
    next-token loss when ``targets`` is given."""

    def __init__(self, cfg: LlamaConfig, device=None, dtype=None) -> None:
        super().__init__()
        kw = {"device": device, "dtype": dtype}
        self.cfg = cfg
        self.embed = nn.Parameter(torch.empty(cfg.vocab_size, cfg.hidden_size, **kw))
        self.layers = nn.ModuleList([LlamaBlock(cfg, i, **kw) for i in range(cfg.num_layers)])
        self.final_norm = nn.Parameter(torch.ones(cfg.hidden_size, **kw))
        if cfg.tie_embeddings:
            self.lm_head = None
        else:
            self.lm_head = nn.Parameter(torch.empty(cfg.vocab_size, cfg.hidden_size, **kw))
        self._rope = None

    def reset_parameters(self, seed: Optional[int] = None) -> None:
        gen = None
        if seed is not None:
            gen = torch.Generator(device=self.embed.device)
            gen.manual_seed(seed)
        nn.init.normal_(self.embed, std=self.cfg.init_std, generator=gen)
        if self.lm_head is not None:
            nn.init.normal_(self.lm_head, std=self.cfg.init_std, generator=gen)
        nn.init.ones_(self.final_norm)
        for layer in self.layers:
            layer.reset_parameters(gen)

    def rope_tables(self, n: int, device):
        if self._rope is None or self._rope[0].shape[0] < n or self._rope[0].device != torch.device(device):
            self._rope = ops.rope_tables(max(n, self.cfg.max_seq_len), self.cfg.head_dim,
                                         self.cfg.rope_theta, device=device)
        return self._rope

    def layer_extra_args(self, tokens: Tensor):
        """Per-step arguments every block receives after the hidden states (RoPE tables)."""
        return self.rope_tables(tokens.shape[1], tokens.device)

    def create_empty_cache(self):
        from ..nn.cache import DynamicCache
        return DynamicCache()

    def embed_tokens(self, tokens: Tensor) -> Tensor:
        return _embedding(tokens, self.embed)

    def head(self, x: Tensor, targets: Optional[Tensor] = None) -> Tensor:
        h = ops.rms_norm(x, self.final_norm, self.cfg.rms_eps)
        w = self.embed if self.lm_head is None else self.lm_head
        logits = ops.linear(h, w)
        if targets is None:
            return logits
        return ops.cross_entropy(logits.view(-1, logits.shape[-1]), targets.reshape(-1))

    def forward(self, tokens: Tensor, targets: Optional[Tensor] = None,
                position_ids: Optional[Tensor] = None, past_key_values=None) -> Tensor:
        B, T = tokens.shape
        if past_key_values is not None and targets is None and 0 < B * T <= 128:
            logits = self._infer_cached(tokens, position_ids, past_key_values)
            if logits is not None:
                return logits
        off = past_key_values.get_seq_length(0) if past_key_values is not None else 0
        cos, sin = self.rope_tables(off + T, tokens.device)
        x = self.embed_tokens(tokens)
        for layer in self.layers:
            x = layer(x, cos, sin, position_ids, past_key_values)
        return self.head(x, targets)


    def _plain_layers(self, dev):
        """Addresses of the layers' weights, six per layer, or None where a layer is not a plain one: another class or
        configuration, a method of its own, a hook, a weight that is not a bf16 parameter of the configured shape."""
        cfg = self.cfg
        H, I, A = cfg.hidden_size, cfg.ffn_size, cfg.num_heads * cfg.head_dim
        shapes = (("attn_norm", (H,)), ("wqkv", (A + 2 * cfg.num_kv_heads * cfg.head_dim, H)), ("wo", (H, A)),
                  ("ffn_norm", (H,)), ("w_gate_up", (2 * I, H)), ("w_down", (H, I)))
        found = []
        for i, layer in enumerate(self.layers):
            if type(layer) is not LlamaBlock or layer.cfg is not cfg or layer.layer_idx != i or layer._forward_hooks \
                    or layer._forward_pre_hooks or layer._compiled_call_impl is not None \
                    or not _BLOCK_METHODS.isdisjoint(layer.__dict__):
                return None
            own = layer._parameters
            for name, shape in shapes:
                w = own.get(name)
                if not _plain(w, shape, dev):
                    return None
                found.append(w.data_ptr())
        return found

    def _infer_cached(self, tokens: Tensor, position_ids: Optional[Tensor], cache) -> Optional[Tensor]:
        """The logits of a few rows over a contiguous cache by one native call, which launches what the pass launches operator
        by operator; None where the model, its layers or the cache are not plain ones or something looks on."""
        cfg = self.cfg
        H, Hq, Hkv, D, I, V = cfg.hidden_size, cfg.num_heads, cfg.num_kv_heads, cfg.head_dim, cfg.ffn_size, cfg.vocab_size
        kind = type(cache)
        if type(self) is not Llama or (kind is not DynamicCache and kind is not StaticCache) or torch.is_grad_enabled() \
                or type(tokens) is not Tensor or not tokens.is_cuda or tokens.dtype is not torch.int64 \
                or D not in (64, 128) or H % 8 or I % 8 or V % 8 or Hq % Hkv or watched() \
                or type(self.layers) is not nn.ModuleList or _methods() != _METHODS \
                or not _MODEL_METHODS.isdisjoint(self.__dict__) or not _CACHE_METHODS.isdisjoint(cache.__dict__) \
                or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
            return None
        dev = tokens.device
        if dev.index != torch._C._cuda_getDevice() or not use_native(tokens):
            return None
        own = self._parameters
        embed, final_norm = own.get("embed"), own.get("final_norm")
        head = own.get("lm_head")
        if head is None and self.lm_head is None:
            head = embed
        if not (_plain(embed, (V, H), dev) and _plain(final_norm, (H,), dev) and _plain(head, (V, H), dev)):
            return None
        weights = self._plain_layers(dev)
        if weights is None:
            return None
        B, T = tokens.shape
        tokens = tokens.contiguous()
        n_layers, rows = len(self.layers), B * T
        past = cache.get_seq_length(0)
        kv_shape = (B, Hkv, T, D)
        for i in range(n_layers):
            buf, vbuf = cache._k.get(i), cache._v.get(i)
            if cache._len.get(i, 0) != past or (buf is not None and not (
                    type(buf) is type(vbuf) is Tensor and buf.dtype is vbuf.dtype is torch.bfloat16 and buf.device == dev
                    and vbuf.device == dev and buf.shape == vbuf.shape and buf.shape[0] == B and buf.shape[1] == Hkv
                    and buf.shape[3] == D and buf.is_contiguous() and vbuf.is_contiguous())):
                return None
        cos, sin = self.rope_tables(past + T, dev)
        for t in (cos, sin):
            if type(t) is not Tensor or t.dtype is not torch.float32 or t.device != dev or not t.is_contiguous() \
                    or t.data_ptr() % 16 or t.dim() != 2 or t.shape[1] != D // 2 or t.shape != cos.shape \
                    or (position_ids is None and t.shape[0] < past + T):
                return None
        pos = flat_positions(position_ids, rows, dev)
        L, Tk = lib(), past + T
        logits = embed.new_empty(B, T, V)
        scratch = logits.new_empty(L.tpb_llama_cached_scratch(rows, H, Hq, Hkv, D, I))
        few = few_rows_sizes(B, T, Tk, Hq, Hkv, D)
        splits = L.tpb_flash_decode_splits(B, T, Tk, Hq, Hkv, D) if few and Tk > 2048 else 0
        lse_stride = (T + 127) // 128 * 128
        part_rows = splits * B * Hq * T   # fp32 partial rows and their sums, as the operator's
        stats = torch.empty(B * Hq * lse_stride + part_rows * (D + 1), dtype=torch.float32, device=dev)
        lse = stats.data_ptr()
        part = lse + 4 * B * Hq * lse_stride if splits else 0
        words = array("q", (
            tokens.data_ptr(), embed.data_ptr(), final_norm.data_ptr(), head.data_ptr(), logits.data_ptr(), cos.data_ptr(),
            sin.data_ptr(), 0 if pos is None else pos.data_ptr(), status_word(dev).data_ptr(), scratch.data_ptr(), part,
            part + 4 * part_rows * D if splits else 0, lse, lse_stride, splits, int(few), B, T, past, H, Hq, Hkv, D, I, V,
            n_layers))
        for i in range(n_layers):
            cache.room(kv_shape, kv_shape, logits, logits, i)
            k = cache._k[i]
            room = k.shape[2]
            if room < Tk:   # buffers of before the cache was allowed more: the append layer by layer refuses
                return None
            words.extend(weights[6 * i:6 * i + 6])
            words.extend((k.data_ptr(), cache._v[i].data_ptr(), room))
        _native.check(L.tpb_llama_cached(words.buffer_info()[0], cfg.rms_eps, 1.0 / math.sqrt(D), stream_ptr()),
                      "tpb_llama_cached")
        _native.launch_count += 3 + n_layers * (10 + (splits > 0))
        for i in range(n_layers):
            cache.advance(T, i)
        return logits


# What a pass operator by operator calls: where one of these was replaced, on a class or on an instance, it is called.
_MODEL_METHODS = frozenset(("embed_tokens", "head", "rope_tables"))
_BLOCK_METHODS = frozenset(("forward", "_attend_cached", "_infer_cached", "_plain_inference", "_weights",
                            "_shapes_as_configured"))
_CACHE_METHODS = frozenset(("update", "get_seq_length"))


def _methods():
    return (Llama.embed_tokens, Llama.head, LlamaBlock.__call__, LlamaBlock.forward, LlamaBlock._attend_cached,
            LlamaBlock._infer_cached, LlamaBlock._plain_inference, LlamaBlock._weights, LlamaBlock._shapes_as_configured,
            DynamicCache.update, DynamicCache.get_seq_length, StaticCache.update,
            StaticCache.get_seq_length, ops.embedding, ops.rms_norm, ops.linear, ops.flash_attention)


_METHODS = _methods()


def _embedding(tokens: Tensor, weight: Tensor) -> Tensor:
    """Row gather; the backward scatter-adds straight into the weight's gradient buffer."""
    return ops.embedding(tokens, weight)
