"""The work that is timed: training passes, inference passes and the single operators under them, each through the
public entry points, at sizes from this repository's configurations and benchmarks or generic ones.

Every kind of work has a range (``draw`` samples it) and one or two listed sizes that stand for it. Inputs are made from
a seed on the GPU; ``exact`` restates the same mathematics in 64-bit PyTorch without this package's operators.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

DEV = "cuda"
BF16 = torch.bfloat16

# One expert-parallel workspace per hidden size, as a model keeps one for all of its layers.
_MOE_TOKENS, _MOE_TOPK, _MOE_EXPERTS = 4096, 8, 128
_workspaces = {}


def listed():
    return [
        # the flagship training step: Llama-3-8B layer shapes and head, one sequence of 4096, forward and backward
        dict(name="llama_train_4096", kind="llama_train", B=1, T=4096, layers=2, hidden=4096, heads=32, kv=8, D=128,
             ffn=14336, vocab=128256),
        # training a smaller decoder on short sequences of odd length
        dict(name="llama_train_ragged", kind="llama_train", B=8, T=309, layers=2, hidden=1024, heads=16, kv=4, D=64,
             ffn=3592, vocab=32000),
        # a 4-layer cut of GPT-2-small, micro-batch 16 of context 1024: LayerNorm, GELU, biases, tied head
        dict(name="gpt2_train", kind="gpt2_train", B=16, T=1024, layers=4, d=768, heads=12, vocab=50257),
        # one expert FFN of the Qwen3-30B-A3B shape, forward and backward, with an uneven load of the experts
        dict(name="moe_ffn_train", kind="moe_ffn", T=4096, hidden=2048, inter=768),
        # reading a prompt: logits of every position, the cache filled
        dict(name="llama_prefill", kind="llama_generate", B=1, prompt=2900, steps=0, layers=2, hidden=4096, heads=32,
             kv=8, D=128, ffn=14336, vocab=128256),
        # batched generation: a prompt per sequence, then token after token over the growing cache
        dict(name="llama_generate_batch", kind="llama_generate", B=16, prompt=1000, steps=12, layers=2, hidden=4096,
             heads=32, kv=8, D=128, ffn=14336, vocab=128256),
        # the smallest generation: one short prompt on a small model, bound by latency and launches
        dict(name="llama_generate_one", kind="llama_generate", B=1, prompt=37, steps=8, layers=2, hidden=1024, heads=16,
             kv=4, D=64, ffn=3592, vocab=32000),
        # attention by itself on a long sequence, forward and backward
        dict(name="attention_train_long", kind="attention_train", B=1, T=8190, heads=32, kv=8, D=128, window=0),
        # attention of one new token per sequence over a long cache
        dict(name="attention_decode", kind="attention_decode", B=8, Tq=1, Tk=16381, heads=32, kv=8, D=128),
        # a 4-bit linear layer while decoding (a few rows) and while reading prompts (hundreds)
        dict(name="weight_only_decode", kind="weight_only", M=5, N=28672, K=8192, bits=4, group=128),
        dict(name="weight_only_prompt", kind="weight_only", M=777, N=14336, K=4096, bits=4, group=128),
        # the optimizer step over a small decoder's parameters (bf16 with fp32 masters and moments)
        dict(name="adamw_step", kind="adamw", layers=2, hidden=2048, ffn=7168, vocab=32000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _decoder(rng):
    hidden = rng.choice([512, 1024, 2048, 4096])
    D = rng.choice([64, 128])
    heads = hidden // D
    return dict(layers=rng.choice([1, 2]), hidden=hidden, heads=heads, kv=heads // rng.choice([1, 2, 4]), D=D,
                ffn=8 * _log(rng, hidden // 4, 7 * hidden // 16), vocab=rng.choice([32000, 50304, 128256]))


def draw(rng):
    kind = rng.choice(["llama_train", "gpt2_train", "moe_ffn", "llama_generate", "llama_generate", "attention_train",
                       "attention_decode", "weight_only", "adamw"])
    if kind == "llama_train":
        # the number of tokens of a training pass is a multiple of 8
        B = rng.choice([1, 2, 4, 8])
        T = max(1, _log(rng, 64, 4096) // 8) * (8 // B)
        return dict(kind=kind, B=B, T=T, **_decoder(rng))
    if kind == "gpt2_train":
        d = rng.choice([256, 512, 768])
        return dict(kind=kind, B=8 * rng.choice([1, 2]), T=_log(rng, 33, 1024), layers=rng.randint(1, 4), d=d, heads=d // 64,
                    vocab=rng.choice([32000, 50257]))
    if kind == "moe_ffn":
        return dict(kind=kind, T=_log(rng, 64, 4096), hidden=2048, inter=rng.choice([384, 768]))
    if kind == "llama_generate":
        B = rng.choice([1, 2, 4, 8, 16])
        return dict(kind=kind, B=B, prompt=_log(rng, 16, 4096 // B), steps=rng.randint(0, 12), **_decoder(rng))
    if kind == "attention_train":
        D, T = rng.choice([64, 128]), _log(rng, 200, 8192)
        heads = rng.choice([8, 16, 32])
        return dict(kind=kind, B=max(1, min(4, 8192 // T)), T=T, heads=heads, kv=heads // rng.choice([1, 2, 4, 8]), D=D,
                    window=rng.choice([0, 0, _log(rng, 64, 2048)]))
    if kind == "attention_decode":
        D, B = rng.choice([64, 128]), _log(rng, 1, 64)
        heads = rng.choice([8, 16, 32, 64])
        kv = heads // rng.choice([1, 2, 4, 8])
        return dict(kind=kind, B=B, Tq=rng.choice([1, 1, 1, rng.randint(2, 8)]),
                    Tk=_log(rng, 128, min(32768, 2 ** 29 // (B * kv * D))), heads=heads, kv=kv, D=D)
    if kind == "weight_only":
        bits = rng.choice([4, 8])
        return dict(kind=kind, M=_log(rng, 1, 1024), N=8 * _log(rng, 128, 3584), K=128 * _log(rng, 8, 64), bits=bits,
                    group=128 if bits == 4 else rng.choice([0, 128]))
    return dict(kind=kind, layers=rng.randint(1, 2), hidden=64 * _log(rng, 2, 40), ffn=8 * _log(rng, 32, 1024),
                vocab=rng.choice([512, 32000, 50257]))


# ----------------------------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def _llama(case, seed):
    from tensorplay_b200.models.llama import Llama, LlamaConfig
    cfg = LlamaConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], num_layers=case["layers"],
                      num_heads=case["heads"], num_kv_heads=case["kv"], head_dim=case["D"], ffn_size=case["ffn"])
    model = Llama(cfg, device=DEV, dtype=BF16)
    model.reset_parameters(seed=seed)
    return model


def _gpt2(case, seed):
    from tensorplay_b200.models.gpt2 import GPT2, GPT2Config
    cfg = GPT2Config(vocab_size=case["vocab"], n_ctx=1024, d_model=case["d"], n_layers=case["layers"], n_heads=case["heads"])
    model = GPT2(cfg, device=DEV, dtype=BF16)
    model.reset_parameters(seed=seed)
    g = _gen(seed + 7)
    with torch.no_grad():   # biases of a model in training are not zero
        for name, p in model.named_parameters():
            if p.dim() == 1 and "_w" not in name:
                p.copy_(_randn(g, *p.shape, std=0.02))
    return model


def _adamw_shapes(case):
    H, I, V = case["hidden"], case["ffn"], case["vocab"]
    out = [(V, H), (V, H), (H,)]
    for _ in range(case["layers"]):
        out += [(H,), (3 * H // 2, H), (H, H), (H,), (2 * I, H), (H, I)]
    return out


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in ("llama_train", "gpt2_train"):
        model = _llama(case, seed) if kind == "llama_train" else _gpt2(case, seed)
        tok, tgt = (torch.randint(0, case["vocab"], (case["B"], case["T"]), generator=g, device=DEV) for _ in range(2))
        return dict(case=case, model=model, tok=tok, tgt=tgt)
    if kind == "llama_generate":
        n = case["prompt"] + case["steps"]
        tok = torch.randint(0, case["vocab"], (case["B"], n), generator=g, device=DEV)
        return dict(case=case, model=_llama(case, seed), tok=tok)
    if kind == "moe_ffn":
        from tensorplay_b200.parallel.moe import MoEWorkspace
        H, I, E, k = case["hidden"], case["inter"], _MOE_EXPERTS, _MOE_TOPK
        if H not in _workspaces:
            _workspaces[H] = MoEWorkspace(_MOE_TOKENS, k, H, E, capacity_factor=1.0)
        logits = torch.randn(case["T"], E, generator=g, device=DEV) + torch.randn(E, generator=g, device=DEV) * 0.5
        w, idx = torch.topk(torch.softmax(logits, -1), k, dim=-1)
        w = (w / w.sum(-1, keepdim=True)).to(BF16)
        return dict(case=case, ws=_workspaces[H], idx=idx, x=_randn(g, case["T"], H).requires_grad_(), w=w.requires_grad_(),
                    gu=_randn(g, E, 2 * I, H, std=0.02).requires_grad_(), down=_randn(g, E, H, I, std=0.02).requires_grad_(),
                    dy=_randn(g, case["T"], H))
    if kind == "attention_train":
        B, T, Hq, Hk, D = (case[k] for k in ("B", "T", "heads", "kv", "D"))
        return dict(case=case, q=_randn(g, B, T, Hq, D).requires_grad_(), k=_randn(g, B, T, Hk, D).requires_grad_(),
                    v=_randn(g, B, T, Hk, D).requires_grad_(), do=_randn(g, B, T, Hq, D))
    if kind == "attention_decode":
        B, Tq, Tk, Hq, Hk, D = (case[k] for k in ("B", "Tq", "Tk", "heads", "kv", "D"))
        # the caches keep [B, H, S, D] with room to grow
        room = Tk + 64
        k, v = (_randn(g, B, Hk, room, D) for _ in range(2))
        return dict(case=case, q=_randn(g, B, Tq, Hq, D), k=k[:, :, :Tk].transpose(1, 2), v=v[:, :, :Tk].transpose(1, 2))
    if kind == "weight_only":
        from tensorplay_b200.quantization import WeightOnlyLinear
        lin = torch.nn.Linear(case["K"], case["N"], bias=False, device=DEV, dtype=BF16)
        with torch.no_grad():
            lin.weight.copy_(_randn(g, case["N"], case["K"], std=0.02))
        return dict(case=case, layer=WeightOnlyLinear(lin, case["bits"], case["group"]), x=_randn(g, case["M"], case["K"]))
    from tensorplay_b200.optim import AdamW
    params = [torch.nn.Parameter(_randn(g, *s, std=0.02)) for s in _adamw_shapes(case)]
    opt = AdamW(params, lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1)
    for p in params:
        p.grad = _randn(g, *p.shape, std=1e-3)
    start = [p.detach().clone() for p in params]
    first = [p.grad for p in params]
    opt.step()
    for p in params:
        p.grad = _randn(g, *p.shape, std=1e-3)
    return dict(case=case, params=params, opt=opt, start=start, grads=(first, [p.grad for p in params]))


# ----------------------------------------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("llama_train", "gpt2_train"):
        model = state["model"]
        model.zero_grad(set_to_none=True)
        loss = model(state["tok"], state["tgt"])
        loss.backward()
        return [loss.detach()] + [p.grad for p in model.parameters()]
    if kind == "llama_generate":
        model, tok, n = state["model"], state["tok"], case["prompt"]
        out = []
        with torch.no_grad():
            cache = model.create_empty_cache()
            out.append(model(tok[:, :n], past_key_values=cache))
            for i in range(n, n + case["steps"]):   # the tokens are given, so that every step's logits can be compared
                out.append(model(tok[:, i:i + 1], past_key_values=cache))
        return out
    if kind == "moe_ffn":
        from tensorplay_b200.parallel.moe import expert_parallel_ffn
        leaves = [state[n] for n in ("x", "w", "gu", "down")]
        y = expert_parallel_ffn(state["x"], state["idx"], state["w"], state["gu"], state["down"], state["ws"], _MOE_EXPERTS)
        return [y.detach()] + list(torch.autograd.grad(y, leaves, state["dy"]))
    if kind in ("attention_train", "attention_decode"):
        from tensorplay_b200 import ops
        q, k, v = state["q"], state["k"], state["v"]
        if kind == "attention_decode":
            with torch.no_grad():
                return ops.flash_attention(q, k, v, causal=True)
        o = ops.flash_attention(q, k, v, causal=True, window=case["window"])
        return [o.detach()] + list(torch.autograd.grad(o, (q, k, v), state["do"]))
    if kind == "weight_only":
        with torch.no_grad():
            return state["layer"](state["x"])
    opt = state["opt"]
    opt.step()
    st = [opt.state[p] for p in state["params"]]
    return [[p.detach() for p in state["params"]], [s["master"] for s in st], [s["exp_avg"] for s in st],
            [s["exp_avg_sq"] for s in st]]


# ----------------------------------------------------------------------------------------------- what it cannot do without

def _pairs(Tq, Tk, window=0):
    """Query-key pairs of a causal mask aligned at the end."""
    if Tq == 1:
        return Tk
    full = Tq * Tk - Tq * (Tq - 1) // 2
    if window and window < Tk:
        cut = Tk - window
        full -= cut * (cut + 1) // 2
    return full


def work(case):
    kind = case["kind"]
    if kind == "llama_train" or kind == "gpt2_train":
        n = case["B"] * case["T"]
        if kind == "llama_train":
            H, D, L, I, V = case["hidden"], case["D"], case["layers"], case["ffn"], case["vocab"]
            mm = L * (H * (case["heads"] + 2 * case["kv"]) * D + case["heads"] * D * H + 3 * H * I) + V * H
            params, width = mm + V * H, case["heads"] * D
        else:
            d, L, V = case["d"], case["layers"], case["vocab"]
            mm = L * 12 * d * d + V * d
            params, width = mm, d
        attn = 4 * L * case["B"] * width * _pairs(case["T"], case["T"])
        return {"bytes": 2 * 2 * params + 16 * n, "flops": 6 * n * mm + 3.5 * attn}
    if kind == "llama_generate":
        B, H, D, L, I, V = (case[k] for k in ("B", "hidden", "D", "layers", "ffn", "vocab"))
        layer = H * (case["heads"] + 2 * case["kv"]) * D + case["heads"] * D * H + 3 * H * I
        calls, n = 1 + case["steps"], case["prompt"] + case["steps"]
        read = sum(range(case["prompt"] + 1, n + 1))   # cached positions read by the single-token steps
        kv = 2 * 2 * L * case["kv"] * D * B
        attn = 4 * L * B * case["heads"] * D * (_pairs(case["prompt"], case["prompt"]) + read)
        return {"bytes": 2 * calls * (L * layer + V * H) + kv * (n + read) + 2 * B * n * V,
                "flops": 2 * B * n * (L * layer + V * H) + attn}
    if kind == "moe_ffn":
        T, H, I, k = case["T"], case["hidden"], case["inter"], _MOE_TOPK
        used = _MOE_EXPERTS if T * k > 4 * _MOE_EXPERTS else min(_MOE_EXPERTS, T * k)
        return {"bytes": 2 * 2 * used * 3 * H * I + 4 * 2 * T * H, "flops": 6 * T * k * 3 * H * I}
    if kind == "attention_train":
        B, T, Hq, Hk, D = (case[k] for k in ("B", "T", "heads", "kv", "D"))
        return {"bytes": 2 * B * T * D * (4 * Hq + 4 * Hk), "flops": 3.5 * 4 * B * Hq * D * _pairs(T, T, case["window"])}
    if kind == "attention_decode":
        B, Tq, Tk, Hq, Hk, D = (case[k] for k in ("B", "Tq", "Tk", "heads", "kv", "D"))
        return {"bytes": 2 * B * D * (2 * Hk * Tk + 2 * Hq * Tq), "flops": 4 * B * Hq * D * _pairs(Tq, Tk)}
    if kind == "weight_only":
        M, N, K = case["M"], case["N"], case["K"]
        groups = N * (K // case["group"] if case["group"] else 1)
        return {"bytes": N * K * case["bits"] // 8 + 2 * groups * (2 if case["bits"] == 4 else 1) + 2 * M * (N + K),
                "flops": 2 * M * N * K}
    n = sum(math.prod(s) for s in _adamw_shapes(case))
    return {"bytes": n * (2 + 3 * 4 + 3 * 4 + 2), "flops": 14 * n}


# ----------------------------------------------------------------------------------------------- tolerance

def tolerance(case):
    # about four times the distance from the 64-bit result that bf16 activations and gradients show at the listed and
    # drawn sizes (0.015-0.029 and 0.012 for the training passes, 0.015 for logits, 0.0042 for the experts, 0.0025 for
    # attention, 0.0022 for the quantised layers, 0.0019 for the bf16 copy of the updated weights)
    return {"rel": {"llama_train": 0.08, "gpt2_train": 0.05, "llama_generate": 0.06, "moe_ffn": 0.016,
                    "attention_train": 0.01, "attention_decode": 0.01, "weight_only": 0.009, "adamw": 0.006}[case["kind"]]}


# ----------------------------------------------------------------------------------------------- 64-bit restatement

def _attend(q, k, v, window=0):
    """Causal attention of ``[T, D]`` matrices of one head in their own precision."""
    Tq, Tk = q.shape[0], k.shape[0]
    s = (q @ k.t()) / math.sqrt(q.shape[1])
    i = torch.arange(Tq, device=q.device).view(-1, 1) + (Tk - Tq)
    j = torch.arange(Tk, device=q.device).view(1, -1)
    hide = j > i
    if window:
        hide |= j < i - window + 1
    return torch.softmax(s.masked_fill(hide, float("-inf")), -1) @ v


def _attention(q, k, v, window=0):
    """``[B, T, H, D]`` grouped-query attention, head by head."""
    B, _, Hq, _ = q.shape
    g = Hq // k.shape[2]
    rows = []
    for b in range(B):
        heads = [checkpoint(_attend, q[b, :, h], k[b, :, h // g], v[b, :, h // g], window, use_reentrant=False)
                 for h in range(Hq)]
        rows.append(torch.stack(heads, 1))
    return torch.stack(rows)


def _rms(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _rotate(x, theta):
    T, D = x.shape[1], x.shape[3]
    inv = theta ** (-torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)
    ang = torch.outer(torch.arange(T, dtype=torch.float64, device=x.device), inv).view(1, T, 1, D // 2)
    a, b = x[..., : D // 2], x[..., D // 2:]
    return torch.cat((a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()), -1)


def _llama_logits(case, p, tok):
    B, T = tok.shape
    Hq, Hk, D, I = case["heads"], case["kv"], case["D"], case["ffn"]
    x = p["embed"][tok]
    for i in range(case["layers"]):
        w = {n: p[f"layers.{i}.{n}"] for n in ("attn_norm", "wqkv", "wo", "ffn_norm", "w_gate_up", "w_down")}
        qkv = (_rms(x, w["attn_norm"]) @ w["wqkv"].t()).view(B, T, Hq + 2 * Hk, D)
        qk = _rotate(qkv[:, :, :Hq + Hk], 500000.0)
        a = _attention(qk[:, :, :Hq], qk[:, :, Hq:], qkv[:, :, Hq + Hk:]).reshape(B, T, Hq * D)
        x = x + a @ w["wo"].t()
        gu = _rms(x, w["ffn_norm"]) @ w["w_gate_up"].t()
        x = x + (F.silu(gu[..., :I]) * gu[..., I:]) @ w["w_down"].t()
    return _rms(x, p["final_norm"]) @ p["lm_head"].t()


def _gpt2_logits(case, p, tok):
    B, T = tok.shape
    d, H = case["d"], case["heads"]
    x = p["wte"][tok] + p["wpe"][:T]
    for i in range(case["layers"]):
        w = {n[len(f"layers.{i}."):]: t for n, t in p.items() if n.startswith(f"layers.{i}.")}
        h = F.layer_norm(x, (d,), w["ln1_w"], w["ln1_b"], 1e-5)
        qkv = (h @ w["w_qkv"].t() + w["b_qkv"]).view(B, T, 3, H, d // H)
        a = _attention(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]).reshape(B, T, d)
        x = x + a @ w["w_o"].t() + w["b_o"]
        h = F.layer_norm(x, (d,), w["ln2_w"], w["ln2_b"], 1e-5)
        x = x + F.gelu(h @ w["w_fc"].t() + w["b_fc"], approximate="tanh") @ w["w_proj"].t() + w["b_proj"]
    return F.layer_norm(x, (d,), p["lnf_w"], p["lnf_b"], 1e-5) @ p["wte"][: case["vocab"]].t()


def exact(case, seed):
    state = prepare(case, seed)
    kind = case["kind"]
    if kind in ("llama_train", "gpt2_train"):
        p = {n: t.detach().double().requires_grad_() for n, t in state["model"].named_parameters()}
        logits = (_llama_logits if kind == "llama_train" else _gpt2_logits)(case, p, state["tok"])
        loss = F.cross_entropy(logits.view(-1, logits.shape[-1]), state["tgt"].view(-1))
        loss.backward()
        return [loss.detach()] + [t.grad for t in p.values()]
    if kind == "llama_generate":
        with torch.no_grad():
            p = {n: t.detach().double() for n, t in state["model"].named_parameters()}
            logits = _llama_logits(case, p, state["tok"])
        n = case["prompt"]
        return [logits[:, :n]] + [logits[:, i:i + 1] for i in range(n, n + case["steps"])]
    if kind == "moe_ffn":
        x, w, gu, down = (state[n].detach().double().requires_grad_() for n in ("x", "w", "gu", "down"))
        I, y = case["inter"], torch.zeros_like(x)
        for e in range(_MOE_EXPERTS):
            tok, slot = (state["idx"] == e).nonzero(as_tuple=True)
            h = x[tok] @ gu[e].t()
            y = y.index_add(0, tok, ((F.silu(h[:, :I]) * h[:, I:]) @ down[e].t()) * w[tok, slot].unsqueeze(-1))
        return [y.detach()] + list(torch.autograd.grad(y, (x, w, gu, down), state["dy"].double()))
    if kind == "attention_train":
        q, k, v = (state[n].detach().double().requires_grad_() for n in ("q", "k", "v"))
        o = _attention(q, k, v, case["window"])
        return [o.detach()] + list(torch.autograd.grad(o, (q, k, v), state["do"].double()))
    if kind == "attention_decode":
        with torch.no_grad():
            return _attention(*(state[n].double() for n in ("q", "k", "v")))
    if kind == "weight_only":
        m = state["layer"]
        q, N, K = m.qweight, case["N"], case["K"]
        if case["bits"] == 4:
            code = torch.stack((q & 0xF, q >> 4), dim=-1).reshape(N, K).double()
        else:
            code = q.double()
        code = code.view(N, m.scale.shape[1], -1)
        if m.zero is not None:
            code = code - m.zero.double().unsqueeze(-1)
        return state["x"].double() @ (code * m.scale.double().unsqueeze(-1)).view(N, K).t()
    out = [[], [], [], []]
    for p0, g1, g2 in zip(state["start"], *state["grads"]):
        p, m, s = p0.double(), 0.0, 0.0
        for t, gr in ((1, g1.double()), (2, g2.double())):
            p = p * (1 - 3e-4 * 0.1)
            m, s = 0.9 * m + 0.1 * gr, 0.95 * s + 0.05 * gr * gr
            p = p - 3e-4 * (m / (1 - 0.9 ** t)) / ((s / (1 - 0.95 ** t)).sqrt() + 1e-8)
        for dst, t in zip(out, (p, p, m, s)):
            dst.append(t)
    return out
