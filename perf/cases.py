"""The work that programs built on this framework spend their time on, as cases that can be timed and checked.

Six kinds, all through public entry points: flash attention forward and backward (``ops.attention``), a Mamba-2 block forward and
backward (``Mamba2Block``), a whole training step of a Llama-family decoder (``TrainEngine.step``), prompts and decode steps of a
served Llama-family decoder, with bf16 or quantised weights (``LlamaPagedRunner``), and decode steps of a served Mamba-2 model
(``StatefulRunner``). Widths, heads and states are those of the presets (``models/config.py``) with fewer layers; lengths and batches
run from a few tokens to the longest sequences that the presets allow.
"""
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

DEV = "cuda"

# (heads, key heads) of the presets; head size 128 except where a case says 64
HEADS = [(8, 2), (16, 16), (28, 4), (32, 8), (32, 32)]
# width, heads, key heads, feed-forward: the small test model, Llama-3 8B / Mistral 7B, Qwen2 7B
WIDTHS = {"tiny": (512, 4, 2, 1024), "8b": (4096, 32, 8, 14336), "qwen2": (3584, 28, 4, 18944)}
# width and groups of the two Mamba-2 presets
MAMBA = {"130m": (768, 1), "2.7b": (2560, 8)}


def listed():
    return [
        # one short, ragged batch: a fine-tuning batch of sentences, bound by launches and host time
        dict(name="attention_short", kind="attention", batch=2, q_len=77, kv_len=77, heads=8, kv_heads=2, dim=128, causal=True, window=0),
        # the attention of the headline training step: Llama-3 8B heads, 4096 tokens
        dict(name="attention_4k", kind="attention", batch=1, q_len=4096, kv_len=4096, heads=32, kv_heads=8, dim=128, causal=True, window=0),
        # long-context training
        dict(name="attention_16k", kind="attention", batch=1, q_len=16384, kv_len=16384, heads=32, kv_heads=8, dim=128, causal=True, window=0),
        # a layer of the 130M Mamba-2 preset on a ragged batch
        dict(name="mamba_block_130m", kind="mamba_block", size="130m", batch=4, tokens=500),
        # a layer of the 2.7B Mamba-2 preset at its training length
        dict(name="mamba_block_2.7b", kind="mamba_block", size="2.7b", batch=1, tokens=8192),
        # a training step of a test-size decoder: hundreds of small launches
        dict(name="train_tiny", kind="train", size="tiny", layers=2, vocab=4096, batch=2, tokens=256),
        # the headline training step with two of its layers
        dict(name="train_8b", kind="train", size="8b", layers=2, vocab=32000, batch=1, tokens=4096),
        # prompts of a served 8B-width decoder, prefilled as one batch of odd length
        dict(name="prefill_8b", kind="serve", size="8b", layers=4, batch=4, context=0, prompt=1511, steps=0, quant=""),
        # one user: decode steps are bound by reading the weights
        dict(name="decode_8b_1", kind="serve", size="8b", layers=4, batch=1, context=1008, prompt=0, steps=16, quant=""),
        # a full decode batch over long contexts: weights and cache
        dict(name="decode_8b_48", kind="serve", size="8b", layers=4, batch=48, context=1808, prompt=0, steps=16, quant=""),
        # a quantised model at a middling batch
        dict(name="decode_8b_int4_16", kind="serve", size="8b", layers=4, batch=16, context=512, prompt=0, steps=16, quant="int4"),
        # decode steps of a served Mamba-2 model
        dict(name="mamba_decode_16", kind="mamba_decode", size="2.7b", layers=8, batch=16, prompt=96, steps=4),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["attention", "attention", "mamba_block", "train", "serve", "serve", "mamba_decode"])
    if kind == "attention":
        heads, kv_heads = rng.choice(HEADS)
        n = _log(rng, 16, 16384)
        kv = n if rng.random() < 0.8 else min(16384, n + _log(rng, 16, 4096))     # queries that follow cached keys
        causal = kv != n or rng.random() < 0.85
        n, kv = (n, kv) if causal else (min(n, 11585), min(kv, 11585))
        most = max(1, min(8, int((1 << 28) * 32 / (kv * kv * heads * (1 if causal else 2)))))
        return dict(kind=kind, batch=rng.randint(1, most), q_len=n, kv_len=kv, heads=heads, kv_heads=kv_heads,
                    dim=64 if rng.random() < 0.2 else 128, causal=causal, window=_log(rng, 64, 4096) if causal and rng.random() < 0.25 else 0)
    if kind == "mamba_block":
        tokens = _log(rng, 16, 8192)
        return dict(kind=kind, size=rng.choice(sorted(MAMBA)), batch=rng.randint(1, max(1, min(8, 8192 // tokens))), tokens=tokens)
    if kind == "train":
        size = rng.choice(sorted(WIDTHS))
        tokens = _log(rng, 32, 4096)
        return dict(kind=kind, size=size, layers=rng.randint(1, 2) if size != "qwen2" else 1, vocab=rng.choice([4096, 32000]),
                    batch=rng.randint(1, max(1, min(8, 4096 // tokens))), tokens=tokens)
    if kind == "serve":
        size, layers = rng.choice(["8b", "qwen2"]), rng.randint(1, 4)
        if rng.random() < 0.4:
            n = _log(rng, 16, 6000)
            return dict(kind=kind, size=size, layers=layers, batch=rng.randint(1, max(1, min(8, 6000 // n))), context=0, prompt=n, steps=0,
                        quant=rng.choice(["", "", "int4", "fp8"]))
        return dict(kind=kind, size=size, layers=layers, batch=_log(rng, 1, 48), context=16 * _log(rng, 1, 112), prompt=0, steps=16,
                    quant=rng.choice(["", "int4", "fp8"]))
    return dict(kind=kind, size=rng.choice(sorted(MAMBA)), layers=rng.randint(2, 8), batch=_log(rng, 1, 16), prompt=_log(rng, 8, 200), steps=4)


# ----------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * std).to(dtype)


def _tokens(seed, vocab, *shape):
    return np.random.RandomState((int(seed) * 31 + 5) % (1 << 31)).randint(0, vocab, shape)


def _llama_weights(case, seed):
    """Weights by parameter name: normal matrices of standard deviation 0.02, norm weights near one."""
    d, h, hk, ff = WIDTHS[case["size"]]
    g, vocab = _gen(seed), case.get("vocab", 32000)
    near_one = lambda: (1 + 0.1 * torch.randn(d, generator=g, device=DEV)).to(torch.bfloat16)
    w = {"embedding.weight": _normal(g, vocab, d, std=0.02)}
    for i in range(case["layers"]):
        p = f"layers.{i}."
        w[p + "attn_norm.weight"] = near_one()
        w[p + "attn.qkv_proj.weight"] = _normal(g, (h + 2 * hk) * 128, d, std=0.02)
        w[p + "attn.o_proj.weight"] = _normal(g, d, h * 128, std=0.02)
        w[p + "mlp_norm.weight"] = near_one()
        w[p + "mlp.gate_up_proj.weight"] = _normal(g, 2 * ff, d, std=0.02)
        w[p + "mlp.down_proj.weight"] = _normal(g, d, ff, std=0.02)
    w["norm.weight"] = near_one()
    w["lm_head.weight"] = _normal(g, vocab, d, std=0.02)
    return w


def _mamba_weights(g, size, prefix=""):
    """Weights of one Mamba-2 block with the published initialisation: decays in [1, 16], step sizes in [1e-3, 1e-1]."""
    d, groups = MAMBA[size]
    inner, heads = 2 * d, 2 * d // 64
    conv = inner + 2 * groups * 128
    uniform = lambda n: torch.rand(n, generator=g, device=DEV)
    dt = torch.exp(uniform(heads) * (math.log(1e-1) - math.log(1e-3)) + math.log(1e-3))
    w = {"in_proj.weight": _normal(g, 2 * inner + 2 * groups * 128 + heads, d, std=0.02),
         "conv_weight": ((torch.rand(conv, 4, generator=g, device=DEV) - 0.5)).to(torch.bfloat16),
         "conv_bias": _normal(g, conv, std=0.02),
         "dt_bias": dt + torch.log(-torch.expm1(-dt)),
         "A_log": torch.log(1 + 15 * uniform(heads)),
         "D": 1 + 0.1 * torch.randn(heads, generator=g, device=DEV),
         "norm.weight": (1 + 0.1 * torch.randn(inner, generator=g, device=DEV)).to(torch.bfloat16),
         "out_proj.weight": _normal(g, d, inner, std=0.02)}
    return {prefix + k: v for k, v in w.items()}


def _mamba_model_weights(case, seed):
    d, _ = MAMBA[case["size"]]
    g = _gen(seed)
    near_one = lambda: (1 + 0.1 * torch.randn(d, generator=g, device=DEV)).to(torch.bfloat16)
    w = {"embedding.weight": _normal(g, 50304, d, std=0.02)}
    for i in range(case["layers"]):
        w[f"layers.{i}.norm.weight"] = near_one()
        w.update(_mamba_weights(g, case["size"], f"layers.{i}.mixer."))
    w["norm.weight"] = near_one()
    return w


def _quantise(w, mode):
    """Packed matrix and scales as checkpoints of quantised models hold them: int4 (offset 8, low nibble first) in groups of 128 along the
    inputs, or e4m3 in blocks of 128 x 128."""
    n, k = w.shape
    w = w.float()
    if mode == "int4":
        blk = w.view(n, k // 128, 128)
        amax = blk.abs().amax(-1, keepdim=True)
        scale = torch.where(amax > 0, amax / 7.0, torch.ones_like(amax))
        q = ((blk / scale).round().clamp(-8, 7) + 8).to(torch.uint8).view(n, k)
        return q[:, ::2] | (q[:, 1::2] << 4), scale.view(n, k // 128)
    blk = F.pad(w, (0, 0, 0, (-n) % 128)).view(-1, 128, k // 128, 128)
    amax = blk.abs().amax((1, 3), keepdim=True)
    scale = torch.where(amax > 0, amax / 448.0, torch.ones_like(amax))
    q = (blk / scale).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    return q.reshape(-1, k)[:n].contiguous(), scale.view(-1, k // 128)


def _dequantised64(w, mode):
    q, scale = _quantise(w, mode)
    n, k = w.shape
    if mode == "int4":
        q = torch.stack([q & 15, q >> 4], -1).view(n, k // 128, 128).double() - 8
        return (q * scale.double()[..., None]).view(n, k)
    return q.view(torch.float8_e4m3fn).double() * scale.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)


def _load(module, weights):
    with torch.no_grad():
        own = dict(module.named_parameters())
        assert sorted(own) == sorted(weights), sorted(set(own) ^ set(weights))
        for k, p in own.items():
            p.copy_(weights[k])
    return module


def _llama(case, seed):
    from sneppx_alg_b200.models import ModelConfig, build_model
    d, h, hk, ff = WIDTHS[case["size"]]
    cfg = ModelConfig(hidden_size=d, num_hidden_layers=case["layers"], num_attention_heads=h, num_key_value_heads=hk, head_dim=128,
                      intermediate_size=ff, vocab_size=case.get("vocab", 32000), max_position_embeddings=8192, rms_norm_eps=1e-5, rope_theta=5e5)
    return _load(build_model(cfg, dtype=torch.bfloat16, device=DEV), _llama_weights(case, seed))


def _attention_inputs(case, seed):
    g = _gen(seed)
    b, n, kv, h, hk, d = (case[k] for k in ("batch", "q_len", "kv_len", "heads", "kv_heads", "dim"))
    return _normal(g, b, n, h, d), _normal(g, b, kv, hk, d), _normal(g, b, kv, hk, d), _normal(g, b, n, h, d)


def _mamba_block_inputs(case, seed):
    d, _ = MAMBA[case["size"]]
    g = _gen(seed)
    w = _mamba_weights(g, case["size"])
    return w, _normal(g, case["batch"], case["tokens"], d), _normal(g, case["batch"], case["tokens"], d)


def _contexts(case):
    """Cached tokens of every sequence, whole blocks of 16: from half of the stated context up to it."""
    c, n = case["context"] // 16, case["batch"]
    return [16 * max(1, c - (i * (c // 2)) // max(1, n)) for i in range(n)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "attention":
        q, k, v, g = _attention_inputs(case, seed)
        return dict(case=case, q=q.requires_grad_(), k=k.requires_grad_(), v=v.requires_grad_(), g=g)
    if kind == "mamba_block":
        from sneppx_alg_b200.nn.ssm import Mamba2Block
        w, u, g = _mamba_block_inputs(case, seed)
        d, groups = MAMBA[case["size"]]
        block = _load(Mamba2Block(d, ngroups=groups, dtype=torch.bfloat16, device=DEV), w)
        return dict(case=case, block=block, u=u.requires_grad_(), g=g, names=[k for k, _ in block.named_parameters()])
    if kind == "train":
        from sneppx_alg_b200.training.engine import TrainEngine
        model = _llama(case, seed)
        ids = torch.from_numpy(_tokens(seed, case["vocab"], case["batch"], case["tokens"])).to(DEV)
        return dict(case=case, engine=TrainEngine(model, lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1, max_grad_norm=1.0), ids=ids)
    if kind == "serve":
        from sneppx_alg_b200.ops.quant import quantize_model_
        from sneppx_alg_b200.serving.kv_cache import PagedKVCache
        from sneppx_alg_b200.serving.llm_engine import LlamaPagedRunner
        model = _llama(case, seed).eval()
        if case["quant"]:           # a quantised checkpoint read into a quantised model
            quantize_model_(model, case["quant"])
            own = model.state_dict()
            for k, v in _llama_weights(case, seed).items():
                if "_proj" in k:
                    for part, t in zip(("qweight", "scales"), _quantise(v, case["quant"])):
                        own[k.replace("weight", part)].copy_(t)
        b, longest = case["batch"], max(case["context"], case["prompt"]) + case["steps"]
        blocks = 2 * b * (longest // 16 + 2)
        cache = PagedKVCache(case["layers"], blocks, 16, WIDTHS[case["size"]][2], 128, device=DEV, enable_prefix_cache=False)
        runner = LlamaPagedRunner(model, cache)
        s = dict(case=case, runner=runner, ids=list(range(b)))
        if case["prompt"]:
            s["prompts"] = _tokens(seed, 32000, b, case["prompt"]).tolist()
            return s
        # conversations whose tokens are cached; a pass continues each of them and drops the continuation
        s["parents"] = list(range(1000, 1000 + b))
        for sid, n, row in zip(s["parents"], _contexts(case), _tokens(seed, 32000, b, case["context"]).tolist()):
            cache.add_sequence(sid)
            runner.prefill(sid, row[:n], 0)
        s["next"] = _tokens(seed + 1, 32000, case["steps"], b).tolist()
        runner.enable_graphs(b, longest)
        for sid, parent in zip(s["ids"], s["parents"]):       # the serving process has captured its step before it takes requests
            cache.fork(parent, sid)
        runner.decode(s["ids"], s["next"][0])
        for sid in s["ids"]:
            cache.free_sequence(sid)
        return s
    if kind == "mamba_decode":
        from sneppx_alg_b200.models import ModelConfig, build_model
        from sneppx_alg_b200.serving.llm_engine import StatefulRunner
        d, groups = MAMBA[case["size"]]
        cfg = ModelConfig(architecture="mamba2", hidden_size=d, num_hidden_layers=case["layers"], vocab_size=50280, ssm_state_size=128, ssm_expand=2,
                          ssm_head_dim=64, ssm_ngroups=groups, ssm_conv_kernel=4, ssm_chunk_size=256, max_position_embeddings=8192,
                          rms_norm_eps=1e-5, tie_word_embeddings=True)
        model = _load(build_model(cfg, dtype=torch.bfloat16, device=DEV).eval(), _mamba_model_weights(case, seed))
        runner, ids = StatefulRunner(model), list(range(case["batch"]))
        for sid, row in zip(ids, _tokens(seed, 50280, case["batch"], case["prompt"]).tolist()):
            runner.prefill(sid, row, 0)
        return dict(case=case, runner=runner, ids=ids, next=_tokens(seed + 1, 50280, case["steps"], case["batch"]).tolist())
    raise ValueError(kind)


# ----------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "attention":
        from sneppx_alg_b200 import ops
        o = ops.attention(state["q"], state["k"], state["v"], causal=case["causal"], window=case["window"])
        dq, dk, dv = torch.autograd.grad(o, (state["q"], state["k"], state["v"]), state["g"])
        return dict(o=o, dq=dq, dk=dk, dv=dv)
    if kind == "mamba_block":
        block, u = state["block"], state["u"]
        y = block(u)
        grads = torch.autograd.grad(y, [u] + list(block.parameters()), state["g"])
        return dict(y=y, grads=dict(zip(["u"] + state["names"], grads)))
    if kind == "train":
        engine, ids = state["engine"], state["ids"]
        loss = engine.step(ids, ids)
        named = list(engine.model.named_parameters())
        return dict(loss=loss, grads={k: p.main_grad for k, p in named}, weights={k: p for k, p in named})
    if kind == "serve":
        runner, ids = state["runner"], state["ids"]
        cache = runner.cache
        if case["prompt"]:
            for sid in ids:
                cache.add_sequence(sid)
            logits = runner.prefill_batch(ids, state["prompts"]) if len(ids) > 1 else runner.prefill(ids[0], state["prompts"][0], 0)
            for sid in ids:
                cache.free_sequence(sid)
            return logits
        for sid, parent in zip(ids, state["parents"]):
            cache.fork(parent, sid)
        out = []
        for tokens in state["next"]:
            logits = runner.decode(ids, tokens)
            logits.argmax(-1).tolist()          # what the scheduler reads to send it to the client; the tokens that follow are given here
            out.append(logits.clone())
        for sid in ids:
            cache.free_sequence(sid)
        return out
    out = []
    for tokens in state["next"]:
        out.append(state["runner"].decode(state["ids"], tokens))
        out[-1].argmax(-1).tolist()
    return out


# ----------------------------------------------------------------------------- what a pass cannot do without
def _pairs(n, kv, causal, window):
    """Visible (query, key) pairs of one head."""
    if not causal:
        return n * kv
    first = kv - n + 1
    if not window:
        return n * first + n * (n - 1) // 2
    return sum(min(window, first + i) for i in range(n))


def _llama_counts(case):
    d, h, hk, ff = WIDTHS[case["size"]]
    return d, h, hk, case["layers"] * (d * (h + 2 * hk) * 128 + h * 128 * d + 3 * d * ff), case.get("vocab", 32000) * d


def _mamba_counts(case):
    d, groups = MAMBA[case["size"]]
    inner = 2 * d
    heads = inner // 64
    return d, inner, heads, groups, d * (2 * inner + 2 * groups * 128 + heads) + inner * d


def work(case):
    kind = case["kind"]
    if kind == "attention":
        b, n, kv, h, hk, d = (case[k] for k in ("batch", "q_len", "kv_len", "heads", "kv_heads", "dim"))
        flops = 14 * b * h * d * _pairs(n, kv, case["causal"], case["window"])         # two products forward, five backward
        return dict(bytes=2 * b * d * (4 * n * h + 4 * kv * hk), flops=flops)          # q, k, v, dO in; o, dq, dk, dv out
    if kind == "mamba_block":
        d, inner, heads, groups, params = _mamba_counts(case)
        rows, state = case["batch"] * case["tokens"], 128
        # projections forward and twice backward; per token and head the recurrence's update and read-out (2 P N each), three times as much backward
        return dict(bytes=2 * (4 * rows * d + 2 * params), flops=6 * rows * params + 4 * rows * heads * 64 * state * 3)
    if kind == "train":
        d, h, hk, layer, head = _llama_counts(case)
        rows = case["batch"] * case["tokens"]
        attn = 14 * case["layers"] * case["batch"] * h * 128 * _pairs(case["tokens"], case["tokens"], True, 0)
        params = layer + 2 * head
        # weights read, gradients written, 32-bit weight and both moments read and written, bf16 weight written
        return dict(bytes=params * (2 + 2 + 24 + 2), flops=6 * rows * (layer + head) + attn)
    if kind == "serve":
        d, h, hk, layer, head = _llama_counts(case)
        wbytes = {"": 2.0, "fp8": 1.0, "int4": 0.5}[case["quant"]]
        if case["prompt"]:
            n, b = case["prompt"], case["batch"]
            attn = 4 * case["layers"] * b * h * 128 * _pairs(n, n, True, 0)
            return dict(bytes=layer * wbytes + 2 * head + 4 * b * 32000 + 4 * case["layers"] * b * n * hk * 128, flops=2 * b * n * layer + 2 * b * head + attn)
        cached = sum(_contexts(case)) * case["steps"] + case["batch"] * case["steps"] * (case["steps"] + 1) // 2
        return dict(bytes=case["steps"] * (layer * wbytes + 2 * head + 4 * case["batch"] * 32000) + 4 * case["layers"] * cached * hk * 128,
                    flops=2 * case["steps"] * case["batch"] * (layer + head) + 4 * case["layers"] * cached * h * 128)
    d, inner, heads, groups, params = _mamba_counts(case)
    n = case["steps"] * case["batch"]
    head = 50280 * d
    state = 2 * 4 * heads * 64 * 128 + 2 * 2 * 3 * (inner + 256 * groups)      # 32-bit state and bf16 convolution inputs, read and written
    return dict(bytes=case["steps"] * 2 * (case["layers"] * params + head) + n * (case["layers"] * state + 4 * 50280),
                flops=2 * n * (case["layers"] * params + head) + n * case["layers"] * 4 * heads * 64 * 128)


def tolerance(case):
    """About four times the distance from the 64-bit result that was measured. Operands and intermediate results are bf16 and sums are 32-bit:
    0.003 for one attention, 0.006 for a Mamba-2 block, 0.02 to 0.03 through the layers of a model; with an e4m3 model up to 256 rows of
    activations are e4m3 too, which gives 0.16."""
    kind = case["kind"]
    if kind == "attention":
        return {"rel": 0.01}
    if kind == "mamba_block":
        return {"rel": 0.025}
    if kind == "train":
        return {"rel": 0.1}
    if kind == "serve":
        return {"rel": 0.6 if case["quant"] == "fp8" else 0.09}
    return {"rel": 0.07}


# ----------------------------------------------------------------------------- the same in 64 bits
def _visible(n, kv, causal, window):
    i = torch.arange(n, device=DEV).view(-1, 1) + kv - n
    j = torch.arange(kv, device=DEV).view(1, -1)
    ok = torch.ones(n, kv, dtype=torch.bool, device=DEV)
    if causal:
        ok &= j <= i
    if window:
        ok &= j > i - window
    return ok


def _exact_attention(case, seed):
    q, k, v, g = (t.double() for t in _attention_inputs(case, seed))
    rep, scale = case["heads"] // case["kv_heads"], 1 / math.sqrt(case["dim"])
    hidden = ~_visible(case["q_len"], case["kv_len"], case["causal"], case["window"])
    o, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for b in range(case["batch"]):
        for h in range(case["heads"]):
            qh, kh, vh, gh = q[b, :, h], k[b, :, h // rep], v[b, :, h // rep], g[b, :, h]
            p = (qh @ kh.t()).mul_(scale).masked_fill_(hidden, -math.inf).softmax(-1)
            oh = p @ vh
            o[b, :, h] = oh
            dv[b, :, h // rep] += p.t() @ gh
            ds = (gh @ vh.t()).sub_((gh * oh).sum(-1, keepdim=True)).mul_(p).mul_(scale)
            dq[b, :, h] = ds @ kh
            dk[b, :, h // rep] += ds.t() @ qh
    return dict(o=o, dq=dq, dk=dk, dv=dv)


def _rms(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * w


def _ssd64(x, dt, A, B, C, D, chunk=64):
    """Chunked state-space recurrence h = exp(dt A) h + dt x B^T, y = C h + D x in 64 bits; returns y and the final state."""
    b, n, h, p = x.shape
    pad = (-n) % chunk
    xp, dtp, Bp, Cp = (F.pad(t, (0, 0) * (t.dim() - 2) + (0, pad)) for t in (x, dt, B, C))
    nc, rep = (n + pad) // chunk, h // B.shape[2]
    xc, dc = xp.view(b, nc, chunk, h, p), dtp.view(b, nc, chunk, h)
    Bc, Cc = (t.view(b, nc, chunk, -1, 128).repeat_interleave(rep, dim=3) for t in (Bp, Cp))
    cs = (dc * A).cumsum(2)
    seg = (cs[:, :, :, None] - cs[:, :, None]).permute(0, 1, 4, 2, 3)                     # [b, nc, h, l, s]
    tril = torch.ones(chunk, chunk, dtype=torch.bool, device=DEV).tril()
    M = torch.einsum("bclhn,bcshn->bchls", Cc, Bc) * seg.masked_fill(~tril, -math.inf).exp()
    xd = xc * dc[..., None]
    y = torch.einsum("bchls,bcshp->bclhp", M, xd)
    S = torch.einsum("bcshp,bcshn->bchpn", xd * (cs[:, :, -1:] - cs).exp()[..., None], Bc)
    tot = cs[:, :, -1].exp()
    state, before = torch.zeros_like(S[:, 0]), []
    for c in range(nc):
        before.append(state)
        state = state * tot[:, c, :, None, None] + S[:, c]
    y = y + torch.einsum("bclhn,bchpn->bclhp", Cc, torch.stack(before, 1)) * cs.exp()[..., None]
    return y.reshape(b, n + pad, h, p)[:, :n] + x * D[:, None], state


def _mamba64(w, u, size):
    d, groups = MAMBA[size]
    inner, heads = 2 * d, 2 * d // 64
    b, n, _ = u.shape
    z, xbc, dt = (u @ w["in_proj.weight"].t()).split([inner, inner + 256 * groups, heads], -1)
    xbc = F.pad(xbc, (0, 0, 3, 0))
    xbc = F.silu(sum(xbc[:, t:t + n] * w["conv_weight"][:, t] for t in range(4)) + w["conv_bias"])
    x, B, C = xbc.split([inner, 128 * groups, 128 * groups], -1)
    y, _ = _ssd64(x.reshape(b, n, heads, 64), F.softplus(dt + w["dt_bias"]), -w["A_log"].exp(), B.reshape(b, n, groups, 128),
                  C.reshape(b, n, groups, 128), w["D"])
    return _rms(y.reshape(b, n, inner) * F.silu(z), w["norm.weight"]) @ w["out_proj.weight"].t()


def _rope64(x):
    """x [b, n, heads, 128], rotate-half, base 5e5."""
    n = x.shape[1]
    inv = 5e5 ** (-torch.arange(0, 128, 2, device=DEV, dtype=torch.float64) / 128)
    a = torch.arange(n, device=DEV, dtype=torch.float64)[:, None] * inv
    c, s = a.cos()[:, None], a.sin()[:, None]
    x1, x2 = x[..., :64], x[..., 64:]
    return torch.cat((x1 * c - x2 * s, x2 * c + x1 * s), -1)


def _llama64(w, case, ids):
    """Hidden states after the last norm, [b, n, d]."""
    d, h, hk, ff = WIDTHS[case["size"]]
    b, n = ids.shape
    x = w["embedding.weight"][ids]
    hidden = ~_visible(n, n, True, 0)
    for i in range(case["layers"]):
        p = f"layers.{i}."
        q, k, v = (_rms(x, w[p + "attn_norm.weight"]) @ w[p + "attn.qkv_proj.weight"].t()).view(b, n, -1, 128).split([h, hk, hk], 2)
        q, k = _rope64(q), _rope64(k).repeat_interleave(h // hk, dim=2)
        s = torch.einsum("bqhd,bkhd->bhqk", q, k) / math.sqrt(128)
        o = torch.einsum("bhqk,bkhd->bqhd", s.masked_fill(hidden, -math.inf).softmax(-1), v.repeat_interleave(h // hk, dim=2))
        x = x + o.reshape(b, n, h * 128) @ w[p + "attn.o_proj.weight"].t()
        gate, up = (_rms(x, w[p + "mlp_norm.weight"]) @ w[p + "mlp.gate_up_proj.weight"].t()).chunk(2, -1)
        x = x + (F.silu(gate) * up) @ w[p + "mlp.down_proj.weight"].t()
    return _rms(x, w["norm.weight"])


def _exact_train(case, seed):
    w = {k: v.double().requires_grad_() for k, v in _llama_weights(case, seed).items()}
    ids = torch.from_numpy(_tokens(seed, case["vocab"], case["batch"], case["tokens"])).to(DEV)
    logits = _llama64(w, case, ids)[:, :-1] @ w["lm_head.weight"].t()
    loss = F.cross_entropy(logits.reshape(-1, case["vocab"]), ids[:, 1:].reshape(-1))
    del logits
    grads = dict(zip(w, torch.autograd.grad(loss, list(w.values()))))
    clip = min(1.0, 1.0 / float(sum(g.square().sum() for g in grads.values()).sqrt() + 1e-6))
    new = {}
    with torch.no_grad():       # the first AdamW step: both bias-corrected moments are those of this gradient alone
        for k in w:
            g = grads[k] * clip
            new[k] = w[k] * (1 - 3e-4 * 0.1) - 3e-4 * g / (g.abs() + 1e-8)
    return dict(loss=loss.detach(), grads=grads, weights=new)


@torch.no_grad()
def _exact_serve(case, seed):
    w = {}
    for k, v in _llama_weights(case, seed).items():
        w[k] = _dequantised64(v, case["quant"]) if case["quant"] and "_proj" in k else v.double()
    head = w["lm_head.weight"].t()
    b = case["batch"]
    if case["prompt"]:
        rows = torch.from_numpy(_tokens(seed, 32000, b, case["prompt"])).to(DEV)
        return torch.cat([_llama64(w, case, rows[i:i + 1])[:, -1] @ head for i in range(b)])
    rows, nxt = _tokens(seed, 32000, b, case["context"]), _tokens(seed + 1, 32000, case["steps"], b)
    out = []
    for i, n in enumerate(_contexts(case)):
        ids = torch.from_numpy(np.concatenate([rows[i, :n], nxt[:, i]])).to(DEV)[None]
        out.append(_llama64(w, case, ids)[0, n:] @ head)
    return list(torch.stack(out, 1))


@torch.no_grad()
def _exact_mamba_decode(case, seed):
    w = {k: v.double() for k, v in _mamba_model_weights(case, seed).items()}
    prompt, nxt = _tokens(seed, 50280, case["batch"], case["prompt"]), _tokens(seed + 1, 50280, case["steps"], case["batch"])
    x = w["embedding.weight"][torch.from_numpy(np.concatenate([prompt, nxt.T], 1)).to(DEV)]
    for i in range(case["layers"]):
        mixer = {k.split("mixer.")[1]: v for k, v in w.items() if k.startswith(f"layers.{i}.mixer.")}
        x = x + _mamba64(mixer, _rms(x, w[f"layers.{i}.norm.weight"]), case["size"])
    logits = _rms(x, w["norm.weight"])[:, case["prompt"]:] @ w["embedding.weight"][:50280].t()
    return list(logits.transpose(0, 1))


def exact(case, seed):
    """What ``run`` returns, in 64 bits."""
    kind = case["kind"]
    if kind == "attention":
        return _exact_attention(case, seed)
    if kind == "mamba_block":
        w, u, g = _mamba_block_inputs(case, seed)
        w, u = {k: v.double().requires_grad_() for k, v in w.items()}, u.double().requires_grad_()
        y = _mamba64(w, u, case["size"])
        grads = torch.autograd.grad(y, [u] + list(w.values()), g.double())
        return dict(y=y.detach(), grads=dict(zip(["u"] + list(w), grads)))
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "serve":
        return _exact_serve(case, seed)
    return _exact_mamba_decode(case, seed)
