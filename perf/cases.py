"""Performance cases: the work this framework does for its users, through its public entry points.

A case names a path (``kind``) and its sizes.  Serving: one decode step and one prompt pass of the engine.  Training: forward and
backward of an attention layer, an attention layer with relative positions, a gated MLP, a biased linear layer, the norms, the
language-model head with its loss, and the optimizer step.  Widths are those of the model configurations in
``tensor_parallel_b200/models`` (and of the smoke test for the smallest); ``draw`` spreads over the same ranges.

``exact`` restates every path in 64-bit PyTorch, with none of this package's code.
"""
import math

import torch
import torch.nn.functional as F

BF16 = torch.bfloat16


def listed():
    return [
        # smallest call: one sequence on the smoke-test model; a step is all launches and latency
        dict(name="decode_tiny", kind="decode", hidden=256, heads=4, kv_heads=4, ffn=688, layers=2, vocab=512, batch=1, context=24),
        # the benchmark's decode step (batch 8 at a 2048-token context), four of the 32 layers
        dict(name="decode_llama", kind="decode", hidden=4096, heads=32, kv_heads=32, ffn=11008, layers=4, vocab=32000, batch=8, context=2048),
        # decode with grouped key / value heads and the parallel attention + MLP block (Falcon-40B widths)
        dict(name="decode_falcon", kind="falcon_decode", hidden=8192, heads=128, kv_heads=8, layers=1, vocab=65024, batch=16, context=1024),
        # prompts of an ordinary, ragged length
        dict(name="prefill_llama", kind="prefill", hidden=4096, heads=32, kv_heads=32, ffn=11008, layers=2, vocab=32000, batch=4, seq=1000),
        # training, micro-batch 4 x 2048: causal attention layer
        dict(name="attention_train", kind="attention", hidden=4096, heads=32, kv_heads=32, batch=4, seq=2048),
        # encoder self-attention with learned relative positions (FLAN-T5-XL widths, 16 x 512)
        dict(name="attention_relative_train", kind="relative_attention", hidden=2048, heads=32, batch=16, seq=512),
        # training, micro-batch 4 x 2048: gated MLP
        dict(name="mlp_train", kind="mlp", hidden=4096, ffn=11008, tokens=8192),
        # a small training call: the first MLP projection of the smallest OPT, 100 tokens, with bias
        dict(name="linear_small_train", kind="linear", inputs=768, outputs=3072, tokens=100),
        # RMSNorm of a training step
        dict(name="rms_norm_train", kind="norm", norm="rms", hidden=4096, rows=8192, dtype="bf16"),
        # LayerNorm in 32 bits (OPT-13B width), an odd number of rows
        dict(name="layer_norm_train", kind="norm", norm="layer", hidden=5120, rows=1999, dtype="fp32"),
        # language-model head fused with the cross-entropy, 4 x 2048 tokens, some of them without a label
        dict(name="head_loss_train", kind="head", hidden=4096, vocab=32000, tokens=8192),
        # optimizer step over the parameters of one 7B decoder layer, with 32-bit master weights
        dict(name="adamw_step", kind="adamw", hidden=4096, ffn=11008),
    ]


def _spread(rng, low, high, step=1):
    """A whole number in [low, high], even over the logarithm, a multiple of ``step``."""
    value = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(low, min(high, int(round(value / step)) * step))


def draw(rng):
    kind = rng.choice(["decode", "decode", "falcon_decode", "prefill", "prefill", "attention", "attention", "relative_attention", "mlp",
                       "linear", "norm", "norm", "head", "adamw"])
    if kind in ("decode", "prefill"):
        heads, head_dim = rng.choice([(4, 64), (12, 64), (16, 128), (32, 128), (40, 128)])
        case = dict(kind=kind, hidden=heads * head_dim, heads=heads, kv_heads=rng.choice([heads, heads // 4]),
                    ffn=_spread(rng, 2 * heads * head_dim, 3 * heads * head_dim, 8), layers=rng.randint(1, 2), vocab=_spread(rng, 512, 50272, 8))
        if kind == "decode":
            return dict(case, batch=_spread(rng, 1, 32), context=_spread(rng, 20, 2500))
        batch = _spread(rng, 1, 8)
        return dict(case, layers=1, batch=batch, seq=_spread(rng, 17, 2048 if batch <= 4 else 1024))
    if kind == "falcon_decode":
        return dict(kind=kind, hidden=8192, heads=128, kv_heads=8, layers=1, vocab=_spread(rng, 4000, 65024, 8), batch=_spread(rng, 1, 16), context=_spread(rng, 20, 1500))
    if kind == "attention":
        heads, head_dim = rng.choice([(12, 64), (16, 128), (32, 128)])
        return dict(kind=kind, hidden=heads * head_dim, heads=heads, kv_heads=rng.choice([heads, heads // 4]), batch=_spread(rng, 1, 4), seq=_spread(rng, 65, 2048))
    if kind == "relative_attention":
        heads = rng.choice([8, 16, 32])
        return dict(kind=kind, hidden=heads * 64, heads=heads, batch=_spread(rng, 1, 16), seq=_spread(rng, 33, 512))
    if kind == "mlp":
        hidden = rng.choice([768, 2048, 4096])
        return dict(kind=kind, hidden=hidden, ffn=_spread(rng, 2 * hidden, 11008, 8), tokens=_spread(rng, 65, 8192))
    if kind == "linear":
        inputs = rng.choice([768, 2048, 4096, 5120])
        return dict(kind=kind, inputs=inputs, outputs=_spread(rng, inputs // 2, 4 * inputs, 8), tokens=_spread(rng, 20, 4096))
    if kind == "norm":
        return dict(kind=kind, norm=rng.choice(["rms", "layer"]), hidden=rng.choice([256, 768, 2048, 4096, 5120, 8192]), rows=_spread(rng, 20, 8192),
                    dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "head":
        return dict(kind=kind, hidden=rng.choice([768, 2048, 4096]), vocab=_spread(rng, 1000, 32000), tokens=_spread(rng, 65, 8192))
    hidden = rng.choice([768, 2048, 4096])
    return dict(kind=kind, hidden=hidden, ffn=_spread(rng, 2 * hidden, 11008, 8))


# -- inputs: every tensor of a case from its seed alone --------------------------------------------------------------


class _Source:
    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=self.gen)

    def ids(self, high, *shape):
        return torch.randint(0, high, shape, generator=self.gen, device="cuda")


def _llama_weights(c, src):
    d, f = c["hidden"], c["ffn"]
    kv = d // c["heads"] * c["kv_heads"]
    w = {"model.embed_tokens.weight": src.normal(c["vocab"], d)}
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (d, d)), ("self_attn.k_proj", (kv, d)), ("self_attn.v_proj", (kv, d)), ("self_attn.o_proj", (d, d)),
                            ("mlp.gate_proj", (f, d)), ("mlp.up_proj", (f, d)), ("mlp.down_proj", (d, f))):
            w[p + name + ".weight"] = src.normal(*shape, std=0.02)
        w[p + "input_layernorm.weight"] = src.normal(d, std=0.1, mean=1.0)
        w[p + "post_attention_layernorm.weight"] = src.normal(d, std=0.1, mean=1.0)
    w["model.norm.weight"] = src.normal(d, std=0.1, mean=1.0)
    w["lm_head.weight"] = src.normal(c["vocab"], d, std=0.02)
    return w


def _falcon_weights(c, src):
    d, hd = c["hidden"], c["hidden"] // c["heads"]
    w = {"transformer.word_embeddings.weight": src.normal(c["vocab"], d, std=0.02)}
    for i in range(c["layers"]):
        p = f"transformer.h.{i}."
        for ln in ("ln_attn", "ln_mlp"):
            w[p + ln + ".weight"] = src.normal(d, std=0.1, mean=1.0)
            w[p + ln + ".bias"] = src.normal(d, std=0.1)
        w[p + "self_attention.query_key_value.weight"] = src.normal((c["heads"] + 2 * c["kv_heads"]) * hd, d, std=0.02)
        w[p + "self_attention.dense.weight"] = src.normal(d, d, std=0.02)
        w[p + "mlp.dense_h_to_4h.weight"] = src.normal(4 * d, d, std=0.02)
        w[p + "mlp.dense_4h_to_h.weight"] = src.normal(d, 4 * d, std=0.02)
    w["transformer.ln_f.weight"] = src.normal(d, std=0.1, mean=1.0)
    w["transformer.ln_f.bias"] = src.normal(d, std=0.1)
    w["lm_head.weight"] = w["transformer.word_embeddings.weight"]
    return w


def _inputs(c, seed):
    src, kind = _Source(seed), c["kind"]
    if kind in ("decode", "falcon_decode", "prefill"):
        w = _falcon_weights(c, src) if kind == "falcon_decode" else _llama_weights(c, src)
        if kind == "prefill":
            return dict(weights=w, ids=src.ids(c["vocab"], c["batch"], c["seq"]))
        shape = (c["batch"], c["kv_heads"], c["context"], c["hidden"] // c["heads"])
        return dict(weights=w, ids=src.ids(c["vocab"], c["batch"]), k=[src.normal(*shape) for _ in range(c["layers"])],
                    v=[src.normal(*shape) for _ in range(c["layers"])])
    if kind == "attention":
        d = c["hidden"]
        kv = d // c["heads"] * c["kv_heads"]
        x, g = (src.normal(c["batch"], c["seq"], d) for _ in range(2))
        return dict(x=x, grad=g, weights=[src.normal(n, d, std=0.02) for n in (d, kv, kv, d)])
    if kind == "relative_attention":
        d = c["hidden"]
        x, g = (src.normal(c["batch"], c["seq"], d) for _ in range(2))
        # un-scaled scores: the query projection is small, as in a trained encoder
        return dict(x=x, grad=g, weights=[src.normal(d, d, std=s) for s in (0.125 / math.sqrt(d), 1 / math.sqrt(d), 0.02, 0.02)], table=src.normal(32, c["heads"]))
    if kind == "mlp":
        d, f = c["hidden"], c["ffn"]
        x, g = (src.normal(c["tokens"], d) for _ in range(2))
        return dict(x=x, grad=g, weights=[src.normal(*s, std=0.02) for s in ((f, d), (f, d), (d, f))])
    if kind == "linear":
        return dict(x=src.normal(c["tokens"], c["inputs"]), grad=src.normal(c["tokens"], c["outputs"]),
                    weight=src.normal(c["outputs"], c["inputs"], std=0.02), bias=src.normal(c["outputs"], std=0.1))
    if kind == "norm":
        dt = torch.float32 if c["dtype"] == "fp32" else BF16
        return dict(x=src.normal(c["rows"], c["hidden"], std=2.0, mean=0.1, dtype=dt), grad=src.normal(c["rows"], c["hidden"], dtype=dt),
                    weight=src.normal(c["hidden"], std=0.1, mean=1.0, dtype=dt), bias=src.normal(c["hidden"], std=0.1, dtype=dt))
    if kind == "head":
        labels = src.ids(c["vocab"], c["tokens"])
        labels[src.ids(10, c["tokens"]) == 0] = -100
        return dict(x=src.normal(c["tokens"], c["hidden"]), weight=src.normal(c["vocab"], c["hidden"], std=0.02), labels=labels)
    if kind == "adamw":
        d, f = c["hidden"], c["ffn"]
        shapes = [(d, d)] * 4 + [(f, d), (f, d), (d, f), (d,), (d,)]
        return dict(params=[src.normal(*s, std=0.02) for s in shapes], grads=[src.normal(*s, std=1e-3) for s in shapes])
    raise ValueError(kind)


# -- what a user's program holds before the call, and the call -------------------------------------------------------


def _engine(c, weights, max_batch, max_seq):
    from tensor_parallel_b200.engine import DecoderEngine
    from tensor_parallel_b200.models.falcon import FalconConfig, FalconForCausalLM
    from tensor_parallel_b200.models.llama import LlamaConfig, LlamaForCausalLM

    with torch.device("meta"):
        if c["kind"] == "falcon_decode":
            model = FalconForCausalLM(FalconConfig(vocab_size=c["vocab"], hidden_size=c["hidden"], n_layer=c["layers"], n_head=c["heads"], n_head_kv=c["kv_heads"]))
        else:
            model = LlamaForCausalLM(LlamaConfig(vocab_size=c["vocab"], hidden_size=c["hidden"], intermediate_size=c["ffn"], num_hidden_layers=c["layers"],
                                                 num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"]))
    model.load_state_dict(weights, assign=True)
    return DecoderEngine(model.eval(), None, max_batch=max_batch, max_seq=max_seq)


def _parameter(module, **tensors):
    for name, t in tensors.items():
        setattr(module, name, torch.nn.Parameter(t))


def prepare(case, seed):
    c, t = case, _inputs(case, seed)
    kind = c["kind"]
    if kind in ("decode", "falcon_decode"):
        b, n = c["batch"], c["context"]
        engine = _engine(c, t["weights"], b, n + 64)
        for i in range(c["layers"]):
            engine.kcache[i][:, :, :n] = t["k"][i]
            engine.vcache[i][:, :, :n] = t["v"][i]
        engine.pos.fill_(n)
        engine.ids.copy_(t["ids"])
        engine.decode_step(b)  # a server captures its step once, before the first request
        return dict(case=c, engine=engine, ids=t["ids"])
    if kind == "prefill":
        return dict(case=c, engine=_engine(c, t["weights"], c["batch"], c["seq"] + 64), ids=t["ids"])
    from tensor_parallel_b200.models import common

    if kind == "attention":
        from tensor_parallel_b200.models.llama import LlamaAttention, LlamaConfig

        with torch.device("meta"):
            module = LlamaAttention(LlamaConfig(hidden_size=c["hidden"], num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"]))
        for name, w in zip(("q_proj", "k_proj", "v_proj", "o_proj"), t["weights"]):
            _parameter(getattr(module, name), weight=w)
        positions = torch.arange(c["seq"], device="cuda")[None].expand(c["batch"], c["seq"])
        return dict(case=c, module=module, x=t["x"].requires_grad_(), grad=t["grad"], positions=positions)
    if kind == "relative_attention":
        from tensor_parallel_b200.models.t5 import T5Attention, T5Config

        with torch.device("meta"):
            module = T5Attention(T5Config(d_model=c["hidden"], d_kv=64, num_heads=c["heads"]), True, False)
        for name, w in zip("qkvo", t["weights"]):
            _parameter(getattr(module, name), weight=w)
        _parameter(module.relative_attention_bias, weight=t["table"])
        return dict(case=c, module=module, x=t["x"].requires_grad_(), grad=t["grad"])
    if kind == "mlp":
        from tensor_parallel_b200.models.llama import LlamaConfig, LlamaMLP

        with torch.device("meta"):
            module = LlamaMLP(LlamaConfig(hidden_size=c["hidden"], intermediate_size=c["ffn"]))
        for name, w in zip(("gate_proj", "up_proj", "down_proj"), t["weights"]):
            _parameter(getattr(module, name), weight=w)
    elif kind == "linear":
        with torch.device("meta"):
            module = common.Linear(c["inputs"], c["outputs"])
        _parameter(module, weight=t["weight"], bias=t["bias"])
    elif kind == "norm":
        with torch.device("meta"):
            module = common.RMSNorm(c["hidden"], 1e-6) if c["norm"] == "rms" else common.LayerNorm(c["hidden"])
        _parameter(module, weight=t["weight"], **({} if c["norm"] == "rms" else {"bias": t["bias"]}))
    elif kind == "head":
        return dict(case=c, x=t["x"].requires_grad_(), weight=t["weight"].requires_grad_(), labels=t["labels"])
    else:
        from tensor_parallel_b200 import optim

        params = [p.requires_grad_() for p in t["params"]]
        for p, g in zip(params, t["grads"]):
            p.grad = g
        return dict(case=c, params=params, optimizer=optim.AdamW(params, lr=1e-5, weight_decay=0.1))
    return dict(case=c, module=module, x=t["x"].requires_grad_(), grad=t["grad"])


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("decode", "falcon_decode"):
        engine, b, n = state["engine"], c["batch"], c["context"]
        engine.pos.fill_(n)  # the next token of this context (a decode step advances position and ids itself)
        engine.ids.copy_(state["ids"])
        engine.decode_step(b)
        return dict(logits=engine.logits_local, k=[k[:, :, n] for k in engine.kcache], v=[v[:, :, n] for v in engine.vcache])
    if kind == "prefill":
        engine, n = state["engine"], c["seq"]
        logits = engine.prefill(state["ids"])
        return dict(logits=logits, k=[k[:, :, :n] for k in engine.kcache], v=[v[:, :, :n] for v in engine.vcache])
    if kind == "adamw":
        state["optimizer"].step()
        moments = [state["optimizer"].state[p] for p in state["params"]]
        return dict(params=state["params"], master=[m["master"] for m in moments], first=[m["exp_avg"] for m in moments], second=[m["exp_avg_sq"] for m in moments])
    x = state["x"]
    x.grad = None
    if kind == "head":
        from tensor_parallel_b200.ops.loss import lm_head_cross_entropy

        state["weight"].grad = None
        loss = lm_head_cross_entropy(x, state["weight"], state["labels"])
        loss.backward()
        return dict(loss=loss.detach(), dx=x.grad, grads=[state["weight"].grad])
    module = state["module"]
    module.zero_grad(set_to_none=True)
    if kind == "attention":
        out = module(x, position_ids=state["positions"])[0]
    elif kind == "relative_attention":
        out = module(x)[0]
    else:
        out = module(x)
    out.backward(state["grad"])
    return dict(out=out.detach(), dx=x.grad, grads=[p.grad for p in module.parameters()])


# -- what a pass cannot do without -----------------------------------------------------------------------------------


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("decode", "prefill", "falcon_decode"):
        d, hd = c["hidden"], c["hidden"] // c["heads"]
        kv = hd * c["kv_heads"]
        layer = d * d * 2 + 2 * kv * d + (8 * d * d if kind == "falcon_decode" else 3 * d * c["ffn"])
        b, s, past = c["batch"], c.get("seq", 1), c.get("context", 0)
        pairs = b * (s * past + s * (s + 1) // 2)
        cache = 2 * b * kv * 2 * (past + s)  # read (the past) and written (the new tokens)
        return dict(bytes=2 * (c["layers"] * layer + c["vocab"] * d) + c["layers"] * cache + 2 * b * s * d + 2 * b * c["vocab"],
                    flops=2 * b * s * c["layers"] * layer + 4 * pairs * d * c["layers"] + 2 * b * c["vocab"] * d)
    if kind in ("attention", "relative_attention"):
        d, b, s = c["hidden"], c["batch"], c["seq"]
        kv = d // c["heads"] * c.get("kv_heads", c["heads"])
        weights, tokens = 2 * d * d + 2 * d * kv, b * s
        pairs = b * s * (s + 1) // 2 if kind == "attention" else b * s * s
        return dict(bytes=2 * (2 * weights + 4 * tokens * d), flops=6 * tokens * weights + 14 * pairs * d)
    if kind == "mlp":
        return dict(bytes=2 * (6 * c["hidden"] * c["ffn"] + 4 * c["tokens"] * c["hidden"]), flops=18 * c["tokens"] * c["hidden"] * c["ffn"])
    if kind == "linear":
        return dict(bytes=2 * (2 * c["inputs"] * c["outputs"] + 2 * c["tokens"] * (c["inputs"] + c["outputs"])), flops=6 * c["tokens"] * c["inputs"] * c["outputs"])
    if kind == "norm":
        return dict(bytes=(4 if c["dtype"] == "fp32" else 2) * 4 * c["rows"] * c["hidden"], flops=20 * c["rows"] * c["hidden"])
    if kind == "head":
        return dict(bytes=2 * (2 * c["vocab"] * c["hidden"] + 2 * c["tokens"] * c["hidden"]), flops=6 * c["tokens"] * c["vocab"] * c["hidden"])
    n = 4 * c["hidden"] ** 2 + 3 * c["hidden"] * c["ffn"] + 2 * c["hidden"]
    return dict(bytes=30 * n, flops=15 * n)  # gradient read; parameter, master copy and both moments read and written


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "falcon_decode", "prefill"):
        return {"rel": 0.02}  # bf16 activations through whole layers, weights rounded once more with the norm folded in
    if kind in ("attention", "relative_attention"):
        return {"rel": 0.02}
    if kind == "adamw":
        return {"rel": 1e-4}  # 32-bit state; a bf16 parameter in a hundred thousand may round the other way
    if kind == "norm" and case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 0.01}


# -- 64-bit restatement ----------------------------------------------------------------------------------------------


def _rope(x, positions):
    half = x.shape[-1] // 2
    freq = 10000.0 ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    angle = positions.double()[:, None] * freq
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)


def _attend(q, k, v, causal, bias=None, scale=None):
    """q [b, s, heads, d], k / v [b, n, kv heads, d]; query i sees the keys up to i + n - s."""
    s, n, rep = q.shape[1], k.shape[1], q.shape[2] // k.shape[2]
    q, k, v = q.transpose(1, 2), k.transpose(1, 2).repeat_interleave(rep, 1), v.transpose(1, 2).repeat_interleave(rep, 1)
    scores = q @ k.transpose(-1, -2) * (1 / math.sqrt(q.shape[-1]) if scale is None else scale)
    if bias is not None:
        scores = scores + bias
    if causal and s > 1:
        scores = scores.masked_fill(torch.ones(s, n, dtype=torch.bool, device=q.device).triu(n - s + 1), -math.inf)
    return (scores.softmax(-1) @ v).transpose(1, 2)


def _exact_serving(c, t):
    d, h, g = c["hidden"], c["heads"], c["kv_heads"]
    hd, b, s, past = d // h, c["batch"], c.get("seq", 1), c.get("context", 0)
    falcon = c["kind"] == "falcon_decode"
    positions = torch.arange(past, past + s, device="cuda")
    w = t["weights"]
    x = w["transformer.word_embeddings.weight" if falcon else "model.embed_tokens.weight"][t["ids"].reshape(b, s)].double()

    def norm(x, name):
        if falcon:
            return F.layer_norm(x, (d,), w[name + ".weight"].double(), w[name + ".bias"].double(), 1e-5)
        return x * (x.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * w[name + ".weight"].double()

    def mul(x, name):
        return x @ w[name + ".weight"].double().t()

    new_k, new_v = [], []
    for i in range(c["layers"]):
        p = f"transformer.h.{i}." if falcon else f"model.layers.{i}."
        if falcon:
            fused = mul(norm(x, p + "ln_attn"), p + "self_attention.query_key_value").view(b, s, g, h // g + 2, hd)
            q, k, v = fused[:, :, :, :-2].reshape(b, s, h, hd), fused[:, :, :, -2], fused[:, :, :, -1]
        else:
            n = norm(x, p + "input_layernorm")
            q, k, v = (mul(n, p + f"self_attn.{j}_proj").view(b, s, -1, hd) for j in "qkv")
        q, k = _rope(q, positions), _rope(k, positions)
        new_k.append(k.transpose(1, 2) if s > 1 else k[:, 0])
        new_v.append(v.transpose(1, 2) if s > 1 else v[:, 0])
        if past:
            k, v = (torch.cat((old[i].double().transpose(1, 2), new), 1) for old, new in ((t["k"], k), (t["v"], v)))
        a = _attend(q, k, v, True).reshape(b, s, d)
        if falcon:
            x = x + mul(a, p + "self_attention.dense") + mul(F.gelu(mul(norm(x, p + "ln_mlp"), p + "mlp.dense_h_to_4h")), p + "mlp.dense_4h_to_h")
        else:
            x = x + mul(a, p + "self_attn.o_proj")
            n = norm(x, p + "post_attention_layernorm")
            x = x + mul(F.silu(mul(n, p + "mlp.gate_proj")) * mul(n, p + "mlp.up_proj"), p + "mlp.down_proj")
    return dict(logits=mul(norm(x[:, -1], "transformer.ln_f" if falcon else "model.norm"), "lm_head"), k=new_k, v=new_v)


def _relative_bias(table, n):
    """Bidirectional buckets of T5: 16 per direction, exact below 8, logarithmic up to a distance of 128."""
    at = torch.arange(n, device=table.device)
    distance = at[None] - at[:, None]
    far = distance.abs()
    large = (8 + (torch.log(far.float().clamp(min=1) / 8) / math.log(16.0) * 8).long()).clamp(max=15)
    bucket = torch.where(far < 8, far, large) + 16 * (distance > 0)
    return table[bucket].permute(2, 0, 1)[None]


def exact(case, seed):
    c, t = case, _inputs(case, seed)
    kind = c["kind"]
    with torch.no_grad() if kind in ("decode", "prefill", "falcon_decode", "adamw") else torch.enable_grad():
        if kind in ("decode", "prefill", "falcon_decode"):
            return _exact_serving(c, t)
        if kind == "adamw":
            out = dict(params=[], master=[], first=[], second=[])
            for p, g in zip(t["params"], t["grads"]):
                p, g = p.double(), g.double()
                new = p * (1 - 1e-5 * 0.1) - 1e-5 * g / (g.abs() + 1e-8)
                for name, v in (("params", new), ("master", new), ("first", 0.1 * g), ("second", 0.001 * g * g)):
                    out[name].append(v)
            return out

        def leaf(v):
            return v.double().requires_grad_()

        x = leaf(t["x"])
        if kind == "attention":
            b, s, d = x.shape
            hd, positions = d // c["heads"], torch.arange(s, device="cuda")
            params = [leaf(w) for w in t["weights"]]
            q, k, v = ((x @ w.t()).view(b, s, -1, hd) for w in params[:3])
            out = _attend(_rope(q, positions), _rope(k, positions), v, True).reshape(b, s, d) @ params[3].t()
        elif kind == "relative_attention":
            b, s, d = x.shape
            params = [leaf(w) for w in t["weights"]] + [leaf(t["table"])]
            q, k, v = ((x @ w.t()).view(b, s, -1, 64) for w in params[:3])
            out = _attend(q, k, v, False, _relative_bias(params[4], s), 1.0).reshape(b, s, d) @ params[3].t()
        elif kind == "mlp":
            params = [leaf(w) for w in t["weights"]]
            out = (F.silu(x @ params[0].t()) * (x @ params[1].t())) @ params[2].t()
        elif kind == "linear":
            params = [leaf(t["weight"]), leaf(t["bias"])]
            out = x @ params[0].t() + params[1]
        elif kind == "norm":
            params = [leaf(t["weight"])]
            if c["norm"] == "rms":
                out = x * (x.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * params[0]
            else:
                params.append(leaf(t["bias"]))
                out = F.layer_norm(x, (c["hidden"],), params[0], params[1], 1e-5)
        else:
            params = [leaf(t["weight"])]
            loss = F.cross_entropy(x @ params[0].t(), t["labels"], ignore_index=-100)
            loss.backward()
            return dict(loss=loss.detach(), dx=x.grad, grads=[params[0].grad])
        out.backward(t["grad"].double())
        return dict(out=out.detach(), dx=x.grad, grads=[p.grad for p in params])
