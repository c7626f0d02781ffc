"""Performance cases: the calls a user of this package makes, over the sizes it is used at.

`listed()` names twelve cases, `draw(rng)` makes another one of the same ranges; `prepare` builds what a program has
in hand before the call, `run` makes one pass through the public entry points and returns what they produce, `work`
is the traffic and arithmetic no implementation can avoid, `tolerance` the rounding difference between two correct
implementations at the same precision.

Sizes are those of the benchmark configurations (hidden 896, 14 query and 2 key/value heads of 64, MLP 4864,
vocabulary 151936, ranks 8 to 64, 4k to 1M rows) and of the tests, with odd token counts between them.
"""
import math

import torch

from metal_candle_b200 import backend
from metal_candle_b200.engine import QwenEngine
from metal_candle_b200.qwen import ModelConfig, Qwen
from metal_candle_b200.training import (AdamW, AdamWConfig, IGNORE_INDEX, LoRAAdapter, LoRAAdapterConfig, LoRAConfig, LoRALayer,
                                        TargetModule, TrainingStep, cross_entropy_loss)

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
TARGETS = {"qv": (TargetModule.QProj, TargetModule.VProj),
           "qkvo": (TargetModule.QProj, TargetModule.KProj, TargetModule.VProj, TargetModule.OProj)}
LR = 1e-4


def listed():
    return [
        # one token through one adapter layer (what a generating program calls per projection): latency and launches
        dict(name="layer_one_token", kind="layer", batch=1, seq=1, inp=512, out=512, rank=8, dtype="f32"),
        # one LoRA linear of a float32 training run, forward and backward (benchmark configuration 1)
        dict(name="linear_f32_512", kind="linear", tokens=512, inp=768, out=768, rank=8, dtype="f32", bias=False),
        # an attention projection of the 0.5B-shaped model on an ordinary batch, forward and backward
        dict(name="linear_896_4096", kind="linear", tokens=4096, inp=896, out=896, rank=16, dtype="bf16", bias=True),
        # the largest LoRA linear of the sweep that fills the GPU for milliseconds
        dict(name="linear_4096_32768", kind="linear", tokens=32768, inp=4096, out=4096, rank=16, dtype="bf16", bias=False),
        # a block's norm over 16 sequences of 2048, forward and backward with the weight's gradient
        dict(name="rmsnorm_32768", kind="rmsnorm", rows=32768, width=896, dtype="bf16"),
        # masked attention scores of a batch whose length no kernel likes, forward and backward
        dict(name="softmax_ragged", kind="softmax", batch=8, heads=14, seq=777, dtype="bf16"),
        # the loss and its gradient over a full vocabulary, some targets ignored
        dict(name="loss_1000", kind="loss", batch=2, seq=500, vocab=151936, dtype="bf16"),
        # grouped-query attention of 8 sequences of 1024 (benchmark configuration 4), forward and backward
        dict(name="attention_1024", kind="attention", batch=8, kv_heads=2, groups=7, seq=1024),
        # the optimizer over the adapters of 24 layers (q, k, v, o; configuration 5): 192 small tensors
        dict(name="adamw_192", kind="adamw", layers=24, hidden=896, kv=128, rank=16, targets="qkvo"),
        # scoring a short prompt batch of odd length with an adapted model: logits of every position
        dict(name="forward_ragged", kind="forward", layers=24, batch=3, seq=111, rank=8, targets="qv"),
        # the trainer's step (forward, loss, backward, optimizer, loss read back) on a small fine-tuning batch
        dict(name="trainer_small", kind="trainer", layers=6, batch=2, seq=256, rank=8, targets="qv"),
        # the whole training step at the headline size (configuration 5), through the engine
        dict(name="step_16x2048", kind="step", layers=24, batch=16, seq=2048, rank=16, targets="qkvo"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "linear", "linear", "rmsnorm", "softmax", "loss", "attention", "adamw", "forward", "trainer", "step"])
    if kind == "layer":
        dtype = rng.choice(["f32", "bf16"])
        step = 8 if dtype == "bf16" else 1
        width = lambda: max(64, _log(rng, 512, 4096) // step * step)  # noqa: E731
        return dict(kind=kind, batch=rng.randint(1, 4), seq=_log(rng, 1, 128), inp=width(), out=width(), rank=rng.choice([4, 8, 16, 32, 64]),
                    dtype=dtype)
    if kind == "linear":
        bias = rng.random() < 0.5
        rank = rng.choice([8, 16, 64])
        if rng.random() < 0.35:
            return dict(kind=kind, tokens=_log(rng, 64, 2048), inp=_log(rng, 256, 1536), out=_log(rng, 128, 1536), rank=rank, dtype="f32",
                        bias=bias)
        inp, out, most = rng.choice([(896, 896, 131072), (896, 128, 131072), (896, 4864, 65536), (4864, 896, 65536), (2048, 2048, 65536),
                                     (4096, 4096, 32768), (4096, 14336, 8192)])
        return dict(kind=kind, tokens=_log(rng, 256, most), inp=inp, out=out, rank=rank, dtype="bf16", bias=bias)
    if kind == "rmsnorm":
        width = rng.choice([896, 2048, 4096, 8 * _log(rng, 32, 512)])
        return dict(kind=kind, rows=_log(rng, 256, min(1 << 20, (1 << 30) // width)), width=width, dtype=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "softmax":
        seq = rng.choice([_log(rng, 64, 2048), 64 * _log(rng, 1, 32)])
        heads = rng.choice([2, 8, 14])
        return dict(kind=kind, batch=max(1, min(_log(rng, 1, 16), (1 << 29) // (heads * seq * seq))), heads=heads, seq=seq,
                    dtype=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "loss":
        vocab = rng.choice([151936, 151936, 32000, 50257])
        return dict(kind=kind, batch=rng.randint(1, 4), seq=_log(rng, 16, 1024), vocab=vocab, dtype=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "attention":
        seq = 128 * _log(rng, 1, 32)
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(16, 32768 // seq))), kv_heads=rng.choice([1, 2, 4]), groups=rng.choice([1, 2, 7]),
                    seq=seq)
    if kind == "adamw":
        return dict(kind=kind, layers=rng.randint(1, 32), hidden=64 * _log(rng, 8, 64), kv=128 * rng.randint(1, 4), rank=rng.choice([4, 8, 16, 32]),
                    targets=rng.choice(["qv", "qkvo"]))
    if kind == "forward":
        return dict(kind=kind, layers=24, batch=rng.randint(1, 4), seq=_log(rng, 16, 512), rank=rng.choice([8, 16]),
                    targets=rng.choice(["qv", "qkvo"]))
    if kind == "trainer":
        return dict(kind=kind, layers=rng.randint(2, 6), batch=rng.randint(1, 4), seq=rng.choice([_log(rng, 32, 512), 128 * rng.randint(1, 4)]),
                    rank=rng.choice([8, 16]), targets=rng.choice(["qv", "qkvo"]))
    seq = 128 * _log(rng, 1, 16)
    return dict(kind=kind, layers=24, batch=_log(rng, 1, 32768 // seq if seq > 2048 else 16), seq=seq, rank=rng.choice([8, 16]),
                targets=rng.choice(["qv", "qkvo"]))


# ---- what a program has in hand before the call --------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, dtype=torch.float32, std=1.0, mean=0.0):
    t = torch.randn(*shape, device="cuda", generator=g)
    return t.mul_(std).add_(mean).to(dtype)


def _adapter_set(case, g, hidden, intermediate, kv):
    """Adapters in mid-training (B is not zero any more), their tensors cut out of one flat buffer."""
    cfg = LoRAAdapterConfig(rank=case["rank"], alpha=2.0 * case["rank"], target_modules=list(TARGETS[case["targets"]]))
    adapter = LoRAAdapter(hidden, intermediate, case["layers"], cfg, "cuda", kv_size=kv, generator=g)
    layers = [layer for _, layer in adapter.layers()]
    flat = torch.empty(sum(t.numel() for layer in layers for t in layer.trainable_variables()), device="cuda")
    at = 0
    for layer in layers:
        layer.lora_a.mul_(math.sqrt(case["rank"] / hidden))
        layer.lora_b.normal_(0.0, 0.02, generator=g)
        for name in ("lora_a", "lora_b"):
            t = getattr(layer, name)
            view = flat[at:at + t.numel()].view_as(t)
            view.copy_(t)
            setattr(layer, name, view)
            at += t.numel()
    return adapter, flat


def _flat_like(tensors):
    """Views with the shapes of `tensors` into one flat buffer of zeros, and that buffer."""
    flat = torch.zeros(sum(t.numel() for t in tensors), device="cuda")
    views, at = [], 0
    for t in tensors:
        views.append(flat[at:at + t.numel()].view_as(t))
        at += t.numel()
    return views, flat


def _model(case, seed):
    cfg = ModelConfig(num_hidden_layers=case["layers"])
    model = Qwen(cfg, "cuda", dtype=torch.bfloat16, seed=seed)
    g = _gen(seed + 1)
    adapter, flat = _adapter_set(case, g, cfg.hidden_size, cfg.intermediate_size, cfg.kv_size)
    model.apply_adapter(adapter)
    shape = (case["batch"], case["seq"])
    ids = torch.randint(0, cfg.vocab_size, shape, device="cuda", generator=g, dtype=torch.int32)
    targets = torch.cat([ids[:, 1:], torch.full_like(ids[:, :1], -1)], 1).contiguous()   # the next token; the last one has none
    return model, adapter, flat, ids, targets


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    g = _gen(seed)
    if kind == "layer":
        layer = LoRALayer(case["inp"], case["out"], LoRAConfig(rank=case["rank"], alpha=2.0 * case["rank"]), "cuda", generator=g)
        layer.lora_b.normal_(0.0, 0.02, generator=g)
        layer.eval()
        s.update(layer=layer, x=_normal(g, case["batch"], case["seq"], case["inp"], dtype=DTYPES[case["dtype"]]))
    elif kind == "linear":
        m, k, n, r, dt = case["tokens"], case["inp"], case["out"], case["rank"], DTYPES[case["dtype"]]
        w = _normal(g, n, k, dtype=dt, std=1.0 / math.sqrt(k))
        s.update(x=_normal(g, m, k, dtype=dt), dy=_normal(g, m, n, dtype=dt), w=w, wt=backend.transpose_2d(w),
                 bias=_normal(g, n, dtype=dt, std=0.1) if case["bias"] else None,
                 a=(torch.rand(k, r, device="cuda", generator=g) * 2 - 1) / math.sqrt(k), b=_normal(g, r, n, std=0.02))
    elif kind == "rmsnorm":
        dt = DTYPES[case["dtype"]]
        s.update(x=_normal(g, case["rows"], case["width"], dtype=dt), dy=_normal(g, case["rows"], case["width"], dtype=dt),
                 w=_normal(g, case["width"], dtype=dt, std=0.1, mean=1.0))
    elif kind == "softmax":
        dt, n = DTYPES[case["dtype"]], case["seq"]
        x = _normal(g, case["batch"], case["heads"], n, n, dtype=dt, std=3.0)
        x.masked_fill_(torch.ones(n, n, dtype=torch.bool, device="cuda").triu_(1), -math.inf)
        s.update(x=x, dy=_normal(g, case["batch"], case["heads"], n, n, dtype=dt))
    elif kind == "loss":
        b, n, v = case["batch"], case["seq"], case["vocab"]
        targets = torch.randint(0, v, (b, n), device="cuda", generator=g)
        targets[torch.rand(b, n, device="cuda", generator=g) < 0.1] = IGNORE_INDEX
        targets[0, 0] = 1
        s.update(logits=_normal(g, b, n, v, dtype=DTYPES[case["dtype"]], std=2.0), targets=targets)
    elif kind == "attention":
        b, hk, gr, n = case["batch"], case["kv_heads"], case["groups"], case["seq"]
        bf = torch.bfloat16
        s.update(q=_normal(g, b * hk, gr * n, 64, dtype=bf), k=_normal(g, b * hk, n, 64, dtype=bf), v=_normal(g, b * hk, n, 64, dtype=bf),
                 do=_normal(g, b * n, hk * gr * 64, dtype=bf))
    elif kind == "adamw":
        adapter, flat = _adapter_set(case, g, case["hidden"], 4 * case["hidden"], case["kv"])
        variables = TrainingStep.collect_trainable_vars(adapter)
        grads, grad_flat = _flat_like(variables)
        grad_flat.copy_(_normal(g, grad_flat.numel(), std=0.1))
        opt = AdamW(AdamWConfig(learning_rate=LR))
        opt.step_vars(variables, grads)   # past the first step: the moments exist
        m, m_flat = _flat_like(variables)
        v, v_flat = _flat_like(variables)
        for i, (key, (m0, v0)) in enumerate(list(opt.state.items())):
            m[i].copy_(m0)
            v[i].copy_(v0)
            opt.state[key] = (m[i], v[i])
        s.update(opt=opt, variables=variables, grads=grads, out=(flat, m_flat, v_flat))
    elif kind == "forward":
        model, _, _, ids, _ = _model(case, seed)
        s.update(model=model, ids=ids)
    elif kind == "trainer":
        model, adapter, flat, ids, targets = _model(case, seed)
        s.update(model=model, adapter=adapter, flat=flat, ids=ids, targets=targets, step=TrainingStep(), opt=AdamW(AdamWConfig(learning_rate=LR)))
    else:
        model, _, flat, ids, targets = _model(case, seed)
        s.update(engine=QwenEngine(model, case["batch"], case["seq"]), flat=flat, ids=ids, targets=targets)
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "layer":
        return s["layer"].forward(s["x"])
    if kind == "linear":
        y, h = backend.lora_linear_forward(s["x"], s["w"], s["bias"], s["a"], s["b"], 2.0)
        dx, da, db = backend.lora_linear_backward(s["x"], s["wt"], s["a"], s["b"], 2.0, s["dy"], h_save=h)
        return y, dx, da, db
    if kind == "rmsnorm":
        y = backend.rms_norm_fused(s["x"], 1e-6, weight=s["w"])
        dx, dw = backend.rms_norm_backward(s["x"], s["w"], s["dy"], 1e-6)
        return y, dx, dw
    if kind == "softmax":
        y = backend.softmax_fused(s["x"])
        return y, backend.softmax_backward(y, s["dy"])
    if kind == "loss":
        return cross_entropy_loss(s["logits"], s["targets"], ignore_index=IGNORE_INDEX, return_grad=True)
    if kind == "attention":
        scale = 1.0 / math.sqrt(64)
        o, lse = backend.attention_causal_forward(s["q"], s["k"], s["v"], case["groups"], scale, kv_heads=case["kv_heads"])
        dq, dk, dv = backend.attention_causal_backward(s["q"], s["k"], s["v"], o, lse, s["do"], case["groups"], scale, kv_heads=case["kv_heads"])
        return o, dq, dk, dv
    if kind == "adamw":
        s["opt"].step_vars(s["variables"], s["grads"])
        return s["out"]
    if kind == "forward":
        return s["model"].forward(s["ids"])
    if kind == "trainer":
        metrics = s["step"].execute(s["ids"], s["targets"], s["adapter"], s["opt"], LR, s["model"].forward_backward)
        return metrics.loss, s["model"].grad_flat(), s["flat"]
    return s["engine"].train_step(s["ids"], s["targets"], LR), s["engine"].model.grad_flat(), s["flat"]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _model_work(case, backward):
    c = ModelConfig(num_hidden_layers=case["layers"])
    h, i, kv, v = c.hidden_size, c.intermediate_size, c.kv_size, c.vocab_size
    m = case["batch"] * case["seq"]
    dims = {TargetModule.QProj: (h, h), TargetModule.OProj: (h, h), TargetModule.KProj: (h, kv), TargetModule.VProj: (h, kv)}
    lora = sum(case["rank"] * sum(dims[t]) for t in TARGETS[case["targets"]]) * case["layers"]
    weights = case["layers"] * (2 * h * h + 2 * h * kv + 3 * h * i) + h * v
    attention = 4.0 * case["batch"] * c.num_attention_heads * case["seq"] ** 2 / 2 * c.head_dim * case["layers"]
    flops = 2.0 * m * (weights + lora) + attention
    bytes_ = 2.0 * (weights + m * h) + 4.0 * lora
    if not backward:
        return {"bytes": bytes_ + 2.0 * m * v, "flops": flops}
    # input gradients of every matrix, both gradients of every adapter, attention's five backward products
    return {"bytes": bytes_ + 4.0 * lora * 7, "flops": flops + 2.0 * m * weights + 4.0 * m * lora + 2.5 * attention}


def work(case):
    kind = case["kind"]
    e = {"f32": 4, "bf16": 2}.get(case.get("dtype"), 2)
    if kind == "layer":
        m, k, n, r = case["batch"] * case["seq"], case["inp"], case["out"], case["rank"]
        return {"bytes": e * m * (k + n) + 4 * r * (k + n), "flops": 2 * m * r * (k + n)}
    if kind == "linear":
        m, k, n, r = case["tokens"], case["inp"], case["out"], case["rank"]
        return {"bytes": e * (2 * m * (k + n) + 2 * n * k) + 4 * 2 * r * (k + n), "flops": 4 * m * k * n + 6 * m * r * (k + n)}
    if kind == "rmsnorm":
        n = case["rows"] * case["width"]
        return {"bytes": 4 * n * e, "flops": 12 * n}   # x is needed by both passes: counted once, with dy, y and dx
    if kind == "softmax":
        n = case["batch"] * case["heads"] * case["seq"] ** 2
        return {"bytes": 4 * n * e, "flops": 8 * n}
    if kind == "loss":
        n = case["batch"] * case["seq"] * case["vocab"]
        return {"bytes": 2 * n * e, "flops": 6 * n}
    if kind == "attention":
        rows = case["batch"] * case["kv_heads"] * case["seq"] * 64
        return {"bytes": 2 * rows * (4 * case["groups"] + 4), "flops": 3.5 * 4 * rows * case["groups"] * case["seq"] / 2}
    if kind == "adamw":
        h, kv, r = case["hidden"], case["kv"], case["rank"]
        per = {TargetModule.QProj: 2 * h, TargetModule.OProj: 2 * h, TargetModule.KProj: h + kv, TargetModule.VProj: h + kv}
        n = case["layers"] * r * sum(per[t] for t in TARGETS[case["targets"]])
        return {"bytes": 28 * n, "flops": 16 * n}
    return _model_work(case, backward=kind != "forward")


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        return {"rel": 1e-6}     # one float32 operation after another
    # Every activation is rounded to bf16 between two kernels, and a difference of one rounding early in the model
    # reaches all that follows: two correct implementations differ by 1.7 % in the logits of 24 layers, by 2.2 % in
    # their adapter gradients and by 1.3 % in those of 6 layers (measured: one element per token moved by one bf16 ulp).
    if kind == "step":
        return {"rel": 3e-2}
    if kind == "forward":
        return {"rel": 2.5e-2}
    if kind == "trainer":
        return {"rel": 2e-2}
    return {"rel": 1e-5} if case.get("dtype") == "f32" else {"rel": 1e-2}
