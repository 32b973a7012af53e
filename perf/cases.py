"""The workloads this framework's speed is judged by: what they are, how one pass of each is run through the public API,
what a pass cannot do without, and what another correct implementation may differ by.

The kinds of work, with the sizes taken from this repository's benchmark, tests and model configurations:

* ``decode``     one token per sequence through a transformer block that keeps its keys and values (serving, latency bound)
* ``prefill``    a small GPT exported to the native graph runtime: token ids in, next-token logits out, host to host
* ``gpt_step``   one optimizer step of a GPT through ``nn.Graph`` with gradient accumulation (the headline training path)
* ``block``      forward and backward of one transformer block (the bulk of GPT and BERT training)
* ``attention``  attention alone, forward and backward: grouped heads, long and unequal lengths
* ``lm_loss``    language-model head and its loss, forward and backward
* ``resnet``     one ResNet-50 training step
* ``dlrm``       one DLRM training step with its embedding engine, then predictions for a held-out batch
"""
from __future__ import annotations

import math
import tempfile

import numpy as np
import torch
import torch.nn as nn
import torch.nn.functional as TF

import oneflow_b200 as flow

DEV = "cuda:0"
F = flow.nn.functional


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call of a serving loop: one sequence, a small model, a short context
        {"name": "decode_one", "kind": "decode", "hidden": 1024, "heads": 16, "kv_heads": 16, "ffn": 4096, "batch": 1, "context": 512},
        # a layer of the 6.7B GPT serving eight sequences whose contexts are full
        {"name": "decode_batch", "kind": "decode", "hidden": 4096, "heads": 32, "kv_heads": 32, "ffn": 16384, "batch": 8, "context": 2048},
        # the exported 4-layer GPT of the graph-runtime benchmark answering prompts
        {"name": "prefill_exported", "kind": "prefill", "layers": 4, "hidden": 1024, "heads": 8, "vocab": 8192, "batch": 4, "seq": 1024},
        # the benchmark's tiny GPT: launches and host work count as much as the kernels
        {"name": "gpt_step_tiny", "kind": "gpt_step", "layers": 2, "hidden": 512, "heads": 4, "vocab": 8192, "seq": 512, "micro": 4, "accum": 2},
        # one layer of BERT-large pre-training, micro-batch 32 of 512 tokens
        {"name": "block_bert_large", "kind": "block", "hidden": 1024, "heads": 16, "ffn": 4096, "batch": 32, "seq": 512, "causal": False},
        # one layer of the 6.7B GPT, micro-batch 4 of 2048 tokens
        {"name": "block_gpt_6_7b", "kind": "block", "hidden": 4096, "heads": 32, "ffn": 16384, "batch": 4, "seq": 2048, "causal": True},
        # fine-tuning of a small model on sequences of a length that fits no tile
        {"name": "block_ragged", "kind": "block", "hidden": 768, "heads": 12, "ffn": 3072, "batch": 3, "seq": 777, "causal": True},
        # long-context training with grouped key / value heads
        {"name": "attention_long_grouped", "kind": "attention", "batch": 1, "heads": 32, "kv_heads": 8, "q_len": 8192, "kv_len": 8192,
         "dim": 128, "causal": True},
        # cross-attention of an encoder-decoder: unequal, odd lengths
        {"name": "attention_cross", "kind": "attention", "batch": 8, "heads": 16, "kv_heads": 16, "q_len": 500, "kv_len": 1100, "dim": 64,
         "causal": False},
        # head and loss of the benchmark's small GPT (hidden 2048) over the full vocabulary
        {"name": "lm_loss", "kind": "lm_loss", "tokens": 4096, "hidden": 2048, "vocab": 50304},
        # the ResNet-50 benchmark's batch of one GPU
        {"name": "resnet50_step", "kind": "resnet", "batch": 256, "image": 224},
        # the DLRM benchmark's batch
        {"name": "dlrm_step", "kind": "dlrm", "batch": 55296},
    ]


def _log(rng, lo, hi, mult=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult))


def _width(rng, lo, hi):
    """(hidden, heads) with a head size of 64 or 128."""
    d = rng.choice((64, 128))
    heads = _log(rng, max(2, lo // d), hi // d)
    return heads * d, heads


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(("decode", "prefill", "gpt_step", "block", "block", "attention", "attention", "lm_loss", "resnet", "dlrm"))
    if kind == "decode":
        hidden, heads = _width(rng, 512, 4096)
        return {"kind": kind, "hidden": hidden, "heads": heads, "kv_heads": heads if heads % 4 or rng.random() < 0.5 else heads // 4,
                "ffn": 4 * hidden, "batch": _log(rng, 1, 64), "context": _log(rng, 64, 4096)}
    if kind == "prefill":
        hidden, heads = _width(rng, 512, 1024)
        return {"kind": kind, "layers": rng.randint(2, 4), "hidden": hidden, "heads": heads, "vocab": _log(rng, 2048, 8192, 8),
                "batch": _log(rng, 1, 4), "seq": _log(rng, 64, 1024)}
    if kind == "gpt_step":
        hidden, heads = _width(rng, 256, 1024)
        return {"kind": kind, "layers": rng.randint(2, 4), "hidden": hidden, "heads": heads, "vocab": _log(rng, 2048, 16384, 64),
                "seq": _log(rng, 128, 1024), "micro": rng.randint(1, 4), "accum": rng.randint(1, 3)}
    if kind == "block":
        hidden, heads = _width(rng, 256, 4096)
        seq = _log(rng, 64, 2048)
        return {"kind": kind, "hidden": hidden, "heads": heads, "ffn": 4 * hidden, "batch": _log(rng, 1, max(1, 8192 // seq)), "seq": seq,
                "causal": rng.random() < 0.6}
    if kind == "attention":
        q = _log(rng, 64, 8192)
        kv = q if rng.random() < 0.6 else _log(rng, q, 8192)
        heads = rng.choice((8, 12, 16, 32))
        return {"kind": kind, "batch": _log(rng, 1, max(1, 16384 // kv)) if heads * kv <= 32 * 4096 else 1, "heads": heads,
                "kv_heads": heads // rng.choice((1, 1, 4)), "q_len": q, "kv_len": kv, "dim": rng.choice((64, 128)),
                "causal": rng.random() < 0.6}
    if kind == "lm_loss":
        return {"kind": kind, "tokens": _log(rng, 64, 4096), "hidden": _log(rng, 256, 2048, 8), "vocab": _log(rng, 2048, 50304, 8)}
    if kind == "resnet":
        return {"kind": kind, "batch": _log(rng, 8, 256), "image": rng.choice((96, 128, 160, 192, 224))}
    return {"kind": "dlrm", "batch": _log(rng, 1024, 55296, 8)}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(shape, device=DEV).normal_(mean, std, generator=g).to(dtype)


def _block_params(g, d, ffn, kv_cols):
    """Weights as they are in the middle of training: LayerNorm gains near one, products that keep the scale of their input."""
    return {"g1": _normal(g, d, std=0.1, mean=1.0), "b1": _normal(g, d, std=0.1),
            "wqkv": _normal(g, d + 2 * kv_cols, d, std=d ** -0.5), "bqkv": _normal(g, d + 2 * kv_cols, std=0.1),
            "wo": _normal(g, d, d, std=0.5 * d ** -0.5), "bo": _normal(g, d, std=0.1),
            "g2": _normal(g, d, std=0.1, mean=1.0), "b2": _normal(g, d, std=0.1),
            "w1": _normal(g, ffn, d, std=d ** -0.5), "c1": _normal(g, ffn, std=0.1),
            "w2": _normal(g, d, ffn, std=0.5 * ffn ** -0.5), "c2": _normal(g, d, std=0.1)}


def _block_inputs(c, seed):
    g = _gen(seed)
    p = _block_params(g, c["hidden"], c["ffn"], c["hidden"])
    rows = c["batch"] * c["seq"]
    return p, _normal(g, rows, c["hidden"]), _normal(g, rows, c["hidden"])


def _decode_inputs(c, seed):
    g = _gen(seed)
    dim = c["hidden"] // c["heads"]
    kv = c["kv_heads"] * dim
    p = _block_params(g, c["hidden"], c["ffn"], kv)
    cache = [_normal(g, c["batch"], c["context"], c["kv_heads"], dim) for _ in range(2)]
    return p, _normal(g, c["batch"], c["hidden"]), cache


def _attention_inputs(c, seed):
    g = _gen(seed)
    q = _normal(g, c["batch"], c["q_len"], c["heads"], c["dim"])
    k, v = (_normal(g, c["batch"], c["kv_len"], c["kv_heads"], c["dim"]) for _ in range(2))
    return q, k, v, _normal(g, c["batch"], c["q_len"], c["heads"], c["dim"])


def _lm_inputs(c, seed):
    g = _gen(seed)
    h, w = _normal(g, c["tokens"], c["hidden"]), _normal(g, c["vocab"], c["hidden"], std=c["hidden"] ** -0.5)
    return h, w, torch.randint(0, c["vocab"], (c["tokens"],), generator=g, device=DEV)


class _Layer(nn.Module):
    def __init__(self, d, heads):
        super().__init__()
        self.ln1, self.qkv, self.proj = nn.LayerNorm(d), nn.Linear(d, 3 * d), nn.Linear(d, d)
        self.ln2, self.fc1, self.fc2 = nn.LayerNorm(d), nn.Linear(d, 4 * d), nn.Linear(4 * d, d)
        self.heads = heads

    def forward(self, x):
        B, S, _ = x.shape
        q, k, v = self.qkv(self.ln1(x)).view(B, S, 3, self.heads, -1).unbind(2)
        a = TF.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=True)
        x = x + self.proj(a.transpose(1, 2).reshape(B, S, -1))
        return x + self.fc2(TF.gelu(self.fc1(self.ln2(x))))


class _NextToken(nn.Module):
    """A user's plain torch GPT that returns the logits of the last position."""

    def __init__(self, c):
        super().__init__()
        d = c["hidden"]
        self.emb, self.pos = nn.Embedding(c["vocab"], d), nn.Embedding(c["seq"], d)
        self.layers = nn.ModuleList([_Layer(d, c["heads"]) for _ in range(c["layers"])])
        self.ln, self.head = nn.LayerNorm(d), nn.Linear(d, c["vocab"], bias=False)

    def forward(self, ids):
        x = self.emb(ids) + self.pos(torch.arange(ids.shape[1], device=ids.device))
        for layer in self.layers:
            x = layer(x)
        return self.head(self.ln(x)[:, -1])


def _prefill_inputs(c, seed):
    g = torch.Generator().manual_seed(seed)
    with torch.device("meta"):
        model = _NextToken(c)
    model = model.to_empty(device="cpu").eval()
    with torch.no_grad():
        for name, p in model.named_parameters():
            std = 0.1 if p.dim() == 1 else (0.5 if name.startswith(("emb", "pos")) else p.shape[1] ** -0.5)
            p.normal_(1.0 if name.endswith("weight") and p.dim() == 1 else 0.0, std, generator=g)
            p.copy_(p.bfloat16())
    return model, torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g)


def _gpt_weight(name, shape, seed):
    """The weights of a ``gpt_step`` case by parameter name (LayerNorm gains near one, products of fan-in scale)."""
    g = _gen(seed * 7919 + sum((i + 1) * b for i, b in enumerate(name.encode())) % 1000003)
    if len(shape) == 1 or name.endswith("bqkv"):
        return _normal(g, *shape, std=0.1, mean=1.0 if name.endswith(("ln1_w", "ln2_w", "lnf_w")) else 0.0)
    std = 0.5 if "embedding" in name else shape[-1] ** -0.5
    return _normal(g, *shape, std=std)


def _gpt_tokens(c, seed):
    return torch.randint(0, c["vocab"], (c["micro"] * c["accum"], c["seq"] + 1), generator=_gen(seed), device=DEV)


LR, WEIGHT_DECAY, BETAS = 1e-3, 0.1, (0.9, 0.95)


def _resnet_weight(name, shape, seed):
    g = _gen(seed * 7919 + sum((i + 1) * b for i, b in enumerate(name.encode())) % 1000003)
    if len(shape) == 1:
        mean = 0.0 if name.endswith("bias") else (0.1 if name.endswith("bn3.weight") else 1.0)
        return _normal(g, *shape, std=0.05, mean=mean)
    fan_in = math.prod(shape[1:])
    w = _normal(g, *shape, std=math.sqrt((1.0 if name.startswith("fc") else 2.0) / fan_in))
    if name == "conv1.weight":
        w[:, 147:] = 0
    return w


def _resnet_inputs(c, seed):
    g = _gen(seed)
    images = _normal(g, c["batch"], c["image"], c["image"], 3)
    return images, torch.randint(0, 1000, (c["batch"],), generator=g, device=DEV)


# ------------------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "decode":
        s["p"], s["x"], s["cache"] = _decode_inputs(case, seed)
    elif kind == "block":
        p, x, s["dy"] = _block_inputs(case, seed)
        p["wqkv"] = p["wqkv"].view(3, case["hidden"], case["hidden"])
        p["bqkv"] = p["bqkv"].view(3, case["hidden"])
        s["p"] = {k: v.requires_grad_() for k, v in p.items()}
        s["x"] = x.requires_grad_()
    elif kind == "attention":
        q, k, v, s["do"] = _attention_inputs(case, seed)
        s["qkv"] = [t.requires_grad_() for t in (q, k, v)]
    elif kind == "lm_loss":
        h, w, s["labels"] = _lm_inputs(case, seed)
        s["hw"] = [h.requires_grad_(), w.requires_grad_()]
    elif kind == "prefill":
        from oneflow_b200.utils import export
        model, ids = _prefill_inputs(case, seed)
        with tempfile.TemporaryDirectory() as d:
            s["graph"] = export.InferenceGraph(export.export_graph(model, (ids,), d), device=0)
        s["ids"] = ids.numpy()
    elif kind == "gpt_step":
        from oneflow_b200.models import gpt, gpt_flow
        cfg = gpt.GPTConfig(vocab_size=case["vocab"], hidden=case["hidden"], layers=case["layers"], heads=case["heads"],
                            ffn=4 * case["hidden"], seq_len=case["seq"])
        s["graph"], s["model"], s["layout"] = gpt_flow.build_gpt_graph(cfg, grad_acc=case["accum"], device_type="cuda", lr=LR,
                                                                       weight_decay=WEIGHT_DECAY, clip_grad=1.0)
        with torch.no_grad():
            for name, p in s["model"].named_parameters():
                p.to_local().copy_(_gpt_weight(name, tuple(p.shape), seed))
        s["tokens"] = _gpt_tokens(case, seed)
    elif kind == "resnet":
        from oneflow_b200.models import resnet
        cfg = resnet.ResNetConfig(image_size=case["image"])
        t = resnet.ResNetTrainer(cfg, DEV, lr=0.1, momentum=0.9, weight_decay=1e-4, seed=0)
        for name, p in t.net.store.named_parameters():
            p.copy_(_resnet_weight(name, tuple(p.shape), seed))
        t.opt.master.copy_(t.net.store.flat)
        s["trainer"] = t
        s["images"], s["labels"] = _resnet_inputs(case, seed)
    else:
        from oneflow_b200.models import dlrm
        cfg = dlrm.DLRMConfig(global_batch=case["batch"], rows_capacity=1 << 22)
        s["trainer"] = dlrm.DLRMTrainer(cfg, torch.device(DEV), seed=seed)
        s["batch"] = tuple(t.to(DEV) for t in dlrm.make_batch(cfg, case["batch"], seed=2 * seed))
        s["held_out"] = tuple(t.to(DEV) for t in dlrm.make_batch(cfg, case["batch"], seed=2 * seed + 1))
    return s


def _run_decode(s):
    c, p = s["case"], s["p"]
    dim = c["hidden"] // c["heads"]
    kv = c["kv_heads"] * dim
    kc, vc = s["cache"]
    with torch.no_grad():
        x = s["x"]
        h = F.layer_norm(x, (c["hidden"],), p["g1"], p["b1"])
        q, k, v = F.linear(h, p["wqkv"], p["bqkv"]).split((c["hidden"], kv, kv), dim=1)
        # the new token takes the last place of the context
        kc[:, -1] = k.view(-1, c["kv_heads"], dim)
        vc[:, -1] = v.view(-1, c["kv_heads"], dim)
        a = F.scaled_dot_product_attention(q.reshape(-1, 1, c["heads"], dim).transpose(1, 2), kc.transpose(1, 2), vc.transpose(1, 2))
        x = flow._C.fused_matmul_bias(a.transpose(1, 2).reshape(-1, c["hidden"]), p["wo"], p["bo"], x)
        h = F.layer_norm(x, (c["hidden"],), p["g2"], p["b2"])
        return {"y": F.mlp(h, p["w1"], p["c1"], p["w2"], p["c2"], act="gelu", residual=x), "k": kc[:, -1], "v": vc[:, -1]}


def _run_block(s):
    c, p, x = s["case"], s["p"], s["x"]
    for t in (x, *p.values()):
        t.grad = None
    h = F.layer_norm(x, (c["hidden"],), p["g1"], p["b1"])
    qkv = F.linear(h, p["wqkv"], p["bqkv"])
    a = flow._C.fused_attention_qkv_packed(qkv, seq_len=c["seq"], head_size=c["hidden"] // c["heads"], causal=c["causal"])
    y = flow._C.fused_matmul_bias(a, p["wo"], p["bo"], x)
    h = F.layer_norm(y, (c["hidden"],), p["g2"], p["b2"])
    y = F.mlp(h, p["w1"], p["c1"], p["w2"], p["c2"], act="gelu", residual=y)
    y.backward(s["dy"])
    return {"y": y.detach(), "dx": x.grad, **{"d_" + k: v.grad for k, v in p.items()}}


def _run_attention(s):
    q, k, v = s["qkv"]
    for t in (q, k, v):
        t.grad = None
    o = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=s["case"]["causal"])
    o = o.transpose(1, 2)
    o.backward(s["do"])
    return {"o": o.detach(), "dq": q.grad, "dk": k.grad, "dv": v.grad}


def _run_lm_loss(s):
    h, w = s["hw"]
    h.grad = w.grad = None
    rows = F.sparse_softmax_cross_entropy(s["labels"], F.linear(h, w))
    rows.mean().backward()
    return {"loss": rows.detach(), "dh": h.grad, "dw": w.grad}


def _run_gpt_step(s):
    from oneflow_b200.models import gpt_flow
    loss = s["graph"](*gpt_flow.make_inputs(s["layout"], s["tokens"])).to_local()
    return {"loss": loss, **{n: p.to_local().detach() for n, p in s["model"].named_parameters()}}


def _run_resnet(s):
    t = s["trainer"]
    loss = t.train_step(s["images"], s["labels"])
    return {"loss": loss, "weights": t.opt.master,
            "running": torch.cat([v for pair in t.net.running.values() for v in pair])}


def _run_dlrm(s):
    t = s["trainer"]
    loss = t.train_step(*s["batch"])
    return {"loss": loss, "grad": t.store.grad, "weights": t.opt.master, "held_out": t.forward(*s["held_out"][:2])}


def run(state):
    kind = state["case"]["kind"]
    if kind == "prefill":
        return state["graph"].run(state["ids"])
    return {"decode": _run_decode, "block": _run_block, "attention": _run_attention, "lm_loss": _run_lm_loss, "gpt_step": _run_gpt_step,
            "resnet": _run_resnet, "dlrm": _run_dlrm}[kind](state)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _pairs(c):
    """Query / key pairs that attend to each other, one head, one sequence (diagonal in the bottom-right corner)."""
    q, kv = c["q_len"], c["kv_len"]
    if not c["causal"]:
        return q * kv
    return q * kv - q * (q - 1) // 2 if kv >= q else kv * (kv + 1) // 2


def work(case):
    c, kind = case, case["kind"]
    if kind == "decode":
        d, b = c["hidden"], c["batch"]
        kv = c["kv_heads"] * d // c["heads"]
        weights = d * (d + 2 * kv) + d * d + 2 * d * c["ffn"]
        return {"bytes": 2 * (weights + 2 * b * c["context"] * kv + 2 * b * d), "flops": 2 * b * weights + 4 * b * c["context"] * d}
    if kind == "block":
        d, rows = c["hidden"], c["batch"] * c["seq"]
        weights = 4 * d * d + 2 * d * c["ffn"]
        pairs = _pairs({"q_len": c["seq"], "kv_len": c["seq"], "causal": c["causal"]})
        # read x, dy and the weights, write y, dx and the weights' gradients; 2 attention products forward, 5 backward
        return {"bytes": 2 * (2 * weights + 4 * rows * d), "flops": 6 * rows * weights + 14 * c["batch"] * pairs * d}
    if kind == "attention":
        q, kv = c["batch"] * c["q_len"] * c["heads"] * c["dim"], c["batch"] * c["kv_len"] * c["kv_heads"] * c["dim"]
        return {"bytes": 2 * (4 * q + 4 * kv), "flops": 14 * c["batch"] * c["heads"] * _pairs(c) * c["dim"]}
    if kind == "lm_loss":
        t, d, v = c["tokens"], c["hidden"], c["vocab"]
        return {"bytes": 2 * (2 * t * d + 2 * v * d), "flops": 6 * t * d * v}
    if kind == "prefill":
        d, rows = c["hidden"], c["batch"] * c["seq"]
        weights = 12 * d * d * c["layers"]
        return {"bytes": 2 * (weights + c["vocab"] * d + rows * d) + 8 * rows,
                "flops": 2 * rows * weights + 2 * c["batch"] * d * c["vocab"] + 2 * c["batch"] * c["seq"] ** 2 * d * c["layers"]}
    if kind == "gpt_step":
        d, rows = c["hidden"], c["micro"] * c["accum"] * c["seq"]
        layers = 12 * d * d * c["layers"]
        params = layers + (2 * c["vocab"] + c["seq"]) * d
        # master weights and two moments read and written in fp32, the bf16 weights read and written
        return {"bytes": params * (6 * 4 + 2 * 2), "flops": 6 * rows * (layers + c["vocab"] * d) + 7 * rows * c["seq"] * d * c["layers"]}
    if kind == "resnet":
        from oneflow_b200.models import resnet
        n, px = c["batch"], c["image"] ** 2
        # every convolution output (about 11.1 M values an image of 224 x 224) written once forward and read once backward
        return {"bytes": int(2 * 2 * n * 11.1e6 * px / 224 ** 2) + 25_600_000 * 4 * 4,
                "flops": int(resnet.ResNetConfig(image_size=c["image"]).flops_per_image() * n)}
    b = c["batch"]
    mlp = 16 * 512 + 512 * 256 + 256 * 128 + 480 * 1024 + 1024 * 1024 + 1024 * 512 + 512 * 256 + 256 * 8
    pairs = 27 * 27 * 128
    # a training batch (forward, backward, row update) and a held-out one (forward): ids, fp32 rows of the tables
    return {"bytes": b * 26 * (8 + 128 * 4) * 2 + b * 26 * 128 * 4 + mlp * 4 * 8, "flops": 2 * b * (4 * mlp + 4 * pairs)}


# ------------------------------------------------------------------------------------------------ 64-bit statements
def _ln64(x, g, b, eps=1e-5):
    return TF.layer_norm(x, (x.shape[-1],), g, b, eps)


def _sdpa64(q, k, v, causal):
    """[B, S, H, D] operands, grouped heads, causal diagonal in the bottom-right corner; one head group at a time."""
    B, Sq, H, D = q.shape
    Sk, Hk = k.shape[1:3]
    mask = torch.ones(Sq, Sk, dtype=torch.bool, device=q.device).tril(Sk - Sq) if causal else None

    def head(q1, k1, v1):
        s = torch.einsum("bqd,bkd->bqk", q1, k1) / math.sqrt(D)
        if mask is not None:
            s = s.masked_fill(~mask, float("-inf"))
        return torch.einsum("bqk,bkd->bqd", s.softmax(-1), v1)
    from torch.utils.checkpoint import checkpoint
    return torch.stack([checkpoint(head, q[:, :, h], k[:, :, h * Hk // H], v[:, :, h * Hk // H], use_reentrant=False)
                        for h in range(H)], 2)


def _block64(x, p, heads, seq, causal):
    d = x.shape[1]
    qkv = (_ln64(x, p["g1"], p["b1"]) @ p["wqkv"].reshape(3 * d, d).t() + p["bqkv"].reshape(-1)).view(-1, seq, 3, heads, d // heads)
    a = _sdpa64(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], causal).reshape(-1, d)
    y = x + a @ p["wo"].t() + p["bo"]
    h = TF.gelu(_ln64(y, p["g2"], p["b2"]) @ p["w1"].t() + p["c1"])
    return y + h @ p["w2"].t() + p["c2"]


def _leaf(t):
    return t.double().requires_grad_()


def _gpt64(case, seed):
    c = case
    d, L = c["hidden"], c["layers"]
    shapes = {"embedding.wte": (c["vocab"], d), "embedding.wpe": (c["seq"], d)}
    layer = {"ln1_w": (d,), "ln1_b": (d,), "wqkv": (3, d, d), "bqkv": (3, d), "wo": (d, d), "bo": (d,), "ln2_w": (d,), "ln2_b": (d,),
             "w1": (4 * d, d), "b1": (4 * d,), "w2": (d, 4 * d), "b2": (d,)}
    for i in range(L):
        shapes.update({f"layers.{i}.{k}": v for k, v in layer.items()})
    shapes.update({"head.lnf_w": (d,), "head.lnf_b": (d,), "head.lm_head": (c["vocab"], d)})
    p = {n: _leaf(_gpt_weight(n, s, seed)) for n, s in shapes.items()}
    tokens = _gpt_tokens(c, seed)
    names = {"g1": "ln1_w", "b1": "ln1_b", "wqkv": "wqkv", "bqkv": "bqkv", "wo": "wo", "bo": "bo", "g2": "ln2_w", "b2": "ln2_b", "w1": "w1",
             "c1": "b1", "w2": "w2", "c2": "b2"}
    losses = []
    for m in range(c["accum"]):
        t = tokens[m * c["micro"]:(m + 1) * c["micro"]]
        x = p["embedding.wte"][t[:, :-1].reshape(-1)] + p["embedding.wpe"].repeat(c["micro"], 1)
        for i in range(L):
            x = _block64(x, {k: p[f"layers.{i}.{v}"] for k, v in names.items()}, c["heads"], c["seq"], True)
        loss = TF.cross_entropy(_ln64(x, p["head.lnf_w"], p["head.lnf_b"]) @ p["head.lm_head"].t(), t[:, 1:].reshape(-1))
        (loss / c["accum"]).backward()
        losses.append(loss.detach())
    out = {"loss": torch.stack(losses)}
    with torch.no_grad():
        # weights and biases are clipped over their own parameter group, then the first AdamW update
        norms = {dec: torch.sqrt(sum((q.grad ** 2).sum() for q in p.values() if (q.dim() >= 2) == dec)) for dec in (True, False)}
        total = torch.sqrt(norms[True] ** 2 + norms[False] ** 2)
        for n, q in p.items():
            g = q.grad * torch.clamp(1.0 / (total + 1e-6), max=1.0)
            out[n] = q * (1 - LR * (WEIGHT_DECAY if q.dim() >= 2 else 0.0)) - LR * g / (g.abs() + 1e-8)
    return out


def _resnet64(case, seed):
    widths, layers = (64, 128, 256, 512), (3, 4, 6, 3)
    specs = [("conv1.weight", (64, 152))]
    cin = 64
    vectors = [("bn1", 64)]
    for i, (n, w) in enumerate(zip(layers, widths)):
        for b in range(n):
            q = f"layer{i + 1}.{b}"
            specs += [(q + ".conv1", (w, 1, 1, cin)), (q + ".conv2", (w, 3, 3, w)), (q + ".conv3", (4 * w, 1, 1, w))]
            vectors += [(q + ".bn1", w), (q + ".bn2", w), (q + ".bn3", 4 * w)]
            if b == 0:
                specs.append((q + ".downsample.0", (4 * w, 1, 1, cin)))
                vectors.append((q + ".downsample.1", 4 * w))
            cin = 4 * w
    bns = [v[0] for v in vectors]
    specs.append(("fc.weight", (1000, 2048)))
    tail = [(b + s, (c,)) for b, c in vectors for s in (".weight", ".bias")] + [("fc.bias", (1000,))]
    p = {n: _leaf(_resnet_weight(n, s, seed)) for n, s in specs + tail}
    images, labels = _resnet_inputs(case, seed)
    running = {}

    def conv(name, x, stride=1):
        w = p[name].permute(0, 3, 1, 2)
        return TF.conv2d(x, w, stride=stride, padding=w.shape[-1] // 2)

    def bn(name, x, res=None, relu=True):
        n = x.numel() // x.shape[1]
        mean, var = x.mean((0, 2, 3)), x.var((0, 2, 3), unbiased=False)
        running[name] = (0.1 * mean.detach(), 0.9 + 0.1 * var.detach() * n / (n - 1))
        y = TF.batch_norm(x, None, None, p[name + ".weight"], p[name + ".bias"], True, 0.0, 1e-5)
        y = y if res is None else y + res
        return TF.relu(y) if relu else y
    x = images.double().permute(0, 3, 1, 2)
    x = TF.conv2d(x, p["conv1.weight"][:, :147].view(64, 7, 7, 3).permute(0, 3, 1, 2), stride=2, padding=3)
    x = TF.max_pool2d(bn("bn1", x), 3, 2, 1)
    for i, n in enumerate(layers):
        for b in range(n):
            q, stride = f"layer{i + 1}.{b}", 2 if b == 0 and i > 0 else 1
            idn = bn(q + ".downsample.1", conv(q + ".downsample.0", x, stride), relu=False) if b == 0 else x
            y = bn(q + ".bn1", conv(q + ".conv1", x))
            y = bn(q + ".bn2", conv(q + ".conv2", y, stride))
            x = bn(q + ".bn3", conv(q + ".conv3", y), res=idn)
    loss = TF.cross_entropy(x.mean((2, 3)) @ p["fc.weight"].t() + p["fc.bias"], labels)
    loss.backward()
    # the trainer's flat layout: decayed tensors first, every tensor padded to a multiple of 64 values; torch's SGD: first step
    pad = lambda t: TF.pad(t.reshape(-1), (0, -t.numel() % 64))  # noqa: E731
    with torch.no_grad():
        wd = {n: 1e-4 for n, _ in specs}
        weights = torch.cat([pad(p[n] - 0.1 * (p[n].grad + wd.get(n, 0.0) * p[n])) for n, _ in specs + tail])
    return {"loss": loss.detach(), "weights": weights, "running": torch.cat([v for b in bns for v in running[b]])}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "decode":
        p, x, (kc, vc) = _decode_inputs(c, seed)
        p = {k: v.double() for k, v in p.items()}
        x, kc, vc = x.double(), kc.double(), vc.double()
        dim = c["hidden"] // c["heads"]
        kv = c["kv_heads"] * dim
        q, k, v = (_ln64(x, p["g1"], p["b1"]) @ p["wqkv"].t() + p["bqkv"]).split((c["hidden"], kv, kv), dim=1)
        kc[:, -1], vc[:, -1] = k.view(-1, c["kv_heads"], dim), v.view(-1, c["kv_heads"], dim)
        a = _sdpa64(q.reshape(-1, 1, c["heads"], dim), kc, vc, False).reshape(-1, c["hidden"])
        x = x + a @ p["wo"].t() + p["bo"]
        h = TF.gelu(_ln64(x, p["g2"], p["b2"]) @ p["w1"].t() + p["c1"])
        return {"y": x + h @ p["w2"].t() + p["c2"], "k": kc[:, -1], "v": vc[:, -1]}
    if kind == "block":
        p, x, dy = _block_inputs(c, seed)
        p, x = {k: _leaf(v) for k, v in p.items()}, _leaf(x)
        y = _block64(x, p, c["heads"], c["seq"], c["causal"])
        y.backward(dy.double())
        d = c["hidden"]
        grads = {"d_" + k: v.grad for k, v in p.items()}
        grads["d_wqkv"], grads["d_bqkv"] = grads["d_wqkv"].view(3, d, d), grads["d_bqkv"].view(3, d)
        return {"y": y.detach(), "dx": x.grad, **grads}
    if kind == "attention":
        q, k, v, do = _attention_inputs(c, seed)
        q, k, v = _leaf(q), _leaf(k), _leaf(v)
        o = _sdpa64(q, k, v, c["causal"])
        o.backward(do.double())
        return {"o": o.detach(), "dq": q.grad, "dk": k.grad, "dv": v.grad}
    if kind == "lm_loss":
        h, w, labels = _lm_inputs(c, seed)
        h, w = _leaf(h), _leaf(w)
        rows = TF.cross_entropy(h @ w.t(), labels, reduction="none")
        rows.mean().backward()
        return {"loss": rows.detach(), "dh": h.grad, "dw": w.grad}
    if kind == "prefill":
        model, ids = _prefill_inputs(c, seed)
        with torch.no_grad():
            return [model.double().to(DEV)(ids.to(DEV)).reshape(-1).cpu().numpy().astype(np.float64)]
    if kind == "gpt_step":
        return _gpt64(c, seed)
    if kind == "resnet":
        return _resnet64(c, seed)
    return None     # the embedding engine's rows start from its own hash of the key


def tolerance(case):
    """About four times the difference between bf16 operands with 32-bit sums and the 64-bit statement. ResNet's gradients are
    noisy (a rounding flips the sign of a few in a thousand of every ReLU's inputs, in 49 layers: 7e-2), but they reach the
    updated weights as a few parts in ten thousand, so that the weights are held to 2e-4."""
    return {"decode": {"rel": 1e-2}, "prefill": {"rel": 2.2e-2}, "gpt_step": {"rel": 2.4e-2}, "block": {"rel": 2.5e-2},
            "attention": {"rel": 1.2e-2}, "lm_loss": {"rel": 8e-3}, "resnet": {"rel": 2e-4, "max": 2e-2}, "dlrm": {"rel": 5e-2}}[case["kind"]]
